"""Components of a nested environment whose shapes differ: ``set_CT`` replaces the plain tensors of an environment alone,
so the components that an earlier nested run left can belong to another boundary dimension.  Such calls are refused
(the product of one component must not be formed with the extents of another), and a new ``set_B`` clears the
components."""
import numpy as np
import pytest

import ipeps_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("chi,other", [(6, 11), (11, 6)])
@pytest.mark.parametrize("parallel", [True, False])
def test_components_of_other_shapes_are_refused(engine, pkg, chi, other, parallel):
    D = 2
    A = O.random_A(D, 2, seed=7).numpy()
    H = [h.numpy() for h in O.heisenberg(1.0)]
    rng = np.random.default_rng(3)
    B = rng.standard_normal(A.shape) + 1j * rng.standard_normal(A.shape)
    cfg = pkg.default_config()
    cfg.update(chi=other, parallel_moves=parallel)
    plain = pkg.CTMTensors(A, dict(cfg), engine=engine)
    for _ in range(3):
        pkg.rg_step(plain)
    CT = [plain.get_CT(k) for k in range(1, 5)]
    plain.close()

    cfg["chi"] = chi
    ts = pkg.CTMTensors(A, dict(cfg), engine=engine)
    pkg.rg_step(ts)
    ts.set_B(B, 0.3, 0.7)
    for _ in range(2):
        pkg.rg_step(ts)
    for k in range(4):
        ts.set_CT(k + 1, *CT[k])
    assert ts.get_CT(1)[0].shape[0] == other
    ts.Params["px"], ts.Params["py"] = 0.3, 0.7
    for call in (lambda: pkg.rg_step(ts), lambda: pkg.get_es_energy(ts, H), lambda: pkg.get_all_norm(ts),
                 lambda: pkg.es_energy_grad(ts, H, 1)):
        with pytest.raises(pkg.host.IPEPSError) as err:
            call()
        assert err.value.code == 4  # invalid argument
    # the plain environment is still there, and starts a nested run afresh
    for k in range(4):
        ts.set_CT(k + 1, *CT[k])
    ts.set_B(B, 0.3, 0.7)
    pkg.rg_step(ts)
    e = pkg.get_es_energy(ts, H)
    ref = pkg.CTMTensors(A, dict(cfg), engine=engine, init=False)
    for k in range(4):
        ref.set_CT(k + 1, *CT[k])
    ref.set_B(B, 0.3, 0.7)
    pkg.rg_step(ref)
    assert abs(e - pkg.get_es_energy(ref, H)) <= 1e-9 * max(1.0, abs(e))
    ts.close()
    ref.close()
