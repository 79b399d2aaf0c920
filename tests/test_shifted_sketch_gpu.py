"""The projector's warm sketches (shifted power iterations from the last calls'
vectors, as many as the direction's last call needed) along CTMRG steps against
the oracle's exact SVDs: the kept corner spectrum of every step.

Bar: a kept triplet is accepted at a residual of 1e-10 s_1, an error of that
size in a value near s_1 and, by second order, less in the small ones; over the
steps the environments differ by the truncation's response to it.  1e-9 s_1
absolute allows a factor ten; values themselves are O(1)."""
import numpy as np
import pytest

import ipeps_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D,chi,seed", [(2, 13, 1), (3, 16, 2), (3, 37, 3), (4, 20, 4)])
def test_spectra_along_steps(engine, pkg, D, chi, seed):
    A = O.random_A(D, 2, seed=seed)
    cfg = O.default_config()
    cfg.update(chi=chi)
    ref = O.make_ctm_tensors(A, cfg)
    ts = pkg.CTMTensors(A.numpy(), cfg, engine=engine)
    for _ in range(9):
        ref, s_ref = O.rg_step(ref, chi)
        ts, s = pkg.rg_step(ts)
        s_ref = s_ref.detach().numpy()
        assert s.shape == s_ref.shape
        assert np.abs(s - s_ref).max() <= 1e-9 * s_ref[0]
    ts.close()
