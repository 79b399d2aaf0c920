"""The complex128 GEMM (DMMA, csrc/gemm_zmma.cu) through ``tcon``: both operand
layouts each, tile edges and remainders, K split inside clusters and over several,
against numpy; its forms with one real operand and the sums of products of nested
tensors through the excited-state pullback at ragged sizes, against the oracle.

Bar per entry of a product: sums of 4 k products of real numbers, 4 k eps (|A| |B|)
with |.| the modulus, and a factor 2."""
import math

import numpy as np
import pytest
import torch

import ipeps_oracle as O

pytestmark = pytest.mark.gpu
EPS = np.finfo(float).eps


def _rand(rng, *shape):
    return rng.standard_normal(shape) + 1j * rng.standard_normal(shape)


@pytest.mark.parametrize("m,n,k", [(1, 1, 1), (16, 32, 16), (17, 33, 31), (66, 66, 128), (128, 66, 130), (48, 432, 48),
                                   (5, 9, 4100), (4096, 4, 16), (130, 190, 1001), (300, 280, 700)])
def test_complex_products(engine, pkg, m, n, k):
    rng = np.random.default_rng(m + 10 * n + 100 * k)
    for ta in (False, True):
        for tb in (False, True):
            A, B = _rand(rng, *((k, m) if ta else (m, k))), _rand(rng, *((n, k) if tb else (k, n)))
            a, b = (A.T if ta else A), (B.T if tb else B)
            la, lb = ([1, -1] if ta else [-1, 1]), ([-2, 1] if tb else [1, -2])
            out = pkg.tcon([A, B], [la, lb], engine=engine)
            bound = 8 * k * EPS * (np.abs(a) @ np.abs(b)) + 1e-300
            assert np.all(np.abs(out - a @ b) <= bound), (ta, tb)
            # the transposed output (the GEMM's roles swapped)
            swap = {-1: -2, -2: -1, 1: 1}
            sw = pkg.tcon([A, B], [[swap[l] for l in la], [swap[l] for l in lb]], engine=engine)
            assert np.all(np.abs(sw.T - a @ b) <= bound), (ta, tb)


@pytest.mark.parametrize("D,chi", [(2, 11), (3, 13)])
def test_nested_pullback_ragged(engine, pkg, D, chi):
    """gH and gN of one vector from a 4-iteration environment; 1e-6 relative, the bar of the nested
    gradient elsewhere (both sides FP64, the environments differ by the projectors' 1e-10 residuals)."""
    A = O.random_A(D, 2, seed=chi)
    H = O.heisenberg(1.0)
    cfg = O.default_config()
    cfg.update(chi=chi, min_iter=4, max_iter=4, rg_tol=0.0, ad_max_iter=2)
    px, py = math.pi, 0.3 * math.pi
    rng = np.random.default_rng(chi)
    B = _rand(rng, D ** 4 * 2)
    ref, _ = O.run_ctm(O.make_ctm_tensors(A, cfg))
    p = dict(cfg)
    p.update(px=px, py=py)
    gH, gN = O.get_es_grad(ref.replace(Params=p), H, torch.from_numpy(B))[:2]
    ts = pkg.CTMTensors(A.numpy(), dict(cfg), engine=engine)
    pkg.run_ctm(ts)
    ts.Params["px"], ts.Params["py"] = px, py
    hH, hN = pkg.get_es_grad(ts, [h.numpy() for h in H], B)
    ts.close()
    for got, want in ((hH, gH.detach().numpy()), (hN, gN.detach().numpy())):
        assert np.linalg.norm(got - want) <= 1e-6 * np.linalg.norm(want)


def test_complex_wide_output(engine, pkg):
    """More column tiles (32 wide) than a grid's y side holds; bar as above."""
    m, n, k = 8, 65535 * 32 + 33, 4
    rng = np.random.default_rng(6)
    A, B = _rand(rng, m, k), np.asfortranarray(_rand(rng, k, n))
    out = pkg.tcon([A, B], [[-1, 1], [1, -2]], engine=engine)
    assert np.all(np.abs(out - A @ B) <= 8 * k * EPS * (np.abs(A) @ np.abs(B)) + 1e-300)
