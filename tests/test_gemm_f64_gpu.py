"""The engine's FP64 GEMM (DMMA tensor-core kernel, gemm_dmma.cu) through the
C ABI against a numpy FP64 product: every op combination, edge tiles (sizes
that are not multiples of the tiles), odd leading dimensions (8-byte copies;
even ones take 16-byte copies),
split-K shapes (few output tiles, long K) and beta != 0.

Bar: |C - C_ref| <= 2 k eps (|A| |B|)_ij + 2 eps |beta C|_ij per entry, the
bound of any FP64 summation order."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EPS = np.finfo(np.float64).eps

CASES = [
    # m, n, k, beta != 0
    (1, 1, 1, 0),
    (7, 5, 3, 1),
    (64, 64, 16, 0),
    (130, 70, 33, 1),
    (2500, 160, 2500, 0),   # projector range finder: few output tiles, long K (split-K)
    (160, 160, 2500, 0),    # Gram matrix shape
    (161, 157, 3001, 1),    # split-K with edge tiles and beta (23 splits)
    (97, 33, 20000, 1),     # two output tiles, 156 splits
    (1000, 1200, 100, 0),   # many output tiles (128x128 kernel)
    (1001, 1203, 101, 1),   # the same with odd sizes (odd leading dimensions)
    (40000, 50, 25, 0),     # tall and narrow (128x64 tiles): the contractions with A
    (40001, 49, 25, 1),     # the same, odd
    (50, 40000, 25, 0),     # short and wide (64x128 tiles)
]


@pytest.mark.parametrize("opA", ["N", "T"])
@pytest.mark.parametrize("opB", ["N", "T"])
@pytest.mark.parametrize("case", CASES)
def test_gemm_f64_matches_numpy(engine, pkg, opA, opB, case):
    m, n, k, pad = case
    rng = np.random.default_rng(m * 7 + n * 3 + k)
    ar, ac = (m, k) if opA == "N" else (k, m)
    br, bc = (k, n) if opB == "N" else (n, k)
    A = np.asfortranarray(rng.standard_normal((ar, ac)))
    B = np.asfortranarray(rng.standard_normal((br, bc)))
    C = rng.standard_normal((m, n))
    alpha, beta = 0.75, (0.0 if pad == 0 else -1.5)
    opa = (lambda x: x) if opA == "N" else (lambda x: x.T)
    opb = (lambda x: x) if opB == "N" else (lambda x: x.T)
    ref = alpha * (opa(A) @ opb(B)) + beta * C
    out = pkg.host.gemm_f64(opA, opB, A, B, alpha=alpha, beta=beta, C=C, engine=engine)
    bound = 2 * k * EPS * abs(alpha) * (np.abs(opa(A)) @ np.abs(opb(B))) + 2 * EPS * np.abs(beta * C) + 1e-300
    assert np.all(np.abs(out - ref) <= bound), float(np.max(np.abs(out - ref) / bound))


def test_gemm_f64_split_k_is_deterministic(engine, pkg):
    """The split-K partial products are summed in split order, whatever order
    the CTAs ran in: repeated products are bitwise equal."""
    rng = np.random.default_rng(5)
    A = np.asfortranarray(rng.standard_normal((2500, 160)))
    B = np.asfortranarray(rng.standard_normal((2500, 160)))
    outs = [pkg.host.gemm_f64("T", "N", A, B, engine=engine) for _ in range(4)]
    for o in outs[1:]:
        assert np.array_equal(o, outs[0])
    ref = A.T @ B
    bound = 2 * 2500 * EPS * (np.abs(A.T) @ np.abs(B))
    assert np.all(np.abs(outs[0] - ref) <= bound)


@pytest.mark.parametrize("op", ["NN", "TN", "NT", "TT"])
@pytest.mark.parametrize("m,n,k,beta", [
    # (the plans named are those of a B200: tile, K chunks, CTAs per cluster)
    (33, 31, 65, 0.0),      # 32 x 32 and its remainders, no split
    (120, 62, 120, 0.5),    # 32 x 32, 2 chunks in a cluster of two
    (37, 37, 150, 0.0),     # 32 x 32, 4 chunks in a cluster of four; odd leading dimensions (8-byte copies)
    (37, 37, 333, 0.0),     # 32 x 32, 8 chunks in a cluster of eight
    (65, 33, 1000, -1.0),   # the same with remainders in both sides
    (2500, 160, 2500, 0.0),  # 64 x 32, clusters of two
    (9, 18, 12321, 0.0),    # 32 x 32, 128 chunks in clusters of eight: their sums through the workspace
    (17, 23, 40001, 2.0),   # 256 chunks with a remainder in K and beta
    (2500, 128, 2500, 1.0),  # 64 x 64, 5 chunks without clusters, all through the workspace
    (2500, 79, 1111, 0.0),  # 128 x 80, 7 chunks without clusters
    (20000, 50, 25, 0.0),   # 64 x 64
    (30000, 64, 40, 0.0),   # 128 x 64
    (100000, 40, 16, 0.0),  # 128 x 48
    (300, 900, 5, 1.0),     # less than one K step
])
def test_gemm_f64_tiles_and_splits(engine, pkg, op, m, n, k, beta):
    """Every tile configuration, and K chunks summed in clusters, through the workspace and both, with remainders;
    bound as above."""
    rng = np.random.default_rng(m + 3 * n + 7 * k)
    A = np.asfortranarray(rng.standard_normal((m, k) if op[0] == "N" else (k, m)))
    B = np.asfortranarray(rng.standard_normal((k, n) if op[1] == "N" else (n, k)))
    C = rng.standard_normal((m, n))
    a, b = (A if op[0] == "N" else A.T), (B if op[1] == "N" else B.T)
    out = pkg.host.gemm_f64(op[0], op[1], A, B, alpha=1.25, beta=beta, C=C, engine=engine)
    bound = 2 * k * EPS * 1.25 * (np.abs(a) @ np.abs(b)) + 2 * EPS * np.abs(beta * C) + 1e-300
    assert np.all(np.abs(out - (1.25 * (a @ b) + beta * C)) <= bound)
    again = pkg.host.gemm_f64(op[0], op[1], A, B, alpha=1.25, beta=beta, C=C, engine=engine)
    assert np.array_equal(out, again)


@pytest.mark.parametrize("op", ["NN", "TT"])
def test_gemm_f64_wide_output(engine, pkg, op):
    """More column tiles than a grid's y side holds (65535; 32-column tiles at this size); bound as above."""
    m, n, k = 4, 65535 * 32 + 33, 17
    rng = np.random.default_rng(5)
    A = np.asfortranarray(rng.standard_normal((m, k) if op[0] == "N" else (k, m)))
    B = np.asfortranarray(rng.standard_normal((k, n) if op[1] == "N" else (n, k)))
    C = rng.standard_normal((m, n))
    a, b = (A if op[0] == "N" else A.T), (B if op[1] == "N" else B.T)
    out = pkg.host.gemm_f64(op[0], op[1], A, B, alpha=1.25, beta=-0.5, C=C, engine=engine)
    bound = 2 * k * EPS * 1.25 * (np.abs(a) @ np.abs(b)) + 2 * EPS * np.abs(0.5 * C) + 1e-300
    assert np.all(np.abs(out - (1.25 * (a @ b) - 0.5 * C)) <= bound)
