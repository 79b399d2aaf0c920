"""The projector's orthonormalisation (shifted CholeskyQR, csrc/projector.cu
`orth`) through ``ipeps_orth``: the range-finder step that stands in for the
Q factor of the reference's full SVD (ctmrg.jl:257).  It exercises the packed
panel Cholesky and triangular solve (k <= 192), the blocked Cholesky with the
row-parallel solve (larger k) and the one-launch kernel of small sketches directly,
against numpy's QR:

* Q^T Q = I to 1e-14 and Q R = Y to 1e-14 relative (sCholQR3 on a
  well-conditioned Y); one pass (shifted) orthogonal to 1e-6, two to 1e-14;
* R equals numpy's R up to the signs of its rows, to 1e-12 relative (R has a
  positive diagonal);
* ill-conditioned Y (singular values 1 .. 1e-12; the first pass is shifted):
  Q^T Q = I to 1e-13 after three passes; rank-deficient Y (rank k/2): Q^T Q = I
  to 1e-10 (the null directions are rounding noise); in both the range of Y
  lies inside range(Q) to 1e-13.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,k", [(300, 5), (1000, 33), (2500, 128), (2500, 160), (1200, 200)])
def test_orth_matches_numpy_qr(engine, pkg, N, k):
    rng = np.random.default_rng(N + k)
    Y = rng.standard_normal((N, k))
    Q, R = pkg.orth(Y, 3, engine=engine)
    assert np.abs(Q.T @ Q - np.eye(k)).max() <= 1e-14 * k ** 0.5
    assert np.linalg.norm(Q @ R - Y) <= 1e-14 * np.linalg.norm(Y) * k ** 0.5
    assert np.allclose(np.tril(R, -1), 0.0)
    assert (np.diag(R) > 0).all()
    _, Rn = np.linalg.qr(Y)
    Rn = Rn * np.sign(np.diag(Rn))[:, None]
    assert np.linalg.norm(R - Rn) <= 1e-12 * np.linalg.norm(Rn)
    # one shifted pass is orthogonal only to the shift's level, ~11 (N k + k^2) u
    # trace(G) / s_min(Y)^2 (a CPU restatement: 1e-11 at k = 5 .. 1e-7 at k = 160);
    # the unshifted second pass restores the rounding level
    for passes, bar in ((1, 1e-6), (2, 1e-14 * k ** 0.5)):
        Qp, Rp = pkg.orth(Y, passes, engine=engine)
        assert np.abs(Qp.T @ Qp - np.eye(k)).max() <= bar, passes
        assert np.linalg.norm(Qp @ Rp - Y) <= 1e-13 * np.linalg.norm(Y)


@pytest.mark.parametrize("k", [64, 160])
def test_orth_ill_conditioned_and_rank_deficient(engine, pkg, k):
    rng = np.random.default_rng(7 * k)
    N = 2000
    # singular values from 1 down to 1e-12 (as a sketch after power iterations)
    U, _ = np.linalg.qr(rng.standard_normal((N, k)))
    V, _ = np.linalg.qr(rng.standard_normal((k, k)))
    Y = (U * np.logspace(0, -12, k)) @ V.T
    Q, R = pkg.orth(Y, 3, engine=engine)
    assert np.abs(Q.T @ Q - np.eye(k)).max() <= 1e-13
    assert np.linalg.norm(Y - Q @ (Q.T @ Y)) <= 1e-13 * np.linalg.norm(Y)
    # rank k/2: the shifted first pass keeps R invertible, Q stays orthonormal
    Yr = rng.standard_normal((N, k // 2)) @ rng.standard_normal((k // 2, k))
    Q, R = pkg.orth(Yr, 3, engine=engine)
    assert np.isfinite(Q).all() and np.isfinite(R).all()
    assert np.abs(Q.T @ Q - np.eye(k)).max() <= 1e-10  # a CPU restatement gives 1.3e-11 at k = 160
    assert np.linalg.norm(Yr - Q @ (Q.T @ Yr)) <= 1e-13 * np.linalg.norm(Yr)


@pytest.mark.parametrize("N,k", [(1, 1), (7, 7), (8, 8), (40, 9), (33, 16), (129, 24), (120, 62), (333, 76), (97, 97),
                                 (1201, 104), (160, 159), (3000, 160), (170, 161)])
def test_orth_block_edges(engine, pkg, N, k):
    """Panel edges of the packed Cholesky and triangular solve (8 columns, 8 rows, 32 columns per
    instance of the solve), square Y among them; the widest packed k follows below.  Bars: two unshifted CholeskyQR passes after the shifted one
    leave rounding, 10 k eps in Q^T Q and in Q R = Y; R against the Cholesky factor of Y^T Y (64-bit,
    backward stable) differs by its conditioning, 100 k eps cond(Y)^2."""
    rng = np.random.default_rng(N * 1000 + k)
    Y = rng.standard_normal((N, k)) + (4.0 * N ** 0.5 * np.eye(N, k) if N < 2 * k else 0.0)
    eps = np.finfo(float).eps
    Q, R = pkg.orth(Y, 3, engine=engine)
    assert np.abs(Q.T @ Q - np.eye(k)).max() <= 10 * k * eps
    assert np.linalg.norm(Q @ R - Y) <= 10 * k * eps * np.linalg.norm(Y)
    assert np.array_equal(np.tril(R, -1), np.zeros((k, k)))
    ref = np.linalg.cholesky(Y.T @ Y).T
    assert np.linalg.norm(R - ref) <= 100 * k * eps * np.linalg.cond(Y) ** 2 * np.linalg.norm(ref)


@pytest.mark.parametrize("n", [2, 17, 38, 39, 40, 41, 47, 48, 64, 66, 81, 97, 113, 144, 160])
def test_projector_jacobi_block_edges(engine, pkg, n):
    """The Jacobi SVD inside the projector at the widths where its kernels change (one CTA below 40
    columns, clusters of 8 CTAs with 16 column blocks from there, odd block widths, rows per lane):
    n x n corners whose sketch is the whole space, singular values 1 .. 1e-4 known by construction.
    Bars: Jacobi and CholeskyQR on an n x n product leave n eps s_1 in each value and, for P1 P2 =
    R2 V S^-1 U^T R1 of the n - 1 leading triplets, that times s_1 / s_n (1e4) and the inverse
    relative gap of the truncated pair (>= 9.2 / n), all with a factor 20."""
    rng = np.random.default_rng(n)
    eps = np.finfo(float).eps
    s = np.logspace(0, -4, n)
    U, _ = np.linalg.qr(rng.standard_normal((n, n)))
    V, _ = np.linalg.qr(rng.standard_normal((n, n)))
    Z, _ = np.linalg.qr(rng.standard_normal((n, n)))
    R1, R2 = (U * np.sqrt(s)) @ Z, Z.T @ (np.sqrt(s)[:, None] * V.T)
    P1, P2, got = pkg.get_projector(R1, R2, n - 1, engine=engine)
    assert got.shape == (n - 1,)
    assert np.abs(got - s[:-1]).max() <= 20 * n * eps
    ref = Z.T[:, :-1] @ Z[:-1]  # R2 V S^-1 U^T R1 on the leading triplets
    assert np.abs(P1 @ P2 - ref).max() <= 20 * n * eps * 1e4 * max(1.0, n / 9.2)


@pytest.mark.parametrize("n,rank", [(62, 5), (100, 20)])
def test_projector_rank_deficient_corners(engine, pkg, n, rank):
    """Corners of exact low rank: the discarded columns of the Jacobi SVD are rounding noise that every
    sweep shrinks further, down to underflow.  The kept values against numpy's (n eps s_1, factor 20)."""
    rng = np.random.default_rng(n)
    # the Gram matrices of the product scale with the fourth power, their pivot guard is absolute at 1e-300
    for scale in (1.0, 1e-20, 1e-40):
        R1 = scale * (rng.standard_normal((n, rank)) @ rng.standard_normal((rank, n)))
        R2 = scale * (rng.standard_normal((n, rank)) @ rng.standard_normal((rank, n)))
        s_ref = np.linalg.svd(R1 / scale @ (R2 / scale), compute_uv=False)
        P1, P2, s = pkg.get_projector(R1, R2, rank, engine=engine)
        assert np.isfinite(P1).all() and np.isfinite(P2).all()
        assert np.abs(s[:rank] / scale ** 2 - s_ref[:rank]).max() <= 20 * n * np.finfo(float).eps * s_ref[0]


# one launch for all passes (no R asked for): one column, ragged rows and columns, the largest, and the first
# sizes beyond it
@pytest.mark.parametrize("N,k", [(1, 1), (8, 8), (13, 13), (64, 31), (120, 41), (127, 97), (128, 128), (129, 9),
                                 (333, 62)])
def test_orth_in_one_launch(engine, pkg, N, k):
    rng = np.random.default_rng(3 * N + k)
    Y = np.asfortranarray(rng.standard_normal((N, k)))
    Qn, Rn = np.linalg.qr(Y)
    Qn = Qn * np.sign(np.diag(Rn))
    # a backward-stable Q moves by rounding times the condition number of Y
    cond = np.linalg.cond(Y)
    for passes, bar in ((1, 1e-6), (2, 1e-14 * k ** 0.5), (3, 1e-14 * k ** 0.5)):
        Q = np.empty((N, k), order="F")
        engine.check(engine.lib.ipeps_orth(engine.h, pkg.host._dp(Y), N, k, passes, pkg.host._dp(Q), None))
        if N > 2 * k:  # (a square Gaussian's condition number is unbounded: the shift then shows)
            assert np.abs(Q.T @ Q - np.eye(k)).max() <= bar, passes
        if passes == 3:
            assert np.abs(Q.T @ Q - np.eye(k)).max() <= 1e-14 * k ** 0.5
            assert np.linalg.norm(Q - Qn) <= 1e-14 * cond * k


@pytest.mark.parametrize("N,k", [(400, 191), (400, 192), (400, 193), (250, 192), (3000, 192)])
def test_orth_largest_packed(engine, pkg, N, k):
    """The widest sketches of the packed Cholesky and solve (192 columns) and the first beyond them; bars as in
    test_orth_block_edges."""
    rng = np.random.default_rng(N + k)
    Y = rng.standard_normal((N, k)) + (4.0 * N ** 0.5 * np.eye(N, k) if N < 2 * k else 0.0)
    eps = np.finfo(float).eps
    Q, R = pkg.orth(Y, 3, engine=engine)
    assert np.abs(Q.T @ Q - np.eye(k)).max() <= 10 * k * eps
    assert np.linalg.norm(Q @ R - Y) <= 10 * k * eps * np.linalg.norm(Y)
    ref = np.linalg.cholesky(Y.T @ Y).T
    assert np.linalg.norm(R - ref) <= 100 * k * eps * np.linalg.cond(Y) ** 2 * np.linalg.norm(ref)


@pytest.mark.parametrize("k,j", [(40, 3), (40, 8), (33, 15), (160, 20), (200, 3)])
def test_orth_failed_pivot(engine, pkg, k, j):
    """A column 1e-25 of the others: the shift of the first pass leaves it at ~1e-21, so its pivot in the second
    pass is below 1e-32 of the trace.  That pass then has R[j, j] = 1 and row j zero, so row j of the product of
    both factors is the first factor's (from its definition, in numpy).  The entries left in the row instead
    would double it.  Rounding: k eps in the sums behind an entry, with a factor 1e3 for their cancellation."""
    N = 2 * k
    rng = np.random.default_rng(k + j)
    Y = rng.standard_normal((N, k))
    Y[:, j] *= 1e-25
    G = Y.T @ Y
    u = 0.5 * np.finfo(float).eps
    R1 = np.linalg.cholesky(G + 11.0 * (N * k + k * (k + 1)) * u * np.trace(G) * np.eye(k)).T
    _, R = pkg.orth(Y, 2, engine=engine)
    bar = 1e3 * k * 2 * u
    assert abs(R[j, j] - R1[j, j]) <= bar * R1[j, j]
    assert np.abs(R[j, j + 1:] - R1[j, j + 1:]).max() <= bar * np.abs(R1[j, j + 1:]).max()
