"""Index permutations (csrc/ops.cu) through ``tcon`` with a factor 1, bit by bit against numpy: the copy of long rows at
the edges of its runs (128 elements per warp and step, 2048 per unit; pairs of doubles where both rows are 16-byte
aligned), rows and element-wise copies beside the lines between them."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n0", [40, 63, 64, 65, 127, 128, 129, 255, 256, 257, 999, 2047, 2048, 2049, 4099])
@pytest.mark.parametrize("complex_", [False, True])
def test_rows(engine, pkg, n0, complex_):
    rng = np.random.default_rng(n0)
    for a, b in ((35, 36), (3, 5)):  # from eight units per SM on, and fewer
        A = rng.standard_normal((n0, a, b))
        if complex_:
            A = A + 1j * rng.standard_normal(A.shape)
        out = pkg.tcon([np.asfortranarray(A), np.ones(1, dtype=A.dtype)], [[-1, -3, -2], [-4]], engine=engine)
        assert np.array_equal(out[..., 0], A.transpose(0, 2, 1))


def test_rows_at_an_odd_offset(engine, pkg):
    """Rows of odd length: every second one starts 8 bytes off a 16-byte boundary."""
    rng = np.random.default_rng(0)
    A = rng.standard_normal((333, 7, 9, 21))
    out = pkg.tcon([np.asfortranarray(A), np.ones(1)], [[-1, -4, -3, -2], [-5]], engine=engine)
    assert np.array_equal(out[..., 0], A.transpose(0, 3, 2, 1))
