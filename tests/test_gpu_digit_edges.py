"""Exact digit products at the edges of their tiles: rows of a drain warp (32) and of a tile
(128), the column halves of the drain warps (16) and of a tile (32), K tiles (64) and chunks."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(31, 16, 63), (32, 17, 64), (33, 31, 65), (127, 32, 128),
                                   (128, 33, 129), (129, 48, 1), (257, 49, 191)])
def test_digit_products_at_tile_edges(ccx, shape):
    """The rounding to nearest of an exact sum, beside the 55-bit digits of the operands and the
    dropped levels below 2^-53 of K max|A| max|B|, and the rounding of C (below 1) after the
    addition, 2^-54 over a largest element of 0.2 or more: within 1e-14 of that element."""
    for seed in (1, 2):
        err, _ = ccx.selftest_tc_gemm([shape, (40, 40, 40)], kind=2, seed=seed)
        assert err < 1e-14, err
