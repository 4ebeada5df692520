"""Tile lists on images of many bands, and on both sides of the line between the two
sort paths: lists, ranges and in-place updates equal the oracle's bit for bit, by the
exact call, by the capacity-sized one, and after a capacity overflow."""
import pytest

from test_gpu_tile_lists import _check, _inputs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,W,H,patches", [
    (3000, 7680, 4320, 11_000_000),   # lists, 68 bands
    (3000, 7680, 4320, 4_000_000),    # as many bands, few patches: radix sort
    (200_000, 3840, 2160, 4_000_000),  # lists, 12 bands
    (900_000, 1920, 1080, 1_300_000),  # few patches per Gaussian: radix sort
    (900_000, 1920, 1080, 3_500_000),
    (5000, 12000, 2000, 9_000_000)])  # rows of 750 tiles, 32 bands
def test_lists_match_oracle(cuda_ok, n, W, H, patches):
    _check(_inputs(n, W, H, seed=n, keys=9000, patches=patches), W, H, patches // 2)
    _check(_inputs(n, W, H, seed=n + 1, keys=9000, patches=patches), W, H, patches // 2)
    _check(_inputs(n, W, H, seed=n + 2, keys=9000, patches=2 * patches), W, H, patches // 2)
