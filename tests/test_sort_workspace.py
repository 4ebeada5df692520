"""Workspace of the tile sort, on the host: whichever path a size takes, it is the
radix sort's -- independent of the Gaussian count, never shrinking as the patches
grow (a buffer sized for the largest render serves the smaller ones), and 16 or 24
bytes per patch plus histograms."""
import ctypes as C

import pytest

from gsplatcu import _lib

SIZES = [(256, 256), (1920, 1080), (3840, 2160), (7680, 4320), (12000, 2000), (60, 9000)]


def _bytes(n, W, H, patches, dkey):
    L = _lib.lib()
    plan = _lib.SplatPlan(patches, dkey, 0)
    exact = int(L.gsb_splat_sort_bytes(n, H, W, C.byref(plan)))
    assert int(L.gsb_splat_sort_capacity_bytes(n, H, W, patches, dkey)) == exact
    return exact


@pytest.mark.parametrize("dkey", [9000, (1 << 17) - 1, (1 << 24) - 1])
@pytest.mark.parametrize("W,H", SIZES)
def test_workspace_is_the_radix_sorts(W, H, dkey):
    tiles = ((W + 15) // 16) * ((H + 15) // 16)
    key = 8 if (tiles - 1).bit_length() + dkey.bit_length() > 32 else 4
    last = 0
    for patches in (1000, 1_199_999, 1_500_000, 1_500_001, 1_900_000, 4_000_000, 20_000_000, 90_000_000):
        need = {_bytes(n, W, H, patches, dkey) for n in (1, 30_000, 1_000_000, 10_000_000)}
        assert len(need) == 1, patches
        need = need.pop()
        hist = 512 * 4 * ((patches + 3071) // 3072) + 512 * 4
        assert 2 * patches * (key + 4) + hist <= need <= 2 * patches * (key + 4) + hist + 6 * 256
        assert need >= last
        last = need
