"""Tile lists filled in depth order (the path of renders with many patches): lists,
ranges and in-place updates equal the oracle's bit for bit, on images whose tiles
split into one and many bands, very wide and very tall ones, Gaussian counts around
a group of 256, tied depth keys, Gaussians behind the camera and off the image;
by the exact and the capacity-sized call, and after a capacity overflow."""
import numpy as np
import pytest
import torch

import gsplatcu as gsc
from oracle import oracle as orc
from helpers import np_of

pytestmark = pytest.mark.gpu

PATCHES = 1_700_000  # above the size from which this path is taken


def _inputs(n, W, H, seed, keys, patches=PATCHES):
    rng = np.random.default_rng(seed)
    side = np.sqrt(patches / n * 256.0) / 2.0  # half extent of `patches / n` tiles
    us = rng.uniform((0, 0), (W, H), size=(n, 2))
    ext = np.ceil(rng.uniform(0.3, 1.9, size=(n, 2)) * side)
    ext = np.maximum(ext, [1, 1])
    if H < 4 * side:  # a low image: widen what the height cuts off
        ext[:, 0] *= max(1.0, 2.2 * side / H)
    if W < 4 * side:
        ext[:, 1] *= max(1.0, 2.2 * side / W)
    depths = rng.integers(1, keys + 1, n) / 1000.0 + 0.3
    depths[rng.random(n) < 0.05] = 0.1                       # culled by depth
    us[rng.random(n) < 0.05] += [4.0 * W + 9e3, 0]           # off the image
    f = lambda x: torch.from_numpy(np.ascontiguousarray(x, np.float32)).cuda()  # noqa: E731
    return dict(us=f(us), cinv=f(np.tile([1.0, 0.0, 1.0], (n, 1))), alphas=f(np.full((n, 1), 0.5)),
                depths=f(depths), feats=f(rng.uniform(0, 1, (n, 1))),
                areas=torch.from_numpy(ext.astype(np.int32)).cuda())


def _check(s, W, H, least):
    us = np_of(s["us"])
    d, a = np_of(s["depths"]).copy(), np_of(s["areas"]).astype(np.int32).copy()
    ref = orc.bin_gaussians(us, a, d, H, W)
    assert len(ref["gsid"]) >= least
    d2, a2 = s["depths"].clone(), s["areas"].clone()
    out = gsc.splat_weight(H, W, 1, s["us"], s["cinv"], s["alphas"], d2, s["feats"], a2)
    assert np.array_equal(np_of(out[4]), ref["gsid"])
    assert np.array_equal(np_of(out[3]), ref["ranges"])
    assert np.array_equal(np_of(d2), d) and np.array_equal(np_of(a2), a)


@pytest.mark.parametrize("n,W,H,keys", [(2000, 1920, 1080, 16000), (4097, 3840, 2160, 300),
                                        (255, 1297, 841, 1), (257, 2000, 1500, 100000),
                                        (20000, 12000, 40, 5000), (9000, 60, 9000, 5000),
                                        (700, 200, 1500, 7)])
def test_lists_match_oracle(cuda_ok, n, W, H, keys):
    tiles = ((W + 15) // 16) * ((H + 15) // 16)
    n = max(n, 20 * PATCHES // tiles // 256 * 256 + n % 256)  # what a border cuts off counts too
    s = _inputs(n, W, H, seed=n, keys=keys)
    _check(s, W, H, 1_500_000)
    _check(s, W, H, 1_500_000)  # sized by the stored capacity, no read-back
    more = _inputs(n, W, H, seed=n + 1, keys=keys, patches=3 * PATCHES)
    _check(more, W, H, 1_500_000)  # (more patches or wider keys than stored: redone)


def test_single_depth_key_and_every_gaussian_everywhere(cuda_ok):
    """Each Gaussian in every tile of a 4K image: one list repeated 32400 times."""
    n, W, H = 64, 3840, 2160
    s = _inputs(n, W, H, seed=5, keys=3)
    s["us"][:] = torch.tensor([W / 2, H / 2], device="cuda")
    s["areas"][:] = 10000
    _check(s, W, H, 1_500_000)
