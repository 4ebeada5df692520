"""Full adjoint with incoming gradients beyond the scalar recursion's range: infinite,
NaN and near the FP32 maximum, at single pixels, in the colour and in the final
transmittance, for images on both sides of the one-pixel line.  Infinities and NaN fall
where the oracle's per-channel FP32 sums have them, with their signs; everything finite
agrees as elsewhere."""
import numpy as np
import pytest
import torch

import gsplatcu as gsc
from oracle import oracle as orc
from test_gpu_cull import _splats
from helpers import np_of, rel_err

pytestmark = pytest.mark.gpu

INF = float("inf")
# (channel, row, column, value); channel -1: the final transmittance's gradient
POKES = {"inf": [(0, 5, 7, INF)], "two signs": [(0, 5, 7, INF), (1, 20, 33, -INF)],
         "one pixel, two channels": [(0, 9, 9, INF), (2, 9, 9, INF)],
         "transmittance": [(-1, 12, 30, -INF)], "nan": [(1, 18, 2, float("nan"))],
         "huge": [(0, 5, 7, 1e35), (1, 5, 7, -3e34), (2, 17, 40, 2e33)],
         "huge transmittance": [(-1, 3, 3, -1e36)]}


@pytest.mark.parametrize("poke", POKES)
@pytest.mark.parametrize("K,n,W,H", [(3, 300, 70, 41), (5, 500, 70, 41), (5, 4000, 640, 272),
                                     (8, 1500, 640, 272)])
def test_extreme_gradients_by_channel(cuda_ok, K, n, W, H, poke):
    s = _splats(n, W, H, 30.0, seed=n + K)
    rng = np.random.default_rng(K)
    feats = torch.from_numpy(rng.uniform(0, 1, (n, K)).astype(np.float32)).cuda()
    out, contrib, tau, ranges, gsid = gsc.splat_weight(H, W, K, s["us"], s["cinv"], s["alphas"],
                                                       s["depths"], feats, s["areas"])
    g = rng.normal(0, 1, (K, H, W)).astype(np.float32)
    gT = rng.normal(0, 1, (H, W)).astype(np.float32)
    for c, y, x, v in POKES[poke]:
        (gT if c < 0 else g[c])[y, x] = v
    got = gsc.splat_weight_B_full(H, W, K, s["us"], s["cinv"], s["alphas"], s["depths"], feats,
                                  contrib, tau, ranges, gsid, torch.from_numpy(g).cuda(),
                                  torch.from_numpy(gT).cuda())
    with np.errstate(all="ignore"):
        ref = orc.draw_backward(H, W, K, np_of(ranges), np_of(gsid), np_of(s["us"]), np_of(s["cinv"]),
                                np_of(s["alphas"]), np_of(feats), np_of(tau), np_of(contrib), g, gT)
    touched = False
    for x, key in zip(got, ("dfeat", "du", "dconic", "dalpha")):
        x, r = np_of(x).reshape(ref[key].shape), ref[key]
        assert np.array_equal(np.isnan(x), np.isnan(r)), key
        inf = np.isinf(r)
        assert np.array_equal(np.isinf(x), inf) and np.array_equal(np.sign(x[inf]), np.sign(r[inf])), key
        ok = np.isfinite(r)
        assert rel_err(x[ok], r[ok]) < 1e-4, key
        touched |= not ok.all() or np.abs(r[ok]).max() > 1e30
    assert touched
