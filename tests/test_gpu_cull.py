"""Culling and skip threshold of the compositing kernels: conics from round to
needle-thin in every orientation, centres inside and outside the image, opacities
around the 0.002 threshold, the 0.99 clamp and above 1, on image sizes with
ragged tiles.  Nothing the reference blends may be dropped, so contributor
indices equal the oracle's; at most two pixels per image may differ, by an ulp
of exp() at a threshold (the oracle uses the host C library's)."""
import numpy as np
import pytest
import torch

import gsplatcu as gsc
from oracle import oracle as orc
from helpers import max_abs, np_of, rel_err

pytestmark = pytest.mark.gpu

MAX_EXP_FLIPS = 2


def _splats(n, W, H, longest, seed):
    """Screen-space Gaussians: axes 0.55 .. `longest` pixels, any orientation."""
    rng = np.random.default_rng(seed)
    us = rng.uniform((-0.3 * W, -0.3 * H), (1.3 * W, 1.3 * H), size=(n, 2))
    ax = np.exp(rng.uniform(np.log(0.55), np.log(longest), size=(n, 2)))
    th = rng.uniform(0, np.pi, n)
    th[: n // 4] = rng.choice([0.0, np.pi / 2, np.pi / 4, 1e-3], n // 4)
    R = np.stack([np.cos(th), -np.sin(th), np.sin(th), np.cos(th)], 1).reshape(n, 2, 2)
    cov = np.einsum("nij,nj,nkj->nik", R, ax ** 2, R)
    inv = np.linalg.inv(cov)
    edge = np.float32(0.002)
    alphas = 1.0 / (1.0 + np.exp(-rng.normal(0, 2, n)))
    alphas[: n // 3] = rng.choice([edge, np.nextafter(edge, np.float32(1)), 0.0021, 0.00199, 0.0,
                                   0.99, 1.0, 1.7, 0.01], n // 3)
    f = lambda x: torch.from_numpy(np.ascontiguousarray(x, np.float32)).cuda()  # noqa: E731
    areas = np.ceil(3 * np.sqrt(np.stack([cov[:, 0, 0], cov[:, 1, 1]], 1)))
    return dict(us=f(us), cinv=f(np.stack([inv[:, 0, 0], inv[:, 0, 1], inv[:, 1, 1]], 1)),
                alphas=f(alphas[:, None]), depths=f(rng.uniform(1, 9, n)),
                areas=torch.from_numpy(areas.astype(np.int32)).cuda(),
                feats=f(rng.uniform(0, 1, (n, 5))))


@pytest.mark.parametrize("n,W,H,longest", [(300, 40, 24, 3.0), (800, 100, 70, 30.0),
                                           (800, 100, 70, 400.0), (3000, 65, 17, 8.0)])
def test_culling_drops_nothing_that_blends(cuda_ok, n, W, H, longest):
    s = _splats(n, W, H, longest, seed=n + W)
    us, cinv, alphas = np_of(s["us"]), np_of(s["cinv"]), np_of(s["alphas"])
    d, a = np_of(s["depths"]).copy(), np_of(s["areas"]).astype(np.int32).copy()
    b = orc.bin_gaussians(us, a, d, H, W)
    ref, rc, rt = orc.draw(H, W, 5, b["ranges"], b["gsid"], us, cinv, alphas, np_of(s["feats"]), 0.0)
    out, contrib, tau, ranges, gsid = gsc.splat_weight(H, W, 5, s["us"], s["cinv"], s["alphas"],
                                                       s["depths"], s["feats"], s["areas"])
    assert np.array_equal(np_of(gsid), b["gsid"])
    same = np_of(contrib) == rc
    assert int((~same).sum()) <= MAX_EXP_FLIPS
    assert max_abs(np_of(out)[:, same], ref[:, same]) < 1e-5
    assert max_abs(np_of(tau)[same], rt[same]) < 1e-5
    g = torch.randn((5, H, W), device="cuda", generator=torch.Generator("cuda").manual_seed(n))
    got = gsc.splat_weight_B_full(H, W, 5, s["us"], s["cinv"], s["alphas"], s["depths"], s["feats"],
                                  contrib, tau, ranges, gsid, g)
    w, = gsc.splat_weight_B(H, W, 5, s["us"], s["cinv"], s["alphas"], s["depths"], s["feats"],
                            contrib, tau, ranges, gsid, g)
    r = orc.draw_backward(H, W, 5, np_of(ranges), np_of(gsid), us, cinv, alphas, np_of(s["feats"]),
                          np_of(tau), np_of(contrib), np_of(g))
    for x, key in ((w, "dfeat"), (got[0], "dfeat"), (got[1], "du"), (got[2], "dconic"),
                   (got[3], "dalpha")):
        assert rel_err(x.reshape(r[key].shape), r[key]) < 1e-4
