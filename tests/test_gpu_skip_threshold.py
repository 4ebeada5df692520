"""The compositing kernels' skip rule against the reference's: a record carries the
smallest exponent p* that still blends, which is exact if expf never decreases.  One
Gaussian per tile, read at the pixel next to its centre, where the form is exactly p:
with a power of two as opacity the image holds 2^j expf(p) exactly, so both the decision
(alpha' < 0.002) and expf itself can be compared float by float.  No mismatch is
allowed."""
import numpy as np
import pytest
import torch

import gsplatcu as gsc
from helpers import np_of

pytestmark = pytest.mark.gpu

W, H = 3840, 2160
GX, GY = W // 16, H // 16
N = GX * GY
MIN, MAX = np.float32(0.002), np.float32(0.99)


def _f32(x):
    return torch.from_numpy(np.ascontiguousarray(x, np.float32)).cuda()


def _render(p, alphas):
    """(blended, value) of each Gaussian's pixel, exponents p <= 0 and opacities [N]."""
    t = np.arange(N)
    us = np.stack([t % GX * 16 + 8, t // GX * 16 + 8], 1)
    qa = -2.0 * p.astype(np.float64)
    out, contrib, _, _, _ = gsc.splat_weight(
        H, W, 1, _f32(us), _f32(np.stack([qa, np.zeros(N), qa], 1)), _f32(alphas[:, None]),
        _f32(np.ones(N)), _f32(np.ones((N, 1))), torch.ones((N, 2), dtype=torch.int32, device="cuda"))
    at = lambda x: np_of(x).reshape(GY, 16, GX, 16)[:, 8, :, 7].reshape(-1)  # noqa: E731
    return at(contrib) > 0, at(out[0])


def _expf(p):
    """The kernels' expf(p), read through a power-of-two opacity."""
    scale = np.exp2(np.floor(np.log2(0.5) - p.astype(np.float64) / np.log(2.0))).astype(np.float32)
    blended, v = _render(p, scale)
    assert blended.all() and v.min() >= 0.2 and v.max() < MAX
    return v / scale  # exact


def _check(p, alphas):
    e = _expf(p)
    ap = np.minimum(MAX, alphas * e)
    blended, v = _render(p, alphas)
    assert np.array_equal(blended, ~(ap < MIN))
    assert np.array_equal(v[blended], ap[blended])
    return e


def _walk(start, n):
    """n consecutive floats downwards from start < 0."""
    return (np.float32(start).view(np.uint32) + np.arange(n, dtype=np.uint32)).view(np.float32)


def test_decisions_around_the_threshold(cuda_ok):
    rng = np.random.default_rng(0)
    a = np.concatenate([[MIN, np.nextafter(MIN, MAX), 0.0020001, 0.00201, 0.99, 1.0, 1.0000001, 1.7],
                        rng.uniform(0.002, 1.0, 96), np.exp(rng.uniform(np.log(0.002), 0.0, 96))])
    a = a.astype(np.float32)
    per = N // len(a)
    alphas = np.ones(N, np.float32)
    p = np.full(N, -1.0, np.float32)
    for i, x in enumerate(a):
        edge = np.float32(min(-1e-30, np.log(np.float64(MIN) / np.float64(x))))
        first = np.int64(edge.view(np.uint32)) - per // 2
        first = max(first, int(np.float32(-1e-38).view(np.uint32)))
        p[i * per:(i + 1) * per] = (np.arange(per) + first).astype(np.uint32).view(np.float32)
        alphas[i * per:(i + 1) * per] = x
    _check(p, alphas)


@pytest.mark.parametrize("start", [-1e-6, -3e-3, -0.03, -0.25, -0.69, -1.0, -1.99, -2.5, -3.9, -5.0,
                                   -6.2, -20.0, -80.0])
def test_expf_never_decreases(cuda_ok, start):
    p = _walk(start, N)
    e = _check(p, np.full(N, 0.3, np.float32))
    assert (np.diff(e) <= 0).all()


def test_expf_never_decreases_over_the_range(cuda_ok):
    rng = np.random.default_rng(1)
    for _ in range(4):
        p = -np.sort(np.exp(rng.uniform(np.log(1e-7), np.log(87.0), N)).astype(np.float32))
        near = np.nextafter(p[::2], np.float32(-100))  # and each second one's neighbour
        p[1::2] = near[:len(p[1::2])]
        p = -np.sort(-p)
        e = _check(p, rng.uniform(0.002, 1.0, N).astype(np.float32))
        assert (np.diff(e) <= 0).all()
