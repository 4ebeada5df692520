"""Parameter shapes of the fused renders are checked on the host before any
launch: every call here is refused, and no kernel runs (the CUDA tensors are
fake ones, without storage)."""
import pytest
import torch
from torch._subclasses.fake_tensor import FakeTensorMode

from palette_b200.render import render_palette, render_palette_views
from palette_b200.scene import Camera
from palette_b200.weights import splat_palette_weights

N = 7


def _views(pws, rots, scales, alphas, cam, **w):
    return render_palette_views(pws, rots, scales, alphas, [cam], **w)


def _weights(pws, rots, scales, alphas, cam, **w):
    return splat_palette_weights(pws, alphas, scales, rots, cam, **w)


ENTRIES = [render_palette, _views, _weights]


def _refused(entry, geometry, weights):
    with FakeTensorMode():
        f = lambda shape: torch.empty(shape, device="cuda")  # noqa: E731
        cam = Camera(0, 64, 48, 50.0, 50.0, 32.0, 24.0, f((3, 3)), f((3,)), twc=f((3,)))
        geo = dict(pws=(N, 3), rots=(N, 4), scales=(N, 3), alphas=(N, 1))
        geo.update(geometry)
        with pytest.raises(ValueError):
            entry(*(f(geo[k]) for k in ("pws", "rots", "scales", "alphas")), cam,
                  **{k: f(s) for k, s in weights.items()})


@pytest.mark.parametrize("entry", ENTRIES)
@pytest.mark.parametrize("A,B", [((N, 5, 3), (N, 1, 15)),   # fewer rows in B than ranks
                                 ((N, 5, 1), (N, 3, 15)),   # more
                                 ((N, 5, 3), (N, 15)), ((N, 5), (N, 1, 15)),
                                 ((N,), (N, 15)), ((N, 5, 3, 1), (N, 3, 15, 1))])
def test_factor_shapes(entry, A, B):
    _refused(entry, {}, dict(dc=(N, 5), A=A, B=B))


@pytest.mark.parametrize("entry", ENTRIES)
@pytest.mark.parametrize("geometry", [dict(rots=(N - 1, 4)), dict(scales=(N, 1)), dict(alphas=(1,)),
                                      dict(rots=(N, 3)), dict(pws=(N, 2))])
def test_geometry_rows(entry, geometry):
    _refused(entry, geometry, dict(shs=(N, 80)))


@pytest.mark.parametrize("entry", ENTRIES)
@pytest.mark.parametrize("short", ["dc", "A", "B", "shs"])
def test_weight_rows(entry, short):
    w = dict(shs=(N, 80)) if short == "shs" else dict(dc=(N, 5), A=(N, 5, 3), B=(N, 3, 15))
    w[short] = (N - 1,) + w[short][1:]
    _refused(entry, {}, w)
