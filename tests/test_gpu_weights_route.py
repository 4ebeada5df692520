"""splat_palette_weights: the fused forward against the operator chain it replaces,
over the weight forms, types and odd sizes it accepts; what it refused or computed
through the operators stays so.  And the one-launch gradient scale against torch."""
import numpy as np
import pytest
import torch

import gsplatcu as gsc
from gsplatcu import _lib
from palette_b200 import loss as pl
from palette_b200 import weights as pw
from palette_b200.render import _weight_args
from palette_b200.scene import look_at, synthetic_scene, to_torch
from helpers import max_abs

pytestmark = pytest.mark.gpu

# (K, rank; 0: full SH, -1: rank-1 factors stored 2-D), dtype, N, W, H
FORMS = [(3, 0), (5, 0), (8, 0), (5, -1), (5, 2), (5, 4), (6, 3), (3, 1), (4, 1)]


def _inputs(K, rank, dtype, n, seed=0):
    full = rank == 0
    sc = synthetic_scene(n, seed=seed, K=K, mode="full" if full else "lowrank", rank=abs(rank) or 1,
                         P=K)
    st = to_torch(sc, "cuda", dtype)
    if full:
        return st, dict(shs=st["shs"])
    A, B = st["A"], st["B"]
    if rank < 0:
        A, B = A[..., 0].contiguous(), B[:, 0].contiguous()
    return st, dict(dc=st["dc"], A=A, B=B)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("K,rank", FORMS)
def test_fused_forward_matches_operator_chain(cuda_ok, K, rank, dtype):
    st, wt = _inputs(K, rank, dtype, 5001)
    cam = look_at((5.0, -5.0, 2.0), width=133, height=70, device="cuda")
    layer, visible = pw.splat_palette_weights(st["pws"], st["alphas"], st["scales"], st["rots"],
                                              cam, **wt)
    w0, A, B, mode, k, P, Q, r = _weight_args(wt.get("shs"), wt.get("dc"), wt.get("A"),
                                              wt.get("B"), None)
    ref, depths = pw._operator_chain(st["pws"], st["alphas"], st["scales"], st["rots"], w0, A, B,
                                     cam, mode, k, Q)
    assert torch.equal(visible, depths > 0.2)
    # weights within a few ulps of each other, sums of at most ~100 terms of size <= 1
    assert max_abs(layer, ref) < 1e-5


def test_other_shapes_and_refusals_stay(cuda_ok):
    st, _ = _inputs(5, 0, torch.float32, 700)
    cam = look_at((0.0, -8.0, 0.0), width=64, height=48, device="cuda")
    geo = (st["pws"], st["alphas"], st["scales"], st["rots"])
    shs = st["shs"][:, :32].contiguous().requires_grad_()  # K = 2: operators only
    layer, _ = pw.splat_palette_weights(*geo, cam, shs=shs)
    assert layer.shape == (2, 48, 64) and float(layer.detach().abs().sum()) > 0
    with pytest.raises(_lib.GsplatError):
        layer.sum().backward()
    with pytest.raises(TypeError):
        pw.splat_palette_weights(st["pws"].double(), *geo[1:], cam, shs=st["shs"])
    with pytest.raises(ValueError):
        pw.splat_palette_weights(*geo, look_at((0.0, -8.0, 0.0), width=64, height=48, device="cpu"),
                                 shs=st["shs"])
    empty = [t[:0] for t in geo]
    layer, visible = pw.splat_palette_weights(*empty, cam, shs=st["shs"][:0])
    assert float(layer.abs().sum()) == 0.0 and visible.numel() == 0


@pytest.mark.parametrize("n", [0, 1, 3, 4, 5, 1023, 4096 * 5 + 2])
@pytest.mark.parametrize("shift", [0, 1])
def test_gradient_scale_matches_torch(cuda_ok, n, shift):
    base = torch.randn(n + shift, device="cuda")
    a, b = base[shift:], torch.randn((3, 5), device="cuda")
    g = torch.randn(4, device="cuda")[1]
    with torch.no_grad():
        x, y = pl._times(g, a, b)
        z, none = pl._times(g, a, None)
    assert torch.equal(x, a * g) and torch.equal(y, b * g) and torch.equal(z, a * g) and none is None


def test_create_graph_still_differentiates_the_scale(cuda_ok):
    layer = torch.rand((5, 16, 16), device="cuda", requires_grad=True)
    pal = torch.rand((5, 3), device="cuda")
    s = torch.tensor(2.0, device="cuda", requires_grad=True)
    loss = s * pl.palette_l1_loss(layer, pal, torch.rand((3, 16, 16), device="cuda"))
    d, = torch.autograd.grad(loss, layer, create_graph=True)
    ds, = torch.autograd.grad(d.sum(), s)
    assert torch.allclose(ds, d.detach().sum() / 2.0, rtol=1e-5)
    assert np.isfinite(float(ds))
