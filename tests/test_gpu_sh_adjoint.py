"""Per-Gaussian adjoint with full SH weights where its blocks of 64 rows can go
wrong: counts around a block, channel counts 3 to 8, both storage types, rows
that are not 16-byte aligned, and gradients added over views.  Gradients against
the oracle's FP64 chain rule within 1e-4 relative (BF16 storage rounds them to 8
bits: 4e-3)."""
import numpy as np
import pytest
import torch

import gsplatcu as gsc
from oracle import oracle as orc
from palette_b200.render import render_palette, render_palette_views
from palette_b200.scene import look_at, synthetic_scene, to_torch
from helpers import forward_ops, np_of, rel_err

pytestmark = pytest.mark.gpu

NAMES = ("pws", "rots", "scales", "alphas", "shs")
W = H = 48


def _leaves(n, K, dtype, seed=3, shift=0):
    st = to_torch(synthetic_scene(n, seed=seed, K=K), "cuda", dtype)
    st["scales"] = st["scales"] * 8.0  # visible at this size
    leaf = {}
    for k in NAMES:
        flat = torch.empty(st[k].numel() + shift, dtype=st[k].dtype, device="cuda")
        flat[shift:] = st[k].reshape(-1)
        leaf[k] = flat[shift:].view(st[k].shape).requires_grad_()
    return st, leaf


def _grads(leaf, cam, g, gT):
    layer, tau, _ = render_palette(leaf["pws"], leaf["rots"], leaf["scales"], leaf["alphas"], cam,
                                   shs=leaf["shs"])
    return torch.autograd.grad((layer * g).sum() + (tau * gT).sum(), [leaf[k] for k in NAMES])


def _upstream(K, seed=1):
    gen = torch.Generator("cuda").manual_seed(seed)
    return (torch.randn((K, H, W), device="cuda", generator=gen),
            torch.randn((H, W), device="cuda", generator=gen))


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("K", [3, 5, 8])
@pytest.mark.parametrize("n", [1, 63, 64, 65, 400])
def test_gradients_match_fp64_chain(cuda_ok, n, K, dtype):
    st, leaf = _leaves(n, K, dtype)
    cam = look_at((0.0, -8.0, 0.0), width=W, height=H, device="cuda")
    g, gT = _upstream(K)
    got = _grads(leaf, cam, g, gT)
    ref = forward_ops(gsc, st, cam)
    f = lambda t: t.detach().double().cpu().numpy()  # noqa: E731
    r = orc.render_weights_backward(f(st["pws"]), f(st["rots"]), f(st["scales"]), f(st["alphas"]),
                                    cam, f(cam.twc), K, shs=f(st["shs"]), lowrank=None,
                                    lists=(np_of(ref["ranges"]), np_of(ref["gsid"])), dout=np_of(g),
                                    dT=np_of(gT))
    for name, d in zip(NAMES, got):
        e = rel_err(d.float().reshape(n, -1), r["d" + name].reshape(n, -1))
        assert e < (4e-3 if name == "shs" and dtype == torch.bfloat16 else 1e-4), (name, e)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_unaligned_rows_and_views_sum(cuda_ok, dtype):
    n, K = 130, 5
    cams = [look_at(e, width=W, height=H, device="cuda") for e in ((0.0, -8.0, 0.0), (5, 5, 3))]
    ups = [_upstream(K, s) for s in (1, 2)]
    _, leaf = _leaves(n, K, dtype)
    _, odd = _leaves(n, K, dtype, shift=1)
    single = [_grads(leaf, c, *u) for c, u in zip(cams, ups)]
    for a, b in zip(single[0], _grads(odd, cams[0], *ups[0])):
        assert rel_err(a, b) < 1e-5  # the compositing adjoint adds in any order
    layers, taus, _ = render_palette_views(leaf["pws"], leaf["rots"], leaf["scales"], leaf["alphas"],
                                           cams, shs=leaf["shs"])
    total = sum((la * g).sum() + (t * gT).sum() for la, t, (g, gT) in zip(layers, taus, ups))
    both = torch.autograd.grad(total, [leaf[k] for k in NAMES])
    tol = 1e-5 if dtype == torch.float32 else 8e-3  # (one rounding to BF16 against two)
    for name, a, b, s in zip(NAMES, single[0], single[1], both):
        assert rel_err(s, np_of(a) + np_of(b)) < (tol if name == "shs" else 1e-5), name
        assert np.isfinite(np_of(s)).all()
