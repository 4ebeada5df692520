"""The losses' backward where its one-launch scale does not apply: batched incoming
gradients, and saved gradients that a hook hands back in another layout or type.
The products are then torch's, as for a loss written in torch."""
import pytest
import torch

from palette_b200 import loss as pl

pytestmark = pytest.mark.gpu

H, W = 20, 33


def _losses():
    gen = torch.Generator("cuda").manual_seed(4)
    rnd = lambda *s: torch.rand(s, device="cuda", generator=gen)  # noqa: E731
    layer, target = rnd(5, H, W), rnd(3, H, W)
    return [(lambda x, p: pl.palette_l1_loss(x, p, target), layer, rnd(5, 3)),
            (lambda x, p: pl.palette_geo_loss(x, p, target), layer, rnd(3, 3)),
            (lambda x, p: pl.palette_l1_ssim_loss(x, p, target), layer, rnd(5, 3))]


@pytest.mark.parametrize("which", range(3))
def test_batched_gradients(cuda_ok, which):
    f, layer, pal = _losses()[which]
    x, p = layer.requires_grad_(), pal.requires_grad_()
    loss = f(x, p)
    one = torch.autograd.grad(loss, (x, p), retain_graph=True)
    scale = torch.tensor([1.0, -2.0, 0.5], device="cuda")
    many = torch.autograd.grad(loss, (x, p), scale, is_grads_batched=True)
    for a, b in zip(one, many):
        assert torch.equal(b, torch.stack([a * s for s in scale]))


def _strided(t):
    wide = torch.zeros(t.shape + (2,), dtype=t.dtype, device=t.device)
    wide[..., 0] = t
    return wide[..., 0]


@pytest.mark.parametrize("unpack", [_strided, lambda t: t.double()], ids=["strided", "double"])
@pytest.mark.parametrize("which", range(3))
def test_saved_tensor_hooks(cuda_ok, which, unpack):
    f, layer, pal = _losses()[which]
    x, p = layer.requires_grad_(), pal.requires_grad_()
    changed = []
    with torch.autograd.graph.saved_tensors_hooks(lambda t: t,
                                                  lambda t: unpack(t) if changed else t):
        loss = f(x, p)
    one = torch.autograd.grad(3.0 * loss, (x, p), retain_graph=True)
    changed.append(True)
    for a, b in zip(one, torch.autograd.grad(3.0 * loss, (x, p))):
        assert torch.equal(a, b.float())
