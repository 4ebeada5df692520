"""splat_palette_weights under saved-tensor hooks that hand back another layout,
alignment or type: the backward reads dense tensors of the saved types, as the
operators' own checks ensured, or refuses.  (Sums differ by the order of the
compositing adjoint's additions only.)"""
import pytest
import torch

from palette_b200.scene import look_at, synthetic_scene, to_torch
from palette_b200.weights import splat_palette_weights
from helpers import rel_err

pytestmark = pytest.mark.gpu


def _strided(t):
    """The same values at twice the stride."""
    wide = torch.zeros(t.shape + (2,), dtype=t.dtype, device=t.device)
    wide[..., 0] = t
    return wide[..., 0]


def _shifted(t):
    flat = torch.empty(t.numel() + 16, dtype=t.dtype, device=t.device)
    flat[16:] = t.reshape(-1)
    return flat[16:].view(t.shape)


def _grads(unpack, rank):
    full = rank == 0
    st = to_torch(synthetic_scene(3000, seed=2, mode="full" if full else "lowrank", rank=rank or 1),
                  "cuda")
    w = {k: st[k].requires_grad_() for k in (("shs",) if full else ("dc", "A", "B"))}
    cam = look_at((0.0, -8.0, 0.0), width=75, height=50, device="cuda")
    with torch.autograd.graph.saved_tensors_hooks(lambda t: t, unpack):
        layer, _ = splat_palette_weights(st["pws"], st["alphas"], st["scales"], st["rots"], cam, **w)
    up = torch.randn(layer.shape, device="cuda", generator=torch.Generator("cuda").manual_seed(3))
    return torch.autograd.grad((layer * up).sum(), list(w.values()))


@pytest.mark.parametrize("rank", [0, 3])
@pytest.mark.parametrize("unpack", [_strided, _shifted], ids=["strided", "shifted"])
def test_other_layouts_are_made_dense(cuda_ok, unpack, rank):
    for a, b in zip(_grads(unpack, rank), _grads(lambda t: t, rank)):
        assert rel_err(a, b) < 1e-5


@pytest.mark.parametrize("kind", [torch.float32, torch.int32])
def test_other_types_are_refused(cuda_ok, kind):
    narrow = {torch.float32: torch.float16, torch.int32: torch.int16}[kind]
    with pytest.raises(TypeError):
        _grads(lambda t: t.to(narrow) if t.dtype == kind else t, 3)
