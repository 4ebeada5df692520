"""Full-SH rows staged in their storage type: a render from BF16 coefficients equals,
bit for bit, the render from the same values in FP32, around the edges of a block of
64 Gaussians, for each row length, on aligned and on unaligned arrays."""
import pytest
import torch

from palette_b200.render import render_palette
from palette_b200.scene import look_at, synthetic_scene, to_torch

pytestmark = pytest.mark.gpu

H, W = 90, 120


def _shifted(t, shift):
    flat = torch.empty(t.numel() + shift, dtype=t.dtype, device="cuda")
    flat[shift:] = t.reshape(-1)
    return flat[shift:].view(t.shape)


@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize("K", [3, 5, 8])
@pytest.mark.parametrize("n", [1, 63, 64, 65, 1000])
def test_bf16_rows_equal_fp32_rows(cuda_ok, n, K, shift):
    st = to_torch(synthetic_scene(n, seed=n + K, K=K), "cuda", torch.bfloat16)
    cam = look_at((0.0, -8.0, 0.0), width=W, height=H, device="cuda")
    with torch.no_grad():
        out = [render_palette(st["pws"], st["rots"], st["scales"] * 8.0, st["alphas"], cam,
                              shs=_shifted(shs, shift))
               for shs in (st["shs"], st["shs"].float())]
    for a, b in zip(*out):
        assert torch.equal(a, b)
