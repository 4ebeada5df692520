"""The L1 + SSIM loss on both sides of the line between its two forms (at most 148
segments of up to six steps: one block per SM), for every channel count and for a
colour image: loss parts and gradients against the FP64 oracle.  Bounds as for the
kernel's other sizes: 2e-6 for the means of values in [0, 1], 1e-4 of the largest
gradient.  Where image and target agree to FP32 rounding (eight products below 2:
1e-6) the sign of the L1 term is not determined in FP32; such pixels are left out."""
import numpy as np
import pytest
import torch

from oracle import oracle as orc
from palette_b200.loss import gau_loss, palette_l1_ssim_loss
from helpers import np_of

pytestmark = pytest.mark.gpu


def _rel(got, want, where=True):
    err = np.abs(np_of(got).astype(np.float64) - want) * where
    return err.max() / np.abs(want).max()


def _off_the_kink(layer, pal, tgt):
    x = np.einsum("kc,khw->chw", pal.astype(np.float64), layer.astype(np.float64))
    return (np.abs(x - tgt) > 1e-6).all(0)


@pytest.mark.parametrize("H,W", [(414, 500), (415, 500),   # 144 segments of six steps; 160
                                 (2, 148 * 32), (3, 148 * 32 + 1), (41, 33)])
@pytest.mark.parametrize("K", range(1, 9))
def test_both_forms_match_oracle(cuda_ok, K, H, W):
    rng = np.random.default_rng(K * 1000 + H)
    layer = rng.normal(0.2, 0.3, (K, H, W)).astype(np.float32)
    pal = rng.random((K, 3)).astype(np.float32)
    tgt = rng.random((3, H, W)).astype(np.float32)
    ref = orc.palette_l1_ssim_loss(layer, pal, tgt, 0.2, 0.5)
    L = torch.from_numpy(layer).cuda().requires_grad_()
    P = torch.from_numpy(pal).cuda().requires_grad_()
    loss, parts = palette_l1_ssim_loss(L, P, torch.from_numpy(tgt).cuda(), 0.2, 0.5, parts=True)
    loss.backward()
    parts = np_of(parts)
    for got, want in ((float(loss.detach()), "loss"), (parts[1], "l1"), (parts[2], "ssim"),
                      (parts[3], "penalty")):
        assert abs(got - ref[want]) < 2e-6, want
    assert _rel(L.grad, ref["dlayer"], _off_the_kink(layer, pal, tgt)) < 1e-4
    assert _rel(P.grad, ref["dpalette"]) < 1e-4


@pytest.mark.parametrize("H,W", [(414, 500), (415, 500)])
def test_colour_image_in_both_forms(cuda_ok, H, W):
    rng = np.random.default_rng(H)
    img, tgt = rng.random((2, 3, H, W)).astype(np.float32)
    ref = orc.palette_l1_ssim_loss(img, np.eye(3, dtype=np.float32), tgt, 0.2, 0.0)
    x = torch.from_numpy(img).cuda().requires_grad_()
    loss = gau_loss(x, torch.from_numpy(tgt).cuda(), 0.2)
    loss.backward()
    assert abs(float(loss.detach()) - ref["loss"]) < 2e-6
    assert _rel(x.grad, ref["dlayer"], _off_the_kink(img, np.eye(3), tgt)) < 1e-4
