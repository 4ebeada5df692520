"""The L1 + SSIM loss kernel at the edges of its strips (32 columns), steps (11 rows)
and segments: loss parts and gradients against the FP64 oracle.  Bounds as derived
for the FP32 kernel elsewhere: 2e-6 for the means of values in [0, 1], 1e-4 of the
largest gradient."""
import numpy as np
import pytest
import torch

from oracle import oracle as orc
from palette_b200.loss import palette_l1_ssim_loss
from helpers import np_of

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("K,H,W", [(5, 2, 31), (4, 3, 32), (5, 11, 33), (2, 13, 64), (3, 14, 65),
                                   (5, 24, 300), (5, 47, 1), (6, 1, 97), (7, 300, 200),
                                   (5, 430, 333), (3, 700, 450)])
def test_strips_and_segments_match_oracle(cuda_ok, K, H, W):
    rng = np.random.default_rng(H * 7 + W)
    layer = rng.normal(0.2, 0.3, (K, H, W)).astype(np.float32)
    pal = rng.random((K, 3)).astype(np.float32)
    tgt = rng.random((3, H, W)).astype(np.float32)
    ref = orc.palette_l1_ssim_loss(layer, pal, tgt, 0.2, 0.5)
    L = torch.from_numpy(layer).cuda().requires_grad_()
    P = torch.from_numpy(pal).cuda().requires_grad_()
    loss, parts = palette_l1_ssim_loss(L, P, torch.from_numpy(tgt).cuda(), 0.2, 0.5, parts=True)
    loss.backward()
    parts = np_of(parts)
    for got, want in ((float(loss), "loss"), (parts[1], "l1"), (parts[2], "ssim"),
                      (parts[3], "penalty")):
        assert abs(got - ref[want]) < 2e-6, want
    for got, want in ((L.grad, "dlayer"), (P.grad, "dpalette")):
        err = np.abs(np_of(got).astype(np.float64) - ref[want]).max() / np.abs(ref[want]).max()
        assert err < 1e-4, want
