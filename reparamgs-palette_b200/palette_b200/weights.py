"""Palette-weight splatting with frozen geometry: the rendered layers of the
operator sequence, with a fused weight-parameter adjoint.

``splat_palette_weights(pws, alphas, scales, rots, cam, shs=... | dc=, A=, B=)``
returns ``(layer [K,H,W], visible [N])`` -- the rendered palette-weight layers
and the ``depths > 0.2`` mask -- and is differentiable in the weight
parameters (geometry is frozen, as in ReparamGS-Palette's finetune stage,
gsplat/gsmodel.py:104-200).  It computes what the reference's own autograd
functions compute, organised differently:

* forward: the operator chain project -> computeCov3D -> computeCov2D ->
  sh2Weight / sh2Weight_fast -> inverseCov2D -> splat_weight as one kernel per
  Gaussian (gsb_render_preprocess, same geometry, tile lists and contributor
  indices bit for bit), tile sort and compositing.  Run as the operators, the
  chain is seven launches that pass their intermediates through HBM: 0.130 ms
  at 1M Gaussians with rank-3 factors against 0.077 ms.
* backward: the weights-only compositing adjoint, then one kernel that
  recomputes the view direction and SH basis per Gaussian and writes dL/dshs
  [N,16K] -- or dL/ddc, dL/dA, dL/dB for rank-r factors -- directly, where the
  reference runs a batched outer product in torch (full weights) or an
  elementwise product plus sh2Weight_fast_B (low rank).

Weight parameters may be FP32 or BF16 (FP32 arithmetic; gradients come back
in the parameter's dtype).  Low-rank factors are ``A [N,P]``/``B [N,Q]``
(rank 1, the reference's layout) or ``A [N,P,r]``/``B [N,r,Q]``.  Supported
shapes are those of the fused kernels (full SH with K in 3..8; low-rank
(K,P,Q,r) in (5,5,15,1..4), (3,3,15,1), (4,4,15,1), (6,6,15,1), (6,6,15,3));
other shapes render through the operators and have no backward here.
"""
import ctypes as C

import torch

import gsplatcu as gsc
from gsplatcu import _lib

from .render import _check_rows, _params, _render_one, _weight_args, camera_struct

_F32, _I32 = torch.float32, torch.int32

# Low-rank shapes (K, P, Q, rank) of the fused kernels; full SH: K in 3..8.
_FUSED_LOWRANK = {(5, 5, 15, 1), (5, 5, 15, 2), (5, 5, 15, 3), (5, 5, 15, 4), (3, 3, 15, 1),
                  (4, 4, 15, 1), (6, 6, 15, 1), (6, 6, 15, 3)}


def _operator_chain(pws, alphas, scales, rots, w0, A, B, cam, mode, K, Q):
    """(layer, depths) through the operators, for shapes without a fused kernel."""
    us, pcs, depths = gsc.project(pws, cam.Rcw, cam.tcw, cam.fx, cam.fy, cam.cx, cam.cy, False)
    cov3, = gsc.computeCov3D(rots, scales, depths, False)
    cov2, = gsc.computeCov2D(cov3, pcs, cam.Rcw, depths, cam.fx, cam.fy, cam.width, cam.height,
                             False)
    if mode == _lib.WEIGHTS_FULL:
        w, = gsc.sh2Weight(w0, pws, cam.twc, False, K)
    else:
        w, = gsc.sh2Weight_fast(w0, A, B, pws, cam.twc, False, K, Q)
    cinv, areas = gsc.inverseCov2D(cov2, depths, False)
    layer = gsc.splat_weight(cam.height, cam.width, K, us, cinv, alphas, depths, w, areas)[0]
    return layer, depths


def _as_saved(t, dtype):
    return t.dtype is dtype and t.is_cuda and t.is_contiguous()


def _saved(t, dtype):
    """A tensor kept from the forward, as the library reads it: saved-tensor hooks
    may have handed back another layout (made dense) or type (refused)."""
    if t is None:
        return None
    if t.dtype != dtype or not t.is_cuda:
        raise TypeError(f"splat_palette_weights: a saved tensor came back as {t.dtype} on "
                        f"{t.device}, saved as {dtype} on a CUDA device")
    return t.contiguous()


class _SplatWeights(torch.autograd.Function):
    @staticmethod
    def forward(ctx, pws, alphas, scales, rots, w0, A, B, cam, mode, K, P, Q, rank):
        fused = 3 <= K <= 8 if mode == _lib.WEIGHTS_FULL else (K, P, Q, rank) in _FUSED_LOWRANK
        ctx.meta = (cam, mode, K, P, Q, rank, w0.dtype)
        if fused:
            layer, tau, depths, state, ranges, gsid, contrib = _render_one(
                pws, rots, scales, alphas, w0, A, B, cam, mode, K, P, Q, rank)
            ctx.save_for_backward(pws, w0, A, B, state, ranges, gsid, contrib, tau)
        else:
            layer, depths = _operator_chain(pws, alphas, scales, rots, w0, A, B, cam, mode, K, Q)
            ctx.save_for_backward(pws, w0, A, B, None, None, None, None, None)
        visible = depths > 0.2
        ctx.mark_non_differentiable(visible)
        return layer, visible

    @staticmethod
    def backward(ctx, dlayer, _dvisible):
        cam, mode, K, P, Q, rank, wt = ctx.meta
        pws, w0, A, B, state, ranges, gsid, contrib, tau = ctx.saved_tensors
        if state is None:
            raise _lib.GsplatError(
                f"splat_palette_weights: unsupported palette parameter shape (K={K}, P={P}, Q={Q}, "
                f"rank={rank}) in the backward (status {_lib.GSB_ERR_UNSUPPORTED})",
                _lib.GSB_ERR_UNSUPPORTED)
        if not (_as_saved(pws, _F32) and _as_saved(tau, _F32) and _as_saved(state, torch.uint8) and
                _as_saved(ranges, _I32) and _as_saved(gsid, _I32) and _as_saved(contrib, _I32) and
                _as_saved(w0, wt) and (A is None or (_as_saved(A, wt) and _as_saved(B, wt))) and
                state.data_ptr() % 256 == 0):
            pws, tau, state = _saved(pws, _F32), _saved(tau, _F32), _saved(state, torch.uint8).clone()
            ranges, gsid, contrib = _saved(ranges, _I32), _saved(gsid, _I32), _saved(contrib, _I32)
            w0, A, B = _saved(w0, wt), _saved(A, wt), _saved(B, wt)
        dev = pws.device
        n = int(pws.shape[0])
        camst, _keep = camera_struct(cam)
        params = _params(mode, K, P, Q, rank, w0, A, B)
        dlayer = dlayer.contiguous()
        dw0 = torch.empty(tuple(w0.shape), dtype=_F32, device=dev)
        dA = torch.empty(tuple(A.shape), dtype=_F32, device=dev) if A is not None else None
        dB = torch.empty(tuple(B.shape), dtype=_F32, device=dev) if B is not None else None
        with _lib.on_device(dev):
            scratch = torch.empty(int(_lib.lib().gsb_render_backward_bytes(n, K)),
                                  dtype=torch.uint8, device=dev)
            st = _lib.stream_of(pws)
            _lib.call("splat_palette_weights.backward", "gsb_render_backward", n, C.byref(camst),
                      _lib.ptr(pws), None, None, None, C.byref(params), _lib.ptr(state),
                      _lib.ptr(ranges), _lib.ptr(gsid), _lib.ptr(contrib), _lib.ptr(tau),
                      _lib.ptr(dlayer), None, _lib.ptr(scratch), None, None, None, None,
                      _lib.ptr(dw0), _lib.ptr(dA), _lib.ptr(dB), st)
            _lib.fetch_device_status(dev, st)
        cast = lambda g, like: None if g is None else g.to(like.dtype)
        return (None, None, None, None, cast(dw0, w0), cast(dA, A), cast(dB, B),
                None, None, None, None, None, None)


def splat_palette_weights(pws, alphas, scales, rots, cam, shs=None, dc=None, A=None, B=None,
                          K=None):
    """Render the palette-weight layers of the operator sequence.  Pass
    ``shs [N,16K]`` (full SH order 3, band-major) or ``dc [N,K], A, B``
    (low rank).  Returns ``(layer [K,H,W], visible [N] bool)``; gradients
    flow to the weight parameters only."""
    for name, t in (("pws", pws), ("alphas", alphas), ("scales", scales), ("rots", rots)):
        if not (isinstance(t, torch.Tensor) and t.is_cuda and t.dtype == _F32):
            raise TypeError(f"splat_palette_weights: {name} must be a CUDA float32 tensor")
    for name in ("Rcw", "tcw", "twc"):
        gsc._cuda("splat_palette_weights", name, getattr(cam, name))
    w0, A, B, mode, K, P, Q, rank = _weight_args(shs, dc, A, B, K)
    _check_rows(pws, rots, scales, alphas, w0, A, B, mode, K, P, Q, rank)
    return _SplatWeights.apply(pws.contiguous(), alphas.contiguous(), scales.contiguous(),
                               rots.contiguous(), w0, A, B, cam, mode, K, P, Q, rank)
