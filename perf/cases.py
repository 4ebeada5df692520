"""Timed workloads of the palette-weight rasterizer and their FP64 values.

Every case goes through the package's public entry points, as a user's program
calls them, with inputs of the distributions that the synthetic scenes use
(means from a mixture of 8 Gaussians, log-scales N(-4.5, 0.8), opacity
sigmoid(N(0, 1.5)), Dirichlet DC weights, small higher orders) drawn on the
device from the seed.  The kinds of call:

  finetune  one finetune step: splat_palette_weights, palette_geo_loss, backward
  render    one view rendered without gradients (render_palette)
  train     render_palette with gradients for every parameter, palette L1 loss
  views     a batch of views (render_palette_views), L1 + SSIM loss, backward
  color     the stage-1 colour path: operators, splat, splatB
  geo_loss  palette_geo_loss on a rendered layer stack, with its gradients
  ssim_loss palette_l1_ssim_loss on a layer stack, with its gradients
  sh        the SH operators alone, with Jacobian outputs and the factor adjoint
  serve     palette-edit requests through PaletteServer

``rank`` 0 means full order-3 SH weights, 1..4 low-rank factors of that rank.
"""
import math
import os
import sys

_PKG = os.path.join(os.getcwd(), "reparamgs-palette_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import torch  # noqa: E402

import gsplatcu as gsc  # noqa: E402
from palette_b200.loss import (palette_geo_loss, palette_l1_loss,  # noqa: E402
                               palette_l1_ssim_loss)
from palette_b200.render import render_palette, render_palette_views  # noqa: E402
from palette_b200.scene import look_at  # noqa: E402
from palette_b200.serve import PaletteServer, Request, Scene  # noqa: E402
from palette_b200.weights import splat_palette_weights  # noqa: E402


def _case(kind, n, w, h, K=5, rank=3, bf16=False, radius=8.0, **more):
    return dict(kind=kind, n=n, width=w, height=h, K=K, rank=rank, bf16=bf16, radius=radius, **more)


def listed():
    return [
        # the smallest scene of the configurations: latency and launches count
        dict(_case("finetune", 20_000, 256, 256, rank=0, clamp=False, loss="mse"),
             name="finetune_20k_256"),
        # the headline finetune step
        dict(_case("finetune", 1_000_000, 1920, 1080, rank=3, clamp=True, loss="l1"),
             name="finetune_1m_1080p"),
        # a photo capture's odd size, seen from close by, rank-1 factors of six anchors
        dict(_case("finetune", 300_000, 1297, 841, K=6, rank=1, radius=6.0, clamp=True, loss="mse"),
             name="finetune_300k_odd"),
        # viewing a finetuned scene kept in BF16
        dict(_case("render", 1_000_000, 1920, 1080, rank=3, bf16=True), name="render_1m_1080p"),
        # the largest scene and resolution that are served
        dict(_case("render", 3_000_000, 3840, 2160, rank=0, bf16=True), name="render_3m_4k"),
        # joint training: gradients of geometry, opacity and weights
        dict(_case("train", 500_000, 1920, 1080, rank=0), name="train_500k_1080p"),
        # the multi-view finetune step, BF16 factors, fewer views
        dict(_case("views", 250_000, 1280, 720, rank=3, bf16=True, views=2, geometry=False),
             name="views_250k_720p"),
        # stage-1 colour training, forward and backward
        dict(_case("color", 400_000, 1600, 1063, K=3, rank=0), name="color_400k"),
        # the two image losses by themselves
        dict(_case("geo_loss", 0, 1920, 1080, clamp=True, loss="l1"), name="geo_loss_1080p"),
        dict(_case("ssim_loss", 0, 1920, 1080), name="ssim_loss_1080p"),
        # the SH operators as the reference's own caller uses them (with Jacobians)
        dict(_case("sh", 1_000_000, 0, 0, rank=1), name="sh_1m"),
        # palette-edit requests at three resolutions against two resident scenes
        dict(_case("serve", 250_000, 1920, 1080, rank=3, requests=6), name="serve_250k"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _size(rng, lo, hi):
    """Width and height of a view whose pixels lie between lo and hi."""
    px = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    aspect = rng.choice([1.0, 4.0 / 3.0, 1.5, 16.0 / 9.0])
    w = max(16, int(math.sqrt(px * aspect)) + rng.randrange(-3, 4))
    return w, max(16, min(int(px / w), hi // w))


def _weights(rng):
    """(K, rank) of a supported weight form."""
    rank = rng.choice([0, 0, 1, 1, 2, 3, 3, 4])
    if rank == 0:
        return rng.choice([3, 4, 5, 5, 6, 7, 8]), 0
    return {1: rng.choice([3, 4, 5, 5, 6]), 2: 5, 3: rng.choice([5, 5, 6]), 4: 5}[rank], rank


def draw(rng):
    kind = rng.choice(["finetune", "finetune", "render", "render", "train", "views", "color",
                       "geo_loss", "ssim_loss", "sh", "serve"])
    K, rank = _weights(rng)
    bf16 = rng.random() < 0.4
    radius = round(rng.uniform(6.0, 14.0), 2)
    px = 1920 * 1080
    if kind == "finetune":
        return _case(kind, _log_int(rng, 5_000, 1_000_000), *_size(rng, 128 * 128, px), K, rank,
                     bf16, radius, clamp=rng.random() < 0.5, loss=rng.choice(["mse", "l1"]))
    if kind == "render":
        return _case(kind, _log_int(rng, 5_000, 2_000_000), *_size(rng, 128 * 128, 4 * px), K, rank,
                     bf16, radius)
    if kind == "train":
        return _case(kind, _log_int(rng, 5_000, 400_000), *_size(rng, 128 * 128, px), K, rank, bf16,
                     radius)
    if kind == "views":
        return _case(kind, _log_int(rng, 5_000, 200_000), *_size(rng, 128 * 128, 1280 * 720), K,
                     rank, bf16, radius, views=rng.choice([2, 3]), geometry=rng.random() < 0.3)
    if kind == "color":
        return _case(kind, _log_int(rng, 5_000, 400_000), *_size(rng, 128 * 128, px), 3, 0, False,
                     radius)
    if kind in ("geo_loss", "ssim_loss"):
        K = rng.choice([4, 5, 5, 6, 7]) if kind == "geo_loss" else rng.choice([3, 4, 5, 5, 6, 8])
        more = dict(clamp=rng.random() < 0.5, loss=rng.choice(["mse", "l1"])) \
            if kind == "geo_loss" else {}
        return _case(kind, 0, *_size(rng, 64 * 64, 2 * px), K, 0, False, 8.0, **more)
    if kind == "sh":
        return _case(kind, _log_int(rng, 5_000, 1_000_000), 0, 0, K, max(rank, 1) if K == 5 else 1,
                     bf16, radius)
    return _case(kind, _log_int(rng, 20_000, 250_000), 1920, 1080, 5, 3, False, radius,
                 requests=rng.choice([2, 4, 6]))


# ---------------------------------------------------------------- inputs
def _anchors(count, gen):
    """Chromatic palette anchors [count,3] of well separated hues, as an extracted palette has."""
    hue, sat, val = torch.rand((3, count), generator=gen, device="cuda")
    hue = (torch.arange(count, device="cuda") + 0.3 * hue) / max(count, 3)
    ramp = (hue[:, None] * 6 + torch.tensor([0.0, 4.0, 2.0], device="cuda")) % 6
    rgb = (torch.abs(ramp - 3) - 1).clamp(0, 1)
    return (0.6 + 0.4 * val[:, None]) * (1 - (0.6 + 0.4 * sat[:, None]) * (1 - rgb))


def _scene(case, gen):
    n, K, rank = case["n"], case["K"], case["rank"]
    dev = "cuda"
    rand = lambda *s: torch.rand(s, generator=gen, device=dev)  # noqa: E731
    randn = lambda *s: torch.randn(s, generator=gen, device=dev)  # noqa: E731
    centres = rand(8, 3) * 6.0 - 3.0
    pick = torch.randint(0, 8, (n,), generator=gen, device=dev)
    sc = dict(pws=centres[pick] + 0.8 * randn(n, 3), scales=torch.exp(0.8 * randn(n, 3) - 4.5))
    q = randn(n, 4)
    sc["rots"] = q / q.norm(dim=1, keepdim=True)
    sc["alphas"] = torch.sigmoid(1.5 * randn(n, 1))
    sc["palette"] = torch.cat([torch.zeros(1, 3, device=dev), torch.ones(1, 3, device=dev),
                               _anchors(max(K - 2, 1), gen)])[:K].contiguous()
    dc = -torch.log(rand(n, K).clamp_min(1e-12))
    dc = dc / dc.sum(dim=1, keepdim=True)
    if rank == 0:
        sc["shs"] = torch.cat([dc[:, None], 0.05 * randn(n, 15, K)], dim=1).reshape(n, 16 * K)
    else:
        sc["dc"] = dc
        sc["A"] = 0.1 * randn(n, K, rank)
        sc["B"] = 0.1 * randn(n, rank, 15)
    if case["bf16"]:
        for k in ("shs", "dc", "A", "B"):
            if k in sc:
                sc[k] = sc[k].to(torch.bfloat16)
    return {k: v.contiguous() for k, v in sc.items()}


def _eye(case, cpu):
    d = torch.randn(3, generator=cpu, dtype=torch.float64)
    return (d / d.norm() * case["radius"]).tolist()


def _weight_args(sc):
    return {k: sc[k] for k in ("shs", "dc", "A", "B") if k in sc}


def _layers(case, gen):
    """A layer stack like a rendered one: mostly convex weights, some below 0."""
    K, h, w = case["K"], case["height"], case["width"]
    x = torch.rand((K, h, w), generator=gen, device="cuda")
    x = x / x.sum(dim=0, keepdim=True)
    return (x + 0.05 * torch.randn((K, h, w), generator=gen, device="cuda")).contiguous()


def prepare(case, seed):
    gen = torch.Generator("cuda").manual_seed(seed)
    cpu = torch.Generator("cpu").manual_seed(seed)
    kind, K, w, h = case["kind"], case["K"], case["width"], case["height"]
    st = dict(case=case)
    image = lambda: torch.rand((3, h, w), generator=gen, device="cuda")  # noqa: E731
    if kind in ("geo_loss", "ssim_loss"):
        st["layer"] = _layers(case, gen).requires_grad_()
        colours = _anchors(max(K - 2, 1), gen)
        if kind == "geo_loss":
            st["chroma"] = colours.requires_grad_()
        else:
            st["palette"] = torch.cat([torch.zeros(1, 3, device="cuda"),
                                       torch.ones(1, 3, device="cuda"), colours])[:K]
            st["palette"] = st["palette"].contiguous().requires_grad_()
        st["target"] = image()
        return st
    sc = st["scene"] = _scene(case, gen)
    eye = _eye(case, cpu)
    if kind == "sh":
        st["twc"] = torch.tensor(eye, dtype=torch.float32, device="cuda")
        dc = torch.rand((case["n"], K), generator=gen, device="cuda")
        sc["shs"] = torch.cat([dc[:, None], 0.05 * torch.randn(
            (case["n"], 15, K), generator=gen, device="cuda")], dim=1).reshape(case["n"], 16 * K)
        sc["shs"] = sc["shs"].to(sc["dc"].dtype).contiguous()
        st["dweights"] = torch.randn((case["n"], K), generator=gen, device="cuda")
        return st
    if kind == "serve":
        return _prepare_serve(case, st, gen, cpu)
    st["cam"] = look_at(eye, width=w, height=h, device="cuda")
    if kind in ("finetune", "train", "views"):
        names = list(_weight_args(sc))
        if kind == "train" or case.get("geometry"):
            names += ["pws", "rots", "scales", "alphas"]
        st["names"] = names
        for k in names:
            sc[k].requires_grad_()
    if kind == "finetune":
        if K > 3:  # (the barycentric loss takes two chromatic anchors or more)
            st["chroma"] = sc["palette"][2:].clone().requires_grad_()
        st["target"] = image()
    elif kind == "train":
        st["target"] = image()
    elif kind == "views":
        st["cams"] = [st["cam"]] + [look_at(_eye(case, cpu), width=w, height=h, device="cuda")
                                    for _ in range(case["views"] - 1)]
        st["targets"] = [image() for _ in st["cams"]]
        sc["palette"].requires_grad_()
    elif kind == "color":
        st["dimage"] = torch.randn((3, h, w), generator=gen, device="cuda") / (3 * h * w)
        st["dtau"] = torch.rand((h, w), generator=gen, device="cuda") / (h * w)
    return st


_RESOLUTIONS = ((1280, 720), (1920, 1080), (3840, 2160))


def _prepare_serve(case, st, gen, cpu):
    full = _scene(dict(case, rank=0), gen)
    low = {k: v.to(torch.bfloat16) if k in ("dc", "A", "B") else v for k, v in st["scene"].items()}
    st["scenes"] = dict(full=full, low=low)
    srv = st["server"] = PaletteServer(hbm_budget=40 << 30, slots=4)
    res = []
    for w, h in _RESOLUTIONS:
        c = look_at((0, -8, 0), width=w, height=h, device="cpu")
        res.append((w, h, c.fx, c.fy, c.cx, c.cy))
    st["requests"] = []
    views = []
    for i in range(case["requests"]):
        w, h, fx, fy, cx, cy = res[i % 3]
        c = look_at(_eye(case, cpu), width=w, height=h, device="cpu")
        views.append((("full", "low")[(i // 3 + i) % 2], c))
    probes = [(c.Rcw.numpy(), c.tcw.numpy()) for _, c in views]
    for sid, s in st["scenes"].items():
        wt = {k: s[k] for k in ("shs", "dc", "A", "B") if k in s}
        if not srv.admit_scene(Scene(sid, s["pws"], s["rots"], s["scales"], s["alphas"], **wt), res,
                               probes):
            raise RuntimeError(srv.last_admit_error)
    for sid, c in views:
        pal = st["scenes"][sid]["palette"].cpu().clone()
        pal[2:] = (pal[2:] + 0.15 * torch.randn(pal[2:].shape, generator=cpu)).clamp(0, 1)
        st["requests"].append(Request(sid, c.Rcw.numpy(), c.tcw.numpy(), c.fx, c.fy, c.cx, c.cy,
                                      c.width, c.height, pal.numpy()))
    srv.prepare(st["requests"])
    return st


# ------------------------------------------------------------------ passes
def _grads(total, tensors):
    return list(torch.autograd.grad(total, tensors))


def run(st):
    case, sc = st["case"], st.get("scene")
    kind = case["kind"]
    if kind == "finetune":
        wt = _weight_args(sc)
        layer, visible = splat_palette_weights(sc["pws"], sc["alphas"], sc["scales"], sc["rots"],
                                               st["cam"], **wt)
        if case["K"] > 3:
            loss = palette_geo_loss(layer, st["chroma"], st["target"], clamp=case["clamp"],
                                    lambda_pos=0.5, kind=case["loss"])
            g = _grads(loss, [sc[k] for k in st["names"]] + [st["chroma"]])
        else:
            loss = palette_l1_loss(layer, sc["palette"], st["target"])
            g = _grads(loss, [sc[k] for k in st["names"]])
        return dict(layer=layer.detach(), visible=visible, loss=loss.detach(), grads=g)
    if kind == "render":
        with torch.no_grad():
            layer, tau, depths = render_palette(sc["pws"], sc["rots"], sc["scales"], sc["alphas"],
                                                st["cam"], **_weight_args(sc))
        return dict(layer=layer, tau=tau, depths=depths)
    if kind == "train":
        layer, tau, _ = render_palette(sc["pws"], sc["rots"], sc["scales"], sc["alphas"], st["cam"],
                                       **_weight_args(sc))
        loss = palette_l1_loss(layer, sc["palette"], st["target"]) + 0.1 * tau.mean()
        return dict(layer=layer.detach(), tau=tau.detach(), loss=loss.detach(),
                    grads=_grads(loss, [sc[k] for k in st["names"]]))
    if kind == "views":
        layers, _, _ = render_palette_views(sc["pws"], sc["rots"], sc["scales"], sc["alphas"],
                                            st["cams"], **_weight_args(sc))
        total = sum(palette_l1_ssim_loss(la, sc["palette"], t) for la, t in
                    zip(layers, st["targets"])) / len(layers)
        return dict(layers=[la.detach() for la in layers], loss=total.detach(),
                    grads=_grads(total, [sc[k] for k in st["names"]] + [sc["palette"]]))
    if kind == "color":
        return _run_color(st)
    if kind == "geo_loss":
        loss = palette_geo_loss(st["layer"], st["chroma"], st["target"], clamp=case["clamp"],
                                lambda_pos=0.5, kind=case["loss"])
        return dict(loss=loss.detach(), grads=_grads(loss, [st["layer"], st["chroma"]]))
    if kind == "ssim_loss":
        loss = palette_l1_ssim_loss(st["layer"], st["palette"], st["target"])
        return dict(loss=loss.detach(), grads=_grads(loss, [st["layer"], st["palette"]]))
    if kind == "sh":
        K = case["K"]
        w, dshs, dpws = gsc.sh2Weight(sc["shs"], sc["pws"], st["twc"], True, K)
        wf, ddc, ylm = gsc.sh2Weight_fast(sc["dc"], sc["A"], sc["B"], sc["pws"], st["twc"], True, K,
                                          15)
        dA, dB = gsc.sh2Weight_fast_B(sc["A"], sc["B"], ylm, st["dweights"], K, 15)
        return dict(w=w, dshs=dshs, dpws=dpws, wf=wf, ddc=ddc, ylm=ylm, dA=dA, dB=dB)
    srv = st["server"]
    for r in st["requests"]:
        srv.submit(r)
    srv.drain()
    srv.done.clear()
    return [r.image for r in st["requests"]]


def _run_color(st):
    sc, cam = st["scene"], st["cam"]
    us, pcs, depths = gsc.project(sc["pws"], cam.Rcw, cam.tcw, cam.fx, cam.fy, cam.cx, cam.cy,
                                  False)
    cov3, = gsc.computeCov3D(sc["rots"], sc["scales"], depths, False)
    cov2, = gsc.computeCov2D(cov3, pcs, cam.Rcw, depths, cam.fx, cam.fy, cam.width, cam.height,
                             False)
    col, = gsc.sh2Color(sc["shs"], sc["pws"], cam.twc, False)
    cinv, areas = gsc.inverseCov2D(cov2, depths, False)
    image, contrib, tau, ranges, gsid = gsc.splat(cam.height, cam.width, us, cinv, sc["alphas"],
                                                  depths, col, areas)
    du, dq, da, dcol = gsc.splatB(cam.height, cam.width, us, cinv, sc["alphas"], depths, col,
                                  contrib, tau, ranges, gsid, st["dimage"], st["dtau"])
    return dict(image=image, contrib=contrib, tau=tau, du=du, dq=dq, da=da, dcol=dcol)


# -------------------------------------------------------------------- work
def work(case):
    """Bytes in and out once, and the arithmetic no form of the path avoids
    (SH sums; the separable SSIM filters)."""
    n, K, rank = case["n"], case["K"], case["rank"]
    px = case["width"] * case["height"]
    el = 2 if case["bf16"] else 4
    wt = (16 * K if rank == 0 else K + K * rank + 15 * rank) * el * n
    geom = 44 * n
    kind = case["kind"]
    sh = 2.0 * 16 * K * n
    if kind == "finetune":
        return dict(bytes=geom + 2 * wt + n + px * (4 * K + 12), flops=2 * sh)
    if kind == "render":
        return dict(bytes=geom + wt + 4 * n + px * (4 * K + 4), flops=sh)
    if kind == "train":
        return dict(bytes=2 * geom + 2 * wt + px * (4 * K + 16), flops=2 * sh)
    if kind == "views":
        v = case["views"]
        return dict(bytes=(2 if case["geometry"] else 1) * geom + 2 * wt + v * px * (4 * K + 12),
                    flops=v * (2 * sh + 1000.0 * px))
    if kind == "color":
        return dict(bytes=geom + wt + 36 * n + px * (12 + 4 + 4 + 12 + 4), flops=sh)
    if kind == "geo_loss":
        return dict(bytes=px * (8 * K + 12), flops=100.0 * px)
    if kind == "ssim_loss":
        return dict(bytes=px * (8 * K + 12), flops=1000.0 * px)
    if kind == "sh":
        low = (K + 2 * K * rank + 30 * rank) * el + 4 * K
        return dict(bytes=n * (16 * K * el + 12 + 4 * (K + 16 + 3 * K) + low + 4 * (2 * K + 15)),
                    flops=4 * sh)
    v = [_RESOLUTIONS[i % 3] for i in range(case["requests"])]
    return dict(bytes=sum(geom + (320 if (i // 3 + i) % 2 == 0 else 130) * n + 12 * w * h
                          for i, (w, h) in enumerate(v)), flops=len(v) * sh)


# ------------------------------------------------------- values in 64 bits
_C1 = 0.4886025119029199
_C2 = (1.0925484305920792, 0.31539156525252005, 0.5462742152960396)
_C3 = (0.5900435899266435, 2.890611442640554, 0.4570457994644658, 0.3731763325901154,
       1.445305721320277)


def _basis(pws, twc):
    """(SH basis [N,16], unit view directions [N,3])."""
    d = pws - twc
    d = d / d.norm(dim=1, keepdim=True)
    x, y, z = d.unbind(1)
    xx, yy, zz = x * x, y * y, z * z
    return torch.stack([
        torch.full_like(x, 0.28209479177387814), -_C1 * y, _C1 * z, -_C1 * x,
        _C2[0] * x * y, -_C2[0] * y * z, _C2[1] * (2 * zz - xx - yy), -_C2[0] * x * z,
        _C2[2] * (xx - yy), -_C3[0] * y * (3 * xx - yy), _C3[1] * x * y * z,
        -_C3[2] * y * (4 * zz - xx - yy), _C3[3] * z * (2 * zz - 3 * xx - 3 * yy),
        -_C3[2] * x * (4 * zz - xx - yy), _C3[4] * z * (xx - yy), -_C3[0] * x * (xx - 3 * yy)],
        dim=1), d


def _through(value, of):
    """`value`, with the gradient of `of` (clamps are not differentiated)."""
    return value.detach() + (of - of.detach())


def _weights64(p, twc):
    Y, _ = _basis(p["pws"], twc)
    n = Y.shape[0]
    if "shs" in p:
        return torch.einsum("nl,nlk->nk", Y, p["shs"].reshape(n, 16, -1))
    C = torch.bmm(p["A"], p["B"]).reshape(n, 15, -1)
    return Y[:, :1] * p["dc"] + torch.einsum("nl,nlk->nk", Y[:, 1:], C)


def _geometry64(p, cam):
    """Projected centres, conics, depths, tile rectangles of one view."""
    R, t = cam.Rcw.double().cuda(), cam.tcw.double().cuda()
    pc = p["pws"] @ R.T + t
    valid = pc[:, 2] >= 0.2
    z = torch.where(valid, pc[:, 2], torch.ones_like(pc[:, 2]))
    u = torch.stack([pc[:, 0] * cam.fx / z + cam.cx, pc[:, 1] * cam.fy / z + cam.cy], dim=1)
    w, x, y, v = p["rots"].unbind(1)
    rot = torch.stack([1 - 2 * (y * y + v * v), 2 * (x * y - v * w), 2 * (x * v + y * w),
                       2 * (x * y + v * w), 1 - 2 * (x * x + v * v), 2 * (y * v - x * w),
                       2 * (x * v - y * w), 2 * (y * v + x * w), 1 - 2 * (x * x + y * y)],
                      dim=1).reshape(-1, 3, 3)
    M = rot * p["scales"][:, None, :]
    cov = M @ M.transpose(1, 2)
    lim = [1.3 * cam.width / (2 * cam.fx), 1.3 * cam.height / (2 * cam.fy)]
    cx = _through((pc[:, 0] / z).clamp(-lim[0], lim[0]) * z, pc[:, 0])
    cy = _through((pc[:, 1] / z).clamp(-lim[1], lim[1]) * z, pc[:, 1])
    o = torch.zeros_like(z)
    J = torch.stack([cam.fx / z, o, -cam.fx * cx / z ** 2, o, cam.fy / z, -cam.fy * cy / z ** 2],
                    dim=1).reshape(-1, 2, 3)
    T = J @ R
    c2 = T @ cov @ T.transpose(1, 2)
    a, b, c = c2[:, 0, 0] + 0.3, c2[:, 0, 1], c2[:, 1, 1] + 0.3
    det = a * c - b * b
    conic = torch.stack([c / det, -b / det, a / det], dim=1)
    with torch.no_grad():
        ext = torch.stack([torch.ceil(3 * a.abs().sqrt()), torch.ceil(3 * c.abs().sqrt())], dim=1)
        g = torch.tensor([(cam.width + 15) // 16, (cam.height + 15) // 16], device="cuda")
        lo = torch.minimum(((u - ext) / 16).trunc().clamp(0, 1e6).long(), g)
        hi = torch.minimum(((u + ext + 15) / 16).trunc().clamp(0, 1e6).long(), g)
        span = (hi - lo).clamp_min(0) * valid[:, None]
        count = span[:, 0] * span[:, 1]
    return u, conic, torch.where(count > 0, pc[:, 2], -torch.ones_like(z)), (lo, span, count)


class _Lists:
    """The tiles' Gaussian lists: by tile, quantised depth, Gaussian index."""

    def __init__(self, cam, depth, rect):
        lo, span, count = rect
        self.gx, self.gy = (cam.width + 15) // 16, (cam.height + 15) // 16
        self.w, self.h = cam.width, cam.height
        gid = torch.repeat_interleave(torch.arange(count.numel(), device="cuda"), count)
        local = torch.arange(gid.numel(), device="cuda") - (count.cumsum(0) - count)[gid]
        tile = (lo[gid, 1] + local // span[gid, 0]) * self.gx + lo[gid, 0] + local % span[gid, 0]
        key = (tile << 32) | (depth.detach().clamp_min(0) * 1000).long()[gid]
        self.gid = gid[torch.sort(key, stable=True)[1]]
        self.count = torch.bincount(tile, minlength=self.gx * self.gy)
        self.start = self.count.cumsum(0) - self.count

    def groups(self):
        """Batches of tiles of like length: (tile ids, list entries, mask)."""
        order = torch.argsort(self.count, descending=True)
        sizes = [c for c in self.count[order].tolist() if c > 0]
        i = 0
        while i < len(sizes):
            L = sizes[i]
            m = max(1, min(len(sizes) - i, (1 << 16) // L))
            t = order[i:i + m]
            i += m
            k = torch.arange(L, device="cuda")[None]
            mask = k < self.count[t][:, None]
            yield t, self.gid[torch.where(mask, self.start[t][:, None] + k, 0)], mask

    def pixels(self, t):
        k = torch.arange(256, device="cuda")[None]
        return (t % self.gx)[:, None] * 16 + k % 16, (t // self.gx)[:, None] * 16 + k // 16


def _blend(u, q, a, f, mask, px, py):
    """One group of tiles: ([T,256,K] blended features, [T,256] final T)."""
    dx, dy = u[..., 0:1] - px[:, None], u[..., 1:2] - py[:, None]
    m = (q[..., 0:1] * dx * dx + q[..., 2:3] * dy * dy + 2 * q[..., 1:2] * dx * dy)
    g = torch.exp(-0.5 * m.detach().clamp_min(0))
    ap = (a * g.detach()).clamp_max(0.99).detach()
    ap = ap + (a - a.detach()) * g - 0.5 * ap * (m - m.detach())
    ap = torch.where((ap >= 0.002) & mask[..., None], ap, torch.zeros_like(ap))
    lg = torch.log1p(-ap)
    before = torch.exp(torch.cumsum(lg, dim=1) - lg)
    alive = (before >= 1e-4).detach()
    w = ap * before * alive
    return torch.einsum("tlp,tlk->tpk", w, f), torch.exp((lg * alive).sum(dim=1))


def _image64(lists, u, q, a, f, tau_empty):
    K = f.shape[1]
    out = torch.zeros((K, lists.gy * 16, lists.gx * 16), dtype=torch.float64, device="cuda")
    tau = torch.full(out.shape[1:], float(tau_empty), dtype=torch.float64, device="cuda")
    with torch.no_grad():
        for t, g, mask in lists.groups():
            px, py = lists.pixels(t)
            o, T = _blend(u[g], q[g], a[g], f[g], mask, px, py)
            out[:, py, px] = o.permute(2, 0, 1)
            tau[py, px] = T
    return out[:, :lists.h, :lists.w].contiguous(), tau[:lists.h, :lists.w].contiguous()


def _image_adjoint64(lists, u, q, a, f, dout, dtau):
    """Gradients of sum(out dout) + sum(tau dtau) w.r.t. u, q, a, f."""
    pad = (0, lists.gx * 16 - lists.w, 0, lists.gy * 16 - lists.h)
    dout = torch.nn.functional.pad(dout, pad)
    dtau = torch.nn.functional.pad(dtau, pad)
    src = [t.detach() for t in (u, q, a, f)]
    total = [torch.zeros_like(t) for t in src]
    for t, g, mask in lists.groups():
        px, py = lists.pixels(t)
        leaf = [s[g].requires_grad_() for s in src]
        o, T = _blend(*leaf, mask, px, py)
        s = (o * dout[:, py, px].permute(1, 2, 0)).sum() + (T * dtau[py, px]).sum()
        for d, e in zip(total, torch.autograd.grad(s, leaf)):
            d.index_add_(0, g.reshape(-1), e.reshape(-1, e.shape[-1]))
    return total


class _Render64(torch.autograd.Function):
    @staticmethod
    def forward(ctx, u, q, a, f, lists, tau_empty):
        ctx.lists = lists
        ctx.save_for_backward(u, q, a, f)
        return _image64(lists, u, q, a, f, tau_empty)

    @staticmethod
    def backward(ctx, dout, dtau):
        with torch.enable_grad():
            return (*_image_adjoint64(ctx.lists, *ctx.saved_tensors, dout, dtau), None, None)


def _view64(p, cam, feats, tau_empty):
    u, q, depth, rect = _geometry64(p, cam)
    lists = _Lists(cam, depth, rect)
    image, tau = _Render64.apply(u, q, p["alphas"].reshape(-1, 1), feats, lists, tau_empty)
    return image, tau, depth


def _bary_weights64(img, chroma, clamp):
    """Barycentric weights [Kc+2, HW] of colours [3, HW] in {black, white, chroma}."""
    Kc = chroma.shape[0]
    errs, raws = [], []
    for i in range(Kc):
        j = (i + 1) % Kc
        A = torch.stack([torch.ones(3, dtype=img.dtype, device=img.device), chroma[i], chroma[j]],
                        dim=1)
        x = (torch.linalg.inv(A) @ img)
        x = torch.cat([1 - x.sum(dim=0, keepdim=True), x])
        s = torch.nn.functional.softplus(x)
        s = s / (s.sum(dim=0, keepdim=True) + 1e-12)
        errs.append(((A @ s[1:] - img) ** 2).sum(dim=0))
        raw = torch.zeros((Kc + 2, img.shape[1]), dtype=img.dtype, device=img.device)
        idx = torch.tensor([0, 1, i + 2, j + 2], device=img.device)
        raws.append(raw.index_add(0, idx, x))
    prob = torch.softmax(-torch.stack(errs) / 1e-9, dim=0)
    W = sum(prob[i] * raws[i] for i in range(Kc))
    if clamp:
        W = W.clamp_min(0)
        W = W / W.sum(dim=0, keepdim=True).clamp_min(1e-8)
    return W


def _geo_loss64(layer, chroma, target, clamp, kind):
    W = _bary_weights64(target.reshape(3, -1), chroma, clamp).reshape(layer.shape)
    d = layer - W
    return (d * d if kind == "mse" else d.abs()).mean() + 0.5 * torch.relu(-layer).mean()


def _l1_loss64(layer, palette, target):
    return (torch.einsum("kc,khw->chw", palette, layer) - target).abs().mean()


def _l1_ssim_loss64(layer, palette, target):
    x = torch.einsum("kc,khw->chw", palette, layer)[:, None]
    y = target[:, None]
    g = torch.exp(-(torch.arange(11, dtype=torch.float64, device="cuda") - 5) ** 2 / 4.5)
    g = g / g.sum()
    blur = lambda t: torch.nn.functional.conv2d(torch.nn.functional.conv2d(  # noqa: E731
        t, g.reshape(1, 1, 1, 11), padding=(0, 5)), g.reshape(1, 1, 11, 1), padding=(5, 0))
    mx, my = blur(x), blur(y)
    sxx, syy, sxy = blur(x * x) - mx * mx, blur(y * y) - my * my, blur(x * y) - mx * my
    ssim = ((2 * mx * my + 1e-4) * (2 * sxy + 9e-4)) / \
        ((mx * mx + my * my + 1e-4) * (sxx + syy + 9e-4))
    return 0.8 * (x - y).abs().mean() + 0.2 * (1 - ssim.mean()) + 0.5 * torch.relu(-layer).mean()


def _double(t):
    return t.detach().double().requires_grad_(t.requires_grad)


def exact(case, seed):
    st = prepare(case, seed)
    sc = st.get("scene")
    kind, K = case["kind"], case["K"]
    if kind in ("geo_loss", "ssim_loss"):
        layer = _double(st["layer"])
        if kind == "geo_loss":
            other = _double(st["chroma"])
            loss = _geo_loss64(layer, other, st["target"].double(), case["clamp"], case["loss"])
        else:
            other = _double(st["palette"])
            loss = _l1_ssim_loss64(layer, other, st["target"].double())
        return dict(loss=loss.detach(), grads=_grads(loss, [layer, other]))
    if kind == "serve":
        out = []
        for r in st["requests"]:
            cam = look_at((0, -8, 0), width=r.width, height=r.height, device="cpu")
            cam.Rcw, cam.tcw = r.Rcw, r.tcw
            p = {k: v.double() for k, v in st["scenes"][r.scene_id].items()}
            with torch.no_grad():
                wt = _weights64(p, r.twc.double().cuda()) @ r.palette.double().cuda()
                out.append(_view64(p, cam, wt, 1.0)[0])
        return out
    p = {k: _double(v) for k, v in sc.items()}
    if kind == "sh":
        return _exact_sh(case, st, p)
    cam = st["cam"]
    twc = cam.twc.double()
    if kind == "render":
        with torch.no_grad():
            layer, tau, depth = _view64(p, cam, _weights64(p, twc), 0.0)
        return dict(layer=layer, tau=tau, depths=depth)
    if kind == "finetune":
        layer, _, depth = _view64(p, cam, _weights64(p, twc), 0.0)
        par = [p[k] for k in st["names"]]
        if K > 3:
            chroma = _double(st["chroma"])
            loss = _geo_loss64(layer, chroma, st["target"].double(), case["clamp"], case["loss"])
            par.append(chroma)
        else:
            loss = _l1_loss64(layer, p["palette"], st["target"].double())
        return dict(layer=layer.detach(), visible=None, loss=loss.detach(), grads=_grads(loss, par))
    if kind == "train":
        layer, tau, _ = _view64(p, cam, _weights64(p, twc), 0.0)
        loss = _l1_loss64(layer, p["palette"], st["target"].double()) + 0.1 * tau.mean()
        return dict(layer=layer.detach(), tau=tau.detach(), loss=loss.detach(),
                    grads=_grads(loss, [p[k] for k in st["names"]]))
    if kind == "views":
        layers = [_view64(p, c, _weights64(p, c.twc.double()), 0.0)[0] for c in st["cams"]]
        total = sum(_l1_ssim_loss64(la, p["palette"], t.double()) for la, t in
                    zip(layers, st["targets"])) / len(layers)
        return dict(layers=[la.detach() for la in layers], loss=total.detach(),
                    grads=_grads(total, [p[k] for k in st["names"]] + [p["palette"]]))
    with torch.no_grad():  # color
        u, q, depth, rect = _geometry64(p, cam)
        col = _weights64(p, twc)
        lists = _Lists(cam, depth, rect)
        a = p["alphas"].reshape(-1, 1)
        image, tau = _image64(lists, u, q, a, col, 1.0)
    du, dq, da, dcol = _image_adjoint64(lists, u, q, a, col, st["dimage"].double(),
                                        st["dtau"].double())
    return dict(image=image, contrib=None, tau=tau, du=du[:, None], dq=dq[:, None], da=da[:, None],
                dcol=dcol[:, None])


def _exact_sh(case, st, p):
    n, K = case["n"], case["K"]
    pws = p["pws"].detach().requires_grad_()
    twc = st["twc"].double()
    Y, d = _basis(pws, twc)
    shs = p["shs"].reshape(n, 16, K)
    w = torch.einsum("nl,nlk->nk", Y, shs)
    # the operator's Jacobian takes d Y_9 / d y as C (3 x^2 - 2 y^2)
    y = d[:, 1]
    quirk = (-_C3[0] * (y * y).detach() * y)[:, None] * shs[:, 9]
    wj = w + quirk - quirk.detach()
    dpws = torch.stack([torch.autograd.grad(wj[:, k].sum(), pws, retain_graph=True)[0]
                        for k in range(K)], dim=1)
    Y = Y.detach()
    C = torch.bmm(p["A"], p["B"]).reshape(n, 15, K)
    wf = Y[:, :1] * p["dc"] + torch.einsum("nl,nlk->nk", Y[:, 1:], C)
    dC = (Y[:, 1:, None] * st["dweights"].double()[:, None]).reshape(n, K, 15)
    return dict(w=w.detach(), dshs=Y[:, None], dpws=dpws, wf=wf,
                ddc=torch.full((n, K), 0.28209479177387814, dtype=torch.float64, device="cuda"),
                ylm=Y[:, 1:], dA=torch.bmm(dC, p["B"].transpose(1, 2)),
                dB=torch.bmm(p["A"].transpose(1, 2), dC))
