"""Timed cases of the per-frame denoiser: its operators, its network and its
whole frame step, through the public entry points, over the sizes this
framework is used at (256x256 clips to 2160p streams).

``listed()`` gives the named cases, ``draw(rng)`` one more case of the same
ranges, ``prepare(case, seed)`` the state a program holds before the call,
``run(state)`` one pass, ``work(case)`` the bytes and operations a pass cannot
do without and ``exact(case, seed)`` the results in 64 bits where there are
such.
"""
from __future__ import annotations

import math

import torch
import torch.nn.functional as F

import __graft_entry__ as ge

cd = ge.load_package()
from cross_denoiser_b200 import ops, step as stepmod, synth, unet as unetmod  # noqa: E402

DEVICE = "cuda:0"


def listed():
    return [
        # an online-trained clip at the small test resolution: every launch
        # of the frame (operators, network, update) counts
        dict(name="step_256_train", op="step", H=256, W=256, B=1, win=17, fwin=11, sp=4, net=True, overlap=False),
        # the production stream: the whole training step of a 1080p frame,
        # the update overlapping the next frame
        dict(name="step_1080p_train", op="step", H=1080, W=1920, B=1, win=15, fwin=11, sp=4, net=True, overlap=True),
        # the largest served stream, operators only (a fixed prediction)
        dict(name="step_2160p_ops", op="step", H=2160, W=3840, B=1, win=15, fwin=11, sp=4, net=False, overlap=False),
        # cross-regression alone: a small clip, and 1080p at the reference's default window
        dict(name="regression_256", op="regression", H=256, W=256, B=1, win=15, sp=4, rs=1),
        dict(name="regression_1080p", op="regression", H=1080, W=1920, B=1, win=17, sp=4, rs=1),
        # differentiable regression on training crops, forward and backward
        dict(name="regression_grad_512x4", op="regression_grad", H=512, W=512, B=4, win=15, sp=4, rs=1),
        # the drop-in filter with its registered gradient on a ragged window
        # of a frame (neither side a multiple of a tile)
        dict(name="filter_grad_719x1277", op="filter_grad", H=719, W=1277, B=1, fwin=11),
        # filter, loss and band gradient of the fused training step
        dict(name="filter_aggregate_1080p", op="filter_aggregate", H=1080, W=1920, B=1, fwin=11),
        # history: reprojection, and erosion + screening
        dict(name="reproject_1080p", op="reproject", H=1080, W=1920, B=1),
        dict(name="screening_1080p", op="screening", H=1080, W=1920, B=1, wc=7),
        # the kernel-predicting network: inference of a stream with frozen
        # weights, and one online update
        dict(name="unet_predict_1080p", op="unet_predict", H=1080, W=1920, B=1),
        dict(name="unet_train_1440p", op="unet_train", H=1440, W=2560, B=1),
    ]


def _size(rng, lo_px, hi_px, mult):
    """Height and width of a frame of log-uniform pixel count and aspect 1:1 to 16:9."""
    px = math.exp(rng.uniform(math.log(lo_px), math.log(hi_px)))
    aspect = rng.uniform(1.0, 16.0 / 9.0)
    h = max(48, int(math.sqrt(px / aspect)))
    w = max(64, int(px / h))
    return max(mult, h // mult * mult), max(mult, w // mult * mult)


def draw(rng):
    op = rng.choice(["step", "regression", "regression_grad", "filter_grad", "filter_aggregate", "reproject",
                     "screening", "unet_predict", "unet_train"])
    small, p1080, p1440, p2160 = 64 * 96, 1080 * 1920, 1440 * 2560, 2160 * 3840
    B = 1
    if op == "step":
        H, W = _size(rng, 192 * 256, p1440, 4)
        return dict(op=op, H=H, W=W, B=1, win=rng.choice([11, 15, 17, 19]), fwin=rng.choice([7, 11]), sp=4,
                    net=rng.random() < 0.5, overlap=rng.random() < 0.5)
    if op == "regression":
        sp = rng.choice([2, 4, 4, 4])
        H, W = _size(rng, small, p2160 if sp == 4 else 720 * 1280, sp)
        return dict(op=op, H=H, W=W, B=1, win=rng.choice([11, 15, 17, 19]), sp=sp, rs=rng.choice([1, 1, 1, 2]))
    if op == "regression_grad":
        H, W = _size(rng, small, 512 * 512, 4)
        return dict(op=op, H=H, W=W, B=rng.choice([1, 2, 4]), win=rng.choice([9, 15]), sp=4, rs=1)
    if op in ("filter_grad", "filter_aggregate"):
        B = rng.choice([1, 1, 2])
        H, W = _size(rng, small, p1440 / B, 1)
        return dict(op=op, H=H, W=W, B=B, fwin=rng.choice([7, 11, 11, 13]))
    if op in ("reproject", "screening"):
        H, W = _size(rng, small, p2160, 1 if rng.random() < 0.5 else 4)
        c = dict(op=op, H=H, W=W, B=1)
        if op == "screening":
            c["wc"] = rng.choice([3, 5, 7, 7])
        return c
    H, W = _size(rng, small, p2160 if op == "unet_predict" else p1440, 4)
    return dict(op=op, H=H, W=W, B=1)


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _frames(case, seed, n):
    """n consecutive frames of a synthetic sequence (a batch: B sequences)."""
    per = []
    for b in range(case["B"]):
        seq = synth.make_sequence(case["H"], case["W"], seed=int(seed) * 16 + b, object_motion=4.0, device=DEVICE,
                                  max_frames=8)
        per.append([seq.frame(t + 1) for t in range(n)])
    return [{k: torch.cat([p[t][k] for p in per]) for k in synth.FRAME_INPUTS} for t in range(n)]


def _prediction(case, seed):
    g = torch.Generator(device=DEVICE).manual_seed(int(seed) + 77)
    shape = (case["B"], case["H"], case["W"])
    band = synth.random_band(shape, g, device=DEVICE)
    return band, torch.sigmoid(torch.randn((*shape, 1), generator=g, device=DEVICE))


def _normal(case, seed, *channels):
    g = torch.Generator(device=DEVICE).manual_seed(int(seed) + 191)
    return [torch.randn((case["B"], case["H"], case["W"], c), generator=g, device=DEVICE) for c in channels]


def _smooth(y):
    """What the regression hands on: the noisy image averaged over a small window."""
    x = F.avg_pool2d(y.permute(0, 3, 1, 2), 5, 1, 2, count_include_pad=False)
    return x.permute(0, 2, 3, 1).contiguous()


def _logs(f):
    return torch.log1p(f["color"]), torch.log1p(f["color2"])


def prepare(case, seed):
    op = case["op"]
    s = {"op": op, "case": case}
    if op == "step":
        fr = _frames(case, seed, 3)
        cfg = stepmod.StepConfig(regression_width=case["win"], filter_width=case["fwin"], sparsity=case["sp"],
                                 fused=True, overlap_training=case["overlap"])
        if case["net"]:
            s["net"] = unetmod.UNet(DEVICE, seed=int(seed) % 1000)
            s["step"] = stepmod.FrameStep(cfg, predictor=s["net"], on_gradients=s["net"].on_gradients)
        else:
            s["step"] = stepmod.FrameStep(cfg)
            s["step"].set_fixed_prediction(*_prediction(case, seed))
        # a stream in flight: the frame before has been denoised
        o1, o2 = (_smooth(y) for y in _logs(fr[0]))
        s["step"].history = stepmod.History(0.5 * (o1 + o2), o1, o2, fr[0]["linearZ"], fr[0]["normal"])
        s["frames"], s["t"] = fr[1:], 0
        return s
    if op == "reproject":
        f0, f1 = _frames(case, seed, 2)
        o1, o2 = (_smooth(y) for y in _logs(f0))
        one = torch.ones((case["B"], case["H"], case["W"], 1), device=DEVICE)
        s["args"] = (f1["mvec"], [0.5 * (o1 + o2), o1, o2], f1["linearZ"], f0["linearZ"], f1["normal"], f0["normal"],
                     f1["pnFwidth"], one, one)
        return s
    if op == "unet_predict" or op == "unet_train":
        f0, f1 = _frames(case, seed, 2)
        o1, o2 = (_smooth(y) for y in _logs(f1))
        p1, p2 = (_smooth(y) for y in _logs(f0))
        s["net"] = unetmod.UNet(DEVICE, seed=int(seed) % 1000)
        s["ins"] = (o1, o2, 0.5 * (p1 + p2), f1["albedo"], f1["normal"])
        if op == "unet_train":
            n = case["B"] * case["H"] * case["W"]
            s["grads"] = [g / n for g in _normal(case, seed, 5, 1)]
        return s
    f0, f1 = _frames(case, seed, 2)
    y1, y2 = _logs(f1)
    if op in ("regression", "regression_grad"):
        s["imgs"] = [y1, y2, f1["albedo"], f1["normal"]]
        if op == "regression_grad":
            s["up"] = _normal(case, seed, 3, 3)
            s["imgs"] = [t.requires_grad_(True) for t in s["imgs"]]
        return s
    o1, o2 = _smooth(y1), _smooth(y2)
    band, alpha = _prediction(case, seed)
    if op == "filter_grad":
        s["imgs"] = (o1, o2, f1["albedo"], f1["normal"])
        s["band"] = band.requires_grad_(True)
        s["up"] = _normal(case, seed, 3, 3, 1, 1)
        return s
    p1, p2 = (_smooth(y) for y in _logs(f0))
    prev = 0.5 * (p1 + p2)
    g = torch.Generator(device=DEVICE).manual_seed(int(seed) + 5)
    mask = torch.rand((case["B"], case["H"], case["W"], 1), generator=g, device=DEVICE) > 0.05
    if op == "screening":
        s["args"] = (o1, o2, prev, p1, p2, mask)
        return s
    keep = torch.rand((case["B"], case["H"], case["W"], 1), generator=g, device=DEVICE) > 0.2
    s["args"] = (o1, o2, f1["albedo"], f1["normal"], band, alpha, mask.float(), keep.float(), prev, f1["opacity"], p1,
                 p2)
    return s


def run(s):
    op, c = s["op"], s["case"]
    if op == "step":
        f = s["frames"][s["t"] % len(s["frames"])]
        s["t"] += 1
        r = s["step"](f)
        out = {k: r[k] for k in ("out", "out_log", "avg_loss", "ols1", "ols2", "g_band", "g_alpha", "success")}
        if "net" in s:
            out["band"], out["alpha"], out["params"] = r["band"], r["alpha"], s["net"].params
        return out
    if op == "regression":
        return ops.cross_regression(*s["imgs"], win_size=c["win"], sparsity=c["sp"], recon_scale=c["rs"])
    if op == "regression_grad":
        o = ops.cross_regression(*s["imgs"], win_size=c["win"], sparsity=c["sp"], recon_scale=c["rs"])
        return [t.detach() for t in o[:2]], torch.autograd.grad(o[:2], s["imgs"], s["up"])
    if op == "filter_grad":
        o = ops.spatial_filter(*s["imgs"], s["band"], win_size=c["fwin"])
        return [t.detach() for t in o], torch.autograd.grad(o, s["band"], s["up"])
    if op == "filter_aggregate":
        return ops.filter_aggregate(*s["args"], win_size=c["fwin"])
    if op == "reproject":
        return ops.Reproject(*s["args"])
    if op == "screening":
        return ops.erode_temporal_screening(*s["args"], c["wc"], 1)
    band, alpha = s["net"](*s["ins"])
    if op == "unet_predict":
        return band, alpha
    s["net"].on_gradients(*s["grads"])
    return band, alpha, s["net"].grads, s["net"].params


# ---------------------------------------------------------------------------
# work
# ---------------------------------------------------------------------------
def _unet_flops(px):
    """Multiply-adds of the network's convolutions per full-resolution pixel, times two."""
    full = 9 * (15 * 8 + 8 * 8 + 24 * 8) + 8 * 6
    half = 9 * (8 * 16 + 16 * 16 + 48 * 16 + 16 * 16) + 16 * 16
    quarter = 9 * (16 * 32 + 32 * 32) + 32 * 32
    return 2.0 * px * (full + half / 4 + quarter / 16)


def _regression_flops(c, px):
    taps = px / c["sp"] ** 2 * c["win"] ** 2
    pairs = px / c.get("rs", 1) ** 2 * (c["win"] / c["sp"]) ** 2
    return 2.0 * (150 * taps + 55 * pairs + 20 * px)


def work(case):
    c, op = case, case["op"]
    px = c["B"] * c["H"] * c["W"]
    if op == "regression":
        out = 24 / c["rs"] ** 2 + 8
        return {"bytes": px * (48 + out), "flops": _regression_flops(c, px)}
    if op == "regression_grad":   # the backward evaluates each pair from both of its sides
        return {"bytes": px * (48 + 24 + 24 + 48), "flops": 4.0 * _regression_flops(c, px)}
    if op == "filter_grad":
        return {"bytes": px * (48 + 20 + 32 + 32 + 20), "flops": px * c["fwin"] ** 2 * 170.0}
    if op == "filter_aggregate":
        return {"bytes": px * (48 + 20 + 4 + 8 + 12 + 4 + 24 + 24 + 20 + 4), "flops": px * c["fwin"] ** 2 * 110.0}
    if op == "reproject":
        return {"bytes": px * (12 + 36 + 24 + 24 + 12 + 8 + 36 + 1.0), "flops": px * 100.0}
    if op == "screening":
        return {"bytes": px * (60 + 1 + 36 + 8.0), "flops": px * 300.0}
    if op == "unet_predict":
        return {"bytes": px * 84.0, "flops": _unet_flops(px)}
    if op == "unet_train":
        return {"bytes": px * (84 + 24.0), "flops": 3.0 * _unet_flops(px)}
    flops = _regression_flops(c, px) + px * (c["fwin"] ** 2 * 110.0 + 400.0)
    n = px * (88 + 60 + 24 + 24 + 48 + 24.0)   # frame, history read and written, prediction
    if c["net"]:
        flops += 3.0 * _unet_flops(px)
    return {"bytes": n, "flops": flops}


# ---------------------------------------------------------------------------
# results in 64 bits
# ---------------------------------------------------------------------------
def _mirror(i, n):
    return torch.where(i >= n, 2 * n - 2 - i, i.abs())


def _ceil_div(a, b):
    """Ceiling division as the operator defines it: C's truncating quotient, plus one on any remainder."""
    q = int(a / b)
    return q + 1 if a - q * b else q


def _variance64(x):
    n = x.permute(0, 3, 1, 2)
    k = torch.ones((1, 1, 3, 3), dtype=x.dtype, device=x.device)
    count = F.conv2d(torch.ones_like(n[:, :1]), k, padding=1) - 1
    mean = (F.conv2d(n, k.expand(3, 1, 3, 3), padding=1, groups=3) - n) / count
    return ((mean - n) ** 2).sum(1, keepdim=True).permute(0, 2, 3, 1)


def _features(f, a, n, sd, fc, ac, nc, sdc):
    """[..., 3 channels, 6 regressors] of a pixel seen from a centre."""
    d1 = (f - fc) / (sd + sdc + 1e-2)
    dn = (n - nc).unsqueeze(-2).expand(*d1.shape, 3)
    return torch.cat([torch.ones_like(d1).unsqueeze(-1), d1.unsqueeze(-1), (a - ac).unsqueeze(-1), dn], -1)


def _weight(f, v, fc, vc):
    return torch.exp(-((f - fc) ** 2).sum(-1, keepdim=True) / (v + vc + 1e-4)) + 1e-7


def _regress64(y, f, v, alb, nrm, c):
    """One image [H,W,.]: the target y predicted from f's features; rows in blocks."""
    H, W, _ = f.shape
    sp, rs, hw = c["sp"], c["rs"], c["win"] // 2
    dev = f.device
    sd = torch.sqrt(v)
    off = torch.arange(-hw, hw + 1, device=dev)
    cy, cx = torch.arange(H // sp, device=dev) * sp, torch.arange(W // sp, device=dev) * sp
    tx = _mirror(cx[:, None] + off, W)
    beta = []
    for rows in torch.split(cy, max(1, 8_000_000 // (tx.numel() * c["win"]))):
        ty = _mirror(rows[:, None] + off, H)
        tap = lambda t: t[ty][:, :, tx].transpose(1, 2).flatten(2, 3)   # [rows, cols, taps, .]
        cen = lambda t: t[rows][:, cx][:, :, None]
        X = _features(tap(f), tap(alb), tap(nrm), tap(sd), cen(f), cen(alb), cen(nrm), cen(sd))
        w = _weight(tap(f), tap(v), cen(f), cen(v))
        wX = X * w.unsqueeze(-1)
        A = torch.einsum("rctki,rctkj->rckij", wX, X) + 1e-3 * torch.eye(6, dtype=f.dtype, device=dev)
        b = torch.einsum("rctki,rctk->rcki", wX, tap(y))
        beta.append(torch.linalg.solve(A, b.unsqueeze(-1)).squeeze(-1))
        del X, wX, w
    beta = torch.cat(beta)                                               # [Hs, Ws, 3, 6]

    def ranges(n, ncen):
        lo = [max(0, _ceil_div(p - hw, sp)) for p in range(0, n, rs)]
        hi = [min((n - 1) // sp, (p + hw) // sp) for p in range(0, n, rs)]
        K = max(h - l + 1 for l, h in zip(lo, hi))
        k = torch.arange(K, device=dev)
        lo, hi = torch.tensor(lo, device=dev)[:, None], torch.tensor(hi, device=dev)[:, None]
        return (lo + k).clamp(max=ncen - 1), lo + k <= hi

    jy, oky = ranges(H, H // sp)
    ix, okx = ranges(W, W // sp)
    fc, ac, nc, vc, sc = (t[cy][:, cx] for t in (f, alb, nrm, v, sd))
    px = torch.arange(0, W, rs, device=dev)
    out = []
    for rows in torch.split(torch.arange(len(jy), device=dev), max(1, 4_000_000 // len(ix))):
        num, den = 0.0, 0.0
        at = lambda t: t[rows * rs][:, px]
        for a in range(jy.shape[1]):
            for b in range(ix.shape[1]):
                cen = lambda t: t[jy[rows, a]][:, ix[:, b]]
                X = _features(at(f), at(alb), at(nrm), at(sd), cen(fc), cen(ac), cen(nc), cen(sc))
                ok = (oky[rows, a][:, None] & okx[:, b][None])[..., None]
                w = _weight(at(f), at(v), cen(fc), cen(vc)) * ok
                num = num + w * (X * cen(beta)).sum(-1)
                den = den + w
        out.append(torch.relu(num / den.clamp(min=1e-7)))
    return torch.cat(out)


def _regression64(imgs, c):
    a, b, alb, nrm = imgs
    va, vb = _variance64(a), _variance64(b)
    oa = torch.stack([_regress64(b[i], a[i], va[i], alb[i], nrm[i], c) for i in range(len(a))])
    ob = torch.stack([_regress64(a[i], b[i], vb[i], alb[i], nrm[i], c) for i in range(len(a))])
    return oa, ob, va, vb


def _filter64(imgs, band, win, partials):
    """Filter sums, and the sums weighted by each of the four distances, of both images."""
    a, b, alb, nrm = imgs
    B, H, W, _ = a.shape
    r = win // 2
    one = torch.ones_like(a[..., :1])
    iy, ix = torch.arange(H, device=a.device), torch.arange(W, device=a.device)
    S = [0.0, 0.0]
    P = [[0.0] * 4 for _ in range(2)]
    for dy in range(-r, r + 1):
        jy = _mirror(iy + dy, H)
        for dx in range(-r, r + 1):
            jx = _mirror(ix + dx, W)
            at = lambda t: t[:, jy][:, :, jx]
            dist = lambda t: ((t - at(t)) ** 2).sum(-1, keepdim=True)
            shared = [dist(alb), dist(nrm), torch.full_like(one, (dy * dy + dx * dx) / (r * r))]
            rest = sum(band[..., 2 + k:3 + k] * d for k, d in enumerate(shared))
            for i, t in enumerate((a, b)):
                d0 = dist(t)
                wc = torch.exp(-(band[..., i:i + 1] * d0 + rest)) * torch.cat([at(t), one], -1)
                S[i] = S[i] + wc
                if partials:
                    for k, d in enumerate([d0] + shared):
                        P[i][k] = P[i][k] + wc * d
    return S, P


def _band_grad64(P, up):
    g = [[-(p * u).sum(-1, keepdim=True) for p in Pi] for Pi, u in zip(P, up)]
    return torch.cat([g[0][0], g[1][0]] + [g[0][k] + g[1][k] for k in (1, 2, 3)], -1)


def _loss64(S, alpha, succ, keep, prev, opacity, labels, prev_labels):
    op = (opacity > 0).to(alpha.dtype)
    sv = succ * keep
    a = sv * alpha + (1 - sv)
    s = S[0] + S[1]
    out = (a * (s[..., :3] / (s[..., 3:] + 1e-4)) + (1 - a) * prev) * op
    loss = 0.0
    for Si, lab, plab in zip(S, labels, prev_labels):
        o = a * (Si[..., :3] / (Si[..., 3:] + 1e-4)) + (1 - a) * prev
        loss = loss + 0.25 * ((o - lab) ** 2 / (lab ** 2 + 1e-2) + (o - plab) ** 2 / (plab ** 2 + 1e-2)) * op
    return out, torch.expm1(out).clamp(min=0.0), loss.mean()


def _unet64(params, ins):
    """band, alpha of the network in float64 (convolutions as Keras defines them)."""
    layers, o = [], 0
    for kind, cin, cout in unetmod.LAYERS:
        shape = unetmod.kernel_shape(kind, cin, cout)
        n = math.prod(shape)
        layers.append((params[o:o + n].reshape(shape), params[o + n:o + n + cout]))
        o += n + cout
    conv = lambda i, x: F.relu(F.conv2d(x, layers[i][0].permute(3, 2, 0, 1), layers[i][1], padding=1))
    pool = lambda x: F.max_pool2d(x, 2)

    def up(i, x):
        K, b = layers[i]
        y = F.conv_transpose2d(x, K[0, 0].t()[:, :, None, None], stride=2, output_padding=1)
        return y + b.view(1, -1, 1, 1)

    x = torch.cat(ins, -1).permute(0, 3, 1, 2)
    c1 = conv(1, conv(0, x))
    c2 = conv(3, conv(2, pool(c1)))
    c3 = conv(5, conv(4, pool(c2)))
    c4 = conv(8, conv(7, torch.cat([up(6, c3), c2], 1)))
    c5 = conv(10, torch.cat([up(9, c4), c1], 1))
    K, b = layers[11]
    p = c5.permute(0, 2, 3, 1) @ K[0, 0] + b
    return 1 / (p[..., :5] ** 2 + 1e-4), torch.sigmoid(p[..., 5:])


def exact(case, seed):
    op = case["op"]
    if op in ("step", "reproject", "screening"):
        return None   # chains of decisions, and moves of data
    s = prepare(case, seed)
    d = lambda t: t.detach().double()
    if op == "regression":
        with torch.no_grad():
            return _regression64([d(t) for t in s["imgs"]], case)
    if op == "regression_grad":
        outs, grads = [], []
        for i in range(case["B"]):   # an image at a time: the batch is independent
            x = [d(t)[i:i + 1].requires_grad_(True) for t in s["imgs"]]
            o = _regression64(x, case)[:2]
            grads.append(torch.autograd.grad(o, x, [d(u)[i:i + 1] for u in s["up"]]))
            outs.append([t.detach() for t in o])
        return [torch.cat(t) for t in zip(*outs)], tuple(torch.cat(t) for t in zip(*grads))
    if op == "filter_grad":
        with torch.no_grad():
            S, P = _filter64([d(t) for t in s["imgs"]], d(s["band"]), case["fwin"], True)
            ga, gb, gwa, gwb = (d(u) for u in s["up"])
            g = _band_grad64(P, [torch.cat([ga, gwa], -1), torch.cat([gb, gwb], -1)])
            return [S[0][..., :3], S[1][..., :3], S[0][..., 3:], S[1][..., 3:]], (g,)
    if op == "filter_aggregate":
        o1, o2, alb, nrm, band, alpha, succ, keep, prev, opacity, p1, p2 = (d(t) for t in s["args"])
        with torch.no_grad():
            S, P = _filter64([o1, o2, alb, nrm], band, case["fwin"], True)
        S = [t.requires_grad_(True) for t in S]
        alpha.requires_grad_(True)
        # labels crossed, as the training step sets them
        out_log, out, avg = _loss64(S, alpha, succ, keep, prev, opacity, (o2, o1), (p2, p1))
        up = torch.autograd.grad(avg, [*S, alpha])
        return out_log.detach(), out.detach(), avg.detach(), _band_grad64(P, up[:2]), up[2]
    params, ins = d(s["net"].params), [d(t) for t in s["ins"]]
    if op == "unet_predict":
        with torch.no_grad():
            return _unet64(params, ins)
    # the parameter gradients sum over bf16 activations, as the network stores
    # them: their distance to 64 bits is that storage's, so they have no value here
    with torch.no_grad():
        return (*_unet64(params, ins), None, None)
