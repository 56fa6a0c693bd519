"""The work that users of this framework have it do, as measurable cases.

A case is a dict of plain values with a "kind":

  plain    one frame pair in host memory through the default (plain, FP64)
           pipeline: a survey script that subtracts one image from another
  plain_dev  the same from device memory to device memory
  mixed    one frame pair in device memory through the mixed pipeline as a
           frame graph, the lowest latency from a new exposure to its
           difference image; "rank" turns the learned substamp order on
  batch    many pairs of a night at once over the workers of a batch,
           device-resident ("host" false) or from and to pinned host memory
  apply    the convolution and subtraction stages of a fitted context, with
           the kernel evaluated per block or ("per_pixel") at every pixel
  stats    the sky level and robust sigma of every stamp of a grid, from the
           entry point that allocates nothing
  score    the ranker's logits of a list of candidate substamps
  train    one training step of the ranker: gradients and an Adam update

Frames are seeded synthetic star fields: pixel-integrated Gaussian stars with
log-uniform fluxes on a Poisson sky with Gaussian read noise; the science
frame has a broader PSF, 1.1 times the flux, a sloped background and a few
variables.  "survey" fields add a PSF that widens across the frame, cosmic
rays on 1 % of the pixels, saturated stars and a detector clip at 6e4 ADU.
"""
import ctypes
import math
import os
import pathlib
import sys

# more hardware queues than CUDA's default of 8, so that the streams of a
# batch's workers do not share them (an application sets it at its start)
os.environ.setdefault("CUDA_DEVICE_MAX_CONNECTIONS", "32")

import numpy as np
import torch

sys.path.insert(0, str(pathlib.Path(__file__).resolve().parent.parent / "thesis-emx-bach_gb300"))

import xbach
from xbach import ranker

# basis of three Gaussians (49 functions, the default) and of four (59)
BASES = {
    49: {},
    59: dict(nGauss=4, dg=[6, 4, 3, 2],
             bg=[1 / (2 * s * s) for s in (0.6, 1.2, 2.4, 4.8)],
             kernelOrder=3, backgroundOrder=2),
}
FLUX_SCALE, SKY, READ_NOISE, CLIP = 1.1, 1000.0, 5.0, 6e4


def listed():
    return [
        # a small cutout pair by the defaults, host arrays in and out
        dict(name="plain_437x611", kind="plain", w=437, h=611, stamps=10, density=0.0057,
             survey=False),
        # one survey frame through the FP64 pipeline
        dict(name="plain_2048", kind="plain_dev", w=2048, h=2048, stamps=16, density=0.0048,
             survey=True),
        # a small cutout as a frame graph: launch latencies and serial chains
        dict(name="mixed_509x541", kind="mixed", w=509, h=541, stamps=8, density=0.0057,
             survey=False, basis=49, rank=False),
        # one survey frame with the learned order, the ordinary alert latency
        dict(name="mixed_2048_rank", kind="mixed", w=2048, h=2048, stamps=16, density=0.0048,
             survey=True, basis=49, rank=True),
        # a crowded field with the wide basis, cubic kernel variation
        dict(name="mixed_3072_wide", kind="mixed", w=3072, h=3072, stamps=20, density=0.0085,
             survey=False, basis=59, rank=False),
        # the largest single frame
        dict(name="mixed_4096_rank", kind="mixed", w=4096, h=4096, stamps=20, density=0.0072,
             survey=True, basis=49, rank=True),
        # a night's throughput: 24 survey pairs in flight on 24 workers
        dict(name="batch_24x2048", kind="batch", frames=24, workers=24, w=2048, h=2048,
             uneven=False, stamps=16, density=0.0048, rank=True, host=False),
        # cutouts of uneven size from and to pinned host memory
        dict(name="batch_16_uneven_host", kind="batch", frames=16, workers=16, w=1900, h=1700,
             uneven=True, stamps=14, density=0.006, rank=False, host=True),
        # the kernel evaluated at every pixel of a fitted frame
        dict(name="apply_per_pixel_2048", kind="apply", w=2048, h=2048, stamps=16, density=0.0048,
             mode="mixed", per_pixel=True),
        # stamp statistics of one frame
        dict(name="stats_16x16", kind="stats", w=2048, h=2048, nx=16, ny=16, width=107),
        # the candidates of a large frame: 400 stamps, 5 candidates each
        dict(name="score_2000", kind="score", n=2000),
        # a step of the ranker's training at its usual batch
        dict(name="train_512", kind="train", n=512),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _frame(rng, lo, hi):
    """Width, height (within a factor of 1.5) and stamp grid of a frame."""
    w = int(_log(rng, lo, hi))
    h = min(hi, max(lo, int(w * _log(rng, 1 / 1.5, 1.5))))
    side = _log(rng, 54, 160)
    return w, h, max(6, min(20, int(min(w, h) / side)))


def draw(rng):
    kind = rng.choice(["plain", "plain_dev", "mixed", "mixed", "mixed", "batch", "batch", "apply",
                       "stats", "score", "train"])
    density = round(_log(rng, 0.004, 0.009), 5)
    if kind in ("plain", "plain_dev"):
        w, h, g = _frame(rng, 340, 2048)
        return dict(kind=kind, w=w, h=h, stamps=min(g, 16), density=density,
                    survey=rng.random() < 0.5)
    if kind == "mixed":
        basis = rng.choice([49, 49, 59])
        w, h, g = _frame(rng, 420 if basis == 49 else 1200, 4096 if basis == 49 else 3072)
        return dict(kind=kind, w=w, h=h, stamps=g if basis == 49 else max(g, 10), density=density,
                    survey=basis == 49 and rng.random() < 0.5, basis=basis,
                    rank=basis == 49 and rng.random() < 0.5)
    if kind == "batch":
        w, h, g = _frame(rng, 500, 2048)
        n = rng.randint(4, 24)
        return dict(kind=kind, frames=n, workers=rng.randint(4, n), w=w, h=h,
                    uneven=rng.random() < 0.5, stamps=min(g, 16), density=density,
                    rank=rng.random() < 0.5, host=rng.random() < 0.5)
    if kind == "apply":
        w, h, g = _frame(rng, 420, 2048)
        return dict(kind=kind, w=w, h=h, stamps=min(g, 16), density=density,
                    mode=rng.choice(["mixed", "mixed", "plain"]), per_pixel=rng.random() < 0.5)
    if kind == "stats":
        width = int(_log(rng, 31, 161)) | 1
        room = (32 << 20) // (9 * (width * width + 1023) + 16 * (width * width // 32 + 1))
        nx = rng.randint(1, max(1, min(20, math.isqrt(room))))
        ny = rng.randint(1, max(1, min(20, room // nx)))
        return dict(kind=kind, w=nx * (width + rng.randint(0, 22)), h=ny * (width + rng.randint(0, 22)),
                    nx=nx, ny=ny, width=width)
    return dict(kind=kind, n=int(_log(rng, 1, 20000) if kind == "score" else _log(rng, 16, 2048)))


# ---- inputs ---------------------------------------------------------------

def _generator(seed, part=0):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed * 1000003 + part)
    return g


def _stars(w, h, xs, ys, flux, sigma):
    """Pixel-integrated Gaussians on an (h, w) frame, summed in fixed point so
    that the frame does not depend on the order of the additions."""
    out = torch.zeros(h * w, dtype=torch.int64, device="cuda")
    r = int(math.ceil(4.0 * float(sigma.max()))) + 1
    off = torch.arange(-r, r + 1, device="cuda")
    for i in range(0, len(xs), 16384):
        x, y, f, s = (v[i:i + 16384, None] for v in (xs, ys, flux, sigma))
        px, py = torch.floor(x).long() + off, torch.floor(y).long() + off
        q = s * math.sqrt(2.0)
        gx = 0.5 * (torch.erf((px + 0.5 - x) / q) - torch.erf((px - 0.5 - x) / q))
        gy = 0.5 * (torch.erf((py + 0.5 - y) / q) - torch.erf((py - 0.5 - y) / q))
        v = ((f * gy)[:, :, None] * gx[:, None, :] * 65536.0).round().long()
        ok = ((py >= 0) & (py < h))[:, :, None] & ((px >= 0) & (px < w))[:, None, :]
        at = py.clamp(0, h - 1)[:, :, None] * w + px.clamp(0, w - 1)[:, None, :]
        out.index_add_(0, at.reshape(-1), (v * ok).reshape(-1))
    return (out.double() / 65536.0).reshape(h, w)


def _pair(w, h, density, survey, gen):
    """A template and a science frame, FP32 on the GPU."""
    n = max(200, int(density * w * h))

    def uniform(lo, hi, k=n):
        return lo + (hi - lo) * torch.rand(k, generator=gen, device="cuda", dtype=torch.float64)

    xs, ys = uniform(0, w - 1), uniform(0, h - 1)
    flux = 10.0 ** uniform(3.0, 6.0)
    if survey:
        k = max(4, n // 500)
        flux[:k] = 10.0 ** uniform(6.5, 7.5, k)
    flux_s = flux * FLUX_SCALE
    flux_s[-15:] *= uniform(0.8, 1.2, 15)
    to_sigma = 1.0 / (2.0 * math.sqrt(2.0 * math.log(2.0)))
    across = xs / max(w - 1, 1) if survey else torch.full_like(xs, 0.3)
    T = _stars(w, h, xs, ys, flux, (2.2 + across) * to_sigma)
    S = _stars(w, h, xs, ys, flux_s, (3.0 + (1.2 if survey else 1.6) * across) * to_sigma)
    S += 50.0 + 0.01 * torch.arange(w, device="cuda", dtype=torch.float64)
    frames = []
    for img in (T, S):
        img = torch.poisson((img + SKY).float(), generator=gen)
        img += READ_NOISE * torch.randn(img.shape, generator=gen, device="cuda")
        if survey:
            hit = torch.rand(img.shape, generator=gen, device="cuda") < 0.01
            img += hit * (5e3 + 4.5e4 * torch.rand(img.shape, generator=gen, device="cuda"))
            img.clamp_(max=CLIP)
        frames.append(img.contiguous())
    return frames


def _params(case, mode, survey):
    p = dict(BASES[case.get("basis", 49)], stampsx=case["stamps"], stampsy=case["stamps"],
             mode=mode)
    # clean fields hold stars above the default threshHigh; both kinds use the
    # level at which their detector clips
    p["threshHigh"] = CLIP if survey else 25000.0
    if case.get("per_pixel"):
        p["convPerPixel"] = 1
    return xbach.default_params(**p)


_kept = {}


def _keep(case, make):
    """The handle that a program keeps from frame to frame: one per workload,
    the last workload's only."""
    key = repr(sorted((k, v) for k, v in case.items() if k != "name"))
    if key not in _kept:
        _kept.clear()
        _kept[key] = make()
    return _kept[key]


def _sizes(case):
    """Frame sizes and stamp grids of a batch: down to a quarter of the
    largest side, odd ones among them, where they are uneven."""
    out = []
    for i in range(case["frames"]):
        f = 1.0 - 0.75 * ((i * 7) % case["frames"]) / case["frames"] if case["uneven"] else 1.0
        w, h = max(340, int(case["w"] * f)), max(340, int(case["h"] * f))
        out.append((w, h, max(6, int(case["stamps"] * max(f, 340 / min(case["w"], case["h"]))))))
    return out


def _candidates(n, gen):
    """Statistics and normalised 2x31x31 windows like those of star
    candidates, accept labels and class weights."""
    ax = torch.arange(31, device="cuda") - 15.0
    c = torch.randn(n, 2, 1, 1, generator=gen, device="cuda")
    s = 1.0 + 0.7 * torch.rand(n, 1, 1, 1, generator=gen, device="cuda")
    r2 = (ax[None, None, :, None] - c[:, :1]) ** 2 + (ax[None, None, None, :] - c[:, 1:]) ** 2
    s = torch.cat([s, 1.35 * s], dim=1)
    pix = torch.exp(-r2 / (2 * s * s)) + 0.03 * torch.randn(n, 2, 31, 31, generator=gen,
                                                           device="cuda")
    stats = torch.randn(n, 16, generator=gen, device="cuda")
    label = (torch.rand(n, generator=gen, device="cuda") > 0.08).float()
    weight = torch.where(label > 0.5, 0.5 / 0.92, 0.5 / 0.08)
    return stats, pix.reshape(n, -1).contiguous(), label, weight


def _weights(seed):
    return ranker.init_weights(seed)


def prepare(case, seed):
    kind = case["kind"]
    gen = _generator(seed)
    if kind in ("plain", "plain_dev", "mixed"):
        mode = xbach.XB_MODE_MIXED if kind == "mixed" else xbach.XB_MODE_PLAIN

        def make():
            ctx = xbach.Context(_params(case, mode, case["survey"]))
            if kind == "mixed":
                if case["rank"]:
                    ranker.enable(ctx, ranker.preset5_weights(), policy=1, tau=0.3)
                ctx.set_option("graph", 1)
            return ctx

        T, S = _pair(case["w"], case["h"], case["density"], case["survey"], gen)
        ctx = _keep(case, make)
        if kind == "plain":
            return dict(kind=kind, ctx=ctx, T=T.cpu().numpy(), S=S.cpu().numpy())
        return dict(kind=kind, ctx=ctx, T=T, S=S, conv=torch.empty_like(T),
                    diff=torch.empty_like(T))
    if kind == "batch":
        sizes = _sizes(case)

        def make():
            b = xbach.Batch(_params(case, xbach.XB_MODE_MIXED, True), workers=case["workers"])
            if case["rank"]:
                for i in range(b.n_workers):
                    ranker.enable(b.worker(i), ranker.preset5_weights(), policy=1, tau=0.3)
            b.set_option("graph", 1)
            b.set_params([_params(dict(case, stamps=g), xbach.XB_MODE_MIXED, True)
                          for _, _, g in sizes])
            return b

        T, S = [], []
        for i, (w, h, _) in enumerate(sizes):
            t, s = _pair(w, h, case["density"], True, _generator(seed, i + 1))
            T.append(t.cpu().pin_memory() if case["host"] else t)
            S.append(s.cpu().pin_memory() if case["host"] else s)
        conv = [torch.empty_like(t, pin_memory=case["host"]) for t in T]
        diff = [torch.empty_like(t, pin_memory=case["host"]) for t in T]
        return dict(kind=kind, batch=_keep(case, make), T=T, S=S, conv=conv, diff=diff,
                    host=case["host"], w=[s[0] for s in sizes], h=[s[1] for s in sizes])
    if kind == "apply":
        mode = xbach.XB_MODE_MIXED if case["mode"] == "mixed" else xbach.XB_MODE_PLAIN
        T, S = _pair(case["w"], case["h"], case["density"], True, gen)
        torch.cuda.synchronize()
        ctx = xbach.Context(_params(case, mode, True))
        ctx.init_device(T.data_ptr(), S.data_ptr(), case["w"], case["h"])
        ctx.sss()
        ctx.cmv()
        ctx.cd()
        ctx.ksc()
        return dict(kind=kind, ctx=ctx, T=T, S=S, shape=(case["h"], case["w"]))
    if kind == "stats":
        w, h, nx, ny, width = (case[k] for k in ("w", "h", "nx", "ny", "width"))
        img = _pair(w, h, 0.0048, True, gen)[0]
        mask = ((img >= CLIP) * 0x82).to(torch.int16)   # saturated and bad input
        geom = torch.tensor([[i % nx * w // nx, i // nx * h // ny,
                              min(width, w - i % nx * w // nx), min(width, h - i // nx * h // ny)]
                             for i in range(nx * ny)], dtype=torch.int32, device="cuda")
        out = torch.empty(2, nx * ny, dtype=torch.float64, device="cuda")
        fn = xbach.lib().xb_stamp_stats_noalloc
        vp, i32, f64 = ctypes.c_void_p, ctypes.c_int, ctypes.c_double
        fn.argtypes = [vp, vp, i32, i32, vp, i32, i32, f64, f64, vp, vp, vp, ctypes.c_char_p,
                       ctypes.c_size_t]
        return dict(kind=kind, fn=fn, img=img, mask=mask, geom=geom, out=out, w=w, h=h, n=nx * ny,
                    width=width)
    stats, pix, label, weight = _candidates(case["n"], gen)
    W = torch.from_numpy(_weights(seed)).cuda()
    state = dict(kind=kind, W=W, stats=stats, pix=pix, n=case["n"])
    if kind == "score":
        return dict(state, logit=torch.empty(case["n"], device="cuda"))
    per = torch.empty(case["n"], W.numel(), device="cuda")
    return dict(state, label=label, weight=weight, per=per, grad=torch.empty_like(W),
                loss=torch.empty(case["n"], device="cuda"), m=torch.zeros_like(W),
                v=torch.zeros_like(W), step=0)


# ---- one pass -------------------------------------------------------------

class _DeviceImage:
    """A context's device image for torch.as_tensor; the tensor holds this
    object and so the context that owns the memory."""

    def __init__(self, ctx, ptr, shape):
        self.ctx = ctx
        self.__cuda_array_interface__ = dict(shape=shape, typestr="<f4", data=(ptr, False),
                                             version=3)


def _view(ctx, ptr, shape):
    t = torch.as_tensor(_DeviceImage(ctx, ptr, shape), device="cuda")
    t.owner = ctx
    return t


def _ok(rc, what):
    if rc:
        raise xbach.XbError(rc, what)


def run(state):
    kind = state["kind"]
    if kind == "plain":
        ctx = state["ctx"]
        ctx.run(state["T"], state["S"])
        return dict(conv=ctx.image(xbach.XB_IMG_CONV), diff=ctx.image(xbach.XB_IMG_DIFF),
                    mask=ctx.mask(), solution=ctx.solution())
    if kind in ("plain_dev", "mixed"):
        T = state["T"]
        h, w = T.shape
        state["ctx"].run_device(T.data_ptr(), state["S"].data_ptr(), w, h,
                                state["conv"].data_ptr(), state["diff"].data_ptr())
        return dict(conv=state["conv"], diff=state["diff"])
    if kind == "batch":
        status, _ = state["batch"].run_ptrs(
            [t.data_ptr() for t in state["T"]], [s.data_ptr() for s in state["S"]], state["w"],
            state["h"], [c.data_ptr() for c in state["conv"]],
            [d.data_ptr() for d in state["diff"]], device=not state["host"])
        return dict(status=np.array(status), conv=state["conv"], diff=state["diff"])
    if kind == "apply":
        ctx = state["ctx"]
        ctx.conv()
        ctx.sub()
        return [_view(ctx, p, state["shape"]) for p in ctx.device_images()]
    stream = torch.cuda.current_stream().cuda_stream
    if kind == "stats":
        err = ctypes.create_string_buffer(256)
        p = (3.0, 1.35)   # sigClipAlpha, iqRange
        sky, sigma = state["out"]
        _ok(state["fn"](state["img"].data_ptr(), state["mask"].data_ptr(), state["w"], state["h"],
                        state["geom"].data_ptr(), state["n"], state["width"], *p, sky.data_ptr(),
                        sigma.data_ptr(), stream, err, 256), err.value)
        return dict(sky=sky, sigma=sigma)
    L = xbach.lib()
    W, stats, pix, n = (state[k] for k in ("W", "stats", "pix", "n"))
    if kind == "score":
        _ok(L.xb_ranker_forward(W.data_ptr(), stats.data_ptr(), pix.data_ptr(), n,
                                state["logit"].data_ptr(), stream), "xb_ranker_forward")
        return state["logit"]
    state["step"] += 1
    _ok(L.xb_ranker_grad(W.data_ptr(), stats.data_ptr(), pix.data_ptr(), state["label"].data_ptr(),
                         state["weight"].data_ptr(), n, state["per"].data_ptr(),
                         state["grad"].data_ptr(), state["loss"].data_ptr(), stream),
        "xb_ranker_grad")
    _ok(L.xb_ranker_adam(W.data_ptr(), state["grad"].data_ptr(), state["m"].data_ptr(),
                         state["v"].data_ptr(), state["step"], ctypes.c_float(3e-3), stream),
        "xb_ranker_adam")
    return dict(grad=state["grad"], loss=state["loss"], W=W, m=state["m"], v=state["v"])


# ---- what a pass cannot do without ------------------------------------------

def _conv_flops(w, h, terms=1):
    return 2 * 441 * w * h * terms


def _frame_work(w, h, stamps, basis=49):
    """Both images in, both out; the convolution, the basis convolutions and
    Gram matrices of one substamp per stamp and direction, and three global
    solves (two test fits and one fit)."""
    n = 293 if basis == 49 else 588
    b = (21 * 31 * 51 * 21 + basis * 961 * 21) * 2 + (basis + 4) ** 2 * 961
    return dict(bytes=16 * w * h,
                flops=_conv_flops(w, h) + 2 * stamps ** 2 * b + 3 * (2 * n ** 3 / 3 + 4 * n * n))


def work(case):
    kind = case["kind"]
    if kind in ("plain", "plain_dev", "mixed"):
        return _frame_work(case["w"], case["h"], case["stamps"], case.get("basis", 49))
    if kind == "batch":
        parts = [_frame_work(*s) for s in _sizes(case)]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    if kind == "apply":
        # images in and out and the mask in and out; a spatially varying
        # kernel at every pixel is one convolution per spatial term
        px = case["w"] * case["h"]
        return dict(bytes=20 * px, flops=_conv_flops(case["w"], case["h"],
                                                    6 if case["per_pixel"] else 1))
    if kind == "stats":
        px = case["nx"] * case["ny"] * case["width"] ** 2
        return dict(bytes=6 * px, flops=8 * px)
    n = case["n"]
    forward = 2 * (196 * 8 * 50 + 36 * 8 * 72 + 16 * 8 * 72 + 32 * 16 + 40)
    if kind == "score":
        return dict(bytes=4 * n * (2 * 961 + 16 + 1), flops=n * forward)
    return dict(bytes=4 * n * (2 * 961 + 16 + 3) + 7 * 4 * 2161, flops=3 * n * forward)


# ---- in 64 bits -------------------------------------------------------------

_SHAPES = [(8, 2, 5, 5), (8,), (8, 8, 3, 3), (8,), (8, 8, 3, 3), (8,), (32, 16), (32,), (40,), (1,)]


def exact(case, seed):
    """The ranker's logits, or its losses, gradients and updated state, in
    FP64 (its weights are BF16 values by definition).  The other kinds fit a
    whole frame or follow a sampled statistic and have no short FP64 form."""
    if case["kind"] not in ("score", "train"):
        return None
    stats, pix, label, weight = _candidates(case["n"], _generator(seed))
    W = torch.from_numpy(_weights(seed)).cuda()
    flat = W.bfloat16().double().requires_grad_(True)
    c1, b1, c2, b2, c3, b3, m1, mb, hw, hb = (
        v.reshape(s) for v, s in zip(flat.split([math.prod(s) for s in _SHAPES]), _SHAPES))

    def conv(a, k, b, stride):
        # windows times weights in FP64
        win = torch.nn.functional.unfold(a, k.shape[-1], stride=stride)
        side = math.isqrt(win.shape[-1])
        return (k.reshape(len(k), -1) @ win + b[:, None]).reshape(len(a), len(k), side, side)

    a = pix.double().reshape(-1, 2, 31, 31)
    for k, b, stride in ((c1, b1, 2), (c2, b2, 2), (c3, b3, 1)):
        a = torch.relu(conv(a, k, b, stride))
    hidden = torch.cat([a.mean(dim=(2, 3)), torch.relu(stats.double() @ m1.T + mb)], dim=1)
    z = hidden @ hw + hb
    if case["kind"] == "score":
        return z.detach()
    loss = weight.double() * torch.nn.functional.binary_cross_entropy_with_logits(
        z, label.double(), reduction="none")
    loss.mean().backward()
    g = flat.grad
    m, v = 0.1 * g, 0.001 * g * g
    step = 3e-3 * (m / 0.1) / ((v / 0.001).sqrt() + 1e-8)
    return dict(grad=g, loss=loss.detach(), W=W.double() - step, m=m, v=v)
