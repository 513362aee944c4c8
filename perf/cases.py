"""The work this framework is used for, as timed cases over its public entry points.

Kinds of case and what each stands for:

  filter   one video frame through a FlowFilter / PyramidalFlowFilter with the frame already on
           the GPU: loadImage (device copy), computeAsync, and the flow read as a device view.
           Eager or replayed from the filter's CUDA graphs (``graphs``), uint8 frames into a
           filter that owns its image or float frames into FlowFilter.on_device (``dtype``).
  host     the reference's own loop: loadImage of a numpy frame, blocking compute(), getFlow().
  batch    one step of many independent video streams of different sizes (BatchFlowFilter).
  infer    the differentiable filter's forward over a clip, gradients off.
  train    the differentiable filter's forward, endpoint-error loss and backward over a clip.
  stages   one level step built from the stage functions, as a user of the stage API wires it,
           with the flow colour-encoded at the end.
  predict  the rotational image predictor (camera flow and Lax-Wendroff propagation).

Frames are blurred noise moved by a smooth random field of Gaussian bumps, with sensor noise on
uint8 frames; filters have run a few frames before the timed pass, so their state is that of a
running video.  ``exact`` restates every path in float64 with plain torch operations.
"""

import math
import os
import random
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "optical-flow-filter_b200"))

import flowfilter_b200 as ffb  # noqa: E402
from flowfilter_b200 import diff, stages  # noqa: E402

WARM = 3   # frames a filter has seen before the first timed pass
RING = 4   # frames the timed passes cycle through
DEV = "cuda"


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # a small camera on a robot: single-level filter, launch and host latency dominate
        dict(name="flow_320x240_L1", kind="filter", H=240, W=320, levels=1, gamma="10", smooth="1", maxflow=4.0,
             border=3, dtype="u8", graphs=False),
        # VGA video, two levels (the configuration the reference's notebook quotes)
        dict(name="flow_640x480_L2", kind="filter", H=480, W=640, levels=2, gamma="10,50", smooth="2,4", maxflow=4.0,
             border=3, dtype="u8", graphs=False),
        # a cropped sensor region: odd sizes at every level, three sub-steps
        dict(name="flow_1001x701_L3", kind="filter", H=701, W=1001, levels=3, gamma="20,20,40", smooth="2,1,3",
             maxflow=3.0, border=3, dtype="u8", graphs=False),
        # full high-speed camera sensor, three levels, frames replayed from CUDA graphs
        dict(name="flow_2048x1088_L3", kind="filter", H=1088, W=2048, levels=3, gamma="5,20,50", smooth="1,2,4",
             maxflow=4.0, border=3, dtype="u8", graphs=True),
        # float images produced on the GPU by an earlier stage, single level
        dict(name="flow_f32_1280x720_L1", kind="filter", H=720, W=1280, levels=1, gamma="0.005", smooth="2",
             maxflow=2.0, border=3, dtype="f32", graphs=False),
        # the reference's blocking loop with host images
        dict(name="host_640x480_L2", kind="host", H=480, W=640, levels=2, gamma="10,50", smooth="2,4", maxflow=4.0,
             border=3, dtype="u8", graphs=False),
        # a few small cameras served together
        dict(name="batch_8", kind="batch", streams=8, sizes="320x240,640x480", mix=7, maxflow=4.0),
        # a server's mix of streams from 320x240 to 1920x1080
        dict(name="batch_64", kind="batch", streams=64, sizes="320x240,640x480,1280x720,1920x1080", mix=100,
             maxflow=4.0),
        # evaluation of a fitted filter on clips of an odd size
        dict(name="infer_8x8x181x243", kind="infer", B=8, T=8, H=181, W=243, levels=2, gamma="0.01,0.005",
             smooth="2,4", maxflow=4.0, every=8),
        # one optimisation step of a fit: checkpointed forward and backward, all gradients
        dict(name="train_16x16x256x256", kind="train", B=16, T=16, H=256, W=256, levels=2, gamma="0.01,0.005",
             smooth="2,4", maxflow=4.0, every=8),
        # a hand-wired delta level on HD frames
        dict(name="stages_1280x720", kind="stages", H=720, W=1280, delta=True, iters=4, smooth=2, maxflow=4.0,
             gamma=10.0, border=3, dtype="u8"),
        # image prediction for a rotating camera
        dict(name="predict_640x480", kind="predict", H=480, W=640, depth=1, iters=4),
    ]


def _size(rng, lo, hi, pixels):
    """A width and height, each log-uniform in [lo, hi], odd half the time, of at most ``pixels``."""
    while True:
        w, h = (int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))))) for _ in range(2))
        if rng.random() < 0.5:
            w, h = (w + 7) // 8 * 8, (h + 7) // 8 * 8
        if w * h <= pixels and w <= 3 * h and h <= 3 * w:
            return w, h


def _join(values):
    return ",".join("%.4g" % v for v in values)


def draw(rng):
    kind = rng.choice(["filter", "filter", "filter", "host", "batch", "infer", "train", "stages", "predict"])
    if kind in ("filter", "host"):
        dtype = "f32" if kind == "filter" and rng.random() < 0.25 else "u8"
        w, h = _size(rng, 64, 2048, 2048 * 1088 if kind == "filter" else 1280 * 720)
        levels = 1 if dtype == "f32" else rng.randint(1, 3)
        lo, hi = (0.002, 0.05) if dtype == "f32" else (2.0, 100.0)
        return dict(kind=kind, H=h, W=w, levels=levels,
                    gamma=_join(math.exp(rng.uniform(math.log(lo), math.log(hi))) for _ in range(levels)),
                    smooth=_join(rng.randint(1, 4) for _ in range(levels)), maxflow=float(rng.randint(1, 4)),
                    border=rng.choice([3, 3, 3, 0, 5]), dtype=dtype, graphs=kind == "filter" and rng.random() < 0.4)
    if kind == "batch":
        n = int(round(math.exp(rng.uniform(math.log(4), math.log(48)))))
        sizes = []
        for _ in range(4):
            w, h = _size(rng, 96, 1920, 1280 * 720)
            sizes.append("%dx%d" % (w, h))
        return dict(kind=kind, streams=n, sizes=",".join(sizes), mix=rng.randrange(1 << 20), maxflow=4.0)
    if kind in ("infer", "train"):
        B, T = rng.randint(1, 16), rng.randint(4, 16)
        w, h = _size(rng, 64, 512, min(512 * 512, 16 * 16 * 256 * 256 // (B * T)))
        levels = rng.randint(1, 3)
        return dict(kind=kind, B=B, T=T, H=h, W=w, levels=levels,
                    gamma=_join(math.exp(rng.uniform(math.log(0.002), math.log(0.05))) for _ in range(levels)),
                    smooth=_join(rng.randint(1, 4) for _ in range(levels)), maxflow=float(rng.randint(1, 4)),
                    every=rng.choice([4, 8, 16]))
    if kind == "stages":
        w, h = _size(rng, 64, 2048, 2048 * 1088)
        dtype = rng.choice(["u8", "f32"])
        return dict(kind=kind, H=h, W=w, delta=rng.random() < 0.5, iters=rng.randint(1, 4), smooth=rng.randint(1, 4),
                    maxflow=4.0, gamma=10.0 if dtype == "u8" else 0.005, border=rng.choice([0, 3]), dtype=dtype)
    w, h = _size(rng, 64, 2048, 1920 * 1080)
    return dict(kind=kind, H=h, W=w, depth=rng.choice([1, 4]), iters=rng.randint(1, 8))


def _floats(text):
    return [float(v) for v in text.split(",")]


def _ints(text):
    return [int(float(v)) for v in text.split(",")]


def _shapes(H, W, levels):
    out = [(H, W)]
    for _ in range(levels - 1):
        out.append((out[-1][0] // 2, out[-1][1] // 2))
    return out


def _streams(case):
    """The streams of a batch: size, levels and seeded parameters of each."""
    rng = random.Random(case["mix"])
    sizes = [tuple(int(v) for v in s.split("x")) for s in case["sizes"].split(",")]
    out = []
    for i in range(case["streams"]):
        w, h = sizes[i * len(sizes) // case["streams"]]
        levels = rng.randint(1, 3)
        out.append(dict(H=h, W=w, levels=levels, maxflow=case["maxflow"], border=3, dtype="u8",
                        gamma=_join(math.exp(rng.uniform(math.log(2.0), math.log(100.0))) for _ in range(levels)),
                        smooth=_join(rng.randint(1, 4) for _ in range(levels))))
    return out


# ------------------------------------------------------------------ inputs
def _bumps(H, W, g, sigma, amp, n=8):
    """A smooth flow field (H, W, 2): n Gaussian bumps with amplitudes in [-amp, amp]."""
    p = torch.rand(n, 4, generator=g, device=DEV)
    x = torch.arange(W, device=DEV).view(1, 1, W) - (p[:, 0] * W).view(n, 1, 1)
    y = torch.arange(H, device=DEV).view(1, H, 1) - (p[:, 1] * H).view(n, 1, 1)
    e = torch.exp(-x * x / (2 * sigma * sigma)) * torch.exp(-y * y / (2 * sigma * sigma))
    return torch.einsum("nhw,nc->hwc", e, (2 * p[:, 2:] - 1) * amp)


def _texture(H, W, g, sigma):
    """Blurred noise (H, W) in [0, 1]."""
    r = int(math.ceil(3 * sigma))
    k = torch.exp(-0.5 * (torch.arange(-r, r + 1, device=DEV) / sigma) ** 2)
    k = k / k.sum()
    t = torch.rand(1, 1, H + 2 * r, W + 2 * r, generator=g, device=DEV)
    for v in (k.view(1, 1, -1, 1), k.view(1, 1, 1, -1)):  # separable, tap by tap
        n = v.numel()
        h, w = (t.shape[2] - n + 1, t.shape[3]) if v.shape[2] > 1 else (t.shape[2], t.shape[3] - n + 1)
        t = sum(v.view(-1)[i] * (t[:, :, i:i + h] if v.shape[2] > 1 else t[:, :, :, i:i + w]) for i in range(n))
    t = t[0, 0]
    return (t - t.min()) / (t.max() - t.min())


def _warp(tex, flow, t):
    """tex sampled at x - t * flow, bilinear, border replicated."""
    H, W = tex.shape
    x = torch.arange(W, device=DEV).view(1, W) - t * flow[..., 0]
    y = torch.arange(H, device=DEV).view(H, 1) - t * flow[..., 1]
    x, y = x.clamp(0, W - 1), y.clamp(0, H - 1)
    x0, y0 = x.floor().clamp(max=max(W - 2, 0)), y.floor().clamp(max=max(H - 2, 0))
    fx, fy = x - x0, y - y0
    i = (y0 * W + x0).long()
    f = tex.reshape(-1)
    return (f[i] * (1 - fx) + f[i + 1] * fx) * (1 - fy) + (f[i + W] * (1 - fx) + f[i + W + 1] * fx) * fy


def _gen(seed, salt=0):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed) * 1009 + salt)
    return g


def _clip(H, W, frames, g, dtype):
    """A clip (frames, H, W): uint8 with sensor noise, or float32 in [0, 1]."""
    tex = _texture(H, W, g, 1.5)
    flow = _bumps(H, W, g, 150.0, 3.0)
    out = []
    for t in range(frames):
        f = _warp(tex, flow, t)
        if dtype == "u8":
            f = (255 * f + 3 * torch.randn(H, W, generator=g, device=DEV)).round().clamp(0, 255).to(torch.uint8)
        out.append(f)
    return torch.stack(out)


def _configure(f, c):
    """Sets a filter's parameters from a case."""
    gamma, smooth = _floats(c["gamma"]), _ints(c["smooth"])
    f.maxflow = c["maxflow"]
    f.gamma = gamma if c["levels"] > 1 else gamma[0]
    f.smoothIterations = smooth if c["levels"] > 1 else smooth[0]
    f.propagationBorder = c["border"]


def _clips(c, seed):
    """Sequences and their true flow for the differentiable filter."""
    g = _gen(seed)
    seqs, truth = [], []
    for _ in range(c["B"]):
        tex = _texture(c["H"], c["W"], g, 1.5)
        flow = _bumps(c["H"], c["W"], g, 40.0, 2.0)
        seqs.append(torch.stack([_warp(tex, flow, t) for t in range(c["T"])]))
        truth.append(flow)
    return torch.stack(seqs), torch.stack(truth)[:, None].expand(c["B"], c["T"], c["H"], c["W"], 2)


def _stage_inputs(c, seed):
    """What a user of the stage functions holds: RING images, the flow, the old image and, for a
    delta level, the delta flow and the coarse flow."""
    g = _gen(seed)
    H, W = c["H"], c["W"]
    imgs = _clip(H, W, RING, g, c["dtype"])
    scale = 1.0 / 255.0 if c["dtype"] == "u8" else 1.0
    return dict(imgs=imgs, flow=_bumps(H, W, g, 150.0, 3.0) + 0.05 * torch.randn(H, W, 2, generator=g, device=DEV),
                old=imgs[0].float() * scale, delta=0.3 * torch.randn(H, W, 2, generator=g, device=DEV),
                coarse=_bumps(max(H // 2, 1), max(W // 2, 1), g, 75.0, 1.5),
                gamma=c["gamma"] / (255.0 * 255.0) if c["dtype"] == "u8" else c["gamma"])


def _predict_inputs(c, seed):
    g = _gen(seed)
    H, W = c["H"], c["W"]
    imgs = torch.stack([_texture(H, W, g, 1.5) for _ in range(RING * c["depth"])]).view(RING, c["depth"], H, W)
    imgs = imgs[:, 0].contiguous() if c["depth"] == 1 else imgs.permute(0, 2, 3, 1).contiguous()
    w = (torch.rand(3, generator=torch.Generator().manual_seed(int(seed))) * 0.008 - 0.004).tolist()
    return imgs, w


CAMERA = dict(focal=8.0, sensor_h=4.8, sensor_w=6.4)  # an 8 mm lens on a 1/2" sensor


def prepare(case, seed):
    c, kind = case, case["kind"]
    if kind in ("filter", "host"):
        clip = _clip(c["H"], c["W"], WARM + RING, _gen(seed), c["dtype"])
        if c["dtype"] == "f32":
            f = ffb.FlowFilter.on_device(torch.zeros_like(clip[0]))
        elif c["levels"] == 1:
            f = ffb.FlowFilter(c["H"], c["W"])
        else:
            f = ffb.PyramidalFlowFilter(c["H"], c["W"], c["levels"])
        _configure(f, c)
        if c["graphs"]:
            f.setGraphs(True)
        for t in range(WARM):
            f.loadImage(clip[t])
            f.computeAsync()
        s = dict(kind=kind, filter=f, at=0)
        if kind == "host":
            s["frames"] = [x.cpu().numpy() for x in clip[WARM:]]
            s["flow"] = np.zeros((c["H"], c["W"], 2), np.float32)
        else:
            s["frames"] = list(clip[WARM:])
        return s
    if kind == "batch":
        streams = _streams(c)
        b = ffb.BatchFlowFilter([(s["H"], s["W"], s["levels"]) for s in streams])
        for i, s in enumerate(streams):
            _configure(b.stream(i), s)
        clips = [_clip(s["H"], s["W"], WARM + RING, _gen(seed, i), "u8") for i, s in enumerate(streams)]
        packed = [b.pack([x[t] for x in clips]) for t in range(WARM + RING)]
        for t in range(WARM):
            b.step(packed[t])
        return dict(kind=kind, batch=b, frames=packed[WARM:], at=0)
    if kind in ("infer", "train"):
        frames, truth = _clips(c, seed)
        f = ffb.diff.DiffPyramidalFlowFilter(c["H"], c["W"], c["levels"], gamma=_floats(c["gamma"]),
                                             smoothIterations=_ints(c["smooth"]), maxflow=c["maxflow"],
                                             checkpoint_every=c["every"])
        if kind == "train":
            frames.requires_grad_(True)
        return dict(kind=kind, filter=f, frames=frames, truth=truth, first=c["T"] // 4)
    if kind == "stages":
        s = _stage_inputs(c, seed)
        s.update(kind=kind, case=dict(c), at=0, color=ffb.FlowToColor(s["flow"], c["maxflow"]))
        return s
    imgs, w = _predict_inputs(c, seed)
    cam = ffb.createPerspectiveCamera(CAMERA["focal"], c["H"], c["W"], CAMERA["sensor_h"], CAMERA["sensor_w"])
    p = ffb.RotationalFlowImagePredictor(cam, imgs[0])
    p.setAngularVelocity(*w)
    p.iterations = c["iters"]
    return dict(kind=kind, predictor=p, imgs=imgs, at=0)


def _next(s, key):
    x = s[key][s["at"] % RING]
    s["at"] += 1
    return x


def run(state):
    s, kind = state, state["kind"]
    if kind == "filter":
        f = s["filter"]
        f.loadImage(_next(s, "frames"))
        f.computeAsync()
        return f.flowTensor()
    if kind == "host":
        f = s["filter"]
        f.loadImage(_next(s, "frames"))
        f.compute()
        return f.getFlow(s["flow"])
    if kind == "batch":
        b = s["batch"]
        b.step(_next(s, "frames"))
        return [b.stream(i).flowTensor() for i in range(len(b))]
    if kind == "infer":
        with torch.no_grad():
            return s["filter"](s["frames"])
    if kind == "train":
        f, frames = s["filter"], s["frames"]
        flows = f(frames)
        loss = diff.endpoint_error(flows, s["truth"], first=s["first"], eps=1e-12)
        grads = torch.autograd.grad(loss, [f.gamma, f.weights, frames])
        return dict(flows=flows, loss=loss, gamma=grads[0], weights=grads[1], frames=grads[2])
    if kind == "stages":
        c, img = s["case"], _next(s, "imgs")
        a0, grad = stages.image_model(img)
        if c["delta"]:
            small = stages.pyramid_down(img)
            f, old, d = stages.propagate_payload(s["flow"], s["old"], s["delta"], c["iters"], c["border"])
            flow, delta, image = stages.delta_update(a0, grad, old, d, s["coarse"], s["gamma"], c["maxflow"])
            out = [small, a0, grad, f, old, d, flow, delta, image]
        else:
            f = stages.propagate(s["flow"], c["iters"], c["border"])
            flow, image = stages.update(a0, grad, s["old"], f, s["gamma"], c["maxflow"])
            out = [a0, grad, f, flow, image]
        smooth = stages.smooth(flow, c["smooth"])
        color = s["color"]
        color.setInputFlow(smooth)
        color.compute()
        return out + [smooth, color.getColorFlow()]
    p = s["predictor"]
    p.setInputImage(_next(s, "imgs"))
    p.compute()
    return [p.getPredictedImage(), p.getOpticalFlow()]


# ------------------------------------------------------------------ compulsory work
# floating-point operations per pixel: an upwind X/Y pair of one channel, the image model, the
# 2x2 solve with its clamps, and one smoothing iteration of a flow field
OP_PAIR, OP_MODEL, OP_SOLVE, OP_SMOOTH = 8, 45, 40, 36


def _level_iters(maxflow, levels):
    out, m = [], maxflow
    for l in range(levels):
        out.append(max(1, int(math.ceil(m))))
        if l < levels - 1:
            m /= 2.0
    return out


def _frame_work(c, state=True):
    """Bytes and operations of one frame of one stream: its image, and the state read and written
    (smoothed flow and old image, plus the delta flow of every level but the top)."""
    item = 1 if c.get("dtype", "f32") == "u8" else 4
    smooth, iters = _ints(c["smooth"]), _level_iters(c["maxflow"], c["levels"])
    nbytes, flops = c["H"] * c["W"] * item, 0
    for l, (h, w) in enumerate(_shapes(c["H"], c["W"], c["levels"])):
        delta = l < c["levels"] - 1
        if state:
            nbytes += h * w * (40 if delta else 24)
        flops += h * w * ((5 if delta else 2) * OP_PAIR * iters[l] + OP_MODEL + OP_SOLVE + OP_SMOOTH * smooth[l])
    return nbytes, flops


def work(case):
    c, kind = case, case["kind"]
    if kind in ("filter", "host"):
        b, f = _frame_work(c)
        return dict(bytes=b, flops=f)
    if kind == "batch":
        w = [_frame_work(s) for s in _streams(c)]
        return dict(bytes=sum(x[0] for x in w), flops=sum(x[1] for x in w))
    n = c["H"] * c["W"]
    if kind in ("infer", "train"):
        n *= c["B"] * c["T"]
        f = _frame_work(c, state=False)[1] * c["B"] * c["T"]
        # frames in, flows out; with gradients also the true flow (one field a clip) and the
        # frames' gradient
        if kind == "infer":
            return dict(bytes=12 * n, flops=f)
        return dict(bytes=16 * n + 8 * n // c["T"], flops=3 * f)
    if kind == "stages":
        item, ch = (1 if c["dtype"] == "u8" else 4), (5 if c["delta"] else 2)
        ins = item + 12 + (8 + 2 if c["delta"] else 0)
        outs = 12 + 8 + 4 + 8 + 4 + 8 + ((12 + 8) + item // 4 if c["delta"] else 0)
        return dict(bytes=n * (ins + outs),
                    flops=n * (ch * OP_PAIR * c["iters"] + OP_MODEL + OP_SOLVE + OP_SMOOTH * c["smooth"]))
    return dict(bytes=n * (8 * c["depth"] + 8), flops=n * (24 + 18 * c["depth"] * c["iters"]))


# ------------------------------------------------------------------ the paths in float64
def _shift(a, axis, k):
    """a (B, H, W, ...) sampled at index + k along dimension ``axis``, clamped to the edge."""
    n = a.shape[axis]
    return a.index_select(axis, (torch.arange(n, device=a.device) + k).clamp(0, n - 1))


def _taps(a, axis, w):
    return sum(w[k] * _shift(a, axis, k - 2) for k in range(5) if not (isinstance(w[k], float) and w[k] == 0.0))


BLUR = [1 / 16, 1 / 4, 3 / 8, 1 / 4, 1 / 16]
DIFF = [-1 / 8, -1 / 4, 0.0, 1 / 4, 1 / 8]


def _model(img):
    by, bx = _taps(img, 1, BLUR), _taps(img, 2, BLUR)
    return _taps(by, 2, BLUR), torch.stack([_taps(by, 2, DIFF), _taps(bx, 1, DIFF)], -1)


def _down(img):
    """One pyramid step; bytes go through the float32 arithmetic that defines their truncation."""
    def half(a, axis):
        n = a.shape[axis] // 2
        at = lambda o: a.index_select(axis, (2 * torch.arange(n, device=a.device) + o).clamp(0, a.shape[axis] - 1))  # noqa: E731
        m, x, p = at(-1), at(0), at(1)
        if a.dtype != torch.uint8:
            return 0.5 * x + 0.25 * (m + p)
        unit = torch.tensor([v / 255.0 for v in range(256)], device=a.device).float()
        m, x, p = (unit[t.long()] for t in (m, x, p))
        s = (0.5 * x.double() + 0.25 * (m + p).double()).float()
        return (255.0 * s).to(torch.uint8)
    return half(half(img, 2), 1)


def _unit(img):
    return img.double() / 255.0 if img.dtype == torch.uint8 else img.double()


def _advect(fields, n, border):
    """n upwind X/Y sub-step pairs of the flow fields[0] and what it carries."""
    f = fields[0]
    H, W = f.shape[1:3]
    y, x = torch.arange(H, device=f.device).view(1, H, 1), torch.arange(W, device=f.device).view(1, 1, W)
    inside = (x >= border) & (x < W - border) & (y >= border) & (y < H - border)
    for _ in range(n):
        for axis, ch in ((2, 0), (1, 1)):
            m, p = _shift(fields[0][..., ch], axis, -1), _shift(fields[0][..., ch], axis, 1)
            v = torch.where(p.abs() - m.abs() > 0, p, m)
            out = []
            for g in fields:
                t, i = (v, inside) if g.dim() == 3 else (v[..., None], inside[..., None])
                d = torch.where(t >= 0, g - _shift(g, axis, -1), _shift(g, axis, 1) - g)
                out.append(torch.where(i, g - t / n * d, g))
            fields = out
    return fields


def _solve(gamma, grad, yt, f):
    ax, ay = grad[..., 0], grad[..., 1]
    r = 1.0 / (gamma * (gamma + ax * ax + ay * ay))
    qx, qy = gamma * f[..., 0] + ax * yt, gamma * f[..., 1] + ay * yt
    n00, n11, n01 = gamma + ay * ay, gamma + ax * ax, -ax * ay
    return torch.stack([(n00 * qx + n01 * qy) * r, (n01 * qx + n11 * qy) * r], -1)


def _upmap(n, nc):
    """The coarse index of every fine index: a normalised coordinate cut to 21 fractional bits."""
    if n == 1:
        return torch.zeros(1, dtype=torch.long, device=DEV)
    u = np.arange(n, dtype=np.float32) / np.float32(n - 1)
    q = np.floor(u * np.float32(2097152.0)).astype(np.int64)
    return torch.from_numpy(np.clip((q * nc) >> 21, 0, nc - 1)).to(DEV)


def _refine(a0, grad, old, d, coarse, gamma, maxflow):
    d = _solve(gamma, grad, old - a0, d).clamp(-0.5 * maxflow, 0.5 * maxflow)
    up = coarse[:, _upmap(a0.shape[1], coarse.shape[1])][:, :, _upmap(a0.shape[2], coarse.shape[2])]
    return (d + 2.0 * up).clamp(-maxflow, maxflow), d


def _box(f, n, w=None):
    for _ in range(n):
        f = _taps(f, 2, [0.2] * 5 if w is None else w)
        f = _taps(f, 1, [0.2] * 5 if w is None else w)
    return f


class _Filter64:
    """The pyramidal filter's recurrence in float64 on (B, H, W) frames."""

    def __init__(self, B, shapes, gamma, smooth, maxflow, border, weights=None):
        self.L, self.gamma, self.smooth, self.border, self.weights = len(shapes), gamma, smooth, border, weights
        self.maxflow = [maxflow / 2 ** l for l in range(self.L)]
        self.iters = _level_iters(maxflow, self.L)
        z = lambda *s: torch.zeros(*s, dtype=torch.float64, device=DEV)  # noqa: E731
        self.state = [(z(B, h, w, 2), None, z(B, h, w, 2)) for h, w in shapes]  # smoothed flow, old image, delta
        self.top = None

    def step(self, img):
        L, imgs = self.L, [img]
        for _ in range(L - 1):
            imgs.append(_down(imgs[-1]))
        new = [None] * L
        w = lambda l: None if self.weights is None else self.weights[l]  # noqa: E731
        for l in reversed(range(L)):
            a0, g = _model(_unit(imgs[l]))
            f, old, d = self.state[l]
            old = a0 if old is None else old
            if l == L - 1:
                (f,) = _advect([f], self.iters[l], self.border)
                m = self.maxflow[l]
                self.top = _solve(self.gamma[l], g, old - a0, f).clamp(-m, m)
                new[l] = (_box(self.top, self.smooth[l], w(l)), a0, d)
            else:
                first = self.state[l][1] is None
                _, s, d = _advect([f, old, d], self.iters[l], self.border)
                coarse = self.top if l == L - 2 else self.state[l + 1][0]
                f, d = _refine(a0, g, a0 if first else s, d, coarse, self.gamma[l], self.maxflow[l])
                new[l] = (_box(f, self.smooth[l], w(l)), a0, d)
        self.state = new
        return new[0][0]


def _video64(c, frames):
    """The smoothed flow after the last of ``frames`` (T, H, W)."""
    k = 255.0 * 255.0 if c["dtype"] == "u8" else 1.0
    f = _Filter64(1, _shapes(c["H"], c["W"], c["levels"]), [g / k for g in _floats(c["gamma"])], _ints(c["smooth"]),
                  c["maxflow"], c["border"])
    for x in frames:
        flow = f.step(x[None])
    return flow[0]


def exact(case, seed):
    c, kind = case, case["kind"]
    if kind in ("filter", "host"):
        flow = _video64(c, _clip(c["H"], c["W"], WARM + RING, _gen(seed), c["dtype"])[:WARM + 1])
        return flow.cpu().numpy() if kind == "host" else flow
    if kind == "batch":
        return [_video64(s, _clip(s["H"], s["W"], WARM + RING, _gen(seed, i), "u8")[:WARM + 1])
                for i, s in enumerate(_streams(c))]
    if kind in ("infer", "train"):
        grads = kind == "train"
        frames, truth = _clips(c, seed)
        with torch.set_grad_enabled(grads):
            frames = frames.double().requires_grad_(grads)
            gamma = torch.tensor(_floats(c["gamma"]), dtype=torch.float64, device=DEV, requires_grad=grads)
            weights = torch.full((c["levels"], 5), 0.2, dtype=torch.float64, device=DEV, requires_grad=grads)
            f = _Filter64(c["B"], _shapes(c["H"], c["W"], c["levels"]), gamma, _ints(c["smooth"]), c["maxflow"], 3,
                          weights)
            flows = []
            for t in range(c["T"]):
                y = f.step(frames[:, t])
                flows.append(y if c["levels"] > 1 else f.top)
            flows = torch.stack(flows, 1)
            if not grads:
                return flows
            d = flows[:, c["T"] // 4:] - truth[:, c["T"] // 4:].double()
            loss = (d.square().sum(-1) + 1e-12).sqrt().mean()
            g = torch.autograd.grad(loss, [gamma, weights, frames])
        return dict(flows=flows.detach(), loss=loss.detach(), gamma=g[0], weights=g[1], frames=g[2])
    if kind == "stages":
        s = _stage_inputs(c, seed)
        img, b = s["imgs"][0], lambda k: s[k].double()[None]
        a0, grad = _model(_unit(img[None]))
        if c["delta"]:
            f, old, d = _advect([b("flow"), b("old"), b("delta")], c["iters"], c["border"])
            flow, delta = _refine(a0, grad, old, d, b("coarse"), s["gamma"], c["maxflow"])
            out = [None if c["dtype"] == "u8" else _down(img.double()[None]), a0, grad, f, old, d, flow, delta, a0]
        else:
            (f,) = _advect([b("flow")], c["iters"], c["border"])
            m = c["maxflow"]
            flow = _solve(s["gamma"], grad, b("old") - a0, f).clamp(-m, m)
            out = [a0, grad, f, flow, a0]
        return [x if x is None else x[0] for x in out + [_box(flow, c["smooth"])]] + [None]
    imgs, w = _predict_inputs(c, seed)
    H, W, n = c["H"], c["W"], c["iters"]
    cx, cy = 0.5 * (W - 1), 0.5 * (H - 1)
    ax, ay = CAMERA["focal"] * (W - 1) / CAMERA["sensor_w"], CAMERA["focal"] * (H - 1) / CAMERA["sensor_h"]
    x = torch.arange(W, device=DEV, dtype=torch.float64).view(1, W).expand(H, W)
    y = torch.arange(H, device=DEV, dtype=torch.float64).view(H, 1).expand(H, W)
    px, py = (x - cx) / ax, (y - cy) / ay
    rx, ry, rz = w[1] - w[2] * py, w[2] * px - w[0], w[0] * py - w[1] * px
    flow = torch.stack([ax * rx + (cx - x) * rz, ay * ry + (cy - y) * rz], -1)
    v = imgs[0].double()[None]
    for _ in range(n):
        for axis, ch in ((1, 1), (2, 0)):
            r = (flow[..., ch] / n)[None]
            r = r if c["depth"] == 1 else r[..., None]
            m, p = _shift(v, axis, -1), _shift(v, axis, 1)
            v = v - 0.5 * r * (p - m) + 0.5 * r * r * (m - 2 * v + p)
    return [v[0], flow]
