"""The slab level kernel against the per-stage kernels: bit-identical at the sizes where its
windows, bands, alignment paths and edge handling change."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SLAB = 3  # setTuningState path


def frames_of(H, W, T, seed):
    rng = np.random.default_rng(seed)
    base = rng.integers(0, 256, (H + T, W + T), dtype=np.uint8)
    k = np.ones(3) / 3
    b = np.apply_along_axis(lambda r: np.convolve(r, k, "same"), 1, base.astype(np.float64))
    b = np.apply_along_axis(lambda r: np.convolve(r, k, "same"), 0, b)
    return [np.ascontiguousarray(np.clip(b[t:t + H, t // 2:t // 2 + W], 0, 255).astype(np.uint8)) for t in range(T)]


def states(f, levels):
    return [f.levelState(l, k) for l in range(levels) for k in (0, 2, 3 if l < levels - 1 else 1)]


def same(a, b):
    return all(np.array_equal(x.view(np.uint32), y.view(np.uint32)) for x, y in zip(a, b))


# sizes at 4-column, window (112 or 104 columns) and warp-run boundaries, and shorter than the halo
SIZES = [(1, 1), (2, 3), (1, 130), (131, 1), (9, 13), (33, 65), (61, 111), (40, 112), (57, 113), (30, 127), (30, 129),
         (70, 225), (100, 227), (260, 337)]
PARAMS = [(1, 1.0, [1], 3), (1, 3.0, [4], 0), (1, 6.0, [6], 1), (2, 4.0, [1, 2], 3), (2, 3.0, [2, 4], 0),
          (2, 2.0, [3, 1], 40), (3, 4.0, [4, 2, 1], 2)]


@pytest.mark.parametrize("H,W", SIZES)
@pytest.mark.parametrize("rows", [0, 1, 7])
def test_slab_equals_per_stage(cuda, H, W, rows):
    import flowfilter_b200 as ffb

    for n, (levels, maxflow, smooth, border) in enumerate(PARAMS):
        if min(H, W) >> (levels - 1) < 1:
            continue
        clip = frames_of(H, W, 4, n)
        out = []
        for tuning in ((0, 0), (SLAB, rows)):
            f = ffb.FlowFilter(H, W) if levels == 1 else ffb.PyramidalFlowFilter(H, W, levels)
            f.maxflow = maxflow
            f.gamma = 8.0 if levels == 1 else [8.0, 20.0, 30.0][:levels]
            f.smoothIterations = smooth if levels > 1 else smooth[0]
            f.propagationBorder = border
            f.setTuningState([tuning] * levels)
            got = []
            for x in clip:
                f.loadImage(x)
                f.compute()
                got.append(states(f, levels))
            out.append(got)
        for t, (a, b) in enumerate(zip(*out)):
            assert same(a, b), (levels, maxflow, smooth, border, t)


@pytest.mark.parametrize("W,pad,shift", [(112, 0, 0), (113, 0, 0), (116, 8, 1), (115, 3, 2)])
def test_slab_float_images_any_alignment(cuda, W, pad, shift):
    """Float images in place: 16-byte aligned rows, and rows at any 4-byte offset; non-finite
    pixels travel as in the per-stage kernels."""
    import flowfilter_b200 as ffb

    torch = cuda
    H = 70
    clip = [torch.from_numpy(x).cuda().float() / 255 for x in frames_of(H, W, 3, 5)]
    clip[1][20, 30], clip[1][33, W - 1], clip[2][50, 0] = float("inf"), float("nan"), -0.0
    out = []
    for tuning in ((0, 0), (SLAB, 0)):
        img = torch.zeros(H * (W + pad) + shift + 8, device="cuda")[shift:shift + H * (W + pad)].view(H, W + pad)[:, :W]
        f = ffb.FlowFilter.on_device(img)
        f.gamma, f.maxflow, f.smoothIterations = 0.005, 3.0, 2
        f.setTuningState([tuning])
        got = []
        for x in clip:
            img.copy_(x)
            f.compute()
            got.append(states(f, 1))
        out.append(got)
    for a, b in zip(*out):
        for x, y in zip(a, b):
            assert np.array_equal(x, y, equal_nan=True)


@pytest.mark.parametrize("dtype", ["u8", "f32"])
def test_slab_delta_filter(cuda, dtype):
    """A standalone delta filter with an external coarse flow of another ratio."""
    import flowfilter_b200 as ffb

    torch = cuda
    H, W = 90, 232
    g = torch.Generator(device="cuda").manual_seed(3)
    coarse = torch.randn((31, 77, 2), device="cuda", generator=g)
    clip = [torch.from_numpy(x).cuda() for x in frames_of(H, W, 3, 6)]
    out = []
    for tuning in ((0, 0), (SLAB, 0)):
        img = torch.zeros((H, W), dtype=torch.uint8 if dtype == "u8" else torch.float32, device="cuda")
        f = ffb.DeltaFlowFilter(img, coarse)
        f.gamma, f.maxflow, f.smoothIterations = (10.0 if dtype == "u8" else 0.001), 4.0, 2
        f.setTuningState([tuning])
        got = []
        for x in clip:
            img.copy_(x if dtype == "u8" else x.float() / 255)
            f.compute()
            got.append([f.levelState(0, k) for k in (0, 2, 3)])
        out.append(got)
    for a, b in zip(*out):
        assert same(a, b)


def clip_flows(torch, H, W, n, seed, pad=0):
    """n float32 fields (H, W, 2) of signed flows with zeros, rows padded by ``pad`` pixels."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    out = []
    for _ in range(n):
        f = torch.randn((H, W + pad, 2), generator=g, device="cuda")
        f[torch.rand((H, W + pad), generator=g, device="cuda") < 0.1] = 0.0
        out.append(f[:, :W])
    return out


@pytest.mark.parametrize("H,W,pad", [(1, 1, 0), (3, 2, 1), (40, 127, 0), (29, 128, 0), (33, 129, 3), (75, 241, 0),
                                     (260, 116, 4)])
@pytest.mark.parametrize("n,border", [(1, 0), (2, 3), (5, 1), (8, 3), (9, 3)])
def test_stages_equal_the_oracle(cuda, H, W, pad, n, border):
    """Propagation, smoothing and image model at slab edges, at the most iterations of one launch
    and one more, on padded rows."""
    import oracle as O
    from flowfilter_b200 import stages

    torch = cuda
    flow, vec = clip_flows(torch, H, W, 2, 7 * H + n, pad)
    sca = torch.rand((H, W + pad), generator=torch.Generator(device="cuda").manual_seed(H + n), device="cuda")[:, :W]
    host = [t.cpu().numpy().copy() for t in (flow, sca, vec)]
    got = stages.propagate(flow, n, border).cpu().numpy()
    assert np.array_equal(got, O.propagate(host[0], n, border))
    got = [t.cpu().numpy() for t in stages.propagate_payload(flow, sca, vec, n, border)]
    assert all(np.array_equal(x, y) for x, y in zip(got, O.propagate_payload(*host, n, border)))
    assert np.array_equal(stages.smooth(flow, n).cpu().numpy(), O.smooth(host[0], n))
    u8 = torch.from_numpy(frames_of(H, W + pad, 1, n)[0]).cuda()[:, :W]
    for img in (u8, u8.float() / 255):
        a0, grad = (t.cpu().numpy() for t in stages.image_model(img))
        wa, wg = O.image_model(img.cpu().numpy().copy())
        assert np.array_equal(a0, wa) and np.array_equal(grad, wg)


@pytest.mark.parametrize("B,H,W,levels", [(1, 37, 53, 1), (3, 33, 128, 2), (1, 31, 132, 2), (2, 70, 240, 3)])
def test_taped_frame_equals_the_stage_functions(cuda, B, H, W, levels):
    """Flows and gradients of the frame node, whose float forward keeps its tape from the slab
    kernel, against one autograd node per stage."""
    from flowfilter_b200 import diff

    torch = cuda
    g = torch.Generator(device="cuda").manual_seed(W)
    frames = torch.rand((B, 3, H, W), generator=g, device="cuda")
    res = []
    for per_stage in (True, False):
        f = diff.DiffPyramidalFlowFilter(H, W, levels, [0.01, 0.02, 0.03][:levels], [2, 1, 3][:levels], maxflow=3.0)
        f.per_stage = per_stage
        x = frames.clone().requires_grad_(True)
        y = f(x)
        y.square().sum().backward()
        res.append((y.detach(), f.gamma.grad, f.weights.grad, x.grad))
    assert torch.equal(res[0][0], res[1][0])
    for a, b in zip(res[0][1:], res[1][1:]):  # the same sums in another order
        assert torch.allclose(a, b, rtol=1e-3, atol=1e-5 * float(a.abs().max()))
