"""The device kernels at the sizes and values where their fast paths end, against the oracle, bit for bit:
every integer sample, lerps between the ends of a depth's range, points on and across the image's border."""
import numpy as np
import pytest

import oracle_lib as O
import twixtor_b200 as tw

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def dev():
    tw.build()
    d = tw.Device(0)
    yield d
    d.close()


def same(a, b):
    return np.asarray(a).view(np.uint8).tobytes() == np.asarray(b).view(np.uint8).tobytes()


def integer_pixels(fmt):
    """Pairs (colour, alpha): all of the 8 bit depth, for 16 bits every alpha with colours around it."""
    if fmt == 0:
        c, a = np.meshgrid(np.arange(256), np.arange(256))
    else:
        a = np.arange(65536).repeat(4).reshape(-1, 4)
        c = np.stack([a[:, 0], a[:, 0] // 2, a[:, 0] * 3 + 1, np.full(65536, 65535)], 1) & 0xffff
    return c.reshape(-1), a.reshape(-1)


@pytest.mark.parametrize("fmt", [0, 1])
def test_every_sample_at_the_image_boundary(dev, fmt):
    c, a = integer_pixels(fmt)
    w = 256
    h = c.size // w
    top = 255 if fmt == 0 else 65535
    wire = np.stack([c, top - c, c ^ 1, a], 1).astype(tw.DTYPES[fmt]).reshape(-1)
    assert same(dev.from_frame(wire, w, h, fmt), O.from_frame(wire, w, h, fmt))
    eng = np.stack([a, c, top - c, c ^ 1], 1).astype(tw.DTYPES[fmt]).reshape(-1)
    assert same(dev.to_frame(eng, w, h, fmt), O.to_frame(eng, w, h, fmt))


@pytest.mark.parametrize("fmt", [0, 1, 2])
@pytest.mark.parametrize("size", [(2, 2), (33, 5), (129, 67)])
@pytest.mark.parametrize("wa,interp", [(0.3, 1), (0.5, 1), (1.5, 1), (0.6, 0)])
def test_warps_between_the_ends_of_the_range(dev, fmt, size, wa, interp):
    """Samples at 0 and at the top of the depth (or random), vectors that reach, touch and cross the border."""
    w, h = size
    rng = np.random.RandomState(w + fmt)
    top = {0: 255, 1: 65535, 2: 1.0}[fmt]
    ends = [(rng.randint(0, 2, w * h * 4) * top).astype(tw.DTYPES[fmt]) for _ in range(2)]
    full = [(rng.random_sample(w * h * 4) * top).astype(tw.DTYPES[fmt]) for _ in range(2)]
    flows = [rng.uniform(-4.0, 4.0, w * h * 2).astype(np.float32) for _ in range(2)]
    for f in flows:
        f[::7] = np.round(f[::7])
        f[::11] = 0.0
    for a, b in (ends, full):
        got = dev.compose_vectors(tw.EngineSettings(), tw.Selection(wa=np.float32(wa), interp=interp), a, b, w, h, fmt,
                                  flows[0], flows[1], (w, h))
        assert same(got, O.compose_vectors(a, b, w, h, fmt, flows[0], flows[1], w, h, np.float32(wa), interp))


@pytest.mark.parametrize("size", [(2, 2), (3, 200), (16, 17), (33, 32), (63, 64), (64, 65), (66, 31), (130, 129)])
@pytest.mark.parametrize("fmt,above_first", [(0, True), (1, False), (2, True), (2, False)])
def test_pyramid_steps_at_the_ends_of_their_tiles(dev, size, fmt, above_first):
    """Planes of one tile of each shape and a pixel more or less; float samples include zeros of both signs and
    magnitudes that the border division by reciprocals leaves to the plain division."""
    w, h = size
    rng = np.random.RandomState(w * 5 + h)
    eng = rng.random_sample(w * h * 4) * {0: 255, 1: 65535, 2: 1}[fmt]
    eng = eng.astype(tw.DTYPES[fmt])
    if fmt == 2:
        eng[rng.randint(0, eng.size, eng.size // 3)] = 0.0
        eng[rng.randint(0, eng.size, eng.size // 8)] = -0.0
        eng[rng.randint(0, eng.size, 3)] = [1e-40, 3e35, -2e-33]
    s = tw.FlowSettings(quality=5, taps_above_first=above_first)
    got = dev.build_pyramid(eng, w, h, fmt, s)
    want = O.build_pyramid(eng, w, h, fmt, quality=5, above_first=above_first)
    assert len(got) == len(want)
    for g, o in zip(got, want):
        assert same(g, o)


@pytest.mark.parametrize("size", [(3, 3), (16, 15), (17, 33), (31, 66), (65, 64), (129, 48), (200, 9)])
@pytest.mark.parametrize("masks", [False, True])
@pytest.mark.parametrize("points", [None, (-1.0, 0.0), (-1.0, -1.0)])
@pytest.mark.parametrize("above_first", [False, True])
def test_solves_at_the_ends_of_their_tiles(dev, size, masks, points, above_first):
    """Levels of one tile of each shape and a pixel more or less, in the one block of the coarse levels and out of
    it. The points put vectors of exactly -1.0, the sentinel of the border rule, near the corners."""
    w, h = size
    rng = np.random.RandomState(w * 3 + h)
    x = np.kron(rng.randint(0, 256, ((h + 2) // 3, (w + 2) // 3, 4)), np.ones((3, 3, 1)))[:h, :w].astype(np.uint8)
    y = np.roll(x, 1, axis=1)
    y[:, 0] = rng.randint(0, 256, (h, 4))
    x, y = np.ascontiguousarray(x).reshape(-1), np.ascontiguousarray(y).reshape(-1)
    mx = my = pairs = None
    if masks:
        mx, my = [(rng.random_sample((h, w)) < 0.9).astype(np.float32).ravel() for _ in range(2)]
    if points:
        at = np.array([[1.0, 1.0], [w - 1.0, 1.0], [1.0, h - 1.0], [w / 2, h / 2]], np.float32)
        pairs = np.concatenate([at, at + np.float32(points)], 1).astype(np.float32)
    kw = dict(quality=5, above_first=above_first)
    want, xl, yl, mxl, myl, ud, uw = O.solve_pyramids_with(x, y, w, h, 0, mx, my, pairs, **kw)
    s = tw.FlowSettings(quality=5, taps_above_first=above_first)
    got, _ = dev.solve_pyramids(s, w, h, xl, yl, mxl, myl, ud, uw)
    assert got.tobytes() == want.tobytes()


@pytest.mark.parametrize("size", [(256, 32), (32, 256), (128, 64), (254, 33), (258, 32), (32, 258), (130, 64)])
@pytest.mark.parametrize("masks", [False, True])
@pytest.mark.parametrize("content", ["blocks", "smooth"])
def test_solves_at_the_limits_of_the_coarse_block(dev, size, masks, content):
    """Levels of exactly 2048 pixels and 128 a side, which one block solves, and the next larger ones, which the
    tiled kernels take: block matching walks lines in several segments there, and walks a segment again where a
    run reaches into it (short runs with blocks of noise, runs across segments with smooth textures)."""
    w, h = size
    rng = np.random.RandomState(w * 3 + h)
    cell = 3 if content == "blocks" else 12
    x = np.kron(rng.randint(0, 256, (h // cell + 1, w // cell + 1, 4)), np.ones((cell, cell, 1)))[:h, :w]
    if content == "smooth":
        for axis in (0, 1):
            x = sum(np.roll(x, k, axis=axis) for k in range(-4, 5)) / 9.0
    y = x.copy()
    for i in range(0, h, 16):  # bands that move on their own
        y[i:i + 16] = np.roll(x[i:i + 16], rng.randint(-5, 6), axis=1)
    y[:, w // 3:w // 2] = np.roll(y[:, w // 3:w // 2], 3, axis=0)
    x, y = (np.ascontiguousarray(np.clip(v, 0, 255)).astype(np.uint8).reshape(-1) for v in (x, y))
    mx = my = None
    if masks:
        mx, my = [(rng.random_sample((h, w)) < 0.98).astype(np.float32).ravel() for _ in range(2)]
    want, xl, yl, mxl, myl, ud, uw = O.solve_pyramids_with(x, y, w, h, 0, mx, my, None, quality=5, above_first=True)
    got, _ = dev.solve_pyramids(tw.FlowSettings(quality=5, taps_above_first=True), w, h, xl, yl, mxl, myl, ud, uw)
    assert got.tobytes() == want.tobytes()


@pytest.mark.parametrize("size", [(2, 2), (2, 33), (32, 32), (33, 65), (66, 31), (129, 97)])
@pytest.mark.parametrize("fmt", [0, 1, 2, "flow"])
@pytest.mark.parametrize("above_first", [False, True])
def test_hole_fill_at_the_ends_of_its_tiles(dev, size, fmt, above_first):
    """Images of one tile and a pixel more or less: sparse holes, all holes and tiles without one, and for floats
    zeros of both signs, infinities and NaNs (signalling ones too) in and beside the holes."""
    w, h = size
    n = w * h
    rng = np.random.RandomState(w + 7 * h)
    channels = 2 if fmt == "flow" else 4
    if fmt in (0, 1):
        img = rng.randint(0, 256 if fmt == 0 else 65536, n * channels).astype(tw.DTYPES[fmt])
    else:
        img = (rng.random_sample(n * channels) * 2 - 1).astype(np.float32)
        img[rng.randint(0, img.size, max(img.size // 9, 1))] = 0.0
        img[rng.randint(0, img.size, max(img.size // 9, 1))] = -0.0
    masks = [(rng.random_sample(n) < p).astype(np.uint8) for p in (0.02, 0.5)] + [np.ones(n, np.uint8)]
    masks.append((np.arange(n) % w < 3).astype(np.uint8))
    for k, mask in enumerate(masks):
        src = img.copy()
        if fmt in (2, "flow") and k % 2:
            src.view(np.uint32)[rng.randint(0, src.size, 3)] = [0x7fc00123, 0xffc04567, 0x7f800001]
            src[rng.randint(0, src.size, 2)] = [np.inf, -np.inf]
        if fmt == "flow":
            got = dev.fill_flow_holes(src.copy(), w, h, mask, taps_above_first=above_first)
            want = O.fill_flow_holes(src.copy(), w, h, mask, 1, above_first)
        else:
            got = dev.fill_holes(src.copy(), w, h, fmt, mask, taps_above_first=above_first)
            want = O.fill_holes(src.copy(), w, h, fmt, mask, 1, above_first)
        assert same(got, want)


@pytest.mark.parametrize("pyramid", [True, False])
@pytest.mark.parametrize("case", ["payload", "rows", "far", "whole"])
def test_forward_warp_where_its_plain_arithmetic_ends(dev, pyramid, case):
    """Samples around and above 10^6, rows closer than 10^-6, corners far outside, vertices on pixels."""
    w, h = 37, 29
    rng = np.random.RandomState(2)
    src = rng.random_sample(w * h * 4).astype(np.float32)
    flow = rng.uniform(-2, 2, (h, w, 2)).astype(np.float32)
    if case == "payload":
        src[rng.randint(0, src.size, 200)] = rng.choice(np.float32([9.99e5, 1e6, -1e6, 3e8, -2e30, 3e38]), 200)
    elif case == "rows":
        flow[..., 1] = np.where(rng.random_sample((h, w)) < 0.5, 0.0, rng.uniform(-3e-6, 3e-6, (h, w)))
        flow[::5, :, 1] -= 1.0
    elif case == "far":
        at = rng.randint(0, h, 12), rng.randint(0, w, 12)
        flow[at] = rng.choice(np.float32([-3e5, 9.9e5, 2e6, -4e7]), (12, 2))
    else:
        flow = np.round(flow)
    flow = flow.astype(np.float32).reshape(-1)
    try:
        want = O.forward_warp(src, w, h, 2, flow, w, h, 1.0, pyramid, True)
    except ValueError:
        with pytest.raises(tw.Unsupported):
            dev.forward_warp(src, w, h, 2, flow, (w, h), 1.0, pyramid, True)
        return
    got = dev.forward_warp(src, w, h, 2, flow, (w, h), 1.0, pyramid, True)
    assert same(got[0], want[0]) and same(got[1], want[1])


@pytest.mark.parametrize("w,h,fw,fh", [(2, 2, 2, 2), (33, 9, 17, 5), (31, 33, 31, 33), (65, 8, 22, 3), (20, 41, 61, 83)])
@pytest.mark.parametrize("smooth", [False, True])
def test_adjoint_at_the_ends_of_its_columns(dev, w, h, fw, fh, smooth):
    """Rows and columns that end inside a warp's strip, vectors that share corners (smooth) and that do not, on
    and beyond the border: within 1e-3 of the double precision gradients (float32 sums of at most a few dozen
    terms in any order), as in test_gpu_adjoint."""
    import torch

    from twixtor_b200 import adjoint
    import os
    import sys
    sys.path.insert(0, os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "oracle"))
    import adjoint_fp64 as A
    n, wa = 2, 0.35
    rng = np.random.RandomState(w * 3 + fh)
    a, b, g = (rng.rand(n, h, w, 4).astype(np.float32) for _ in range(3))
    fab, fba = ((np.full((n, fh, fw, 2), 1.25) + rng.uniform(-0.01, 0.01, (n, fh, fw, 2)) if smooth
                 else rng.uniform(-9, 9, (n, fh, fw, 2))).astype(np.float32) for _ in range(2))
    host = (a, b, fab, fba)
    xs = [torch.from_numpy(x).cuda().requires_grad_(True) for x in host]
    out = adjoint.warp_blend(*xs, wa, dev)
    out.backward(torch.from_numpy(g).cuda())
    for i in range(n):
        _, _, *refs = A.warp_blend_grads(*[x[i].reshape(-1) for x in host], w, h, fw, fh, wa, pos32=True,
                                         grad_out=g[i].reshape(-1))
        for x, ref in zip(xs, refs):
            got = x.grad[i].cpu().numpy().astype(np.float64)
            assert np.linalg.norm(got.reshape(-1) - np.asarray(ref).reshape(-1)) <= 1e-3 * max(np.linalg.norm(ref), 1e-6)


@pytest.mark.parametrize("value", [0x7f800000, 0xff800000, 0x7fc00000, 0x7fc00001], ids=hex)
@pytest.mark.parametrize("push", [(500.0, 0.25), (0.25, -500.0), (-500.0, 500.0)])
@pytest.mark.parametrize("where", ["gradient", "frame"])
def test_adjoint_of_clamped_positions_with_values_that_are_not_finite(dev, value, push, where):
    """An axis on which every position is clamped has no gradient: exactly 0, also where the output's gradient or
    the frames hold infinities and NaNs (of any payload); the other axis has NaNs then."""
    import torch

    from twixtor_b200 import adjoint
    w, h, fw, fh = 40, 37, 20, 19
    rng = np.random.RandomState(4)
    a, b, g = (rng.rand(1, h, w, 4).astype(np.float32) for _ in range(3))
    for x in (g,) if where == "gradient" else (a, b):
        x.reshape(-1).view(np.uint32)[rng.randint(0, x.size, x.size // 4)] = value
    fab, fba = (np.tile(np.array(push, np.float32), (1, fh, fw, 1)) for _ in range(2))
    xs = [torch.from_numpy(x).cuda().requires_grad_(True) for x in (a, b, fab, fba)]
    adjoint.warp_blend(*xs, 0.35, dev).backward(torch.from_numpy(g).cuda())
    for f in xs[2:]:
        for axis in range(2):
            if abs(push[axis]) > 1.0:
                assert (f.grad[..., axis] == 0.0).all()
            else:
                assert torch.isnan(f.grad[..., axis]).any()


@pytest.mark.parametrize("size", [(3, 3), (3, 40), (33, 4), (5, 5), (32, 32), (33, 33), (65, 34), (97, 66)])
@pytest.mark.parametrize("fmt", [0, 2])
@pytest.mark.parametrize("density", [0.02, 0.3, 0.7])
def test_sharpening_mask_at_the_ends_of_its_tiles(dev, size, fmt, density):
    """Weighted Blend compositions of frames that differ in scattered blocks, single pixels and along the border:
    the difference mask's clean-up across tiles of 32 x 32, with borders on, before and after a tile's edge."""
    w, h = size
    rng = np.random.RandomState(w + 5 * h)
    top = 255 if fmt == 0 else 1.0
    a = rng.random_sample((h, w, 4)) * top * 0.3
    a[..., 0] = top
    b = a.copy()
    on = rng.random_sample((h, w)) < density
    on |= np.kron(rng.random_sample((h // 4 + 1, w // 4 + 1)) < density / 2, np.ones((4, 4)))[:h, :w] > 0
    on[:, 0] |= rng.random_sample(h) < 0.5
    on[-1] |= rng.random_sample(w) < 0.5
    b[on, 1:] = top
    a, b = (x.reshape(-1).astype(tw.DTYPES[fmt]) for x in (a, b))
    flows = [rng.uniform(-1.5, 1.5, w * h * 2).astype(np.float32) for _ in range(2)]
    sel = tw.Selection(wa=np.float32(0.4), interp=2)
    cs = tw.EngineSettings(taps_above_first=True)
    got = dev.compose_vectors(cs, sel, a, b, w, h, fmt, flows[0], flows[1], (w, h))
    assert same(got, O.compose_vectors3(a, b, w, h, fmt, flows[0], flows[1], w, h, sel, cs))


def test_algorithmic_bytes_of_a_level(dev):
    """The bytes a level's kernels cannot do without, as the profiler counts them (what the layout adds, such as the
    determinant beside the tensor, is not among them): per pixel 44 for the level's start, 36 for an iteration, 60
    where it makes the next one's B, and 32 for the B after the finest level's block matching."""
    w, h = 33, 65  # one level above the coarse ones, in 16 x 16 tiles
    rng = np.random.RandomState(1)
    x, y = (rng.randint(0, 256, w * h * 4).astype(np.uint8) for _ in range(2))
    s = tw.FlowSettings(quality=5)
    for kernel, launches, per_pixel in [("k_level_init_16x16", 1, 44), ("k_level_iter_16x16", 3, 60 + 36 + 36),
                                        ("k_calc_b_pitched", 1, 32)]:
        dev.profile_begin(kernel)
        dev.solve(x, y, w, h, 0, s)
        _, n, b = dev.profile_end()
        assert (n, b) == (launches, per_pixel * w * h)
