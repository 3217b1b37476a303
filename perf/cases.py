"""The work a program has the library do, as cases that a benchmark can time: each listed case is one
call (or one training step) through the public entry points of ``twixtor_b200``, over the sizes,
depths and options of the effects it serves.

A case is a dict of plain values with a ``kind``:

* ``frame``    one output frame of `retime` from host buffers (``Device.retime_frame``)
* ``clip``     a clip of `retime`, in device memory or host memory (``retime_clip_device``, ``retime_clip``)
* ``batch``    several float clips of uneven size in one call (``retime_batch_device``)
* ``solve``    the flows of an image pair, the estimator seam of the engine (``Device.solve_pair``)
* ``vectors``  Create Vectors over a clip in host memory (``create_vectors_clip``)
* ``layers``   retime-fgbg with FG matte layers over a clip in host memory (``retime_layers_clip``)
* ``vecin``    Vectors In over clips in device memory (``vectors_in_clip_device``)
* ``adjoint``  the gradients of warp + blend, the fused L1 step or a backward pass of autograd

Depth codes: 0 is 8 bpc, 1 is 16 bpc, 2 is float. The clips are a value noise background that moves
by a sub-pixel step per frame and textured ellipses on top that move on their own.
"""
import math

import torch

import twixtor_b200 as tw
from twixtor_b200 import adjoint

DTYPE = {0: torch.uint8, 1: torch.uint16, 2: torch.float32}
BYTES = {0: 4, 1: 8, 2: 16}  # of one pixel
BATCH_SIZES = ((1280, 720), (1440, 1080), (1920, 1080), (3840, 2160))

_DEV = None


def _device():
    """The process's handle, opened once as a program does, on torch's stream."""
    global _DEV
    if _DEV is None:
        _DEV = tw.Device(0)
    _DEV.set_stream(torch.cuda.current_stream().cuda_stream)
    return _DEV


def listed():
    return [
        # one in-between frame of a thumbnail sized clip: the smallest call, all latency
        dict(name="frame 64x48 u8", kind="frame", w=64, h=48, fmt=0, interp=1, warp=0, speed=40.0),
        # the interactive preview: a short small clip at half speed, frames in host memory
        dict(name="clip 160x96 u8 host", kind="clip", w=160, h=96, fmt=0, interp=1, warp=0, speed=50.0, nout=47, host=True),
        # the usual render: HD footage at 40 %, resident on the device, ten output frames
        dict(name="clip 1080p u8", kind="clip", w=1920, h=1080, fmt=0, interp=1, warp=0, speed=40.0, nout=10, host=False),
        # Smart Blend with its hole fill on 16 bpc footage of a ragged size
        dict(name="smart blend 1279x717 u16", kind="clip", w=1279, h=717, fmt=1, interp=1, warp=1, speed=40.0, nout=5,
             host=False),
        # Weighted Blend of float footage at standard definition
        dict(name="weighted 720x486 f32", kind="clip", w=720, h=486, fmt=2, interp=2, warp=0, speed=30.0, nout=10,
             host=False),
        # a render queue: clips of uneven size in one call, float, keyed speed (the largest case)
        dict(name="batch 720p-2160p f32", kind="batch", scale=1.0, njobs=4, nout=4),
        # the estimator alone behind the engine's stage seam, at full resolution on an odd size
        dict(name="solve pair 853x481 f32 full", kind="solve", w=853, h=481, fmt=2, quality=5),
        # motion vectors of HD 16 bpc footage, frame to previous frame
        dict(name="create vectors 1080p u16", kind="vectors", w=1920, h=1080, fmt=1, full=False, npairs=6),
        # three FG matte layers over HD footage
        dict(name="fgbg 1080p u8 3 layers", kind="layers", w=1920, h=1080, fmt=0, nfg=3, warp=0, nout=3),
        # the defaults of Vectors In (Warping Forward) with holes in both vector layers
        dict(name="vectors in 1080p u8", kind="vecin", w=1920, h=1080, fmt=0, warping=2, both=True, nout=4),
        # photometric flow refinement: loss and gradients of a batch of frame triples
        dict(name="adjoint L1 1280x720 x16", kind="adjoint", w=1280, h=720, batch=16, l1=True),
        # a training step of two small ragged images through autograd, forward and backward
        dict(name="adjoint autograd 333x217 x2", kind="adjoint", w=333, h=217, batch=2, l1=False),
    ]


def _size(rng, lo, hi, aspects=(4 / 3, 16 / 9, 1.0, 1.85, 0.75)):
    """A width spread over its logarithm and a height of a usual aspect, odd sizes among them."""
    w = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    h = max(int(round(w / rng.choice(aspects))), 24)
    return w, min(h, w) if w > 1500 else h


def draw(rng):
    kind = rng.choice(["frame", "clip", "clip", "clip", "batch", "solve", "vectors", "layers", "vecin", "adjoint"])
    fmt = rng.choice([0, 0, 1, 2])
    if kind == "frame":
        w, h = _size(rng, 48, 1920)
        return dict(kind=kind, w=w, h=h, fmt=fmt, interp=rng.choice([0, 1, 1]), warp=rng.choice([0, 0, 1]),
                    speed=rng.choice([25.0, 40.0, 60.0]))
    if kind == "clip":
        w, h = _size(rng, 64, 2560)
        return dict(kind=kind, w=w, h=h, fmt=fmt, interp=rng.choice([0, 1, 1, 2]), warp=rng.choice([0, 0, 0, 1]),
                    speed=rng.choice([30.0, 40.0, 50.0, 70.0]), nout=rng.randint(2, 8), host=rng.random() < 0.4)
    if kind == "batch":
        return dict(kind=kind, scale=round(rng.uniform(0.2, 0.95), 3), njobs=rng.randint(2, 4), nout=rng.randint(2, 4))
    if kind == "solve":
        w, h = _size(rng, 64, 1920)
        return dict(kind=kind, w=w, h=h, fmt=fmt, quality=rng.choice([3, 4, 4, 5]))
    if kind == "vectors":
        w, h = _size(rng, 96, 1920)
        return dict(kind=kind, w=w, h=h, fmt=fmt, full=rng.random() < 0.3, npairs=rng.randint(2, 6))
    if kind == "layers":
        w, h = _size(rng, 96, 1920)
        return dict(kind=kind, w=w, h=h, fmt=rng.choice([0, 0, 1]), nfg=rng.randint(1, 3), warp=rng.choice([0, 0, 1]),
                    nout=rng.randint(2, 3))
    if kind == "vecin":
        w, h = _size(rng, 96, 1920)
        return dict(kind=kind, w=w, h=h, fmt=fmt, warping=rng.choice([1, 2, 2]), both=rng.random() < 0.7,
                    nout=rng.randint(2, 4))
    w, h = _size(rng, 64, 1280)
    return dict(kind=kind, w=w, h=h, batch=rng.randint(1, 8), l1=rng.random() < 0.5)


# ---- inputs ----------------------------------------------------------------------------------------

def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed) * 7919 + 17)


def _uniform(g, n, lo, hi):
    return [float(v) for v in (torch.rand(n, generator=g, device="cuda") * (hi - lo) + lo).tolist()]


def _noise(g, w, h):
    """Three octaves of value noise around 0.5."""
    v = 0.0
    for cell, amp in ((24, 1.0), (10, 0.55), (4, 0.3)):
        lat = torch.randn((1, 1, h // cell + 4, w // cell + 4), generator=g, device="cuda")
        v = v + amp * torch.nn.functional.interpolate(lat, size=(h, w), mode="bicubic", align_corners=False)[0, 0]
    return (0.5 + 0.157 * (v - v.mean()) / v.std()).clamp(0.0, 1.0)


def _shift(t, dx, dy):
    """The (periodic) plane moved by a sub-pixel step, bilinear."""
    ix, iy = math.floor(dx), math.floor(dy)
    fx, fy = dx - ix, dy - iy
    r = lambda ox, oy: torch.roll(t, shifts=(iy + oy, ix + ox), dims=(0, 1))  # noqa: E731
    return (r(0, 0) * (1 - fx) + r(1, 0) * fx) * (1 - fy) + (r(0, 1) * (1 - fx) + r(1, 1) * fx) * fy


def _wire(r, g, b, a, fmt):
    """One wire frame: interleaved RGBA bytes or words, or float planes G, B, R, A."""
    if fmt == 2:
        return torch.stack([g, b, r, a]).to(torch.float32).reshape(-1)
    top = 255.0 if fmt == 0 else 65535.0
    px = torch.stack([r, g, b, a], -1).clamp(0, 1).mul(top).round()
    return px.to(torch.uint8).reshape(-1) if fmt == 0 else px.to(torch.int32).to(torch.uint16).reshape(-1)


def _scene(g, w, h, n, fmt, nell=3, soft_alpha=False):
    """``n`` wire frames of the moving scene, and the ellipses' coverage per frame (top one first)."""
    step = max(0.5, min(6.0, w / 320.0))  # pixels a frame, in proportion to the frame
    bg = _noise(g, w, h)
    vx, vy = _uniform(g, 2, -step, step)
    y, x = torch.meshgrid(torch.arange(h, device="cuda", dtype=torch.float32),
                          torch.arange(w, device="cuda", dtype=torch.float32), indexing="ij")
    ells = []
    for _ in range(nell):
        ax, ay = _uniform(g, 2, 0.08 * min(w, h), 0.25 * min(w, h))
        cx, cy = _uniform(g, 1, 0.25 * w, 0.75 * w)[0], _uniform(g, 1, 0.25 * h, 0.75 * h)[0]
        ux, uy = _uniform(g, 2, -1.5 * step, 1.5 * step)
        ells.append((ax, ay, cx, cy, ux, uy, _noise(g, w, h)))
    alpha = 0.4 + 0.6 * _noise(g, w, h) if soft_alpha else torch.ones_like(bg)
    frames, cover = [], [[] for _ in range(nell)]
    for t in range(n):
        lum = _shift(bg, vx * t, vy * t)
        r, gg, b = lum, 0.85 * lum + 0.08, 1.0 - 0.6 * lum
        for k in reversed(range(nell)):
            ax, ay, cx, cy, ux, uy, tex = ells[k]
            m = ((x - cx - ux * t) / ax) ** 2 + ((y - cy - uy * t) / ay) ** 2 <= 1.0
            tl = _shift(tex, ux * t, uy * t)
            r, gg, b = torch.where(m, tl, r), torch.where(m, 0.5 * tl + 0.3, gg), torch.where(m, 1.0 - tl, b)
            cover[k].append(m)
        frames.append(_wire(r, gg, b, alpha, fmt))
    return torch.cat(frames), cover, (vx, vy)


def _pinned(t):
    """A page-locked copy and its numpy view."""
    p = torch.empty(t.shape, dtype=t.dtype, pin_memory=True)
    p.copy_(t)
    return p, p.numpy()


def _selections(case, nout, **kw):
    tp = tw.TimeParams(speed_percent=case.get("speed", 40.0), frame_interp=case.get("interp", 1) + 1, **kw)
    return [tw.select(tp, n, case["w"], case["h"]) for n in range(nout)]


def _vector_field(g, w, h, n, fmt, velocity, md):
    """``n`` frames of a vector layer: the displacement with a slow ripple, discs of alpha 0 in it."""
    y, x = torch.meshgrid(torch.arange(h, device="cuda", dtype=torch.float32),
                          torch.arange(w, device="cuda", dtype=torch.float32), indexing="ij")
    rad = 0.037 * min(w, h)
    out = []
    for t in range(n):
        u = velocity[0] + 0.1 * torch.sin(x / 97.0 + t)
        v = velocity[1] + 0.1 * torch.cos(y / 61.0 - t)
        a = torch.ones_like(u)
        for cx, cy in zip(_uniform(g, 12, 0, w), _uniform(g, 12, 0, h)):
            a[(x - cx) ** 2 + (y - cy) ** 2 < rad * rad] = 0.0
        if fmt == 2:
            out.append(_wire((u / md + 1) / 2, (v / md + 1) / 2, torch.zeros_like(u), a, fmt))
        else:
            half, top = (127.0, 255.0) if fmt == 0 else (32767.0, 65535.0)
            code = lambda c: torch.floor((c / md + 1) * half + 0.5) / top  # noqa: E731
            out.append(_wire(code(u), code(v), torch.zeros_like(u), a, fmt))
    return torch.cat(out)


def prepare(case, seed):
    g = _gen(seed)
    kind = case["kind"]
    s = dict(kind=kind, case=case)
    if kind == "batch":
        tp = tw.TimeParams(keys=[(0.0, 100.0, 1), (12.0, 25.0, 1), (24.0, 100.0, 1)])
        s["jobs"], s["keep"], s["outs"] = [], [], []
        for bw, bh in BATCH_SIZES[:case["njobs"]]:
            w, h = max(int(bw * case["scale"]), 32), max(int(bh * case["scale"]), 32)
            sels = [tw.select(tp, n, w, h) for n in range(10, 10 + case["nout"])]
            first = min(min(x.a, x.b) for x in sels)
            n = max(max(x.a, x.b) for x in sels) - first + 1
            frames, _, _ = _scene(g, w, h, n, 2)
            out = torch.empty(case["nout"] * w * h * 4, dtype=torch.float32, device="cuda")
            s["keep"].append(frames)
            s["outs"].append(out)
            s["jobs"].append(dict(settings=tw.RetimeSettings(), frames=frames.data_ptr(), nframes=n,
                                  sels=tw.rebase(sels, first, first + n), width=w, height=h, fmt=2, out=out.data_ptr()))
        s["dev"] = _device()
        return s
    w, h = case["w"], case["h"]
    if kind == "adjoint":
        n, fw, fh = case["batch"], max(w // 2, 2), max(h // 2, 2)
        # a sequence around the middle frame, and smooth flows of up to about ten pixels
        tex = [torch.stack([_noise(g, w, h) for _ in range(3)] + [torch.ones((h, w), device="cuda")], -1) for _ in range(n)]
        d = torch.stack([torch.stack([(_noise(g, max(fw // 6, 8), max(fh // 6, 8)) - 0.5) for _ in range(2)]) for _ in range(n)])
        d = torch.nn.functional.interpolate(d * min(10.0, w / 64.0), size=(fh, fw), mode="bicubic", align_corners=True)
        vx, vy = _uniform(g, 2, -2.0, 2.0)
        a = [torch.stack([_shift(t[..., c], vx, vy) for c in range(4)], -1) for t in tex]
        b = [torch.stack([_shift(t[..., c], -vx, -vy) for c in range(4)], -1) for t in tex]
        s["a"], s["b"], s["m"] = (torch.stack(v).contiguous() for v in (a, b, tex))
        d = d.permute(0, 2, 3, 1).contiguous()
        s["f_ab"], s["f_ba"] = d, (-d + 0.01 * torch.randn(d.shape, generator=g, device="cuda")).contiguous()
        if not case["l1"]:
            s["g"] = torch.randn(s["a"].shape, generator=g, device="cuda")
            for k in ("a", "b", "f_ab", "f_ba"):
                s[k].requires_grad_(True)
        s["dev"] = _device()
        return s
    fmt = case["fmt"]
    fs = w * h * 4
    if kind == "frame":
        sel = next(x for x in _selections(case, 8) if not x.exact)
        frames, _, _ = _scene(g, w, h, 2, fmt)
        s["keep"] = _pinned(frames), _pinned(torch.empty(fs, dtype=DTYPE[fmt]))
        clip, s["out"] = s["keep"][0][1], s["keep"][1][1]
        s["args"] = (tw.RetimeSettings(compose=tw.EngineSettings(warp_mode=case["warp"])), sel, clip[:fs], clip[fs:], w, h, fmt)
    elif kind == "clip":
        sels = _selections(case, case["nout"])
        n = max(max(x.a, x.b) for x in sels) + 1
        frames, _, _ = _scene(g, w, h, n, fmt, soft_alpha=fmt == 1)
        out = torch.empty(case["nout"] * fs, dtype=DTYPE[fmt], device="cuda")
        settings = tw.RetimeSettings(compose=tw.EngineSettings(warp_mode=case["warp"]))
        if case["host"]:
            s["keep"] = _pinned(frames), _pinned(out)
            s["args"] = (settings, s["keep"][0][1], n, sels, w, h, fmt)
            s["out"] = s["keep"][1][1]
        else:
            s["keep"] = frames
            s["args"] = (settings, frames.data_ptr(), n, sels, w, h, fmt, out.data_ptr())
            s["out"] = out.view(torch.int16) if fmt == 1 else out  # torch indexes no unsigned words on the GPU
    elif kind == "solve":
        frames, _, _ = _scene(g, w, h, 2, fmt)
        wire = frames.cpu().numpy()
        dev = _device()
        a, b = (dev.from_frame(wire[k * fs:(k + 1) * fs], w, h, fmt) for k in range(2))
        s["args"] = (a, b, w, h, fmt, tw.FlowSettings(quality=case["quality"]))
    elif kind == "vectors":
        n = case["npairs"] + 1
        frames, _, _ = _scene(g, w, h, n, fmt)
        s["keep"] = _pinned(frames), _pinned(torch.empty(case["npairs"] * fs, dtype=DTYPE[fmt]))
        s["out"] = s["keep"][1][1]
        pairs = [tw.vectors_pair(k, 1) for k in range(1, n)]
        s["args"] = (tw.vectors_settings(vector_resolution=2 if case["full"] else 1), s["keep"][0][1], n, pairs, w, h, fmt)
    elif kind == "layers":
        sels = _selections(case, case["nout"] + 1)[1:]
        n = max(max(x.a, x.b) for x in sels) + 1
        frames, cover, _ = _scene(g, w, h, n, fmt, nell=case["nfg"])
        one = torch.ones((h, w), device="cuda")
        mattes = [torch.cat([_wire(m.float(), 0 * one, 0 * one, one, fmt) for m in c]) for c in cover]
        s["keep"] = [_pinned(t) for t in [frames] + mattes] + [_pinned(torch.empty(case["nout"] * fs, dtype=DTYPE[fmt]))]
        host = [k[1] for k in s["keep"]]
        s["out"] = host[-1]
        s["args"] = (tw.RetimeSettings(compose=tw.EngineSettings(warp_mode=case["warp"], gouraud=True)), host[0], n, host[1:-1],
                     [1] * case["nfg"], [tw.percent_param(70.0)] * (case["nfg"] + 1), sels, w, h, fmt)
    elif kind == "vecin":
        tp = tw.TimeParams(fps=(30, 1), speed_percent=40.0)
        both = [tw.select_vectors_in(tp, k, w, h, has_prev=case["both"]) for k in range(case["nout"])]
        n = max(max(v.a, v.b) for _, v in both) + 1
        md = 32.0
        frames, _, vel = _scene(g, w, h, n, fmt)
        nxt = _vector_field(g, w, h, n, fmt, vel, md)
        prv = _vector_field(g, w, h, n, fmt, (-vel[0], -vel[1]), md)
        out = torch.empty(case["nout"] * fs, dtype=DTYPE[fmt], device="cuda")
        s["keep"], s["out"] = (frames, nxt, prv), out.view(torch.int16) if fmt == 1 else out
        s["args"] = (tw.vectors_in_settings(warping=case["warping"]), frames.data_ptr(), n, nxt.data_ptr(), n,
                     prv.data_ptr() if case["both"] else 0, n if case["both"] else 0, [x for x, _ in both],
                     [v for _, v in both], md, w, h, fmt, out.data_ptr())
    s["dev"] = _device()
    return s


# ---- one pass --------------------------------------------------------------------------------------

def run(s):
    dev, kind = s["dev"], s["kind"]
    if kind == "batch":
        dev.retime_batch_device(s["jobs"])
        return s["outs"]
    if kind == "adjoint":
        if s["case"]["l1"]:
            return adjoint.l1_loss_and_grads(dev, s["a"], s["b"], s["f_ab"], s["f_ba"], s["m"], 0.5)
        leaves = [s[k] for k in ("a", "b", "f_ab", "f_ba")]
        for t in leaves:
            t.grad = None
        out = adjoint.warp_blend(*leaves, 0.4, dev)
        out.backward(s["g"])
        return [out.detach()] + [t.grad for t in leaves]
    if kind == "solve":
        f_ab, f_ba, _ = dev.solve_pair(*s["args"])
        return f_ab, f_ba
    if kind == "frame":
        dev.retime_frame(*s["args"], out=s["out"])
    elif kind == "clip" and s["case"]["host"]:
        dev.retime_clip(*s["args"], out=s["out"])
    elif kind == "clip":
        dev.retime_clip_device(*s["args"])
    elif kind == "vectors":
        dev.create_vectors_clip(*s["args"], out=s["out"])
    elif kind == "layers":
        dev.retime_layers_clip(*s["args"], out=s["out"])
    elif kind == "vecin":
        dev.vectors_in_clip_device(*s["args"])
    return s["out"]


# ---- what a pass cannot do without -----------------------------------------------------------------

# Operations per pixel of a solver level: the two band pyramids (30), gradient and tensor with its
# blur (143), three iterations (the B step 25, its blur 88, the displacement 20, the flow's blur 64),
# four sweeps of two block costs (832), the range check and the upsample (40). A pyramid's levels
# hold 4/3 of its finest one. The composition of a pixel: two warps of four channels and the blend.
SOLVE_OPS, COMPOSE_OPS = 1640.0, 150.0


def _solve_ops(w, h, quality, solves):
    fw, fh, _ = tw.flow_geometry(tw.FlowSettings(quality=quality), w, h)
    return solves * SOLVE_OPS * fw * fh * 4.0 / 3.0


def _clip_work(sels, w, h, px, solves=2, layers=1):
    used = {f for x in sels for f in ((x.a,) if x.exact else (x.a, x.b))}
    moved = [x for x in sels if not x.exact]
    flops = len(moved) * layers * (_solve_ops(w, h, 4, solves) + COMPOSE_OPS * w * h)
    return px * w * h * (len(used) + len(sels)), flops


def work(case):
    kind = case["kind"]
    if kind == "batch":
        tp = tw.TimeParams(keys=[(0.0, 100.0, 1), (12.0, 25.0, 1), (24.0, 100.0, 1)])
        b = f = 0.0
        for bw, bh in BATCH_SIZES[:case["njobs"]]:
            w, h = max(int(bw * case["scale"]), 32), max(int(bh * case["scale"]), 32)
            x, y = _clip_work([tw.select(tp, n, w, h) for n in range(10, 10 + case["nout"])], w, h, 16)
            b, f = b + x, f + y
        return {"bytes": b, "flops": f}
    w, h = case["w"], case["h"]
    if kind == "adjoint":
        # both frames, the target (or the output's gradient, and the output) and the frames' gradients;
        # the two flows and their gradients at half size; about 350 operations a pixel
        n = case["batch"]
        return {"bytes": n * (w * h * (80.0 if case["l1"] else 96.0) + (w // 2) * (h // 2) * 32.0), "flops": n * w * h * 350.0}
    px = BYTES[case["fmt"]]
    if kind == "solve":
        fw, fh, _ = tw.flow_geometry(tw.FlowSettings(quality=case["quality"]), w, h)
        return {"bytes": 2.0 * px * w * h + 16.0 * fw * fh, "flops": _solve_ops(w, h, case["quality"], 2)}
    if kind == "vectors":
        n = case["npairs"]
        return {"bytes": px * w * h * (2.0 * n + 1), "flops": n * _solve_ops(w, h, 5 if case["full"] else 4, 1)}
    if kind == "vecin":
        n = case["nout"]
        return {"bytes": px * w * h * (3.0 * (int(0.4 * (n - 1)) + 2) + n), "flops": n * w * h * 600.0}
    if kind == "frame":
        return {"bytes": 3.0 * px * w * h,
                "flops": _solve_ops(w, h, 4, 1 if case["interp"] == 0 else 2) + COMPOSE_OPS * w * h}
    layers = case.get("nfg", 0) + 1
    sels = _selections(case, case["nout"] + 1)[1:] if kind == "layers" else _selections(case, case["nout"])
    b, f = _clip_work(sels, w, h, px, 1 if case.get("interp") == 0 else 2, layers)
    return {"bytes": b * layers if kind == "layers" else b, "flops": f}


# ---- the same in 64 bits ---------------------------------------------------------------------------

def _cell(x, n):
    i = torch.floor(x)
    f = x - i
    i = i.long()
    f = torch.where(i >= n - 1, torch.ones_like(f), f)
    return i.clamp(0, n - 2), f


def _bilinear(img, x, y):
    h, w = img.shape[:2]
    ix, fx = _cell(x, w)
    iy, fy = _cell(y, h)
    fx, fy = fx[..., None], fy[..., None]
    top = img[iy, ix] + (img[iy, ix + 1] - img[iy, ix]) * fx
    bot = img[iy + 1, ix] + (img[iy + 1, ix + 1] - img[iy + 1, ix]) * fx
    return top * (1 - fy) + bot * fy


def _warp64(img, flow, amount):
    h, w = img.shape[:2]
    fh, fw = flow.shape[:2]
    y, x = torch.meshgrid(torch.arange(h, device="cuda", dtype=torch.float64),
                          torch.arange(w, device="cuda", dtype=torch.float64), indexing="ij")
    rx, ry = (fw - 1) / (w - 1), (fh - 1) / (h - 1)
    uv = _bilinear(flow, x * rx, y * ry)
    return _bilinear(img, (x + uv[..., 0] * (amount / rx)).clamp(0, w - 1), (y + uv[..., 1] * (amount / ry)).clamp(0, h - 1))


def exact(case, seed):
    """The gradients of warp + blend by plain autograd in double precision. The other outputs are whole
    values, or come out of the estimator, whose block matching decides between vectors by comparing
    costs, step after step along every line: in 64 bits it takes other decisions, and minutes."""
    if case["kind"] != "adjoint":
        return None
    s = prepare(case, seed)
    res = [[], [], [], [], []]
    for k in range(case["batch"]):
        a, b, fab, fba = (s[n][k].detach().double().requires_grad_(True) for n in ("a", "b", "f_ab", "f_ba"))
        wa = 0.5 if case["l1"] else float(torch.tensor(0.4, dtype=torch.float32))
        ta, tb = _warp64(a, fba, 1.0 - wa), _warp64(b, fab, wa)
        out = ta + (tb - ta) * (1.0 - wa)
        if case["l1"]:
            first = (out - s["m"][k].double()).abs().sum()
            first.backward()
        else:
            first = out
            out.backward(s["g"][k].double())
        for r, t in zip(res, (first.detach(), a.grad, b.grad, fab.grad, fba.grad)):
            r.append(t)
    res = [torch.stack(r) for r in res]
    return tuple(res) if case["l1"] else res
