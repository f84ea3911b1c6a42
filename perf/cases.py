"""The calls a user of this framework makes, as measurable cases.

Each case is one pass through a public entry point on inputs that are already on the GPU: a frame
through a stitcher's ``process``, a captured multi-stream job through ``Batch.launch``, a burst of
requests through ``StitchServer``, a frame pair through ``Stabilizer.run`` and an image pair through
``hmp_blend2_noalloc``. Rigs are N pinhole cameras on a horizontal arc, projected onto a cylindrical
canvas as Hugin exports them (CV_16U nearest-neighbour tables, 65535 where nothing maps); seams are
random walks inside the overlaps; frames are camera frames (smooth content with sensor noise, alpha
255). Rigs, seams and frames all come from the seed.
"""
import ctypes as C
import math
import os
import sys

import numpy as np
import torch
import torch.nn.functional as F

sys.path.insert(0, os.path.join(os.getcwd(), "hm-cupano_gb300"))
import hmpano  # noqa: E402
from hmpano import _lib, pano  # noqa: E402

HFOV = math.radians(65.0)


def stitch(name=None, n=2, kind=2, w=2200, h=800, levels=6, pixels="rgba", storage="f32", filter="refbox", batch=1,
           overlap=0.14, minimize=True):
    c = dict(do="stitch", n=n, kind=kind, w=w, h=h, levels=levels, pixels=pixels, storage=storage, filter=filter,
             batch=batch, overlap=overlap, minimize=minimize)
    return dict(c, name=name) if name else c


def listed():
    return [
        # Two 720p cameras onto a 2200x800 canvas, hard seam: the smallest configuration, one launch.
        stitch("hard2_2200x800", levels=0),
        # A live preview: small two-camera canvas of odd size, a shallow blend, two frames a call.
        stitch("blend2_2203x797_l3_b2", w=2203, h=797, levels=3, batch=2),
        # The production frame: two 5K cameras onto 8500x3300, six levels.
        stitch("blend2_8500x3300_l6", w=8500, h=3300, levels=6, overlap=0.07),
        # The same frame through the 5-tap filter.
        stitch("binomial2_8500x3300_l6", w=8500, h=3300, levels=6, overlap=0.07, filter="binomial5"),
        # The same frame from RGB sources (decoders without an alpha plane).
        stitch("rgb2_8500x3300_l6", w=8500, h=3300, levels=6, overlap=0.07, pixels="rgb"),
        # Three cameras, half-precision pyramid storage (the batched job's other stream).
        stitch("blend3_6000x1800_l6_f16", n=3, kind=3, w=6000, h=1800, levels=6, overlap=0.2, storage="f16"),
        # Eight cameras, the widest rig.
        stitch("blend8_9000x2400_l6", n=8, kind=1, w=9000, h=2400, levels=6, overlap=0.25),
        # Five RGB cameras on an odd-sized canvas.
        stitch("rgb5_4999x1201_l5", n=5, kind=1, w=4999, h=1201, levels=5, overlap=0.22, pixels="rgb"),
        # Four streams of eight frames (two two-camera, two three-camera), one captured job.
        dict(name="batch_4streams_f16", do="batch", w2=4250, h2=1650, w3=3000, h3=900, frames=8, per_call=4, levels=6),
        # A burst of requests over three resident configurations.
        dict(name="serve_24_requests", do="serve", w=2200, h=800, w3=3000, h3=900, requests=24, slots=4),
        # Camera shake taken out of a 4K greyscale pair.
        dict(name="stabilize_3840x2160", do="stabilize", w=3840, h=2160, window=15, features=False, cap=0),
        # A host plugin's blend of two remapped HD frames, no device allocation.
        dict(name="noalloc_1920x1080_l6", do="noalloc", w=1920, h=1080, levels=6, batch=1),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choices(["stitch", "stabilize", "noalloc", "batch", "serve"], [14, 3, 2, 1, 1])[0]
    if kind == "stabilize":
        h = _log(rng, 480, 2160)
        return dict(do="stabilize", w=min(3840, int(h * rng.choice([4 / 3, 16 / 9])) + rng.randint(0, 3)), h=h,
                    window=rng.choice([15, 15, 15, 21, 9]), features=rng.random() < 0.5,
                    cap=rng.choice([0, 0, 500, 4000]))
    if kind == "noalloc":
        h = _log(rng, 240, 1080)
        return dict(do="noalloc", w=int(h * 16 / 9) + rng.randint(0, 3) * (h < 1000), h=h, levels=rng.randint(1, 6),
                    batch=rng.choice([1, 1, 2]) if h < 700 else 1)
    if kind == "batch":
        h2, h3 = _log(rng, 600, 1650), _log(rng, 500, 900)
        return dict(do="batch", w2=int(2.58 * h2), h2=h2, w3=int(3.33 * h3), h3=h3, frames=8,
                    per_call=rng.choice([1, 2, 4, 8]), levels=rng.randint(3, 6))
    if kind == "serve":
        h, h3 = _log(rng, 600, 1200), _log(rng, 500, 900)
        return dict(do="serve", w=int(2.75 * h), h=h, w3=int(3.33 * h3), h3=h3, requests=rng.choice([12, 24, 32]),
                    slots=rng.choice([2, 4, 8]))
    n = rng.choice([2, 2, 2, 2, 3, 3, 4, 5, 6, 8])
    h = _log(rng, 700, 3300 if n == 2 else 2400)
    w = min(9000, int(h * (2.1 + 0.55 * (n - 2) * rng.uniform(0.8, 1.0) + rng.uniform(0.3, 0.6))) + rng.randint(0, 7))
    pixels = rng.choice(["rgba", "rgba", "rgba", "rgb"])
    levels = rng.choice([0, 1, 2, 3, 4, 5, 6, 6, 6])
    batch = rng.choice([1, 1, 1, 2, 3]) if w * h < 6e6 else 1
    storage = rng.choice(["f32", "f32", "f16"]) if pixels == "rgba" else "f32"
    filt = "binomial5" if pixels == "rgba" and levels > 1 and n <= 3 and rng.random() < 0.2 else "refbox"
    minimize = not (n != 3 and w * h < 4e6 and rng.random() < 0.2)
    kind = {2: 2, 3: rng.choice([3, 3, 1])}.get(n, 1)
    return stitch(None, n, kind, w, h, levels, pixels, storage, filt, batch, rng.uniform(0.12, 0.25), minimize)


# ---- inputs ----

def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) % (1 << 62))
    return g


def _overlap(w, n, overlap):
    """Overlap as a fraction of a footprint that leaves room for the two-image blend strip's margin."""
    return max(overlap, 40.0 / w * n)


def _rig(n, kind, w, h, overlap, seed):
    """Tables (numpy uint16), positions, the seam and the source size of an n-camera rig."""
    g = _gen(seed * 7919 + 17)
    fw = w / (n - (n - 1) * _overlap(w, n, overlap))
    step = (w - fw) / (n - 1)
    src_h = int(round(h * 0.875)) // 2 * 2
    src_w = src_h * 16 // 9
    fc = fw / HFOV
    fs = (src_w / 2) / math.tan(HFOV / 2)
    fcv = 0.97 * h * fs / src_h
    rolls = ((torch.rand(n, generator=g, device="cuda") * 2 - 1) * math.radians(2.0)).tolist()
    cols, rows, pos, spans = [], [], [], []
    v = ((torch.arange(h, device="cuda", dtype=torch.float64) - h / 2) / fcv)[:, None]
    for i in range(n):
        centre = fw / 2 + i * step
        c0 = 0 if i == 0 else int(centre - fw / 2)
        c1 = w if i == n - 1 else int(centre + fw / 2)
        t = (torch.arange(c0, c1, device="cuda", dtype=torch.float64) - centre) / fc
        x, z, cr, sr = torch.sin(t)[None, :], torch.cos(t)[None, :], math.cos(rolls[i]), math.sin(rolls[i])
        px = torch.floor(fs * (cr * x - sr * v) / z + src_w / 2 + 0.5)
        py = torch.floor(fs * (sr * x + cr * v) / z + src_h / 2 + 0.5)
        ok = (px >= 0) & (px < src_w) & (py >= 0) & (py < src_h)
        for out, p in ((cols, px), (rows, py)):
            out.append(torch.where(ok, p, 65535.0).to(torch.int32).cpu().numpy().astype(np.uint16))
        pos.append(hmpano.SpatialTiff(float(c0), 0.0))
        spans.append((c0, c1))
    label = torch.zeros((h, w), dtype=torch.uint8, device="cuda")
    u = torch.arange(w, device="cuda")[None, :]
    for i in range(n - 1):
        lo, hi = spans[i + 1][0], spans[i][1]
        walk = torch.cumsum(torch.randint(-1, 2, (h,), generator=g, device="cuda"), 0)
        walk = ((lo + hi) // 2 + walk).clamp(lo + (hi - lo) // 6, hi - (hi - lo) // 6)
        label += (u >= walk[:, None]).to(torch.uint8)
    seam = (label == 0).to(torch.uint8) if kind == 2 else label
    return cols, rows, pos, seam.cpu().numpy(), src_w, src_h


def _masks(kind, cols, rows, pos, seam):
    if kind == 2:
        return hmpano.ControlMasks(cols[0], rows[0], cols[1], rows[1], seam, pos)
    if kind == 3:
        return hmpano.ControlMasks3(cols[0], rows[0], cols[1], rows[1], cols[2], rows[2], seam, pos)
    return hmpano.ControlMasksN(cols, rows, seam, pos)


def _frames(batch, h, w, channels, seed):
    """Camera frames [batch, h, w, channels] uint8: smooth content with sensor noise, alpha 255."""
    g = _gen(seed * 104729 + 5)
    grid = torch.rand((batch, 3, h // 24 + 3, w // 24 + 3), generator=g, device="cuda") * 255
    out = F.interpolate(grid, size=(h, w), mode="bilinear", align_corners=False)
    out += torch.randn((batch, 3, h, w), generator=g, device="cuda") * 3
    out = out.clamp_(0, 255).to(torch.uint8).permute(0, 2, 3, 1)
    if channels == 4:
        out = torch.cat([out, torch.full_like(out[..., :1], 255)], dim=-1)
    return out.contiguous()


def _grey_pair(h, w, seed):
    """A greyscale float pair of 8-bit values: one scene, the second frame moved by a few pixels and a
    fraction, independent sensor noise."""
    g = _gen(seed * 15485863 + 3)
    grid = torch.rand((1, 1, h // 6 + 12, w // 6 + 12), generator=g, device="cuda") * 220 + 16
    r = torch.rand(4, generator=g, device="cuda").tolist()
    shift = (round(r[0] * 8 - 4) + 0.6 * r[1] - 0.3, round(r[2] * 8 - 4) + 0.6 * r[3] - 0.3)
    gh, gw = grid.shape[2:]
    frames = []
    for dx, dy in ((0.0, 0.0), shift):
        xs = ((torch.arange(w, device="cuda") - dx) / 6 + 4) / (gw - 1) * 2 - 1
        ys = ((torch.arange(h, device="cuda") - dy) / 6 + 4) / (gh - 1) * 2 - 1
        at = torch.stack(torch.broadcast_tensors(xs[None, :], ys[:, None]), -1)[None]
        f = F.grid_sample(grid, at, mode="bicubic", align_corners=True)[0, 0]
        f = (f + torch.randn((h, w), generator=g, device="cuda") * 1.5).round().clamp(0, 255)
        frames.append(f.contiguous())
    return frames


def _stitcher(kind, batch, levels, masks, minimize=True, **kw):
    if kind == 2:
        return hmpano.CudaStitchPano(batch, levels, masks, quiet=True, minimize_blend=minimize, **kw)
    if kind == 3:
        return hmpano.CudaStitchPano3(batch, levels, masks, quiet=True, **kw)
    return hmpano.CudaStitchPanoN(batch, levels, masks, quiet=True, minimize_blend=minimize, **kw)


def _checked(st):
    if not st.status.ok():
        raise hmpano.CudaStatusError(st.status)
    return st


def prepare(case, seed):
    c = case
    if c["do"] == "stitch":
        *tables, sw, sh = _rig(c["n"], c["kind"], c["w"], c["h"], c["overlap"], seed)
        st = _checked(_stitcher(c["kind"], c["batch"], c["levels"], _masks(c["kind"], *tables), c["minimize"],
                                storage=c["storage"], filter=c["filter"]))
        ch = 3 if c["pixels"] == "rgb" else 4
        ins = [_frames(c["batch"], sh, sw, ch, seed * 31 + i) for i in range(c["n"])]
        canvas = torch.zeros((c["batch"], c["h"], c["w"], ch), dtype=torch.uint8, device="cuda")
        if ch == 3:  # the stitcher of a pixel type is made on its first frame; a program makes it before its loop
            st.process(ins, canvas) if c["kind"] == 1 else st.process(*ins, canvas)
        return dict(case=c, st=st, ins=ins, canvas=canvas)
    if c["do"] == "batch":
        job, sts, outs = hmpano.Batch(), [], []
        for s, (kind, w, h) in enumerate([(2, c["w2"], c["h2"])] * 2 + [(3, c["w3"], c["h3"])] * 2):
            *tables, sw, sh = _rig(kind, kind, w, h, 0.15, seed * 4 + s)
            st = _checked(_stitcher(kind, c["per_call"], c["levels"], _masks(kind, *tables), storage="f16"))
            ins = [_frames(c["frames"], sh, sw, 4, seed * 131 + 10 * s + i) for i in range(kind)]
            for k in range(0, c["frames"], c["per_call"]):
                canvas = torch.zeros((c["per_call"], h, w, 4), dtype=torch.uint8, device="cuda")
                job.add(st, [t[k:k + c["per_call"]] for t in ins], canvas, stream_index=s)
                outs.append(canvas)
            sts.append(st)
        torch.cuda.synchronize()
        job.capture()
        torch.cuda.synchronize()
        return dict(case=c, job=job, sts=sts, outs=outs)
    if c["do"] == "serve":
        srv = hmpano.StitchServer(20 << 30, slots=c["slots"], max_instances_per_config=2)
        configs, requests = [], []
        for i, (kind, w, h, levels) in enumerate([(2, c["w"], c["h"], 0), (2, c["w"], c["h"], 3),
                                                  (3, c["w3"], c["h3"], 6)]):
            *tables, sw, sh = _rig(kind, kind, w, h, 0.15, seed * 3 + i)
            cid = srv.add_config(kind, _masks(kind, *tables), levels)
            configs.append((cid, [_frames(1, sh, sw, 4, seed * 53 + 10 * i + k) for k in range(kind)], w, h))
        for k in range(c["requests"]):
            cid, ins, w, h = configs[k % 3]
            requests.append((cid, ins, torch.zeros((1, h, w, 4), dtype=torch.uint8, device="cuda")))
        s = dict(case=c, srv=srv, requests=requests)
        torch.cuda.synchronize()
        for _ in range(2):  # resident stitchers, as a server in service has them
            run(s)
        return s
    if c["do"] == "stabilize":
        prev, nxt = _grey_pair(c["h"], c["w"], seed)
        st = hmpano.Stabilizer(c["w"], c["h"], c["cap"])
        return dict(case=c, st=st, prev=prev, next=nxt, out=torch.zeros_like(prev))
    h, w, b = c["h"], c["w"], c["batch"]
    g = _gen(seed * 6151 + 9)
    walk = w // 2 + torch.cumsum(torch.randint(-1, 2, (h,), generator=g, device="cuda"), 0)
    seam = (torch.arange(w, device="cuda")[None, :] < walk[:, None]).to(torch.uint8).contiguous()
    t = [_frames(b, h, w, 4, seed * 3 + 1), _frames(b, h, w, 4, seed * 3 + 2)]
    out = torch.zeros_like(t[0])
    return dict(case=c, keep=(t, seam), out=out, images=[pano._image(x) for x in (*t, out)], seam=C.c_void_p(seam.data_ptr()))


# ---- one pass ----

def run(state):
    s, c = state, state["case"]
    if c["do"] == "stitch":
        if c["kind"] == 1:
            return s["st"].process(s["ins"], s["canvas"])
        return s["st"].process(*s["ins"], s["canvas"])
    if c["do"] == "batch":
        s["job"].launch()
        return s["outs"]
    if c["do"] == "serve":
        for cid, ins, canvas in s["requests"]:
            s["srv"].submit(cid, ins, canvas)
        status = s["srv"].drain()
        if not status.ok():
            raise hmpano.CudaStatusError(status)
        return [canvas for _, _, canvas in s["requests"]]
    if c["do"] == "stabilize":
        s["st"].run(s["prev"], s["next"], s["out"], window_size=c["window"])
        if not c["features"]:
            return s["out"]
        xy, flow, m = s["st"].features()  # a program that logs the motion reads it back
        return [s["out"], xy, flow, m.dx, m.dy, m.corners]
    a, b, out = s["images"]
    st = _lib.lib().hmp_blend2_noalloc(C.byref(a), C.byref(b), s["seam"], c["w"], c["levels"], c["batch"], C.byref(out),
                                       C.c_void_p(torch.cuda.current_stream().cuda_stream))
    if st.code:
        raise RuntimeError(st.message.decode())
    return s["out"]


# ---- what a pass cannot do without ----

def _stitch_work(n, w, h, levels, channels, batch, overlap):
    """Per canvas pixel one table entry, one source pixel and one canvas pixel; with a blend, the seam
    and the second image's entry and pixel in the overlaps too. The pyramid's arithmetic: about 40
    operations per channel and overlap pixel (a mean, two upsamples and a blend, times 4/3)."""
    ov = _overlap(w, n, overlap)
    fw = w / (n - (n - 1) * ov)
    both = (n - 1) * ov * fw * h if levels else 0
    px = float(w) * h
    return dict(bytes=px * (4 + (levels > 0) + 2 * channels * batch) + both * (4 + channels * batch),
                flops=40.0 * channels * both * batch)


def work(case):
    c = case
    if c["do"] == "stitch":
        return _stitch_work(c["n"], c["w"], c["h"], c["levels"], 3 if c["pixels"] == "rgb" else 4, c["batch"], c["overlap"])
    if c["do"] == "batch":
        parts = [_stitch_work(2, c["w2"], c["h2"], c["levels"], 4, c["frames"], 0.15)] * 2
        parts += [_stitch_work(3, c["w3"], c["h3"], c["levels"], 4, c["frames"], 0.15)] * 2
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    if c["do"] == "serve":
        each = [_stitch_work(2, c["w"], c["h"], 0, 4, 1, 0.15), _stitch_work(2, c["w"], c["h"], 3, 4, 1, 0.15),
                _stitch_work(3, c["w3"], c["h3"], 6, 4, 1, 0.15)]
        return {k: sum(each[i % 3][k] for i in range(c["requests"])) for k in ("bytes", "flops")}
    px = float(c["w"]) * c["h"]
    if c["do"] == "stabilize":
        # Both frames in, one out; about 60 operations a pixel for the response, and per corner (one
        # pixel in 40 on these frames) one window of gradients and sums.
        corners = min(px / 40, c["cap"] or px)
        return dict(bytes=12 * px, flops=60 * px + corners * c["window"] ** 2 * 15)
    # Two images and the seam in, one image out.
    return dict(bytes=px * (12 * c["batch"] + 1), flops=160.0 * px * c["batch"])


# ---- the stabiliser in 64 bits (every other output is whole numbers) ----

def _shift_of(v):
    return torch.sign(v) * torch.floor(v.abs() + 0.5)


def exact(case, seed):
    if case["do"] != "stabilize":
        return None
    c, (prev, nxt) = case, _grey_pair(case["h"], case["w"], seed)
    p, q = prev.double(), nxt.double()
    h, w = p.shape
    gx, gy = torch.zeros_like(p), torch.zeros_like(p)
    gx[1:-1, 1:-1] = (p[:-2, 2:] + 2 * p[1:-1, 2:] + p[2:, 2:]) - (p[:-2, :-2] + 2 * p[1:-1, :-2] + p[2:, :-2])
    gy[1:-1, 1:-1] = (p[:-2, :-2] + 2 * p[:-2, 1:-1] + p[:-2, 2:]) - (p[2:, :-2] + 2 * p[2:, 1:-1] + p[2:, 2:])

    def box(a):
        return F.conv2d(a[None, None], torch.ones((1, 1, 3, 3), dtype=a.dtype, device=a.device))[0, 0]

    sxx, sxy, syy = box(gx * gx), box(gx * gy), box(gy * gy)
    resp = torch.zeros_like(p)
    resp[1:-1, 1:-1] = sxx * syy - sxy * sxy - 0.04 * (sxx + syy) ** 2
    inner = resp[1:-1, 1:-1]
    top = F.max_pool2d(resp[None, None], 3, 1)[0, 0]
    yx = torch.nonzero((inner > 1e6) & (inner >= top)) + 1
    xy = torch.stack([yx[:, 1], yx[:, 0]], 1)
    found = xy.shape[0]
    kept = xy[:c["cap"]] if c["cap"] else xy
    half = c["window"] // 2
    o = torch.arange(-half, half + 1, device=p.device)
    flows = []
    for part in kept.split(16384):
        x = (part[:, 0, None, None] + o[None, None, :]).expand(-1, len(o), -1)
        y = (part[:, 1, None, None] + o[None, :, None]).expand(-1, -1, len(o))
        own = (x >= 1) & (x < w - 1) & (y >= 1) & (y < h - 1)
        xc, yc = x.clamp(1, w - 2), y.clamp(1, h - 2)
        ix, iy = (p[yc, xc + 1] - p[yc, xc - 1]) / 2, (p[yc + 1, xc] - p[yc - 1, xc]) / 2
        base = p[yc, xc]
        d = torch.zeros((part.shape[0], 2), dtype=torch.float64, device=p.device)
        live = torch.ones(part.shape[0], dtype=torch.bool, device=p.device)
        for _ in range(10):
            r = _shift_of(d).long()
            xn, yn = x + r[:, 0, None, None], y + r[:, 1, None, None]
            m = (own & (xn >= 0) & (xn < w - 1) & (yn >= 0) & (yn < h - 1)).double()
            it = q[yn.clamp(0, h - 1), xn.clamp(0, w - 1)] - base
            a, b, e = (ix * ix * m).sum((1, 2)), (ix * iy * m).sum((1, 2)), (iy * iy * m).sum((1, 2))
            tx, ty = (ix * it * m).sum((1, 2)), (iy * it * m).sum((1, 2))
            det = a * e - b * b
            live &= det.abs() >= 1e-6
            step = torch.stack([(-e * tx + b * ty) / det, (b * tx - a * ty) / det], 1)
            d = torch.where(live[:, None], d + step, d)
            live &= torch.where(live, step.norm(dim=1) >= 0.01, live)
            if not live.any():
                break
        flows.append(d)
    flow = torch.cat(flows) if flows else torch.zeros((0, 2), dtype=torch.float64, device=p.device)
    mean = flow.mean(0) if len(flow) else torch.zeros(2, dtype=torch.float64, device=p.device)
    sx, sy = (int(v) for v in _shift_of(mean).tolist())
    out = torch.zeros_like(q)
    y0, y1, x0, x1 = max(0, sy), min(h, h + sy), max(0, sx), min(w, w + sx)
    if y1 > y0 and x1 > x0:
        out[y0:y1, x0:x1] = q[y0 - sy:y1 - sy, x0 - sx:x1 - sx]
    if not c["features"]:
        return out
    return [out, kept.int(), flow, float(mean[0]), float(mean[1]), found]
