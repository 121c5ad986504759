"""Performance cases: the work that a user of this package has it do, over its range of sizes and options.

listed() names the cases, draw() makes more of the same ranges, prepare() builds what a program holds before the
call (inputs in device memory or host frames, and the filters it keeps), run() is one pass through the public entry
points, work() the bytes and operations a pass cannot do without, and exact() the same outputs in 64 bits in plain
torch.

Kinds of case:
  window   one frame window of one filter (BM3D, the stacked accumulators with radius > 0) on device buffers
  twopass  both BM3Dv2 passes of one frame on device buffers: pass 1 writes the reference half that pass 2 reads
  fused    one output frame of the temporal filter: one new window and the aggregation of the stacks around it
  batch    one window each of several clips of unequal sizes in one call
  host     a whole short clip of host frames through BM3Dv2 twice, frame after frame
  pilot    the learned pilot's estimate of one plane
  train    the loss gradients of one batch at the start of the pilot's training
"""
import ctypes
import math
import os
import struct
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(ROOT, "vapoursynth-zipcu_b200")
if PKG not in sys.path:
    sys.path.insert(0, PKG)

import zb3d  # noqa: E402
from zb3d import _native as N  # noqa: E402
from zb3d import pilot as P  # noqa: E402
from zb3d.device import DeviceFilter, process_batch  # noqa: E402

EXTRACTOR_EXP = 3  # the deterministic mode
PS_NUM, PS_RANGE = 2, 4
HARD_FACTOR = struct.unpack("<f", struct.pack("<I", 0x3F021BB6))[0]
WIENER_FACTOR = struct.unpack("<f", struct.pack("<I", 0x3E40C0C1))[0]
FUSED_FRAMES_EACH_SIDE = 2  # radius of the fused cases
BATCH_CLIPS = (  # width, height, format, chroma, radius, sigma (scaled by the case's own scale)
    (720, 480, "yuv420", False, 0, 14.0),
    (1280, 720, "yuv444", True, 0, 8.0),
    (1280, 720, "yuv420", False, 1, 10.0),
    (3840, 2160, "yuv420", False, 0, 17.0),
)


def _case(kind, w, h, **kw):
    c = dict(kind=kind, w=w, h=h, fmt="gray", chroma=False, sigma=10.0, bs=8, rng=9, radius=0, final=False,
             metric="ssd", t2d="dct", t1d="dct", precision=False, bits=0, frames=1)
    c.update(kw)
    return c


def listed():
    return [
        # the smallest call: a thumbnail of odd size through both passes, default search; launches and latency
        dict(_case("twopass", 77, 53), name="tiny_twopass"),
        # standard definition gray, weak noise, the default search (block_step 8, bm_range 9), one pass
        dict(_case("window", 640, 480, sigma=3.0), name="gray640"),
        # the headline job: both passes of a 1080p YUV420 frame, block_step 4, bm_range 12
        dict(_case("twopass", 1920, 1080, fmt="yuv420", bs=4, rng=12), name="twopass1080"),
        # joint colour filtering (CBM3D) of a 720p YUV444 frame that came from 8-bit video
        dict(_case("window", 1280, 720, fmt="yuv444", chroma=True, bs=4, rng=12, bits=8), name="cbm3d720"),
        # VBM3D: 1080p gray, radius 2, sigma 15, per output frame one window and one aggregation
        dict(_case("fused", 1920, 1080, sigma=15.0, radius=2), name="vbm3d1080"),
        # the second (Wiener) temporal pass on 720p YUV420, radius 1, block_step 4, with a basic estimate as ref
        dict(_case("window", 1280, 720, fmt="yuv420", bs=4, rng=12, radius=1, final=True), name="temporal_final720"),
        # the other distance and transforms on an odd-sized plane: sad, haar 2D, wht across the group
        dict(_case("window", 959, 541, bs=4, rng=12, sigma=20.0, metric="sad", t2d="haar", t1d="wht"),
             name="sad_haar540"),
        # the tensor-core precision form of the filter, Wiener pass on a 1080p plane
        dict(_case("window", 1920, 1080, bs=8, rng=9, sigma=15.0, final=True, precision=True),
             name="precision1080"),
        # host frames: a 20-frame 720p YUV420 clip from 8-bit video through BM3Dv2 twice, uploads and downloads
        dict(_case("host", 1280, 720, fmt="yuv420", bs=4, rng=12, bits=8, frames=20), name="host720"),
        # clips of unequal sizes, one window each, in one batch call
        dict(_case("batch", 3840, 2160, fmt="yuv420", bs=4, rng=12), name="batch_uneven"),
        # the shipped pilot network on a 1080p luma plane (bf16 tensor-core inference)
        dict(_case("pilot", 1920, 1080), name="pilot1080"),
        # gradients of one batch of the pilot's training recipe: 32 crops of 64 x 64
        dict(_case("train", 64, 64, frames=32), name="pilot_train"),
    ]


def _log_size(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _cost(c):
    """A rough measure of a case's work: candidate distances and filtered values."""
    if c["kind"] in ("pilot", "train"):
        return 0.0
    planes = {"gray": 1.0, "yuv420": 1.5, "yuv444": 3.0}[c["fmt"]]
    blocks = c["w"] * c["h"] / (c["bs"] * c["bs"]) * planes
    cand = (2 * c["rng"] + 1) ** 2 + 2 * c["radius"] * PS_NUM * (2 * PS_RANGE + 1) ** 2
    passes = {"twopass": 2, "host": 2 * c["frames"]}.get(c["kind"], 1)
    return passes * blocks * (cand + 500 * (1 + c["final"]))


def draw(rng):
    top = 1.2 * 3840 * 2160 / 16 * 1.5 * 1125  # the 4K clip of the batch, and something for the others
    while True:
        kind = rng.choice(["window", "window", "window", "twopass", "twopass", "fused", "batch", "host", "pilot",
                           "train"])
        if kind == "pilot":
            return _case("pilot", _log_size(rng, 64, 1920), _log_size(rng, 48, 1080), sigma=rng.uniform(5.0, 25.0))
        if kind == "train":
            side = rng.choice([48, 56, 64])
            return _case("train", side, side, frames=rng.randint(8, 32), sigma=rng.uniform(5.0, 25.0))
        if kind == "batch":
            # the same clips scaled down by up to four
            w = rng.randint(960, 3840)
            return _case("batch", w, w * 9 // 16, fmt="yuv420", bs=4, rng=12, sigma=rng.uniform(5.0, 15.0))
        bs = rng.choice([4, 4, 8, 8, 3, 5, 6])
        c = _case(kind, _log_size(rng, 48, 1920), _log_size(rng, 40, 1080), bs=bs,
                  rng=rng.choice([12, 9, 16]) if bs in (4, 8) else rng.choice([7, 9]),
                  sigma=rng.uniform(3.0, 25.0), bits=rng.choice([0, 0, 8]))
        if kind == "fused":
            c["radius"] = FUSED_FRAMES_EACH_SIDE
        elif kind == "host":
            c.update(fmt="yuv420", frames=rng.randint(18, 21))
        else:
            c["fmt"] = rng.choice(["gray", "yuv420", "yuv444"])
        if kind == "window":
            c["chroma"] = c["fmt"] == "yuv444" and rng.random() < 0.6
            c["radius"] = rng.choice([0, 0, 0, 1, 2]) if c["fmt"] != "yuv444" else 0
            c["final"] = rng.random() < 0.5
            what = rng.random()
            if what < 0.2:
                c["metric"] = "sad"
            elif what < 0.4:
                c.update(t2d=rng.choice(["haar", "wht"]), t1d=rng.choice(["dct", "haar", "wht"]))
            elif what < 0.6:
                c["precision"] = True
        if c["fmt"] == "yuv420":  # even luma sizes, as the format asks; the chroma planes may be odd
            c["w"], c["h"] = max(96, c["w"] // 2 * 2), max(80, c["h"] // 2 * 2)
        if _cost(c) <= top:
            return c


# ---- inputs ------------------------------------------------------------------------------------

def _planes_of(case):
    """(width, height) of each plane."""
    w, h = case["w"], case["h"]
    if case["fmt"] == "gray":
        return [(w, h)]
    if case["fmt"] == "yuv420":
        return [(w, h), (w // 2, h // 2), (w // 2, h // 2)]
    return [(w, h)] * 3


def _scene(w, h, seed, frames):
    """Clean moving planes [frames][h][w] (float32, device): a gradient, rectangles and a sinusoidal texture that
    translate by a few pixels per frame."""
    r = np.random.default_rng(seed)
    gx, gy = (int(v) for v in r.integers(0, 4, 2))
    xs = torch.arange(w, device="cuda", dtype=torch.float32)
    ys = torch.arange(h, device="cuda", dtype=torch.float32)
    rects = [(int(r.integers(-w // 8, w)), int(r.integers(-h // 8, h)), int(r.integers(4, max(5, w // 3))),
              int(r.integers(4, max(5, h // 3))), float(r.uniform(0.0, 1.0))) for _ in range(20)]
    period, theta = r.uniform(6.0, 40.0), r.uniform(0.0, np.pi)
    out = torch.empty((frames, h, w), device="cuda", dtype=torch.float32)
    for t in range(frames):
        sx, sy = gx * t, gy * t
        img = 0.25 + 0.25 * ((xs + sx)[None, :] / w + (ys + sy)[:, None] / h)
        for x0, y0, rw, rh, v in rects:
            xa, xb = max(x0 - sx, 0), min(x0 - sx + rw, w)
            ya, yb = max(y0 - sy, 0), min(y0 - sy + rh, h)
            if xa < xb and ya < yb:
                img[ya:yb, xa:xb] = v
        phase = (xs + sx)[None, :] * math.cos(theta) + (ys + sy)[:, None] * math.sin(theta)
        out[t] = img + 0.1 * torch.sin(2.0 * math.pi / period * phase)
    return out


def _noisy(clean, sigma, seed, bits):
    """The clean planes with Gaussian noise of sigma / 255; from 8-bit video: clamped and rounded to k / 255."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    x = clean + torch.randn(clean.shape, generator=g, device="cuda", dtype=torch.float32) * (sigma / 255.0)
    if bits:
        top = float((1 << bits) - 1)
        x = (x.clamp(0.0, 1.0) * top).round() / top
    return x


def _frames(case, seed, count):
    """Per plane [count][h][w]: the noisy planes, and a basic estimate of them (the clean ones with a quarter of
    the noise)."""
    noisy, basic = [], []
    for p, (w, h) in enumerate(_planes_of(case)):
        clean = _scene(w, h, 1000 * seed + p, count)
        noisy.append(_noisy(clean, case["sigma"], 1000 * seed + 10 + p, case["bits"]))
        basic.append(_noisy(clean, case["sigma"] / 4.0, 1000 * seed + 20 + p, 0))
    return noisy, basic


def _family(case):
    if case["fmt"] == "gray":
        return N.GRAY, (0, 0)
    return N.YUV, (1, 1) if case["fmt"] == "yuv420" else (0, 0)


def _options(case):
    return dict(sigma=[case["sigma"]] * len(_planes_of(case)), block_step=case["bs"], bm_range=case["rng"],
                radius=case["radius"], ps_num=PS_NUM, ps_range=PS_RANGE, chroma=int(case["chroma"]),
                extractor_exp=EXTRACTOR_EXP, bm_error_s=case["metric"], transform_2d_s=case["t2d"],
                transform_1d_s=case["t1d"])


def _device_filter(case, ref):
    family, sub = _family(case)
    return DeviceFilter(case["w"], case["h"], family=family, subsampling=sub, num_frames=2 * case["radius"] + 1,
                        ref=ref, num_streams=1, filter_form=int(case["precision"]), **_options(case))


def _window_source(f, noisy, basic, ref):
    """One window's source buffer: [clips][planes][frames][h][pitch] per entry."""
    src = torch.zeros(f.src_elems, device="cuda", dtype=torch.float32)
    for lay in f.entries:
        v = src[lay.src_offset:lay.src_offset + lay.src_elems].view(lay.nclips, lay.nplanes, lay.tw, lay.height,
                                                                    lay.pitch)
        for i in range(lay.nplanes):
            v[lay.nclips - 1, i, :, :, :lay.width] = noisy[lay.plane[i]]
            if ref:
                v[0, i, :, :, :lay.width] = basic[lay.plane[i]]
    return src


def _window_result(f, dst):
    """Every entry's output without the padding columns."""
    out = []
    for lay in f.entries:
        v = dst[lay.dst_offset:lay.dst_offset + lay.dst_elems]
        v = v.view(lay.nplanes, lay.height, lay.pitch) if lay.tw == 1 else \
            v.view(lay.nplanes, lay.tw, 2, lay.height, lay.pitch)
        out.append(v[..., :lay.width])
    return out


def _batch_cases(case):
    """The batch's clips, scaled with the case's width (3840 = as listed in BATCH_CLIPS)."""
    out = []
    for w, h, fmt, chroma, radius, sigma in BATCH_CLIPS:
        w, h = max(96, w * case["w"] // 3840 // 2 * 2), max(80, h * case["h"] // 2160 // 2 * 2)
        out.append(_case("window", w, h, fmt=fmt, chroma=chroma, radius=radius, bs=case["bs"], rng=case["rng"],
                         sigma=sigma * case["sigma"] / 10.0))
    return out


def _network_inputs(case, seed):
    """Noisy planes [n][h][w], their targets and noise levels for the pilot."""
    n = case["frames"]
    clean = torch.stack([_scene(case["w"], case["h"], 1000 * seed + i, 1)[0] for i in range(n)])
    noisy = _noisy(clean, case["sigma"], 1000 * seed + 500, 0)
    target = _noisy(clean, case["sigma"] / 8.0, 1000 * seed + 501, 0)
    return noisy, target, torch.full((n,), case["sigma"], device="cuda", dtype=torch.float32)


def _initial_state(seed):
    """Random weights of the shipped architecture, as at the start of training (2 real inputs, 1 real output)."""
    r = np.random.default_rng(seed)
    out, shapes = {}, P.arch(32, 7)
    for l, (cin, cout) in enumerate(shapes):
        rin, rout = 2 if l == 0 else cin, 1 if l == len(shapes) - 1 else cout
        w, b = np.zeros((cout, 3, 3, cin), np.float32), np.zeros(cout, np.float32)
        w[:rout, :, :, :rin] = r.normal(0.0, math.sqrt(2.0 / (9 * rin)), (rout, 3, 3, rin))
        b[:rout] = r.normal(0.0, 0.05, rout)
        out["w%d" % l], out["b%d" % l] = w, b
    return out


def prepare(case, seed):
    kind = case["kind"]
    s = {"kind": kind, "stream": torch.cuda.Stream()}
    if kind == "window":
        noisy, basic = _frames(case, seed, 2 * case["radius"] + 1)
        f = s["filter"] = _device_filter(case, case["final"])
        s["src"] = _window_source(f, noisy, basic, case["final"])
        s["dst"] = torch.zeros(f.dst_elems, device="cuda", dtype=torch.float32)
    elif kind == "twopass":
        noisy, _ = _frames(case, seed, 1)
        s["first"], s["second"] = _device_filter(case, False), _device_filter(case, True)
        s["bufs"], s["outs"] = [], []
        for lay in s["first"].entries:  # per plane [basic | noisy]
            b = torch.zeros((2, lay.height, lay.pitch), device="cuda", dtype=torch.float32)
            b[1, :, :lay.width] = noisy[lay.plane[0]][0]
            s["bufs"].append(b)
            s["outs"].append(torch.zeros((lay.height, lay.pitch), device="cuda", dtype=torch.float32))
    elif kind == "fused":
        r = case["radius"]
        tw = 2 * r + 1
        f = s["filter"] = _device_filter(case, False)
        lay = s["lay"] = f.entries[0]
        noisy, _ = _frames(case, seed, 4 * r + 1)
        s["frames"] = torch.zeros((4 * r + 1, lay.height, lay.pitch), device="cuda", dtype=torch.float32)
        s["frames"][:, :, :lay.width] = noisy[0]
        s["stacks"] = [torch.zeros((tw, 2, lay.height, lay.pitch), device="cuda", dtype=torch.float32)
                       for _ in range(tw)]
        s["out"] = torch.zeros((lay.height, lay.pitch), device="cuda", dtype=torch.float32)
        torch.cuda.synchronize()
        for m in range(tw - 1):  # the stacks that earlier output frames left
            f.run_entry(0, s["frames"][m].data_ptr(), s["stacks"][m].data_ptr(), s["stream"].cuda_stream)
        nf = 4 * r + 1  # the output frame is the middle one of the clip: no clamping at its ends
        s["ptrs"] = (ctypes.c_void_p * tw)(*[t.data_ptr() for t in s["stacks"]])
        s["zs"] = (ctypes.c_int * tw)(*[N.lib().zb3d_agg_z(i, 2 * r, nf, r) for i in range(tw)])
    elif kind == "batch":
        s["jobs"] = []
        for i, c in enumerate(_batch_cases(case)):
            noisy, basic = _frames(c, seed + 100 * i, 2 * c["radius"] + 1)
            f = _device_filter(c, False)
            s["jobs"].append((f, _window_source(f, noisy, basic, False),
                              torch.zeros(f.dst_elems, device="cuda", dtype=torch.float32)))
    elif kind == "host":
        noisy, _ = _frames(case, seed, case["frames"])
        host = [p.cpu().numpy() for p in noisy]
        family, sub = _family(case)
        frames = [[p[i] for p in host] for i in range(case["frames"])]
        clip = zb3d.Clip.from_frames(frames, family=family, subsampling=sub, pinned=True)
        first = zb3d.BM3Dv2(clip, **_options(case))
        s["clip"] = zb3d.BM3Dv2(clip, ref=first, **_options(case))
        s["count"] = case["frames"]  # more frames than a Clip keeps (16): every pass computes every frame
    else:
        if kind == "pilot":
            s["net"] = P.shipped()
        else:
            s["net"] = P.PilotNet()
            s["net"].load_state(_initial_state(seed))
        s["noisy"], s["target"], s["sigma"] = _network_inputs(case, seed)
    torch.cuda.synchronize()
    return s


def run(s):
    kind, st = s["kind"], s["stream"].cuda_stream
    if kind == "window":
        s["filter"].run(s["src"].data_ptr(), s["dst"].data_ptr(), st)
        return _window_result(s["filter"], s["dst"])
    if kind == "twopass":
        for e, lay in enumerate(s["first"].entries):
            buf, out = s["bufs"][e], s["outs"][e]
            s["first"].run_entry(e, buf[1].data_ptr(), buf[0].data_ptr(), st)
            s["second"].run_entry(e, buf.data_ptr(), out.data_ptr(), st)
        return [v[..., :lay.width] for lay, b, o in zip(s["first"].entries, s["bufs"], s["outs"]) for v in (b[0], o)]
    if kind == "fused":
        lay, tw = s["lay"], len(s["stacks"])
        s["filter"].run_entry(0, s["frames"][tw - 1].data_ptr(), s["stacks"][tw - 1].data_ptr(), st)
        if N.lib().zb3d_vaggregate_device(s["ptrs"], s["zs"], tw, lay.width, lay.height, lay.pitch, 1, 1,
                                          s["out"].data_ptr(), ctypes.c_void_p(st)) != 0:
            raise RuntimeError("zb3d_vaggregate_device failed")
        return [s["out"][:, :lay.width], s["stacks"][tw - 1][..., :lay.width]]
    if kind == "batch":
        process_batch([(f, src.data_ptr(), dst.data_ptr()) for f, src, dst in s["jobs"]], st)
        return [_window_result(f, dst) for f, _, dst in s["jobs"]]
    if kind == "host":
        return [s["clip"].get_frame(n) for n in range(s["count"])]
    if kind == "pilot":
        return s["net"].forward(s["noisy"], s["sigma"])[0]
    dws, dbs, loss, y = s["net"].gradients(s["noisy"], s["target"], s["sigma"])
    return {"dw": dws, "db": dbs, "loss": loss, "y": y}


# ---- what a pass cannot do without -------------------------------------------------------------

def _candidates(w, h, bs, rng):
    def axis(n):
        at = np.minimum(np.arange((n - 8 + bs - 1) // bs + 1) * bs, n - 8)
        return float((np.minimum(at + rng, n - 8) - np.maximum(at - rng, 0) + 1).sum()), len(at)
    (cx, nx), (cy, ny) = axis(w), axis(h)
    return cx * cy, nx * ny


def _pass_work(case, final):
    """Bytes and operations of one filter pass over one window.  Per candidate 64 differences, squares and sums;
    per group 24 eight-point transforms of 64 lines (44 operations each) per 3D transform pair, and the shrinkage."""
    tw = 2 * case["radius"] + 1
    dims = _planes_of(case)
    moved = sum(w * h for w, h in dims) * 4.0 * (tw * (1 + final) + (2 * tw if tw > 1 else 1))
    ops = 0.0
    for i, (w, h) in enumerate(dims):
        cand, blocks = _candidates(w, h, case["bs"], case["rng"])
        if i == 0 or not case["chroma"]:
            ops += 192.0 * (cand + blocks * (tw - 1) * PS_NUM * (2 * PS_RANGE + 1) ** 2)
        ops += blocks * ((3 if final else 2) * 8448.0 + 4 * 512.0)
    return moved, ops


def work(case):
    kind = case["kind"]
    if kind in ("pilot", "train"):
        net = P.arch(32, 7)
        px = float(case["w"] * case["h"] * case["frames"])
        macs = sum(9 * a * b for a, b in net)
        weights = 4.0 * sum(9 * a * b + b for a, b in net)
        return {"bytes": 8.0 * px + weights / 2, "flops": 2.0 * macs * px} if kind == "pilot" else \
            {"bytes": 12.0 * px + weights, "flops": 6.0 * macs * px}
    if kind == "batch":
        each = [_pass_work(c, False) for c in _batch_cases(case)]
        return {"bytes": sum(b for b, _ in each), "flops": sum(o for _, o in each)}
    if kind in ("twopass", "host"):
        (b1, o1), (b2, o2) = _pass_work(case, False), _pass_work(case, True)
        return {"bytes": (b1 + b2) * case["frames"], "flops": (o1 + o2) * case["frames"]}
    b, o = _pass_work(case, case["final"])
    if kind == "fused":
        b += 4.0 * case["w"] * case["h"] * (2 * (2 * case["radius"] + 1) + 1)
    return {"bytes": b, "flops": o}


# ---- the same outputs in 64 bits ---------------------------------------------------------------

def _transform(name):
    """(forward, inverse) 8 x 8 matrices of the filter's unnormalised 1D transforms."""
    if name == "dct":
        k, n = np.arange(8)[:, None], np.arange(8)[None, :]
        m = 4.0 * np.where(k == 0, math.sqrt(1 / 8), math.sqrt(2 / 8)) * np.cos(math.pi * (2 * n + 1) * k / 16)
        return m, m.T
    r2 = math.sqrt(2.0)
    if name == "haar":
        f = np.zeros((8, 8))
        f[0], f[1] = r2, r2 * np.repeat([1, -1], 4)
        f[2, :4], f[3, 4:] = 2 * np.repeat([1, -1], 2), 2 * np.repeat([1, -1], 2)
        for i in range(4):
            f[4 + i, 2 * i:2 * i + 2] = 2 * r2 * np.array([1, -1])
        # the inverse takes coefficients 2 and 4 for every detail, as the filter defines it
        inv = np.zeros((8, 8))
        inv[:, 0], inv[:, 1] = r2, r2 * np.repeat([1, -1], 4)
        inv[:, 2], inv[:, 4] = 2 * np.tile([1, 1, -1, -1], 2), 2 * r2 * np.tile([1, -1], 4)
        return f, inv
    s = np.array([[1, 1, 1, 1, 1, 1, 1, 1], [1, 1, 1, 1, -1, -1, -1, -1], [1, 1, -1, -1, -1, -1, 1, 1],
                  [1, 1, -1, -1, 1, 1, -1, -1], [1, -1, -1, 1, 1, -1, -1, 1], [1, -1, -1, 1, -1, 1, 1, -1],
                  [1, -1, 1, -1, -1, 1, -1, 1], [1, -1, 1, -1, 1, -1, 1, -1]], float) * r2  # wht
    return s, s


def _score(d, metric):
    return d.abs() if metric == "sad" else d * d


def _match64(planes, case):
    """Match lists (x, y, z), each [blocks][8], of the reference blocks of planes[radius]: planes [tw][h][w]."""
    tw, h, w = planes.shape
    r, bs, rng, dev = tw // 2, case["bs"], case["rng"], planes.device

    def axis(n):
        return torch.clamp(torch.arange((n - 8 + bs - 1) // bs + 1, device=dev) * bs, max=n - 8)
    xs, ys = axis(w), axis(h)
    mid, nb = planes[r], len(xs) * len(ys)
    rows = (ys[:, None] + torch.arange(8, device=dev)).reshape(-1)
    cols = (xs[:, None] + torch.arange(8, device=dev)).reshape(-1)
    side = 2 * rng + 1
    dist = torch.full((side * side, nb), math.inf, device=dev, dtype=torch.float64)
    for dy in range(-rng, rng + 1):
        oy = (ys + dy >= 0) & (ys + dy <= h - 8)
        cand = mid[(rows + dy).clamp(0, h - 1)]
        ref = mid[rows]
        for dx in range(-rng, rng + 1):
            ox = (xs + dx >= 0) & (xs + dx <= w - 8)
            d = _score(ref - cand[:, (torch.arange(w, device=dev) + dx).clamp(0, w - 1)], case["metric"])
            d = d.view(len(ys), 8, w).sum(1)[:, cols].view(len(ys), len(xs), 8).sum(2)
            k = (dy + rng) * side + dx + rng
            dist[k] = torch.where(oy[:, None] & ox[None, :], d, d.new_tensor(math.inf)).reshape(-1)
    e, k = torch.sort(dist, dim=0, stable=True)
    e, k = e[:8].T.contiguous(), k[:8].T.contiguous()
    del dist
    bx, by = xs.repeat(len(ys)), ys.repeat_interleave(len(xs))
    gx, gy = bx[:, None] + k % side - rng, by[:, None] + k // side - rng
    gz = torch.full_like(gx, r)
    i8 = torch.arange(8, device=dev)
    if r:
        pr = 2 * PS_RANGE + 1
        oy = torch.arange(pr, device=dev).repeat_interleave(pr) - PS_RANGE
        ox = torch.arange(pr, device=dev).repeat(pr) - PS_RANGE
        ge, sx, sy = e, gx.clone(), gy.clone()
        for way in (-1, 1):
            lx, ly = sx[:, :PS_NUM], sy[:, :PS_NUM]
            for t in range(1, r + 1):
                z = r + way * t
                cx = (lx[:, :, None] + ox).reshape(nb, -1)
                cy = (ly[:, :, None] + oy).reshape(nb, -1)
                ok = (cx >= 0) & (cx <= w - 8) & (cy >= 0) & (cy <= h - 8)
                px, py = cx.clamp(0, w - 8), cy.clamp(0, h - 8)
                d = torch.empty(cx.shape, device=dev, dtype=torch.float64)
                flat = planes[z].reshape(-1)
                for a in range(0, nb, 8192):
                    b = slice(a, a + 8192)
                    acc = torch.zeros(cx[b].shape, device=dev, dtype=torch.float64)
                    for i in range(8):
                        for j in range(8):
                            ref = mid[by[b] + i, bx[b] + j]
                            acc += _score(ref[:, None] - flat[(py[b] + i) * w + px[b] + j], case["metric"])
                    d[b] = acc
                d = torch.where(ok, d, d.new_tensor(math.inf))
                fe, k = torch.sort(d, dim=1, stable=True)
                fe, k = fe[:, :PS_NUM], k[:, :PS_NUM]
                lx, ly = cx.gather(1, k), cy.gather(1, k)
                ge, k = torch.sort(torch.cat([ge, fe], 1), dim=1, stable=True)
                ge, k = ge[:, :8], k[:, :8]
                gx = torch.cat([gx, lx], 1).gather(1, k)
                gy = torch.cat([gy, ly], 1).gather(1, k)
                gz = torch.cat([gz, torch.full_like(lx, z)], 1).gather(1, k)
    # the block itself is always in its group
    absent = ~((gx == bx[:, None]) & (gy == by[:, None]) & (gz == r)).any(1, keepdim=True)
    at = torch.where(absent, (i8 - 1).clamp(min=0), i8)
    own = absent & (i8 == 0)
    return (torch.where(own, bx[:, None], gx.gather(1, at)), torch.where(own, by[:, None], gy.gather(1, at)),
            torch.where(own, torch.full_like(gz, r), gz.gather(1, at)))


def _filter64(clips, case, final):
    """Accumulators (num, den) [planes][tw][h][w] of one pass over [clips][planes][tw][h][w] in float64."""
    nplanes, tw, h, w = clips.shape[1:]
    lx, ly, lz = _match64(clips[0, 0], case)
    f2, i2 = (torch.from_numpy(np.ascontiguousarray(m)).to(clips.device) for m in _transform(case["t2d"]))
    f1, i1 = (torch.from_numpy(np.ascontiguousarray(m)).to(clips.device) for m in _transform(case["t1d"]))
    sigma = case["sigma"] * (WIENER_FACTOR if final else HARD_FACTOR)
    num = torch.zeros((nplanes, tw * h * w), device=clips.device, dtype=torch.float64)
    den = torch.zeros_like(num)
    i8 = torch.arange(8, device=clips.device)
    inside = i8[:, None] * w + i8[None, :]

    def forward(g):
        return torch.einsum("pq,rs,ct,nqst->nprc", f1, f2, f2, g)

    for a in range(0, len(lx), 16384):
        at = ((lz[a:a + 16384] * h + ly[a:a + 16384]) * w + lx[a:a + 16384])[:, :, None, None] + inside
        for p in range(nplanes):
            g = forward(clips[-1, p].reshape(-1)[at])
            if final:
                b = forward(clips[0, p].reshape(-1)[at]).square()
                c = b / (b + sigma * sigma)
                c[:, 0, 0, 0] = 1.0
                weight = 1.0 / c.square().sum((1, 2, 3))
            else:
                c = (g.abs() >= sigma).double()
                c[:, 0, 0, 0] = 1.0
                weight = 1.0 / c.sum((1, 2, 3))
            g = torch.einsum("qp,sr,tc,nprc->nqst", i1, i2, i2, g * c / 4096.0)
            num[p].index_add_(0, at.reshape(-1), (g * weight[:, None, None, None]).reshape(-1))
            den[p].index_add_(0, at.reshape(-1), weight[:, None, None, None].expand_as(g).reshape(-1))
    return num.view(nplanes, tw, h, w), den.view(nplanes, tw, h, w)


def _entries(case):
    """Plane numbers of each separately filtered entry."""
    n = len(_planes_of(case))
    return [list(range(n))] if case["chroma"] else [[p] for p in range(n)]


def _window64(case, noisy, basic, final):
    out = []
    for planes in _entries(case):
        clips = torch.stack([torch.stack([c[p] for p in planes]) for c in ([basic, noisy] if final else [noisy])])
        num, den = _filter64(clips.double(), case, final)
        out.append((num / den)[:, 0] if case["radius"] == 0 else torch.stack([num, den], 2))
    return out


def _twopass64(case, noisy):
    first = _window64(case, noisy, None, False)
    second = _window64(case, noisy, [f for f in first], True)
    return first, second


def _network64(state, noisy, sigma):
    """The network with these weights in float64: (weights, biases, estimate)."""
    layers = 7
    ws = [torch.from_numpy(state["w%d" % l]).double().cuda().requires_grad_(True) for l in range(layers)]
    bs = [torch.from_numpy(state["b%d" % l]).double().cuda().requires_grad_(True) for l in range(layers)]
    x = torch.zeros((len(noisy), 16) + tuple(noisy.shape[1:]), device=noisy.device, dtype=torch.float64)
    x[:, 0] = noisy.double()
    x[:, 1] = (sigma.double() / 255.0 * P.LEVEL_SCALE)[:, None, None]
    for l, (w, b) in enumerate(zip(ws, bs)):
        x = torch.nn.functional.conv2d(x, w.permute(0, 3, 1, 2), b, padding=1)
        if l < layers - 1:
            x = x.relu()
    return ws, bs, noisy.double() + x[:, 0]


def exact(case, seed):
    kind = case["kind"]
    if kind == "window":
        noisy, basic = _frames(case, seed, 2 * case["radius"] + 1)
        return _window64(case, noisy, basic, case["final"])
    if kind == "twopass":
        noisy, _ = _frames(case, seed, 1)
        first, second = _twopass64(case, noisy)
        return [v[0] for pair in zip(first, second) for v in pair]
    if kind == "fused":
        r = case["radius"]
        tw = 2 * r + 1
        noisy, _ = _frames(case, seed, 4 * r + 1)
        acc, last = 0.0, None
        for m in range(tw):  # the window around frame m + r holds the output frame 2 r in its slot 2 r - m
            num, den = _filter64(noisy[0][None, None, m:m + tw].double(), case, False)
            acc = acc + torch.stack([num[0, 2 * r - m], den[0, 2 * r - m]])
            last = torch.stack([num[0], den[0]], 1)
        return [acc[0] / acc[1], last]
    if kind == "batch":
        out = []
        for i, c in enumerate(_batch_cases(case)):
            noisy, basic = _frames(c, seed + 100 * i, 2 * c["radius"] + 1)
            out.append(_window64(c, noisy, basic, False))
        return out
    if kind == "host":
        noisy, _ = _frames(case, seed, case["frames"])
        out = []
        for i in range(case["frames"]):
            _, second = _twopass64(case, [p[i:i + 1] for p in noisy])
            out.append([p[0].cpu() for p in second])
        return out
    noisy, target, sigma = _network_inputs(case, seed)
    if kind == "pilot":
        with torch.no_grad(), np.load(P.WEIGHTS) as f:
            return _network64(f, noisy, sigma)[2]
    ws, bs, y = _network64(_initial_state(seed), noisy, sigma)
    loss = (y - target.double()).square().mean()
    grads = torch.autograd.grad(loss * P.LOSS_SCALE, ws + bs)
    return {"dw": list(grads[:len(ws)]), "db": list(grads[len(ws):]), "loss": float(loss.detach()), "y": y.detach()}
