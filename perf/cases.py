"""The work that users of the front-end give it, through its public entry points.

One camera (host u8 frames, the reference's host f32 frames, frames already in
device memory), feature sets kept and matched by the caller, batches from host
frames and over resident frames (one size, many sizes, the cfg profile, 4K
brute force), the served form, RANSAC scoring and triangulation.  Sizes are
those of the benchmark, the tests and the smoke check, and odd ones.

Frames are seeded scenes of the benchmark's recipe (rectangles, checkerboards,
noise; a warped second view, or a camera moving over a textured plane), drawn
here on the GPU because 3840x2160 scenes take seconds on the host.  The BRIEF
table is an input of the library; a seeded Gaussian table of the same reach
stands in for a caller's.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from uni_slam_gb300 import Batch, Context, FeatureSet, Frontend, Server, capi, synth
from uni_slam_gb300.capi import FEATURE_DTYPE, MATCH_DTYPE, iptr, ptr

# frames of the mixed batch: the benchmark's uneven workload, (width, height, pairs)
MIXED = ((640, 480, 16), (752, 480, 16), (1280, 720, 8), (1920, 1080, 4), (3840, 2160, 2))
SERVED = ((640, 480), (752, 480), (1280, 720))


def listed():
    return [
        # the smallest call: a low-resolution camera tracked frame by frame against its keyframe
        {"name": "stream_320x240_u8", "kind": "stream", "w": 320, "h": 240, "levels": 6, "source": "u8"},
        # the drop-in path: EuRoC-sized frames as the reference holds them (f32 u8 / 255)
        {"name": "stream_752x480_f32", "kind": "stream", "w": 752, "h": 480, "levels": 6, "source": "f32"},
        # a full-HD camera whose frames a decoder leaves in device memory
        {"name": "stream_1920x1080_device", "kind": "stream", "w": 1920, "h": 1080, "levels": 6, "source": "device"},
        # a caller that keeps its own feature sets: two frames detected, then matched; odd size
        {"name": "sets_637x479", "kind": "sets", "w": 637, "h": 479, "levels": 6},
        # an offline run over host frames in small batches: upload, work, download, read
        {"name": "batch_12x640x480_host", "kind": "host_batch", "w": 640, "h": 480, "levels": 6, "frames": 12},
        # the headline workload: 64 consecutive resident frames, consecutive pairs
        {"name": "batch_64x752x480", "kind": "batch", "w": 752, "h": 480, "levels": 6, "frames": 64},
        # many cameras of different sizes in one work table, per-cell caps
        {"name": "batch_mixed", "kind": "mixed", "levels": 6, "cell_cap": 8, "scale": 1.0},
        # the cfg profile (FAST 9-of-16 with NMS) with the brute-force matcher on the integer pipes
        {"name": "cfg_16x752x480", "kind": "cfg", "w": 752, "h": 480, "levels": 6, "frames": 16, "matcher": 1},
        # 4K frames, 20000 features each, brute force on the tensor cores
        {"name": "stress_3840x2160", "kind": "stress", "w": 3840, "h": 2160, "levels": 8, "pairs": 4,
         "frame_cap": 20000, "matcher": 2},
        # one frame from each of 16 served cameras at the same moment
        {"name": "served_16", "kind": "served", "streams": 16, "levels": 6, "cap": 333},
        # the step after matching: hypotheses scored over a pair's matches
        {"name": "ransac_500x1640", "kind": "ransac", "hyps": 500, "matches": 1640, "masks": True},
        # the step after that: two-view triangulation of several pairs at once
        {"name": "triangulate_8x1500", "kind": "triangulate", "pairs": 8, "rows": 1500},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _size(rng, lo, hi):
    w = _log(rng, lo, hi)
    return w, max(48, int(w * rng.uniform(0.5, 0.8)))


def draw(rng):
    kind = rng.choice(["stream", "stream", "sets", "host_batch", "batch", "batch", "mixed", "cfg", "stress", "served",
                       "ransac", "triangulate"])
    if kind == "stream":
        w, h = _size(rng, 96, 1920)
        return {"kind": kind, "w": w, "h": h, "levels": rng.choice([4, 6, 8]),
                "source": rng.choice(["u8", "f32", "device"])}
    if kind == "sets":
        w, h = _size(rng, 96, 1920)
        return {"kind": kind, "w": w, "h": h, "levels": rng.choice([4, 6, 8])}
    if kind == "host_batch":
        w, h = _size(rng, 160, 1280)
        return {"kind": kind, "w": w, "h": h, "levels": 6, "frames": rng.randint(2, 12)}
    if kind == "batch":
        w, h = _size(rng, 200, 1000)
        most = max(2, min(96, int(64 * 752 * 480 / (w * h))))
        return {"kind": kind, "w": w, "h": h, "levels": 6, "frames": _log(rng, 2, most)}
    if kind == "mixed":
        return {"kind": kind, "levels": 6, "cell_cap": rng.choice([0, 4, 8]), "scale": round(rng.uniform(0.3, 0.95), 3)}
    if kind == "cfg":
        w, h = _size(rng, 200, 800)
        return {"kind": kind, "w": w, "h": h, "levels": 6, "frames": rng.randint(2, 16), "matcher": rng.choice([1, 2])}
    if kind == "stress":
        w, h = _size(rng, 1000, 3200)
        return {"kind": kind, "w": w, "h": h, "levels": 8, "pairs": rng.randint(1, 4),
                "frame_cap": _log(rng, 2000, 20000), "matcher": rng.choice([1, 2])}
    if kind == "served":
        return {"kind": kind, "streams": rng.randint(1, 32), "levels": 6, "cap": rng.choice([200, 333, 500])}
    if kind == "ransac":
        return {"kind": kind, "hyps": _log(rng, 20, 2000), "matches": _log(rng, 16, 4000), "masks": rng.random() < 0.5}
    return {"kind": "triangulate", "pairs": rng.randint(1, 12), "rows": _log(rng, 12, 2500)}


# ------------------------------------------------------------------- inputs

def _pattern():
    rs = np.random.RandomState(256)
    p = np.clip(np.rint(rs.normal(0.0, 6.2, (256, 4))), -13, 13).astype(np.int32)
    p[0] = (13, 13, -13, -13)  # the reach of a 31 x 31 patch rotated
    return p


def _sub(seed, i):
    return (seed * 1009 + i) % (1 << 32)


def _inliers(seed, n, outliers=0.0):
    """n correspondences of a two-view scene as (prev_x, prev_y, curr_x, curr_y)."""
    rows = synth.two_view_scene(seed, n, outlier_frac=outliers)[0][:, 1:5].astype(np.float64)
    return np.ascontiguousarray(rows[np.arange(n) % len(rows)])


def _content(rs, w, h, rects, checks):
    img = np.full((h, w), 128.0, np.float32)
    size = rs.randint(8, 81, (rects, 2))
    val = rs.randint(0, 256, rects)
    at = rs.random_sample((rects, 2))
    for (rw, rh), v, (u, t) in zip(size, val, at):
        x, y = int(u * w) - rw // 2, int(t * h) - rh // 2
        img[max(y, 0):max(y + rh, 0), max(x, 0):max(x + rw, 0)] = v
    for _ in range(checks):
        cell = rs.randint(2, 7)
        side = 8 * cell
        x, y = rs.randint(-side // 2, w - side // 2), rs.randint(-side // 2, h - side // 2)
        v = rs.randint(0, 256, 2).astype(np.float32)
        k = np.arange(side) // cell
        board = v[(k[:, None] + k[None, :]) & 1]
        xs, ys, xe, ye = max(x, 0), max(y, 0), min(x + side, w), min(y + side, h)
        if xe > xs and ye > ys:
            img[ys:ye, xs:xe] = board[ys - y:ye - y, xs - x:xe - x]
    return torch.from_numpy(img).cuda()


def _counts(w, h):
    f = w * h / (752.0 * 480.0)
    return max(4, round(200 * f)), max(2, round(50 * f))


def _noise(gen, w, h, sigma, smooth):
    n = torch.randn(h, w, device="cuda", generator=gen) * sigma
    if smooth:
        k = [math.exp(-0.5 * i * i) for i in range(-3, 4)]
        s = sum(k)
        for axis in (0, 1):
            n = sum(torch.roll(n, i - 3, axis) * (v / s) for i, v in enumerate(k))
    return n


def _view(img, w, h, cx, cy, ang, scale):
    """The w x h view of img whose pixel (x, y) looks at the centre (cx, cy) + scale R(ang) (x - w / 2, y - h / 2)."""
    H, W = img.shape
    yy, xx = torch.meshgrid(torch.arange(h, device="cuda", dtype=torch.float32) - (h - 1) / 2,
                            torch.arange(w, device="cuda", dtype=torch.float32) - (w - 1) / 2, indexing="ij")
    c, s = math.cos(ang) * scale, math.sin(ang) * scale
    u, v = cx + c * xx - s * yy, cy + s * xx + c * yy
    grid = torch.stack([2 * u / (W - 1) - 1, 2 * v / (H - 1) - 1], -1)[None]
    return torch.nn.functional.grid_sample((img - 128.0)[None, None], grid, align_corners=True)[0, 0] + 128.0


def _u8(img):
    return img.round().clamp(0, 255).to(torch.uint8)


def _pair(seed, w, h, rects=None, checks=None):
    """A frame and a view of it turned up to 5 degrees, moved up to 10 pixels and scaled up to 3 %."""
    rs = np.random.RandomState(seed)
    nr, nc = _counts(w, h)
    img = _content(rs, w, h, rects or nr, checks or nc)
    gen = torch.Generator("cuda").manual_seed(seed)
    dx, dy = rs.uniform(-10, 10, 2)
    second = _view(img, w, h, (w - 1) / 2 + dx, (h - 1) / 2 + dy, math.radians(rs.uniform(-5, 5)), rs.uniform(0.97, 1.03))
    return _u8(img + _noise(gen, w, h, 4.0, True)), _u8(second + _noise(gen, w, h, 4.0, True))


def _sequence(seed, n, w, h):
    """A camera moving over a textured plane: 5 to 12 texels and 0.5 to 2 degrees a frame."""
    rs = np.random.RandomState(seed)
    side = max(2048, 2 * max(w, h) + 24 * n)
    tex = _content(rs, side, side, *_counts(side, side))
    gen = torch.Generator("cuda").manual_seed(seed)
    cx = cy = side / 2
    ang, way = rs.uniform(0, 2 * math.pi), rs.uniform(0, 2 * math.pi)
    frames = []
    for _ in range(n):
        frames.append(_u8(_view(tex, w, h, cx, cy, ang, 1.087) + _noise(gen, w, h, 3.0, False)))
        way += rs.uniform(-0.3, 0.3)
        step = rs.uniform(5, 12)
        cx, cy, ang = cx + step * math.cos(way), cy + step * math.sin(way), ang + math.radians(rs.uniform(0.5, 2))
    return frames


class _Handles:
    """The library's handles of one program, given back in reverse order with their last holder."""

    def __init__(self):
        self.held = []

    def __del__(self):
        for handle in reversed(self.held):
            handle.close()


class _DeviceBytes:
    """Device memory of a batch, for torch.as_tensor, whose tensor keeps this object and so the batch."""

    def __init__(self, address, nbytes, handles):
        self.handles = handles
        self.__cuda_array_interface__ = {"shape": (nbytes // 4,), "typestr": "<i4", "data": (address, False),
                                         "version": 3}


class _State:
    """What a program holds between calls."""

    def __init__(self, kind):
        self.kind, self.handles = kind, _Handles()

    def own(self, handle):
        self.handles.held.append(handle)
        return handle


def _resident(s, sizes, pairs, frames, **options):
    """A batch with its frames in device memory, and its outputs (counts, features, matches) as they lie there: the
    region behind the inputs that download() copies out."""
    ctx = s.own(Context(_pattern(), max_width=max(w for w, _ in sizes), max_height=max(h for _, h in sizes), **options))
    s.batch = s.own(Batch(ctx, sizes, pairs))
    for i, f in enumerate(frames):
        s.batch.set_frame(i, f.cpu().numpy())
    s.batch.upload()
    s.batch.sync()
    h2d, d2h = s.batch.io_bytes()
    s.out = torch.as_tensor(_DeviceBytes(s.batch.input_device(0)[0] + h2d, d2h, s.handles), device="cuda")


class _Read:
    """Buffers a caller reads features and matches into through the C ABI, sized for the largest result."""

    def __init__(self, ctx, case, frames, pairs):
        rows = max(1, case["levels"] * (case["w"] * case["h"] // 250))
        self.check, self.lib = ctx.check, capi.load()
        self.feats, self.match = np.zeros((frames, rows), FEATURE_DTYPE), np.zeros((pairs, rows), MATCH_DTYPE)
        self.kept, self.raw = np.zeros((frames, case["levels"]), np.int32), np.zeros((frames, case["levels"]), np.int32)
        self.n = np.zeros(pairs, np.int32)

    def features(self, name, *who, at=0):
        f = self.feats[at]
        self.check(getattr(self.lib, name)(*who, ptr(f), len(f), iptr(self.kept[at]), iptr(self.raw[at])), name)

    def matches(self, name, *who, at=0):
        m = self.match[at]
        self.check(getattr(self.lib, name)(*who, ptr(m), len(m), iptr(self.n[at:])), name)

    def out(self):
        return {"features": self.feats.view(np.int32), "kept": self.kept, "raw": self.raw,
                "matches": self.match.view(np.int32), "n": self.n}


def _mixed_sizes(case):
    return [(max(64, int(w * case["scale"])), max(48, int(h * case["scale"])), n) for w, h, n in MIXED]


def _served_sizes(case):
    return [SERVED[(7 * i) % 3] for i in range(case["streams"])]


def prepare(case, seed):
    kind, s = case["kind"], _State(case["kind"])
    if kind == "stream":
        w, h = case["w"], case["h"]
        key, frame = _pair(seed, w, h)
        ctx = s.own(Context(_pattern(), levels=case["levels"], max_width=w, max_height=h))
        s.front, s.source = s.own(Frontend(ctx, w, h)), case["source"]
        s.read = _Read(ctx, case, 1, 1)
        s.front.process(key.cpu().numpy())
        s.device = frame.contiguous()
        s.frame = frame.cpu().numpy()
        if s.source == "f32":
            s.frame = s.frame.astype(np.float32) / np.float32(255)
        s.front.process(frame.cpu().numpy())  # the key frame is the reference set from here on
    elif kind == "sets":
        w, h = case["w"], case["h"]
        s.frames = [f.cpu().numpy() for f in _pair(seed, w, h)]
        s.ctx = s.own(Context(_pattern(), levels=case["levels"], max_width=w, max_height=h))
        s.read = _Read(s.ctx, case, 1, 1)
        s.sets = [s.own(FeatureSet(s.ctx, w, h)) for _ in range(2)]
    elif kind == "host_batch":
        w, h, n = case["w"], case["h"], case["frames"]
        s.frames = [f.cpu().numpy() for f in _sequence(seed, n, w, h)]
        ctx = s.own(Context(_pattern(), levels=case["levels"], max_width=w, max_height=h))
        s.batch = s.own(Batch(ctx, [(w, h)] * n, [(i, i + 1) for i in range(n - 1)]))
        s.read = _Read(ctx, case, n, n - 1)
    elif kind == "batch":
        w, h, n = case["w"], case["h"], case["frames"]
        _resident(s, [(w, h)] * n, [(i, i + 1) for i in range(n - 1)], _sequence(seed, n, w, h), levels=case["levels"])
    elif kind == "mixed":
        frames = []
        for k, (w, h, n) in enumerate(_mixed_sizes(case)):
            for i in range(n):
                frames += _pair(_sub(seed, 40 * k + i), w, h)
        sizes = [(f.shape[1], f.shape[0]) for f in frames]
        _resident(s, sizes, [(2 * i, 2 * i + 1) for i in range(len(frames) // 2)], frames, levels=case["levels"],
                  cell_cap=case["cell_cap"])
    elif kind == "cfg":
        w, h, n = case["w"], case["h"], case["frames"]
        _resident(s, [(w, h)] * n, [(i, i + 1) for i in range(n - 1)], _sequence(seed, n, w, h), levels=case["levels"],
                  detector=1, matcher=case["matcher"], ratio=0.8)
    elif kind == "stress":
        w, h, cap = case["w"], case["h"], case["frame_cap"]
        f = w * h / (3840.0 * 2160.0)
        frames = []
        for i in range(case["pairs"]):
            frames += _pair(_sub(seed, i), w, h, max(50, round(5000 * f)), max(10, round(500 * f)))
        _resident(s, [(w, h)] * len(frames), [(2 * i, 2 * i + 1) for i in range(case["pairs"])], frames,
                  levels=case["levels"], cap_per_level=cap, frame_cap=cap, matcher=case["matcher"], ratio=0.8)
    elif kind == "served":
        sizes = _served_sizes(case)
        n, rows = len(sizes), case["cap"] * case["levels"]
        views = [_pair(_sub(seed, i), w, h) for i, (w, h) in enumerate(sizes)]
        ctx = s.own(Context(_pattern(), levels=case["levels"], max_width=1280, max_height=720, cap_per_level=case["cap"]))
        s.server = s.own(Server(ctx, list(SERVED), hbm_budget_bytes=6 << 30, max_batch=64))
        s.streams = [s.server.open_stream(w, h) for w, h in sizes]
        for sid, (key, _) in zip(s.streams, views):
            t = s.server.submit(sid, key.cpu().numpy())
            s.server.wait(t)
            s.server.release(t)
        s.frames = [f.cpu().numpy() for _, f in views]
        s.feats, s.matches = np.zeros((n, rows), FEATURE_DTYPE), np.zeros((n, rows), MATCH_DTYPE)
        s.kept, s.raw = np.zeros((n, case["levels"]), np.int32), np.zeros((n, case["levels"]), np.int32)
    elif kind == "ransac":
        n, m = case["matches"], case["hyps"]
        rows = _inliers(seed, n, 0.2)
        s.prev, s.curr = np.ascontiguousarray(rows[:, :2]), np.ascontiguousarray(rows[:, 2:])
        rng = np.random.default_rng(seed)
        at = rng.integers(0, len(rows), (m, 8))
        p, q = s.prev[at], s.curr[at]
        one = np.ones((m, 8, 1))
        a = np.concatenate([q[..., 0:1] * p, q[..., 0:1], q[..., 1:2] * p, q[..., 1:2], p, one], 2)
        s.fmats = np.ascontiguousarray(np.linalg.svd(a)[2][:, -1])
        s.ctx, s.masks = s.own(Context(_pattern(), max_width=752, max_height=480)), case["masks"]
    else:
        s.px = [_inliers(_sub(seed, i), case["rows"]) for i in range(case["pairs"])]
        s.cam = synth.SCENE_CAMERA
        s.ctx = s.own(Context(_pattern(), max_width=752, max_height=480))
    return s


# --------------------------------------------------------------------- runs

def run(s):
    if s.kind == "stream":
        if s.source == "u8":
            s.front.process(s.frame)
        elif s.source == "f32":
            s.front.process_f32(s.frame)
        else:
            s.front.enqueue(s.device.data_ptr(), s.device.shape[1])
            s.front.sync()
        s.read.features("uslam_frontend_features", s.front.h, 0)
        s.read.matches("uslam_frontend_matches", s.front.h)
        return s.read.out()
    if s.kind == "sets":
        for fs, f in zip(s.sets, s.frames):
            fs.detect(f)
        s.read.features("uslam_featset_features", s.sets[1].h)
        s.read.matches("uslam_match_sets", s.ctx.h, s.sets[0].h, s.sets[1].h)
        return s.read.out()
    if s.kind == "host_batch":
        s.batch.process(s.frames)
        for i in range(len(s.frames)):
            s.read.features("uslam_batch_features", s.batch.h, i, at=i)
        for p in range(len(s.frames) - 1):
            s.read.matches("uslam_batch_matches", s.batch.h, p, at=p)
        return s.read.out()
    if s.kind in ("batch", "mixed", "cfg", "stress"):
        s.batch.run()
        s.batch.sync()
        return s.out
    if s.kind == "served":
        tickets = [s.server.submit(sid, f) for sid, f in zip(s.streams, s.frames)]
        for i, t in enumerate(tickets):
            s.server.wait(t)
            s.server.result_into(t, s.feats[i], s.matches[i], s.kept[i], s.raw[i])
            s.server.release(t)
        return {"features": s.feats.view(np.int32), "matches": s.matches.view(np.int32), "kept": s.kept, "raw": s.raw}
    if s.kind == "ransac":
        got = s.ctx.ransac_score(s.fmats, s.prev, s.curr, 3.84, masks=s.masks)
        return {"counts": got[0], "masks": got[1].view(np.int32)} if s.masks else {"counts": got}
    return _poses(s.ctx.triangulate(s.px, s.cam))


def _poses(got):
    """One row per pair of what triangulation returns, and each pair's landmarks."""
    return {"rotation": np.stack([r["rotation"] for r in got]), "translation": np.stack([r["translation"] for r in got]),
            "stats": np.array([[r["mean_reprojection_error_px"], r["rotation_angle_rad"]] for r in got]),
            "counts": np.array([[r["input_matches"], r["landmark_count"], r["cheirality_passes"], r["pose_recovered"]]
                                for r in got], np.int64),
            "landmarks": [r["landmarks"] for r in got], "keep": [r["keep"] for r in got]}


# --------------------------------------------------------------------- work

def _frame_work(w, h, levels, cap):
    """(bytes, operations, features) of detecting and describing one u8 frame: the frame read, the records written; a
    tap a pyramid pixel, the circle test, and the blurred samples (a sample a pixel or 512 a feature, where fewer)."""
    px = sum(int(w / 1.2 ** l) * int(h / 1.2 ** l) for l in range(levels))
    feats = 0.9 * levels * cap
    return w * h + 48 * feats, 24 * px + 90 * min(px, 512 * feats) + 12 * 512 * feats, feats


def work(case):
    kind = case["kind"]
    if kind in ("stream", "sets", "host_batch", "batch", "mixed", "cfg", "stress", "served"):
        levels = case["levels"]
        if kind == "mixed":
            frames = [(w, h, 0) for w, h, n in _mixed_sizes(case) for _ in range(2 * n)]
            pairs = len(frames) // 2
        elif kind == "served":
            frames = [(w, h, case["cap"]) for w, h in _served_sizes(case)]
            pairs = len(frames)
        else:
            n = {"stream": 1, "sets": 2, "stress": 2 * case.get("pairs", 0)}.get(kind) or case["frames"]
            frames = [(case["w"], case["h"], case.get("frame_cap", 0) / levels)] * n
            pairs = {"stream": 1, "sets": 1, "stress": case.get("pairs", 0)}.get(kind) or n - 1
        b = f = feats = 0.0
        for w, h, cap in frames:
            fb, ff, fn = _frame_work(w, h, levels, cap or w * h / 250)
            b, f, feats = b + fb * (4 if kind == "stream" and case["source"] == "f32" else 1), f + ff, feats + fn
        feats /= len(frames)
        # a distance is 512 operations; the window holds 4 % of three levels' features
        dist = feats * feats if kind in ("cfg", "stress") else feats * feats / levels * 3 * 0.04
        return {"bytes": b + pairs * (64 * feats + 16 * feats / 5), "flops": f + pairs * 512 * dist}
    if kind == "ransac":
        h, n = case["hyps"], case["matches"]
        return {"bytes": 72 * h + 32 * n + 4 * h + (h * n / 8 if case["masks"] else 0), "flops": 40.0 * h * n}
    n = case["pairs"] * case["rows"]
    # undistortion, the 9 x 9 normal matrix, four 4 x 4 null vectors and the filter of a row
    return {"bytes": 73.0 * n, "flops": n * (2 * 6 * 30 + 2 * 45 + 4 * 400 + 100.0)}


# -------------------------------------------------------------------- exact

def exact(case, seed):
    """Triangulation in numpy (binary64, LAPACK singular value decompositions); every other result is whole numbers."""
    if case["kind"] != "triangulate":
        return None
    return _poses([_triangulate(_inliers(_sub(seed, i), case["rows"]), synth.SCENE_CAMERA) for i in range(case["pairs"])])


def _distort(x, y, cam):
    r2 = x * x + y * y
    rad = 1 + cam[4] * r2 + cam[5] * r2 * r2
    return rad, 2 * cam[6] * x * y + cam[7] * (r2 + 2 * x * x), cam[6] * (r2 + 2 * y * y) + 2 * cam[7] * x * y


def _rays(px, cam):
    x0, y0 = (px[:, 0] - cam[2]) / cam[0], (px[:, 1] - cam[3]) / cam[1]
    x, y, live = x0.copy(), y0.copy(), np.ones(len(px), bool)
    for _ in range(20):
        rad, dx, dy = _distort(x, y, cam)
        nx, ny = np.where(live, (x0 - dx) / rad, x), np.where(live, (y0 - dy) / rad, y)
        live &= np.hypot(nx - x, ny - y) >= 1e-9
        x, y = nx, ny
    return np.stack([x, y], 1)


def _hartley(p):
    c = p.mean(0)
    s = math.sqrt(2) / np.linalg.norm(p - c, axis=1).mean()
    return np.array([[s, 0, -s * c[0]], [0, s, -s * c[1]], [0, 0, 1]])


def _project(p, cam):
    x, y = p[:, 0] / p[:, 2], p[:, 1] / p[:, 2]
    rad, dx, dy = _distort(x, y, cam)
    return np.stack([cam[0] * (x * rad + dx) + cam[2], cam[1] * (y * rad + dy) + cam[3]], 1)


def _triangulate(px, cam):
    n = len(px)
    p, q = _rays(px[:, :2], cam), _rays(px[:, 2:], cam)
    tp, tq = _hartley(p), _hartley(q)
    a, b = p @ tp[:2, :2] + tp[:2, 2], q @ tq[:2, :2] + tq[:2, 2]
    one = np.ones((n, 1))
    rows = np.concatenate([b[:, :1] * a, b[:, :1], b[:, 1:] * a, b[:, 1:], a, one], 1)
    u, w, vt = np.linalg.svd(np.linalg.svd(rows)[2][8].reshape(3, 3)) if n < 2000 else \
        np.linalg.svd(np.linalg.svd(np.linalg.qr(rows, "r"))[2][8].reshape(3, 3))
    e = tq.T @ (u @ np.diag([(w[0] + w[1]) / 2] * 2 + [0]) @ vt) @ tp
    u, _, vt = np.linalg.svd(e)
    u[:, 2] *= np.linalg.det(u)
    vt[2] *= np.linalg.det(vt)
    turn = np.array([[0.0, -1, 0], [1, 0, 0], [0, 0, 1]])
    best, found = -1, None
    for r in (u @ turn @ vt, u @ turn.T @ vt):
        for t in (u[:, 2], -u[:, 2]):
            m = np.zeros((n, 4, 4))
            m[:, 0, 0] = m[:, 1, 1] = -1
            m[:, :2, 2] = p
            cam2 = np.concatenate([r, t[:, None]], 1)
            m[:, 2:] = q[:, :, None] * cam2[2] - cam2[:2]
            x = np.linalg.svd(m)[2][:, 3]
            near = x[:, :3] / x[:, 3:]
            far = near @ r.T + t
            front = int(((near[:, 2] > 0) & (far[:, 2] > 0)).sum())
            if front > best:
                best, found = front, (r, t, near, far)
    r, t, near, far = found
    z = np.stack([near[:, 2], far[:, 2]], 1)
    ok = ((z >= 1e-3) & (z <= 1e3)).all(1)
    err = np.full(n, np.inf)
    err[ok] = (np.linalg.norm(_project(near[ok], cam) - px[ok, :2], axis=1)
               + np.linalg.norm(_project(far[ok], cam) - px[ok, 2:], axis=1)) / 2
    ok &= err <= 4.0
    lm = np.zeros((n, 4))
    lm[ok] = np.concatenate([far[ok], err[ok, None]], 1)
    return {"rotation": r, "translation": t, "input_matches": n, "landmark_count": int(ok.sum()),
            "cheirality_passes": best, "pose_recovered": bool(ok.any()), "keep": ok, "landmarks": lm,
            "mean_reprojection_error_px": float(err[ok].mean()) if ok.any() else 0.0,
            "rotation_angle_rad": math.acos(min(max((np.trace(r) - 1) / 2, -1), 1))}
