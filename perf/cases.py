"""The work that an encoder or decoder built on this framework has it do, as cases to time.

Each case is one pass through the public entry points (the classes of ``imagecodingutils_gb300`` or the C ABI they
wrap) on inputs of the repository's own kind: smooth textures under a quarter-pel pan with moving objects and sensor
noise (synth.py's sequences, made here on the GPU), Laplacian residuals, and natural-looking colour planes.  Resolutions
are those of the benchmark (QCIF, CIF, 720p, 1080p, 4K) and ragged ones between them.  Everything the library computes
is whole numbers, so no case has a 64-bit reference of its own.

  me      frame pairs of a sequence through one estimator handle, device planes (vppgpu_me_estimate_device)
  host    the drop-in class on host planes, as a codec written against the reference calls it (Estimate())
  coded   a mixed-resolution batch with its coding stage (MotionEstimatorBatch: vectors, residual, levels, recon)
  tq      forward transform + quantisation and its inverse over the planes of 4:2:0 frames, one launch
  rgb2yuv / yuv2rgb   capture-side and display-side colour conversion of frames
  mc      decoder-side motion compensation of 4:2:0 frames
"""
import ctypes as C
import math
import random

import torch

import imagecodingutils_gb300 as vpp
from imagecodingutils_gb300 import _lib

ESTIMATORS = {"full": _lib.ME_FULL, "full_sad": _lib.ME_FULL_SAD, "multires": _lib.ME_MULTIRES,
              "multires_cross": _lib.ME_MULTIRES_CROSS, "multires_cross_v2": _lib.ME_MULTIRES_CROSS_V2}
MIX = [(176, 144), (352, 288), (1280, 720), (1920, 1080), (3840, 2160)]
DEV = "cuda"


def listed():
    return [
        # the smallest call: one QCIF frame of the integer-pel SAD search, +-16 pels (video telephony)
        {"name": "sad_qcif", "path": "me", "est": "full_sad", "w": 176, "h": 144, "range": 64, "pairs": 1},
        # a codec's unchanged call on host planes, CIF, +-32 pels
        {"name": "full_cif_host", "path": "host", "est": "full", "w": 352, "h": 288, "range": 128, "pairs": 1},
        # the headline: full-search quarter-pel estimation of a 1080p sequence, planes on the device
        {"name": "full_1080p", "path": "me", "est": "full", "w": 1920, "h": 1080, "range": 128, "pairs": 8},
        # the pyramid full search with the predictor, 1080p
        {"name": "multires_1080p", "path": "me", "est": "multires", "w": 1920, "h": 1080, "range": 128, "pairs": 4},
        # the cross pyramid without and with the predictor: 720p, and a ragged window-sized source
        {"name": "cross_720p", "path": "me", "est": "multires_cross", "w": 1280, "h": 720, "range": 128, "pairs": 8},
        {"name": "cross_v2_ragged", "path": "me", "est": "multires_cross_v2", "w": 848, "h": 478, "range": 96,
         "pairs": 4},
        # a transcoder's tick: sequences of every resolution estimated and coded together (the largest case)
        {"name": "coded_mix", "path": "coded", "largest": 4, "seqs": 10, "pairs": 3, "qp": 28},
        # the residual round trip of 16 1080p frames in one launch
        {"name": "tq_1080p", "path": "tq", "w": 1920, "h": 1080, "frames": 16, "qp": 28, "intra": 0},
        # the same for a few small intra frames, sizes that are no multiple of 16
        {"name": "tq_small", "path": "tq", "w": 712, "h": 488, "frames": 4, "qp": 35, "intra": 1},
        # capture: 16 RGB frames to YUV 4:2:0; display: 16 frames back
        {"name": "rgb2yuv_1080p", "path": "rgb2yuv", "kind": _lib.RGB_FIXED_POINT, "w": 1920, "h": 1080, "frames": 16},
        {"name": "yuv2rgb_1080p", "path": "yuv2rgb", "kind": _lib.YUV_REAL_IMPL2, "w": 1920, "h": 1080, "frames": 16},
        # a decoder's motion compensation, frame after frame
        {"name": "mc_1088p", "path": "mc", "w": 1920, "h": 1088, "frames": 8},
    ]


def _log_size(rng, lo, hi, step):
    return max(step, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))) / step)) * step)


def draw(rng):
    path = rng.choice(["me", "me", "me", "me", "host", "coded", "tq", "rgb2yuv", "yuv2rgb", "mc"])
    w = _log_size(rng, 176, 3840, 16)
    h = max(96, min(2160, int(w * rng.uniform(0.45, 0.8))))
    most = max(1, min(8, 16588800 // (w * h)))  # frames: at most eight of 1080p's area
    if path == "me":
        return {"path": path, "est": rng.choice(sorted(ESTIMATORS)), "w": w, "h": h,
                "range": rng.choice([64, 80, 96, 128]), "pairs": rng.randint(1, most)}
    if path == "host":
        return {"path": path, "est": rng.choice(["full", "multires", "multires_cross"]), "w": w, "h": h,
                "range": rng.choice([64, 128]), "pairs": 1}
    if path == "coded":
        return {"path": path, "largest": rng.randint(1, 4), "seqs": rng.randint(2, 10), "pairs": rng.randint(1, 3),
                "qp": rng.randint(18, 40)}
    if path == "tq":
        return {"path": path, "w": max(712, w) + 8 * rng.randint(0, 1), "h": max(488, h) // 8 * 8,
                "frames": rng.randint(2, max(4, 2 * most)), "qp": rng.randint(0, 36), "intra": rng.randint(0, 1)}
    w, h = w + 2 * rng.randint(0, 3), h // 2 * 2
    if path == "rgb2yuv":
        return {"path": path, "kind": rng.choice([_lib.RGB_FIXED_POINT, _lib.RGB_FIXED_POINT, _lib.RGB_REAL]), "w": w,
                "h": h, "frames": rng.randint(1, 2 * most)}
    if path == "yuv2rgb":
        return {"path": path, "kind": rng.choice([_lib.YUV_REAL, _lib.YUV_REAL_IMPL2, _lib.YUV_CCIR601]), "w": w,
                "h": h, "frames": rng.randint(1, 2 * most)}
    return {"path": "mc", "w": w // 16 * 16, "h": h // 16 * 16, "frames": rng.randint(1, most)}


# ---- inputs ------------------------------------------------------------------


def _generator(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed))
    return g


def _texture(g, h, w):
    """Uniform noise under a 5x5 box filter (synth.smooth_texture's distribution), as floats."""
    x = torch.randint(0, 256, (1, 1, h + 4, w + 4), generator=g, device=DEV, dtype=torch.uint8).float()
    return torch.floor(torch.round(torch.nn.functional.avg_pool2d(x, 5, 1)[0, 0] * 25) / 25)


def _tap(x, frac, dim):
    """The H.264 luma interpolation of one axis at frac quarters, from rows / columns 2 .. n-4."""
    n = x.shape[dim] - 6
    at = lambda k: x.narrow(dim, k, n)  # noqa: E731
    if frac == 0:
        return at(2)
    half = (at(0) - 5 * at(1) + 20 * at(2) + 20 * at(3) - 5 * at(4) + at(5)) / 32
    return half if frac == 2 else (half + at(2 if frac == 1 else 3)) / 2


def _crop(base, y, x, h, w):
    """h x w samples of base from quarter-pel position (y, x), interpolated."""
    r = base[(y >> 2) - 2:(y >> 2) + h + 4, (x >> 2) - 2:(x >> 2) + w + 4]
    return _tap(_tap(r, x & 3, 1), y & 3, 0)


def _sequence(seed, w, h, n):
    """n int16 frames: one texture under a quarter-pel random-walk pan of up to 16 pels a frame, two textured objects
    moving on their own, and Gaussian noise of sigma 2."""
    g, rng, m = _generator(seed), random.Random(seed), 72
    base = _texture(g, h + 2 * m, w + 2 * m)
    y = x = 4 * m
    objs = []
    for _ in range(2):
        oh, ow = h // 4, w // 4
        objs.append([_texture(g, oh, ow), rng.randint(0, h - oh), rng.randint(0, w - ow)])
    frames = torch.empty((n, h, w), dtype=torch.int16, device=DEV)
    for t in range(n):
        f = _crop(base, y, x, h, w).clone()
        for o in objs:
            f[o[1]:o[1] + o[0].shape[0], o[2]:o[2] + o[0].shape[1]] = o[0]
            o[1] = min(max(o[1] + rng.randint(-8, 8), 0), h - o[0].shape[0])
            o[2] = min(max(o[2] + rng.randint(-8, 8), 0), w - o[0].shape[1])
        f += torch.round(torch.randn((h, w), generator=g, device=DEV) * 2)
        frames[t] = torch.clamp(torch.round(f), 0, 255).to(torch.int16)
        y = min(max(y + rng.randint(-64, 64), 16), 8 * m - 24)
        x = min(max(x + rng.randint(-64, 64), 16), 8 * m - 24)
    return frames


def _laplacian(g, n):
    """n residual samples, Laplacian of scale 6, clipped to +-255."""
    u = torch.rand(n, generator=g, device=DEV) - 0.5
    v = -6.0 * torch.sign(u) * torch.log(torch.clamp(1 - 2 * u.abs(), min=1e-30))
    return torch.clamp(torch.round(v), -255, 255).to(torch.int16)


def _plane(g, frames, h, w, mean, sigma):
    """Smooth shading plus fine texture around `mean`, 0..255."""
    low = torch.randn((frames, 1, max(2, h // 32), max(2, w // 32)), generator=g, device=DEV) * sigma
    x = torch.nn.functional.interpolate(low, size=(h, w), mode="bilinear", align_corners=False)[:, 0]
    return torch.clamp(torch.round(x + mean + torch.randn((frames, h, w), generator=g, device=DEV) * 4), 0, 255)


def _ptr(t):
    return C.c_void_p(t.data_ptr())


class _Handle:
    """A C ABI handle that a program keeps, given back with the state."""

    def __init__(self, h, destroy):
        self.h, self.destroy = h, destroy

    def __del__(self):
        self.destroy(self.h)


class _TqJob(C.Structure):
    """vppgpu_tq_job (include/vppgpu.h)."""
    _fields_ = [("residual", C.c_void_p), ("levels", C.c_void_p), ("recon", C.c_void_p), ("width", C.c_int),
                ("height", C.c_int), ("stride", C.c_int), ("qp", C.c_int), ("intra", C.c_int)]


def _mbs(w, h):
    return (w // 16) * (h // 16)


def _coded_jobs(case):
    """(sequence, pair, width, height) of the batch: sequence i has size i modulo the resolutions up to `largest`."""
    for s in range(case["seqs"]):
        w, h = MIX[s % (case["largest"] + 1)]
        for t in range(case["pairs"]):
            yield s, t, w, h


# ---- one state per path --------------------------------------------------------


def prepare(case, seed):
    ctx, lib = vpp.get_context(), vpp.load()
    path = case["path"]
    s = {"path": path, "ctx": ctx, "lib": lib, "case": case}
    if path in ("me", "host"):
        w, h = case["w"], case["h"]
        s["frames"] = _sequence(seed, w, h, case["pairs"] + 1)
        included = torch.rand(_mbs(w, h), generator=_generator(seed + 1), device=DEV) < 0.9
    if path == "host":
        cls = {"full": vpp.MotionEstimatorH264ImplFull, "multires": vpp.MotionEstimatorH264ImplMultires,
               "multires_cross": vpp.MotionEstimatorH264ImplMultiresCross}[case["est"]]
        f = s.pop("frames").cpu().numpy()
        s["me"] = cls(f[1], f[0], w, h, case["range"], pDistortionIncluded=included.cpu().numpy(), ctx=ctx)
        assert s["me"].Create() == 1
    elif path == "me":
        hd = C.c_void_p()
        _lib.check(lib.vppgpu_me_create(ctx.handle, ESTIMATORS[case["est"]], w, h, case["range"], C.byref(hd)), "create")
        if case["est"].startswith("multires"):
            _lib.check(lib.vppgpu_me_set_mode(hd, 2), "mode")
        s["me"] = _Handle(hd, lib.vppgpu_me_destroy)
        s["included"] = included.to(torch.uint8)
        s["mv"] = torch.zeros((case["pairs"], _mbs(w, h), 2), dtype=torch.int16, device=DEV)
        s["dist"] = torch.zeros((case["pairs"], _mbs(w, h)), dtype=torch.int32, device=DEV)
        s["avg"] = torch.zeros(case["pairs"], dtype=torch.int64, device=DEV)
    elif path == "coded":
        jobs = list(_coded_jobs(case))
        seqs = {}
        for q, _, w, h in jobs:
            if q not in seqs:
                seqs[q] = _sequence(seed + 1000 * q, w, h, case["pairs"] + 1)
        # one buffer for each kind of result, the jobs' parts one after the other at 16-byte boundaries
        at_mv, at_px, parts = 0, 0, []
        for _, _, w, h in jobs:
            parts.append((at_mv, at_px))
            at_mv += -(-_mbs(w, h) // 4) * 4
            at_px += w * h
        s["mv"] = torch.zeros((at_mv, 2), dtype=torch.int16, device=DEV)
        s["planes"] = [torch.zeros(at_px, dtype=torch.int16, device=DEV) for _ in range(3)]
        s["seqs"] = seqs
        s["jobs"] = [(seqs[q][t + 1].data_ptr(), seqs[q][t].data_ptr(), w, h, 128, s["mv"].data_ptr() + 4 * m, None, None,
                      *[p.data_ptr() + 2 * x for p in s["planes"]], case["qp"])
                     for (q, t, w, h), (m, x) in zip(jobs, parts)]
        s["batch"] = vpp.MotionEstimatorBatch(streams=8, ctx=ctx)
    elif path == "tq":
        w, h, n = case["w"], case["h"], case["frames"]
        per = w * h * 3 // 2
        s["res"] = _laplacian(_generator(seed), n * per)
        s["lev"], s["rec"] = torch.zeros_like(s["res"]), torch.zeros_like(s["res"])
        jobs = (_TqJob * (3 * n))()
        for f in range(n):
            at = f * per
            for k, (pw, ph) in enumerate(((w, h), (w // 2, h // 2), (w // 2, h // 2))):
                jobs[3 * f + k] = _TqJob(*[s[x].data_ptr() + 2 * at for x in ("res", "lev", "rec")], pw, ph, pw,
                                         case["qp"], case["intra"])
                at += pw * ph
        s["njobs"] = 3 * n
        s["jobs"] = torch.frombuffer(bytearray(bytes(jobs)), dtype=torch.uint8).to(DEV)
    elif path in ("rgb2yuv", "yuv2rgb"):
        w, h, n, g = case["w"], case["h"], case["frames"], _generator(seed)
        if path == "rgb2yuv":
            s["rgb"] = torch.stack([_plane(g, n, h, w, m, 45) for m in (110, 120, 130)], -1).to(torch.uint8)
            s["y"] = torch.zeros((n, h, w), dtype=torch.int16, device=DEV)
            s["u"] = torch.zeros((n, h // 2, w // 2), dtype=torch.int16, device=DEV)
            s["v"] = torch.zeros_like(s["u"])
        else:
            s["y"] = _plane(g, n, h, w, 120, 45).to(torch.int16)
            s["u"], s["v"] = (_plane(g, n, h // 2, w // 2, 128, 20).to(torch.int16) for _ in range(2))
            s["rgb"] = torch.zeros((n, h, w, 3), dtype=torch.uint8, device=DEV)
    else:  # mc
        w, h, n, g, rng = case["w"], case["h"], case["frames"], _generator(seed), random.Random(seed)
        y, u, v = _plane(g, n, h, w, 120, 45), _plane(g, n, h // 2, w // 2, 128, 20), _plane(g, n, h // 2, w // 2, 128, 20)
        s["ref"] = torch.cat([p.reshape(n, -1) for p in (y, u, v)], 1).to(torch.int16)
        s["out"] = torch.zeros_like(s["ref"])
        # a pan per frame, a quarter of the macroblocks with motion of their own, a tenth still
        pan = torch.tensor([[rng.randint(-64, 64), rng.randint(-64, 64)] for _ in range(n)], device=DEV)
        own = torch.randint(-63, 64, (n, _mbs(w, h), 2), generator=g, device=DEV)
        pick = torch.rand((n, _mbs(w, h), 1), generator=g, device=DEV)
        s["mv"] = torch.where(pick < 0.25, pan[:, None] + own, pan[:, None].expand_as(own))
        s["mv"] = torch.where(pick > 0.9, 0, s["mv"]).to(torch.int16).contiguous()
        hd = C.c_void_p()
        _lib.check(lib.vppgpu_mc_create(ctx.handle, w, h, 32, C.byref(hd)), "create")
        s["mc"] = _Handle(hd, lib.vppgpu_mc_destroy)
    return s


def run(s):
    case, lib, ctx, path = s["case"], s["lib"], s["ctx"].handle, s["path"]
    if path == "host":
        mv, avg = s["me"].Estimate()
        return mv, s["me"].last_mb_distortion, avg
    if path == "me":
        for t in range(case["pairs"]):
            _lib.check(lib.vppgpu_me_estimate_device(s["me"].h, _ptr(s["frames"][t + 1]), _ptr(s["frames"][t]),
                                                     _ptr(s["included"]), None, _ptr(s["mv"][t]), _ptr(s["dist"][t]),
                                                     _ptr(s["avg"][t])), "vppgpu_me_estimate_device")
        return s["mv"], s["dist"], s["avg"]
    if path == "coded":
        status, _ = s["batch"].run(s["jobs"])
        return s["mv"], s["planes"], status
    if path == "tq":
        _lib.check(lib.vppgpu_tq_roundtrip_planes_device(ctx, _ptr(s["jobs"]), s["njobs"], _lib.INV_ROWS_FIRST, None),
                   "vppgpu_tq_roundtrip_planes_device")
        return s["lev"], s["rec"]
    if path == "rgb2yuv":
        _lib.check(lib.vppgpu_rgb24_to_yuv420_frames_device(ctx, case["kind"], _ptr(s["rgb"]), case["frames"], case["w"],
                                                            case["h"], 128, 0, _ptr(s["y"]), _ptr(s["u"]),
                                                            _ptr(s["v"])), "vppgpu_rgb24_to_yuv420_frames_device")
        return s["y"], s["u"], s["v"]
    if path == "yuv2rgb":
        _lib.check(lib.vppgpu_yuv420_to_rgb24_frames_device(ctx, case["kind"], _ptr(s["y"]), _ptr(s["u"]), _ptr(s["v"]),
                                                            case["frames"], case["w"], case["h"], -128, 0, 0,
                                                            _ptr(s["rgb"])), "vppgpu_yuv420_to_rgb24_frames_device")
        return s["rgb"]
    for t in range(case["frames"]):
        _lib.check(lib.vppgpu_mc_compensate_device(s["mc"].h, _ptr(s["ref"][t]), _ptr(s["mv"][t]), _ptr(s["out"][t])),
                   "vppgpu_mc_compensate_device")
    return s["out"]


# ---- what a pass cannot do without ------------------------------------------------


def _search_terms(est, rng):
    """Pixel differences per macroblock: every candidate of a full search over 256 pixels; for the pyramids a coarse
    search, +-2 at the finer levels, and 16 sub-pel points."""
    side = 2 * (rng // 4 - 1) + 1
    sub = 0 if est == "full_sad" else 16 * 256
    if est in ("full", "full_sad"):
        return side * side * 256 + sub
    coarse = 2 * (rng // 16) + 1
    top = coarse * coarse if est == "multires" else 4 * max(1, int(math.log2(coarse)))
    return top * 16 + 25 * 64 + 25 * 256 + sub


def work(case):
    path = case["path"]
    if path in ("me", "host"):
        w, h = case["w"], case["h"]
        return {"bytes": case["pairs"] * (4 * w * h + 8 * _mbs(w, h)),
                "flops": 2 * case["pairs"] * _mbs(w, h) * _search_terms(case["est"], case["range"])}
    if path == "coded":
        jobs = list(_coded_jobs(case))
        return {"bytes": sum(10 * w * h + 4 * _mbs(w, h) for _, _, w, h in jobs),
                "flops": sum(2 * _mbs(w, h) * (_search_terms("full", 128) + 256 * 20) for _, _, w, h in jobs)}
    px = case["w"] * case["h"] * case["frames"]
    if path == "tq":
        return {"bytes": 9 * px, "flops": 1.5 * px * 20}
    return {"bytes": 6 * px, "flops": 20 * px}
