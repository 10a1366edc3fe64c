"""GPU RGB24 -> YUV420 parity with the reference's golden fixtures and the
CPU oracle (bit-exact for the integer and both IEEE-double converters)."""
import numpy as np
import pytest

from imagecodingutils_gb300 import synth

pytestmark = pytest.mark.gpu


def convert(vpp, ctx, kind, bgr, co, flip):
    h, w, _ = bgr.shape
    y = np.empty((h, w), np.int16)
    u = np.empty((h // 2, w // 2), np.int16)
    v = np.empty((h // 2, w // 2), np.int16)
    c = vpp.FastGpuRGB24toYUV420Converter(w, h, co, kind=kind, ctx=ctx)
    c.SetFlip(flip)
    c.Convert(bgr, y, u, v)
    return y, u, v


def test_against_golden(vpp, ctx, golden):
    g = golden("colour.npz")
    for kind in (0, 1, 2):
        for flip in (0, 1):
            for co in (0, 128):
                y, u, v = convert(vpp, ctx, kind, g["bgr"], co, flip)
                np.testing.assert_array_equal(y, g[f"k{kind}_f{flip}_c{co}_y"])
                np.testing.assert_array_equal(u, g[f"k{kind}_f{flip}_c{co}_u"])
                np.testing.assert_array_equal(v, g[f"k{kind}_f{flip}_c{co}_v"])


@pytest.mark.parametrize("kind", [0, 1, 2])
@pytest.mark.parametrize("w,h", [(1920, 1080), (1922, 6), (2, 2), (1000, 750)])
def test_against_oracle(vpp, ctx, orc, kind, w, h):
    bgr = synth.rgb_frame(w + h + kind, w, h)
    for co in (0, 128):
        got = convert(vpp, ctx, kind, bgr, co, 0)
        want = orc.rgb_to_yuv(kind, bgr, co, 0)
        for a, b in zip(got, want):
            np.testing.assert_array_equal(a, b)


def test_extreme_colours(vpp, ctx, orc):
    """Saturated primaries exercise every clamp of the luma and chroma ranges."""
    vals = np.array([0, 1, 127, 128, 254, 255], np.uint8)
    b, g, r = np.meshgrid(vals, vals, vals, indexing="ij")
    px = np.stack([b.ravel(), g.ravel(), r.ravel()], -1)  # 216 colours
    bgr = np.repeat(np.repeat(px.reshape(6, 36, 3), 2, 0), 2, 1)  # each colour fills a 2x2 block
    for kind in (0, 1, 2):
        got = convert(vpp, ctx, kind, bgr, 128, 0)
        want = orc.rgb_to_yuv(kind, bgr, 128, 0)
        for a, bb in zip(got, want):
            np.testing.assert_array_equal(a, bb)


@pytest.mark.parametrize("kind", [0, 1, 2])
def test_every_colour(vpp, ctx, orc, kind):
    """Each of the 2^24 colours once: the luma of the real converters is formed from integers except where its exact
    value is a whole number, and every 2x2 block has four colours (its chroma sum, likewise)."""
    i = np.arange(1 << 24, dtype=np.uint32)
    j = (i * np.uint32(2654435761)) & np.uint32(0xffffff) if kind == 2 else i  # an odd factor: every colour once
    bgr = np.stack([j & 255, (j >> 8) & 255, j >> 16], -1).astype(np.uint8).reshape(4096, 4096, 3)
    for a, b in zip(convert(vpp, ctx, kind, bgr, 128, 0), orc.rgb_to_yuv(kind, bgr, 128, 0)):
        np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("kind", [1, 2])
def test_chroma_sums_on_a_whole_number(vpp, ctx, orc, kind):
    """Blocks whose exact chroma sum is a truncation boundary (multiples of 1, of 4 shifted by 2, and 0), where the
    double's last bits decide."""
    vals = [(b, g, r) for b in range(0, 256, 5) for g in range(0, 256, 3) for r in range(0, 256, 3)
            if (436 * b - 289 * g - 147 * r) % 250 == 0 or (615 * r - 515 * g - 100 * b) % 250 == 0]
    n = len(vals) // 16 * 16
    px = np.array(vals[:n], np.uint8).reshape(-1, 16, 3)
    bgr = np.repeat(np.repeat(px, 2, 0), 2, 1)
    for flip in (0, 1):
        for a, b in zip(convert(vpp, ctx, kind, bgr, 0, flip), orc.rgb_to_yuv(kind, bgr, 0, flip)):
            np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("kind", [0, 1, 2])
@pytest.mark.parametrize("w,h,off,yoff", [(8, 2, 0, 0), (10, 4, 0, 0), (10, 4, 1, 2), (22, 6, 3, 0), (24, 4, 2, 2),
                                          (24, 4, 8, 8), (14, 2, 0, 1), (6, 4, 0, 0), (64, 4, 4, 0)])
def test_widths_and_alignments(vpp, ctx, orc, kind, w, h, off, yoff):
    """Frames on the device at any byte, planes at any sample: the wide, the narrow and the sample-by-sample path."""
    import ctypes as C
    torch = pytest.importorskip("torch")
    from imagecodingutils_gb300 import _lib
    L = vpp.load()
    nf, n = 3, w * h
    bgr = np.stack([synth.rgb_frame(7 * w + f + kind, w, h) for f in range(nf)])
    src = torch.zeros(nf * n * 3 + 16, dtype=torch.uint8, device="cuda")
    src[off:off + nf * n * 3] = torch.from_numpy(bgr.reshape(-1)).cuda()
    out = [torch.full((nf * m + 16,), 77, dtype=torch.int16, device="cuda") for m in (n, n // 4, n // 4)]
    torch.cuda.synchronize()
    _lib.check(L.vppgpu_rgb24_to_yuv420_frames_device(ctx.handle, kind, C.c_void_p(src.data_ptr() + off), nf, w, h, 128,
                                                      0, *[C.c_void_p(t.data_ptr() + 2 * yoff) for t in out]), "convert")
    ctx.synchronize()
    for f in range(nf):
        for t, want in zip(out, orc.rgb_to_yuv(kind, bgr[f], 128, 0)):
            m = want.size
            np.testing.assert_array_equal(t[yoff + f * m:yoff + (f + 1) * m].cpu().numpy(), want.reshape(-1))
    for t, m in zip(out, (n, n // 4, n // 4)):
        assert (t[:yoff] == 77).all() and (t[yoff + nf * m:] == 77).all()


@pytest.mark.parametrize("kind", [1, 2])
@pytest.mark.parametrize("w,h,nf,flip", [(1280, 720, 1, 1), (1280, 720, 2, 0), (1280, 720, 2, 1), (1920, 1080, 1, 1)])
def test_real_kinds_at_the_change_of_kernel(vpp, ctx, orc, kind, w, h, nf, flip):
    """Aligned frames too small to fill the GPU by eight pixels a thread, and large enough; colours in steps of 25, so
    that many terms lie on whole numbers."""
    import ctypes as C
    torch = pytest.importorskip("torch")
    from imagecodingutils_gb300 import _lib
    bgr = np.stack([synth.rgb_frame(31 + f, w, h) // 25 * 25 for f in range(nf)])
    src = torch.from_numpy(bgr).cuda()
    out = [torch.zeros(nf * m, dtype=torch.int16, device="cuda") for m in (w * h, w * h // 4, w * h // 4)]
    torch.cuda.synchronize()
    _lib.check(vpp.load().vppgpu_rgb24_to_yuv420_frames_device(ctx.handle, kind, C.c_void_p(src.data_ptr()), nf, w, h, 128,
                                                               flip, *[C.c_void_p(t.data_ptr()) for t in out]), "convert")
    ctx.synchronize()
    for f in range(nf):
        for t, want in zip(out, orc.rgb_to_yuv(kind, bgr[f], 128, flip)):
            np.testing.assert_array_equal(t.cpu().numpy()[f * want.size:(f + 1) * want.size], want.reshape(-1))


def test_real_kinds_on_small_frames(vpp, ctx):
    """Colours whose terms lie on whole numbers, each a chain of doubles: eight pixels a thread made a small frame of
    them 3.7 times as long as a noisy one."""
    import ctypes as C
    import time
    torch = pytest.importorskip("torch")
    from imagecodingutils_gb300 import _lib
    w, h = 176, 144
    noise = synth.rgb_frame(3, w, h)
    out = [torch.zeros(m, dtype=torch.int16, device="cuda") for m in (w * h, w * h // 4, w * h // 4)]
    for _ in range(4):  # other work may share the machine
        best = []
        for bgr in (noise, noise // 50 * 50):
            src = torch.from_numpy(np.ascontiguousarray(bgr)).cuda()
            torch.cuda.synchronize()
            t = []
            for _ in range(6):
                t0 = time.perf_counter()
                for _ in range(200):
                    _lib.check(vpp.load().vppgpu_rgb24_to_yuv420_frames_device(
                        ctx.handle, 1, C.c_void_p(src.data_ptr()), 1, w, h, 128, 0, *[C.c_void_p(x.data_ptr()) for x in out]),
                        "convert")
                ctx.synchronize()
                t.append(time.perf_counter() - t0)
            best.append(min(t))
        if best[1] < 2.6 * best[0]:
            break
    assert best[1] < 2.6 * best[0]
