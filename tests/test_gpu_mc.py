"""GPU MotionCompensatorH264ImplStd (vppgpu_mc_*): the compensated 4:2:0 frame
bit-exact with the reference's golden fixtures and with the oracle on further
sizes; in-place host semantics and the device entry point with a separate
output; the add-with-clip and subtract plane helpers against the oracle; and
the encoder loop prediction + residual = input for a zero-quantisation step."""
import ctypes as C

import numpy as np
import pytest

from imagecodingutils_gb300 import synth

pytestmark = pytest.mark.gpu

CASES = ["qcif_r16", "cif_r32", "small_r8"]


def compensate(vpp, ctx, y, u, v, mv, rg):
    h, w = y.shape
    yuv = np.concatenate([np.ravel(y), np.ravel(u), np.ravel(v)]).astype(np.int16)
    mc = vpp.MotionCompensatorH264ImplStd(rg, ctx=ctx)
    assert mc.Create(yuv, w, h) == 1
    mc.Compensate(mv)
    n, c = w * h, (w // 2) * (h // 2)
    return yuv[:n].reshape(h, w), yuv[n:n + c].reshape(h // 2, w // 2), yuv[n + c:].reshape(h // 2, w // 2)


@pytest.mark.parametrize("case", CASES)
def test_against_golden(vpp, ctx, golden, case):
    g = golden("mc.npz")
    w, h, rg = (int(v) for v in g[f"{case}_meta"])
    y, u, v = (g[f"{case}_{k}"].astype(np.int16) for k in ("y", "u", "v"))
    cy, cu, cv = compensate(vpp, ctx, y, u, v, g[f"{case}_mv"], rg)
    np.testing.assert_array_equal(cy, g[f"{case}_cy"])
    np.testing.assert_array_equal(cu, g[f"{case}_cu"])
    np.testing.assert_array_equal(cv, g[f"{case}_cv"])


@pytest.mark.parametrize("seed,w,h,rg", [(71, 1920, 1088, 32), (72, 208, 120, 24), (73, 640, 368, 16)])
def test_against_oracle(vpp, ctx, orc, seed, w, h, rg):
    y = synth.pan_sequence(seed, w, h, 1)[0]
    u = synth.pan_sequence(seed + 1, w // 2, h // 2, 1)[0]
    v = synth.pan_sequence(seed + 2, w // 2, h // 2, 1)[0]
    nmb = (w // 16) * (h // 16)
    mv = ((synth.splitmix64(seed, 2 * nmb) % np.uint64(8 * rg + 1)).astype(np.int64) - 4 * rg).astype(np.int16)
    mv = mv.reshape(nmb, 2)
    got = compensate(vpp, ctx, y, u, v, mv, rg)
    for a, b in zip(got, orc.mc_compensate(y, u, v, mv, rg)):
        np.testing.assert_array_equal(a, b)


def test_device_entry_and_plane_helpers(vpp, ctx, orc):
    """Device compensation into a separate frame, then residual = input - prediction
    and reconstruction = clip(prediction + residual) == input."""
    torch = pytest.importorskip("torch")
    from imagecodingutils_gb300 import _lib
    L = vpp.load()
    dev = torch.device("cuda", 0)
    w, h, rg = 352, 288, 32
    fr = synth.pan_sequence(74, w, h, 2)
    u = synth.pan_sequence(75, w // 2, h // 2, 1)[0]
    v = synth.pan_sequence(76, w // 2, h // 2, 1)[0]
    mv_o, _, _ = orc.me_full(fr[1], fr[0], 128)
    ref = torch.from_numpy(np.concatenate([fr[0].ravel(), u.ravel(), v.ravel()]).astype(np.int16)).to(dev)
    pred = torch.empty_like(ref)
    mv = torch.from_numpy(mv_o).to(dev)
    mc = C.c_void_p()
    _lib.check(L.vppgpu_mc_create(ctx.handle, w, h, rg, C.byref(mc)), "create")
    _lib.check(L.vppgpu_mc_compensate_device(mc, C.c_void_p(ref.data_ptr()), C.c_void_p(mv.data_ptr()),
                                             C.c_void_p(pred.data_ptr())), "compensate")
    ctx.synchronize()
    oy, ou, ov = orc.mc_compensate(fr[0], u, v, mv_o, rg)
    n = w * h
    np.testing.assert_array_equal(pred[:n].cpu().numpy().reshape(h, w), oy)
    np.testing.assert_array_equal(pred[n:].cpu().numpy(), np.concatenate([ou.ravel(), ov.ravel()]))
    np.testing.assert_array_equal(ref.cpu().numpy()[:n].reshape(h, w), fr[0])  # input untouched
    # residual of the luma and back
    inp = torch.from_numpy(fr[1].astype(np.int16).ravel()).to(dev)
    res = inp.clone()
    _lib.check(L.vppgpu_sub_device(ctx.handle, C.c_void_p(res.data_ptr()), C.c_void_p(pred.data_ptr()), n), "sub")
    rec = pred[:n].clone()
    _lib.check(L.vppgpu_add_clip255_device(ctx.handle, C.c_void_p(rec.data_ptr()), C.c_void_p(res.data_ptr()), n),
               "add")
    ctx.synchronize()
    np.testing.assert_array_equal(res.cpu().numpy(), orc.sub(fr[1].ravel(), oy.ravel()))
    np.testing.assert_array_equal(rec.cpu().numpy(), fr[1].ravel())
    # odd length: the tail path of the plane helpers
    a = torch.from_numpy(np.arange(-500, 499, dtype=np.int16)).to(dev)
    b = torch.from_numpy(np.full(999, 37, np.int16)).to(dev)
    ah = a.cpu().numpy()
    _lib.check(L.vppgpu_add_clip255_device(ctx.handle, C.c_void_p(a.data_ptr()), C.c_void_p(b.data_ptr()), 999), "add")
    ctx.synchronize()
    np.testing.assert_array_equal(a.cpu().numpy(), orc.add_clip255(ah, np.full(999, 37, np.int16)))
    L.vppgpu_mc_destroy(mc)


@pytest.mark.parametrize("spread", ["bytes", "hard", "some", "all"])
@pytest.mark.parametrize("w,h,shift", [(16, 16, 0), (48, 34, 0), (48, 34, 1), (112, 64, 4), (176, 80, 0)])
def test_sample_ranges_and_alignments(vpp, ctx, orc, spread, w, h, shift):
    """The packed path and the one that takes any samples, against the oracle: bytes (also only 0 and 255, where the
    6-tap sums are largest), a few samples outside 0..255, any shorts; frames that are 16-byte aligned or not; every
    quarter case, vectors of zero and ones that leave the picture."""
    torch = pytest.importorskip("torch")
    from imagecodingutils_gb300 import _lib
    L = vpp.load()
    ny, nc, nmb = w * h, (w // 2) * (h // 2), (w // 16) * (h // 16)
    n = ny + 2 * nc
    r = synth.splitmix64(800 + w + shift, n)
    yuv = (r % np.uint64(256)).astype(np.int64)
    if spread == "hard":
        yuv = np.where(yuv < 128, 0, 255)
    elif spread == "some":
        yuv = np.where(r >> np.uint64(40) & np.uint64(511), yuv, 256 - 2 * yuv)
    elif spread == "all":
        yuv = (r % np.uint64(65536)).astype(np.int64) - 32768
        yuv //= 8  # the chroma weights sum to 64: the reference's int holds it either way
    yuv = yuv.astype(np.int16)
    planes = yuv[:ny].reshape(h, w), yuv[ny:ny + nc].reshape(h // 2, w // 2), yuv[ny + nc:].reshape(h // 2, w // 2)
    rg = 8
    mc = C.c_void_p()
    _lib.check(L.vppgpu_mc_create(ctx.handle, w, h, rg, C.byref(mc)), "create")
    try:
        src = torch.zeros(n + 16, dtype=torch.int16, device="cuda")
        out = torch.zeros(n + 16, dtype=torch.int16, device="cuda")
        src[shift:shift + n] = torch.from_numpy(yuv).cuda()
        for seed in range(3):
            mv = ((synth.splitmix64(900 + seed, 2 * nmb) % np.uint64(8 * rg + 1)).astype(np.int64) - 4 * rg)
            mv = mv.astype(np.int16).reshape(nmb, 2)
            mv[seed::5] = 0
            mv[1::4] //= 8
            d_mv = torch.from_numpy(mv).cuda()
            torch.cuda.synchronize()
            _lib.check(L.vppgpu_mc_compensate_device(mc, C.c_void_p(src.data_ptr() + 2 * shift),
                                                     C.c_void_p(d_mv.data_ptr()),
                                                     C.c_void_p(out.data_ptr() + 2 * shift)), "compensate")
            ctx.synchronize()
            got = out[shift:shift + n].cpu().numpy()
            want = np.concatenate([np.ravel(p) for p in orc.mc_compensate(*planes, mv, rg)])
            np.testing.assert_array_equal(got, want)
    finally:
        L.vppgpu_mc_destroy(mc)


def test_samples_of_any_range_cost_no_second_pass(vpp, ctx):
    """Frames of samples outside 0..255 against frames of bytes: read and staged twice they took 1.6 times as long."""
    import time

    torch = pytest.importorskip("torch")
    from imagecodingutils_gb300 import _lib
    L = vpp.load()
    w, h = 1920, 1088
    n, nmb = w * h * 3 // 2, (w // 16) * (h // 16)
    r = synth.splitmix64(990, n).astype(np.int64)
    mv = torch.from_numpy((synth.splitmix64(991, 2 * nmb) % np.uint64(128)).astype(np.int16) - 64).cuda()
    mc = C.c_void_p()
    _lib.check(L.vppgpu_mc_create(ctx.handle, w, h, 32, C.byref(mc)), "create")
    for _ in range(4):  # other work may share the machine
        best = []
        for yuv in (r % 256, r % 4096 - 2048):
            src = torch.from_numpy(yuv.astype(np.int16)).cuda()
            out = torch.empty_like(src)
            torch.cuda.synchronize()
            t = []
            for _ in range(6):
                t0 = time.perf_counter()
                for _ in range(200):
                    _lib.check(L.vppgpu_mc_compensate_device(mc, C.c_void_p(src.data_ptr()), C.c_void_p(mv.data_ptr()),
                                                             C.c_void_p(out.data_ptr())), "compensate")
                ctx.synchronize()
                t.append(time.perf_counter() - t0)
            best.append(min(t))
        if best[1] < 1.35 * best[0]:
            break
    L.vppgpu_mc_destroy(mc)
    assert best[1] < 1.35 * best[0]
