"""The kernels that prepare an estimate's planes from resident 16-bit samples, against the CPU oracle, bit-exact:
samples at every alignment the device call accepts (4 bytes; the wide loads take 8 and 16), widths whose bordered
copies are no whole number of words, heights that leave part of a macroblock row, and values outside 0..255 in the
input's or the reference's first and last samples refused."""
import ctypes as C

import numpy as np
import pytest

from imagecodingutils_gb300 import synth

pytestmark = pytest.mark.gpu

KINDS = [("ME_FULL", "me_full", {}), ("ME_MULTIRES_CROSS", "me_multires_cross", {"mode": 2}),
         ("ME_MULTIRES", "me_multires", {"mode": 2})]


def place(torch, plane, shift):
    buf = torch.zeros(plane.size + 16, dtype=torch.int16, device="cuda")
    buf[shift:shift + plane.size] = torch.from_numpy(plane.reshape(-1)).cuda()
    return buf, C.c_void_p(buf.data_ptr() + 2 * shift)


@pytest.mark.parametrize("w,h", [(16, 18), (80, 52), (176, 144)])
@pytest.mark.parametrize("s_src,s_ref", [(0, 0), (2, 4), (4, 2), (8, 6)])
@pytest.mark.parametrize("kind", range(len(KINDS)))
def test_alignment(vpp, ctx, orc, kind, s_src, s_ref, w, h):
    torch = pytest.importorskip("torch")
    from imagecodingutils_gb300 import _lib
    L = vpp.load()
    name, fn, extra = KINDS[kind]
    h4 = h // 4 * 4  # the oracle's pyramid takes whole level-2 rows
    fr = synth.pan_sequence(500 + w, w, h4, 2)
    nmb = (w // 16) * (h4 // 16)
    mv_o, dist_o, _ = getattr(orc, fn)(fr[1], fr[0], 64, **extra)
    keep_s, src = place(torch, fr[1], s_src)
    keep_r, ref = place(torch, fr[0], s_ref)
    mv = torch.empty((nmb, 2), dtype=torch.int16, device="cuda")
    dist = torch.empty(nmb, dtype=torch.int32, device="cuda")
    handle = C.c_void_p()
    _lib.check(L.vppgpu_me_create(ctx.handle, getattr(_lib, name), w, h4, 64, C.byref(handle)), "create")
    try:
        if extra:
            _lib.check(L.vppgpu_me_set_mode(handle, extra["mode"]), "mode")
        run = lambda: L.vppgpu_me_estimate_device(handle, src, ref, None, None, C.c_void_p(mv.data_ptr()),
                                                  C.c_void_p(dist.data_ptr()), None)
        torch.cuda.synchronize()
        _lib.check(run(), "estimate")
        ctx.synchronize()
        np.testing.assert_array_equal(mv.cpu().numpy(), mv_o)
        np.testing.assert_array_equal(dist.cpu().numpy(), dist_o)
        assert L.vppgpu_me_last_status(handle) == 0
        for buf, at, v in ((keep_s, s_src, 256), (keep_s, s_src + w * h4 - 1, -1), (keep_r, s_ref, -1),
                           (keep_r, s_ref + w * h4 - 1, 256)):
            was = int(buf[at])
            buf[at] = v
            torch.cuda.synchronize()
            run()
            ctx.synchronize()
            assert L.vppgpu_me_last_status(handle) != 0
            buf[at] = was
    finally:
        L.vppgpu_me_destroy(handle)


AVG_KINDS = [("ME_FULL", "me_full", None), ("ME_MULTIRES", "me_multires", 2), ("ME_MULTIRES_CROSS_V2", "me_multires_cross_v2", 2),
             ("ME_MULTIRES_CROSS", "me_multires_cross", 1), ("ME_CROSS", "me_cross", 0),
             ("ME_H263_MULTIRES_CROSS", "me_h263_multires_cross", 2), ("ME_FULL_SAD", "me_full_intpel", None)]


@pytest.mark.parametrize("w,h", [(16, 16), (176, 150), (1040, 520), (1040, 516)])
@pytest.mark.parametrize("kind", range(len(AVG_KINDS)))
def test_average_on_the_device(vpp, ctx, orc, kind, w, h):
    """The average that a device call writes, from the included macroblocks' distortions: every estimator that shares
    the cluster resolve or the pyramid search, below and above the 2048 macroblocks where the SAD stage's launches
    change, with a part of a macroblock row below the last whole one, on one handle twice and with none included."""
    torch = pytest.importorskip("torch")
    from imagecodingutils_gb300 import _lib
    L = vpp.load()
    name, fn, mode = AVG_KINDS[kind]
    fr = synth.pan_sequence(520 + w, w, h, 3)
    nmb = (w // 16) * (h // 16)
    incl = (synth.splitmix64(w + h, nmb) % np.uint64(3) != 0).astype(np.uint8)
    planes = [torch.from_numpy(f).cuda() for f in fr]
    mv = torch.empty((nmb, 2), dtype=torch.int16, device="cuda")
    avg = torch.full((3,), -7, dtype=torch.int64, device="cuda")
    d_incl = torch.from_numpy(incl).cuda()
    handle = C.c_void_p()
    _lib.check(L.vppgpu_me_create(ctx.handle, getattr(_lib, name), w, h, 64, C.byref(handle)), "create")
    try:
        if mode is not None:
            _lib.check(L.vppgpu_me_set_mode(handle, mode), "mode")
        torch.cuda.synchronize()
        for t, inc in ((1, d_incl), (2, d_incl), (2, torch.zeros_like(d_incl))):
            _lib.check(L.vppgpu_me_estimate_device(handle, C.c_void_p(planes[t].data_ptr()),
                                                   C.c_void_p(planes[t - 1].data_ptr()), C.c_void_p(inc.data_ptr()), None,
                                                   C.c_void_p(mv.data_ptr()), None, C.c_void_p(avg.data_ptr() + 8)), "run")
            ctx.synchronize()
            mask = inc.cpu().numpy()
            if name == "ME_FULL_SAD":
                d = orc.me_full_intpel(fr[t], fr[t - 1], 64, metric=1)[1][mask.astype(bool)]
                want = int(d.sum()) // d.size if d.size else 0
            else:
                want = getattr(orc, fn)(fr[t], fr[t - 1], 64, dist_incl=mask, **({} if mode is None else {"mode": mode}))[2]
            assert avg.tolist() == [-7, want, -7]
    finally:
        L.vppgpu_me_destroy(handle)
