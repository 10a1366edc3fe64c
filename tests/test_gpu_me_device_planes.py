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
