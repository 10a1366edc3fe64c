"""Autotuning (vppgpu_me_autotune): for every estimator kind the tuner picks a
launch shape / relaxation policy, and estimates afterwards still give the
oracle's vectors and distortions."""
import numpy as np
import pytest

from imagecodingutils_gb300 import synth

pytestmark = pytest.mark.gpu

KINDS = [("MotionEstimatorH264ImplFull", "me_full", {}),
         ("MotionEstimatorH264ImplMultires", "me_multires", {"mode": 0}),
         ("MotionEstimatorH264ImplMultiresCross", "me_multires_cross", {"mode": 0}),
         ("MotionEstimatorH264ImplMultiresCrossVer2", "me_multires_cross_v2", {"mode": 0})]


@pytest.mark.parametrize("cls,ofn,kw", KINDS)
def test_autotune_keeps_results(vpp, ctx, orc, cls, ofn, kw):
    w, h = 640, 368
    fr = synth.pan_sequence(95, w, h, 3)
    me = getattr(vpp, cls)(fr[1], fr[0], w, h, 128, ctx=ctx)
    assert me.Create() == 1
    me.SetMode(0)
    before = me.tuning()
    t = me.Autotune(reps=1)
    assert t["choice"] >= 0
    assert set(t) >= set(before)
    for k in (1, 2):
        me._src, me._ref = fr[k], fr[k - 1]
        mv, _ = me.Estimate()
        mv_o, dist_o, _ = getattr(orc, ofn)(fr[k], fr[k - 1], 128, **kw)
        np.testing.assert_array_equal(mv, mv_o)
        np.testing.assert_array_equal(me.last_mb_distortion, dist_o)


@pytest.mark.parametrize("kind,mode,src_off", [
    ("ME_MULTIRES_CROSS", 1, 1), ("ME_MULTIRES_CROSS", 2, 1), ("ME_H263_MULTIRES_CROSS", 2, 1),
    ("ME_H263_MULTIRES_CROSS_V2", 2, 1), ("ME_MULTIRES_CROSS_V2", 2, 0), ("ME_MULTIRES", 2, 0), ("ME_FULL", 0, 0)])
def test_planes_at_any_sample(vpp, ctx, orc, kind, mode, src_off):
    """A tuning call takes planes whose first sample is at any even address (the input's only where it is not packed by
    pairs: there it is refused), and the estimate after it is the same."""
    import ctypes as C
    torch = pytest.importorskip("torch")
    from imagecodingutils_gb300 import _lib
    L = vpp.load()
    w, h = 176, 144
    fr = synth.pan_sequence(97, w, h, 2)
    n = w * h
    dev = []
    for f, off in ((fr[1], src_off), (fr[0], 1)):
        t = torch.zeros(n + 8, dtype=torch.int16, device="cuda")
        t[off:off + n] = torch.from_numpy(f.reshape(-1)).cuda()
        dev.append((t, C.c_void_p(t.data_ptr() + 2 * off)))
    torch.cuda.synchronize()
    hd = C.c_void_p()
    _lib.check(L.vppgpu_me_create(ctx.handle, getattr(_lib, kind), w, h, 64, C.byref(hd)), "create")
    try:
        L.vppgpu_me_set_mode(hd, mode)
        mv = [np.zeros((n // 256, 2), np.int16) for _ in range(2)]
        avg = C.c_long()
        for i in range(2):
            _lib.check(L.vppgpu_me_estimate(hd, fr[1].ctypes.data, fr[0].ctypes.data, None, None, mv[i].ctypes.data, None,
                                            C.byref(avg)), "estimate")
            if i == 0:
                idx = C.c_int()
                _lib.check(L.vppgpu_me_autotune(hd, dev[0][1], dev[1][1], 1, C.byref(idx)), "autotune")
        np.testing.assert_array_equal(mv[0], mv[1])
        if src_off == 0:
            assert L.vppgpu_me_autotune(hd, C.c_void_p(dev[0][0].data_ptr() + 2), dev[1][1], 1, None) == \
                _lib.ERR_INVALID_ARG
    finally:
        L.vppgpu_me_destroy(hd)


@pytest.mark.parametrize("cls", ["MotionEstimatorH264ImplFull", "MotionEstimatorH264ImplMultires",
                                 "MotionEstimatorH264ImplMultiresCrossVer2", "MotionEstimatorH264ImplCross"])
def test_autotune_times_each_launch_sequence_once(vpp, ctx, cls):
    """A small frame has four of them (0, 1, 2 and 4 sweeps before the cluster: any grid holds all of it), a candidate a
    warm-up and a timed estimate each; the sweeps that only the statistics and the Lagrangian overload read stay."""
    w, h = 176, 144
    fr = synth.pan_sequence(96, w, h, 2)
    me = getattr(vpp, cls)(fr[1], fr[0], w, h, 128, ctx=ctx)
    assert me.Create() == 1
    me.Estimate()
    n0 = ctx.launch_count()
    me.Estimate()
    n1 = ctx.launch_count()
    before = me.tuning()
    after = me.Autotune(reps=1)
    assert ctx.launch_count() - n1 <= 4 * 2 * (n1 - n0 + 3)  # (up to three more sweeps than the estimate's one)
    assert after["relax_sweeps"] == before["relax_sweeps"]
    assert after["grid_sweeps"] in (0, 1, 2, 4)
