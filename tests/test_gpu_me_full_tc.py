"""The tensor-core table of the SSD full search where it can go wrong: frames smaller than a tile, widths around the
64-column windows and heights around the 16-row tiles, ranges from one pel to +-31, and samples at both ends of their
range (the largest cross terms and energies).  Bit-exact against the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _planes(kind, seed, w, h):
    rng = np.random.default_rng(seed)
    if kind == "extremes":  # 0 and 255 only: |sample - 128| at its largest everywhere
        return (rng.integers(0, 2, (h, w)) * 255).astype(np.int16), (rng.integers(0, 2, (h, w)) * 255).astype(np.int16)
    if kind == "white":     # every candidate of one half the same: ties decided by the scan
        a = np.full((h, w), 255, np.int16)
        b = a.copy()
        b[: h // 2] = 0
        return a, b
    return rng.integers(0, 256, (h, w)).astype(np.int16), rng.integers(0, 256, (h, w)).astype(np.int16)


@pytest.mark.parametrize("w,h,mr,kind", [
    (16, 16, 128, "noise"), (48, 31, 128, "noise"), (64, 64, 128, "extremes"), (80, 47, 4, "noise"),
    (96, 80, 128, "white"), (112, 97, 20, "extremes"), (128, 112, 100, "noise"), (176, 144, 64, "extremes"),
    (240, 130, 128, "extremes"), (1040, 64, 128, "noise"), (32, 528, 128, "noise"), (320, 272, 36, "white"),
])
def test_table_edges_against_oracle(vpp, ctx, orc, w, h, mr, kind):
    src, ref = _planes(kind, w * h + mr, w, h)
    incl = np.ones((w // 16) * (h // 16), np.uint8)
    me = vpp.MotionEstimatorH264ImplFull(src, ref, w, h, mr, pDistortionIncluded=incl, ctx=ctx)
    assert me.Create() == 1
    mv, avg = me.Estimate()
    want_mv, want_dist, want_avg = orc.me_full(src, ref, mr, dist_incl=incl)
    np.testing.assert_array_equal(mv, want_mv)
    np.testing.assert_array_equal(me.last_mb_distortion, want_dist)
    assert avg == want_avg
