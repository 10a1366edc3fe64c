"""The lane-per-candidate search of the multi-resolution estimators against the CPU oracle, bit-exact, where it
can go wrong: pictures of one macroblock and row pitches that are no multiple of four (every read then starts at
another byte of its word), windows that reach past the reference copy, hard 0/255 content (6-tap sums at their
extremes, partial distortions that reject late), half-pel shifts (winners beside the incomplete row and column of
the sub-pel window) and content rich in ties."""
import numpy as np
import pytest

from imagecodingutils_gb300 import synth

pytestmark = pytest.mark.gpu

ESTIMATORS = [("MotionEstimatorH264ImplMultiresCross", "me_multires_cross", 1, {}),
              ("MotionEstimatorH264ImplMultiresCrossVer2", "me_multires_cross_v2", 1, {}),
              ("MotionEstimatorH264ImplMultires", "me_multires", 1, {}),
              ("MotionEstimatorH263ImplMultiresCross", "me_h263_multires_cross", 2, {}),
              ("MotionEstimatorH263ImplMultiresCrossVer2", "me_h263_multires_cross_ver2", 2, {}),
              ("MotionEstimatorH264ImplMultiresCrossVer2", "me_multires_cross_v2_lambda", 1, {"lam": 1.5})]


def frames(kind, seed, w, h):
    big = synth.splitmix64(seed, (h + 8) * (w + 8)).reshape(h + 8, w + 8)
    if kind == "hard":  # blocks of black and white, every eighth sample of the second frame its own
        a = np.repeat(np.repeat((big[::2, ::2] & np.uint64(1)) * np.uint64(255), 2, 0), 2, 1)[:h + 8, :w + 8]
        b = np.where(big[1:h + 1, 2:w + 2] & np.uint64(0x700), a[3:h + 3, 2:w + 2], big[1:h + 1, 2:w + 2] & np.uint64(255))
        return a[2:h + 2, 2:w + 2].astype(np.int16), b.astype(np.int16)
    if kind == "ties":
        a = (big & np.uint64(1)) + np.uint64(100)
        return a[:h, :w].astype(np.int16), a[2:h + 2, 2:w + 2].astype(np.int16)
    y, x = np.mgrid[0:h + 8, 0:w + 8]
    s = 128 + 60 * np.sin(x / 3.1) * np.cos(y / 2.7) + (big & np.uint64(31)).astype(np.float64)
    a = np.clip(s, 0, 255).astype(np.int64)
    b = (a[:-1, :-1] + a[1:, :-1] + a[:-1, 1:] + a[1:, 1:] + 2) >> 2  # half a pel both ways
    return a[2:h + 2, 2:w + 2].astype(np.int16), b[3:h + 3, 1:w + 1].astype(np.int16)


@pytest.mark.parametrize("kind", ["hard", "ties", "half"])
@pytest.mark.parametrize("w,h,mr,mode", [(16, 16, 32, 2), (48, 36, 64, 2), (32, 50, 64, 1), (112, 68, 128, 2)])
@pytest.mark.parametrize("est", range(len(ESTIMATORS)))
def test_against_oracle(vpp, ctx, orc, est, w, h, mr, mode, kind):
    cls, fn, div, extra = ESTIMATORS[est]
    ref, src = frames(kind, 300 + w, w, h)
    me = getattr(vpp, cls)(src, ref, w, h, mr // div, ctx=ctx)
    assert me.Create() == 1
    me.SetMode(mode)
    mv, avg = me.Estimate(param=extra["lam"]) if extra else me.Estimate()
    args = (src, ref, mr // div) + tuple(extra.values())
    mv_o, dist_o, avg_o = getattr(orc, fn)(*args, mode=mode)
    np.testing.assert_array_equal(mv, mv_o)
    np.testing.assert_array_equal(me.last_mb_distortion, dist_o)
    assert avg == avg_o


@pytest.mark.parametrize("kind,w,h,mr", [("half", 848, 478, 128), ("ties", 48, 38, 64), ("hard", 32, 50, 64),
                                         ("half", 48, 37, 64), ("hard", 80, 19, 32)])
@pytest.mark.parametrize("est", range(len(ESTIMATORS)))
def test_heights_of_odd_levels(vpp, ctx, orc, est, kind, w, h, mr):
    """Three levels of pictures whose height is no multiple of four: the last row of a level, and of its bordered copy,
    comes from fewer rows than two."""
    test_against_oracle(vpp, ctx, orc, est, w, h, mr, 2, kind)
