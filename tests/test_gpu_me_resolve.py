"""The predictor resolve's cluster kernel at the shapes where its layout changes: one, four, eight and sixteen CTAs,
bands that do not divide the rows, single rows and columns, distortions beside the vectors or in global memory.
Bit-exact against the oracle; a +-1 pel search on half-related textures keeps the predictions moving."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _pair(seed, w, h):
    """Two smooth textures of a 512-sample period, the second half the first and half one of its own: every
    macroblock's best candidate is another."""
    from imagecodingutils_gb300 import synth
    a, b = synth.smooth_texture(seed, 512, 512), synth.smooth_texture(seed + 1, 512, 512)
    tiled = lambda t: np.ascontiguousarray(np.tile(t, (-(-h // 512), -(-w // 512)))[:h, :w].astype(np.int16))
    return tiled(a), tiled((np.roll(a, (1, -1), axis=(0, 1)).astype(np.int32) + b) // 2)


@pytest.mark.parametrize("w,h", [
    (16, 16), (16, 1040), (2048, 16), (352, 288),  # one CTA
    (528, 272), (1024, 500),                       # four, the last band short or empty
    (1936, 1090), (1040, 2064),                    # eight
    (8192, 3600),                                  # sixteen, distortions in shared memory
    (8192, 8192),                                  # sixteen, distortions in global memory
])
def test_resolve_shapes_against_oracle(vpp, ctx, orc, w, h):
    src, ref = _pair(w + h, w, h)
    n = (w // 16) * (h // 16)
    incl = (np.arange(n) % 3 != 0).astype(np.uint8)
    me = vpp.MotionEstimatorH264ImplFull(src, ref, w, h, 8, pDistortionIncluded=incl, ctx=ctx)
    assert me.Create() == 1
    mv, avg = me.Estimate()
    want_mv, want_dist, want_avg = orc.me_full(src, ref, 8, dist_incl=incl)
    np.testing.assert_array_equal(mv, want_mv)
    np.testing.assert_array_equal(me.last_mb_distortion, want_dist)
    assert avg == want_avg
