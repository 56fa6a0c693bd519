"""The mixed convolution (csrc/xb_mixed.cu) against the plain mode's over frame
sizes whose last kernel blocks and rows are cut (one to 21 pixels left, groups of
seven rows), with masked and saturated pixels, background orders and an input
mask, by the mixed path's acceptance (1e-3 of the pixel noise; masks equal but
where the FP32 good-fraction test sits on 0.99).  Blocks per CTA change nothing."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h,bg", [(512, 503, 1), (504, 512, 0), (492, 511, 2), (505, 493, 1), (491, 494, 2)])
def test_conv_and_mask_match_plain(w, h, bg):
    import xbach
    from xbach.accuracy import is_bad
    from xbach.synth import make_pair
    T, S, info = make_pair(1)
    T, S = T[:h, :w].copy(), S[:h, :w].copy()
    rng = np.random.default_rng(w)
    for im in (T, S):
        im[rng.integers(h, size=20), rng.integers(w, size=20)] = 0
    inp = (rng.uniform(size=(h, w)) < 0.0002).astype(np.uint8)
    res = []
    for mode, v in ((xbach.XB_MODE_PLAIN, 0), (xbach.XB_MODE_MIXED, 0), (xbach.XB_MODE_MIXED, 1),
                    (xbach.XB_MODE_MIXED, 2)):
        ctx = xbach.Context(xbach.default_params(mode=mode, stampsx=info["stamps"], stampsy=info["stamps"],
                                                 backgroundOrder=bg, threshHigh=info["threshHigh"]),
                            trace=True)
        ctx.set_option("tune_variant", v)
        ctx.set_input_mask(inp)
        ctx.run_all(T, S)
        res.append([np.asarray(x).reshape(h, w) for x in (
            ctx.image(xbach.XB_IMG_CONV), ctx.image(xbach.XB_IMG_DIFF), ctx.array("mask", np.uint16))])
        ct = ctx.scalar("convTemplate")
        ctx.close()
    (cp, dp, mp), (cm, dm, mm) = res[0], res[1]
    target = S if ct else T
    ok = ~is_bad(dp) & ~is_bad(dm)
    assert ok.mean() > 0.3
    sigma = np.sqrt(np.abs(target) + np.abs(cp) + 2 * 5.0 ** 2)
    assert (np.abs(dm - dp)[ok] / sigma[ok]).max() <= 1e-3
    assert np.mean(mp != mm) < 1e-4
    for other in res[2:]:
        for a, b in zip(res[1], other):
            assert np.array_equal(a, b)
