"""The mixed per-pixel convolution (csrc/xb_mixed.cu) on low frames whose last
CTA of a row holds one to five kernel blocks past the frame, with fewer block rows
than that, and with bad pixels in the last columns and rows (whose clamped copies
fill those blocks): against the plain mode's, by the mixed path's acceptance (1e-3
of the pixel noise; masks equal but where the FP32 good-fraction test sits on
0.99), and the same bits from a context that has held other frames."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h,order", [(1012, 84, 1), (1029, 80, 0), (1030, 84, 1), (1050, 92, 1), (1092, 105, 1),
                                       (1113, 84, 1)])
def test_low_frames_match_plain(w, h, order):
    import xbach
    from xbach.accuracy import is_bad
    from xbach.synth import make_pair
    T, S, info = make_pair(1, size=w, n_src=int(0.009 * w * w))
    T, S = T[:h].copy(), S[:h].copy()
    rng = np.random.default_rng(w)
    for im in (T, S):
        im[rng.integers(h, size=20), rng.integers(w, size=20)] = 0
    T[:, -1] = S[-1] = 0
    kw = dict(stampsx=w // 84, stampsy=1, hSStampWidth=7, kernelOrder=order, backgroundOrder=0,
              threshHigh=info["threshHigh"], convPerPixel=1)
    res = []
    for mode in (xbach.XB_MODE_PLAIN, xbach.XB_MODE_MIXED):
        ctx = xbach.Context(xbach.default_params(mode=mode, **kw), trace=True)
        for t, s in ([(T, S)] if mode == xbach.XB_MODE_PLAIN else [(T, S), (T[::-1], S[::-1]), (T, S)]):
            ctx.run_all(np.ascontiguousarray(t), np.ascontiguousarray(s))
            res.append([np.asarray(x).reshape(h, w) for x in (
                ctx.image(xbach.XB_IMG_CONV), ctx.image(xbach.XB_IMG_DIFF), ctx.array("mask", np.uint16))])
        ct = ctx.scalar("convTemplate")
        ctx.close()
    (cp, dp, mp), first, _, again = res
    cm, dm, mm = first
    ok = ~is_bad(dp) & ~is_bad(dm)
    assert ok.mean() > 0.3
    sigma = np.sqrt(np.abs(S if ct else T) + np.abs(cp) + 2 * 5.0 ** 2)
    assert (np.abs(dm - dp)[ok] / sigma[ok]).max() <= 1e-3
    assert np.mean(mp != mm) < 1e-4
    for a, b in zip(first, again):
        assert np.array_equal(a, b)
