"""The stamp statistics against the FP64 oracle over stamp sizes (good pixels in
shared memory, in the scratch slice with chunk sums in shared
memory and without) and pixel contents: sky and sources, a constant, a dynamic
range whose plain sums are not exact in 53 bits, pixels around zero, NaN pixels
and mostly masked stamps.  Sky, width and mask are identical."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _frames(size, stamps):
    from xbach.synth import make_pair
    T, S, info = make_pair(2, frame=size, size=size, n_src=int(0.006 * size * size), stamps=stamps)
    rng = np.random.default_rng(size)
    cell = size // stamps
    out = []
    for im in (T, S):
        im = np.array(im, np.float32)
        for k in range(stamps * stamps):
            y, x = (k // stamps) * cell, (k % stamps) * cell
            c = im[y:y + cell, x:x + cell]
            kind = k % 7 if stamps > 2 else 0
            if kind == 1:
                c[:] = 1000
            elif kind == 2:
                c[:] = np.exp(rng.normal(0, 3.5, c.shape))
            elif kind == 3:
                c[:] = rng.normal(0, 30, c.shape)
            elif kind == 4:
                c[rng.uniform(size=c.shape) < 0.05] = np.nan
            elif kind == 5:
                c[rng.uniform(size=c.shape) < 0.999] = 0
        out.append(im)
    return out[0], out[1], info


@pytest.mark.parametrize("size,stamps,f64", [
    (330, 5, False), (330, 5, True), (400, 3, False), (632, 4, False), (504, 3, False),
    (640, 3, False), (708, 3, False), (705, 3, False), (720, 3, False), (720, 3, True),
    (900, 3, False), (300, 1, False)])
def test_sky_and_width_equal_the_oracle(oracle, size, stamps, f64):
    import xbach
    T, S, info = _frames(size, stamps)
    kw = dict(stampsx=stamps, stampsy=stamps, threshHigh=info["threshHigh"], threshLow=-1e9)
    ctx = xbach.Context(xbach.default_params(**kw), trace=True)
    ctx.init(*((T.astype(np.float64), S.astype(np.float64)) if f64 else (T, S)))
    ctx.sss()
    ref = oracle.run(oracle.default_params(**kw), T.astype(np.float64), S.astype(np.float64))
    for k in ("sky0", "fwhm0", "sky1", "fwhm1"):
        a, b = ctx.array(k, np.float64), ref.array(k, np.float64)
        assert a.size > 0 and np.array_equal(a.view(np.uint64), b.view(np.uint64)), k
    assert np.array_equal(ctx.array("mask_sss", np.uint16), ref.array("mask_sss", np.uint16))
    ctx.close()
