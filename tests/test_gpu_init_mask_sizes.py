"""The init masks (csrc/xb_ctx.cu) against NumPy over frame widths around the
32-pixel words and the 256-pixel rows of a warp, spreads within one word and over
several, both pixel types, thresholds between two floats, and an input mask."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h,hk,factor,f64", [
    (256, 40, 10, 1.0, False), (257, 33, 10, 0.1, False), (31, 50, 3, 1.0, False),
    (289, 70, 10, 3.0, False), (300, 90, 20, 3.3, False), (700, 120, 20, 7.0, True),
    (64, 65, 16, 4.0, False), (1000, 9, 10, 0.0, True)])
def test_mask_and_spread_equal_numpy(w, h, hk, factor, f64):
    import xbach
    rng = np.random.default_rng(w)
    dt = np.float64 if f64 else np.float32
    th, tl = 1200.0000001, 800.00000001  # between two floats
    T = rng.uniform(810, 1190, (h, w)).astype(dt)
    S = rng.uniform(810, 1190, (h, w)).astype(dt)
    for im in (T, S):
        for v in (0, 1200, np.nextafter(np.float32(1200), np.float32(2000)), 800,
                  np.nextafter(np.float32(800), np.float32(2000)), np.nan, np.inf, -np.inf):
            im[rng.integers(h), rng.integers(w)] = v
    inp = (rng.uniform(size=(h, w)) < 0.0005).astype(np.uint8)
    ctx = xbach.Context(xbach.default_params(hKernelWidth=hk, inSpreadMaskFactor=factor, threshHigh=th,
                                             threshLow=tl, stampsx=1, stampsy=1), trace=True)
    ctx.set_input_mask(inp)
    ctx.init(T, S)
    got = ctx.array("mask_init", np.uint16).reshape(h, w)
    border = ctx.params.hSStampWidth + hk
    ref = np.zeros((h, w), np.uint16)
    a, b = T.astype(np.float64), S.astype(np.float64)
    ref[(a == 0) | (b == 0)] |= 1 << 7 | 1 << 0
    ref[(a >= th) | (b >= th)] |= 1 << 7 | 1 << 1
    ref[(a <= tl) | (b <= tl)] |= 1 << 7 | 1 << 2
    y, x = np.mgrid[:h, :w]
    ref[(x < border) | (x >= w - border) | (y < border) | (y >= h - border)] |= 1 << 8 | 1 << 10
    ref[inp > 0] |= 1 << 5 | 1 << 7
    r = int(hk * np.float64(factor)) // 2
    bad = (ref & 1 << 7) > 0
    assert bad.any()
    near = np.zeros_like(bad)
    for yy, xx in zip(*np.nonzero(bad)):
        near[max(yy - r, 0):yy + r + 1, max(xx - r, 0):xx + r + 1] = True
    if r:
        ref[near & ~bad] |= 1 << 6
    assert np.array_equal(got, ref)
    ctx.close()
