"""The substamp search with lists of candidates that fill exactly (csrc/xb_sss.cu:
2048 at a time, 512 in stamps of 189 and 190 px, collected 512 words of 32 pixels
at a time), one below and one above, as the first list of a stamp and as a resumed
one.  Every listed candidate has a bad pixel in its window and one good substamp
lies behind them, in words that the list did not reach.  Substamps, values and
mask equal the FP64 oracle's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

STAMP, SIDE = 4, 3   # the middle one of 3 x 3 stamps


def _frame(width, counts, rows, star):
    """Candidates counts[i] in the rows rows[i] of the middle stamp, zeros on a
    grid of seven pixels down to ten rows above the star."""
    size = 3 * (width + 21)
    rng = np.random.default_rng(width + sum(counts))
    T = 1000 + 30 * rng.uniform(-1, 1, (size, size))
    y, x = np.mgrid[:size, :size]
    c = width + 21
    for sy in range(3):
        for sx in range(3):
            cy, cx = sy * c + (star if (sy, sx) == (1, 1) else 100), sx * c + 100
            T += 2.82e4 * np.exp(-((y - cy) ** 2 + (x - cx) ** 2) / 4.5)
    s = T[c:c + width, c:c + width]   # a view of the middle stamp
    zero = np.zeros(s.shape, bool)
    zero[3:star - 10:7, 3::7] = True
    s[zero] = 0
    for n, (r0, r1) in zip(counts, rows):
        free = np.flatnonzero(~zero[r0:r1].ravel())
        at = r0 * width + rng.choice(free, n, replace=False)
        s[np.unravel_index(at, s.shape)] = rng.uniform(2.75e4, 2.85e4, n)
    return T.astype(np.float32)


@pytest.mark.parametrize("width,counts,rows,star", [
    (183, (2047,), [(0, 85)], 150), (183, (2048,), [(0, 85)], 150), (183, (2049,), [(0, 85)], 150),
    (183, (2048, 2048), [(0, 70), (70, 150)], 172), (183, (2048, 2047), [(0, 70), (70, 150)], 172),
    (189, (511,), [(0, 85)], 150), (189, (512,), [(0, 85)], 150), (189, (513,), [(0, 85)], 150),
    (189, (512, 512), [(0, 70), (70, 150)], 172), (189, (512, 513), [(0, 70), (70, 150)], 172)])
def test_full_list_equals_the_oracle(oracle, width, counts, rows, star):
    import xbach
    T = _frame(width, counts, rows, star)
    S = (T * np.float32(1.02)).astype(np.float32)
    kw = dict(stampsx=SIDE, stampsy=SIDE, threshHigh=3e4, hSStampWidth=7, threshKernFit=6)
    ref = oracle.run(oracle.default_params(**kw), T.astype(np.float64), S.astype(np.float64))
    assert ref.scalar("fStampWidth") == width
    for im in "01":  # the star is the middle stamp's only substamp
        n = ref.array("ss_count_all" + im, np.int32)
        xy = ref.array("ss_xy_all" + im, np.int32).reshape(len(n), -1, 2)
        assert n[STAMP] == 1 and tuple(xy[STAMP, 0]) == (width + 21 + 100, width + 21 + star)
    ctx = xbach.Context(xbach.default_params(**kw), trace=True)
    ctx.init(T, S)
    ctx.sss()
    for im in "01":
        for k in ("ss_count_all", "ss_xy_all"):
            assert np.array_equal(ctx.array(k + im, np.int32), ref.array(k + im, np.int32)), k + im
        a, b = ctx.array("ss_val_all" + im, np.float64), ref.array("ss_val_all" + im, np.float64)
        assert np.array_equal(a.view(np.uint64), b.view(np.uint64)), im
    assert np.array_equal(ctx.array("mask_sss", np.uint16), ref.array("mask_sss", np.uint16))
    ctx.close()
