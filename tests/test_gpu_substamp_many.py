"""The substamp search with far more candidates per stamp than one list of it
holds (csrc/xb_sss.cu, 2048 at a time, 512 in the largest stamps), most of them
with a bad window, against the FP64 oracle: substamps, values and mask are
identical."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size,stamps,dens,clean", [(420, 3, 0.2, 60), (560, 3, 0.15, 60), (400, 2, 0.2, 50),
                                                    (300, 2, 0.22, 60), (630, 3, 0.15, 60), (633, 3, 0.15, 60)])
def test_many_candidates_equal_the_oracle(oracle, size, stamps, dens, clean):
    import xbach
    rng = np.random.default_rng(size + clean)
    T = rng.normal(1000, 20, (size, size))
    up = rng.uniform(size=T.shape) < dens
    T[up] += rng.uniform(2000, 4000, up.sum())
    # a bad pixel in most windows, but none in the lower right corner of each stamp
    c = size // stamps
    y, x = np.mgrid[:size, :size]
    T[(rng.uniform(size=T.shape) < 0.01) & ~((y % c > c - clean) & (x % c > c - clean))] = 0
    T = T.astype(np.float32)
    S = (T * np.float32(1.02)).astype(np.float32)
    kw = dict(stampsx=stamps, stampsy=stamps, threshHigh=3e4, hSStampWidth=7, threshKernFit=3)
    ctx = xbach.Context(xbach.default_params(**kw), trace=True)
    ctx.init(T, S)
    ctx.sss()
    ref = oracle.run(oracle.default_params(**kw), T.astype(np.float64), S.astype(np.float64))
    for im in "01":
        for k in ("ss_count_all", "ss_xy_all"):
            assert np.array_equal(ctx.array(k + im, np.int32), ref.array(k + im, np.int32)), k + im
        a, b = ctx.array("ss_val_all" + im, np.float64), ref.array("ss_val_all" + im, np.float64)
        assert np.array_equal(a.view(np.uint64), b.view(np.uint64)), im
    assert np.array_equal(ctx.array("mask_sss", np.uint16), ref.array("mask_sss", np.uint16))
    ctx.close()
