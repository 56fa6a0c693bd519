"""The substamp search against the FP64 oracle over stamp and window sizes: row
winners of windows narrower than a task's eight columns and wider than a warp,
one to six words per bit row, stamps that just fit in shared memory and ones
that take the maps in global memory.  Substamp sets, values and the mask are
identical."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size,stamps,hss", [
    (330, 5, 2), (330, 5, 3), (330, 5, 4), (330, 5, 7), (400, 5, 15), (500, 4, 16), (640, 5, 20),
    (632, 4, 15), (600, 3, 15), (630, 3, 15), (660, 3, 15)])
def test_substamps_equal_the_oracle(oracle, size, stamps, hss):
    import xbach
    from xbach.synth import make_pair
    T, S, info = make_pair(2, frame=size, size=size, n_src=int(0.006 * size * size), stamps=stamps)
    kw = dict(stampsx=stamps, stampsy=stamps, threshHigh=info["threshHigh"], hSStampWidth=hss)
    ctx = xbach.Context(xbach.default_params(**kw), trace=True)
    ctx.init(T, S)
    ctx.sss()
    p = oracle.default_params(**kw)
    ref = oracle.run(p, T.astype(np.float64), S.astype(np.float64))
    for k in ("nstamps0", "nstamps1"):
        assert ctx.scalar(k) == ref.scalar(k) and ctx.scalar(k) > 0, k
    for im in "01":
        for k in ("ss_count_all", "ss_xy_all"):
            assert np.array_equal(ctx.array(k + im, np.int32), ref.array(k + im, np.int32)), k + im
        a, b = ctx.array("ss_val_all" + im, np.float64), ref.array("ss_val_all" + im, np.float64)
        assert np.array_equal(a.view(np.uint64), b.view(np.uint64)), im
    assert np.array_equal(ctx.array("mask_sss", np.uint16), ref.array("mask_sss", np.uint16))
