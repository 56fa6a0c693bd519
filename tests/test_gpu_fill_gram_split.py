"""The fused fill + Gram kernel on short lists, where four CTAs share a stamp by
output rows (csrc/xb_fill_gram.cu), against the separate kernels, bit for bit:
substamps of one row block (ranks without rows) up to four, stamps at the frame's
edges, and frames whose rows are no 16-byte multiples."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ARRAYS = {"Wf0": np.float32, "Wlo0": np.float32, "Wf1": np.float32, "Wlo1": np.float32,
          "Q0": np.float64, "Q1": np.float64, "B0": np.float64, "B1": np.float64}


@pytest.mark.parametrize("size,stamps,hss", [(400, 3, 2), (400, 3, 3), (401, 4, 4), (400, 3, 7),
                                             (402, 3, 8), (400, 3, 11), (400, 2, 12), (500, 4, 15),
                                             (700, 8, 15), (503, 3, 15), (720, 9, 15)])
def test_short_lists_equal_separate_kernels(size, stamps, hss):
    import xbach
    from xbach.synth import make_pair
    T, S, info = make_pair(2, frame=size, size=size, n_src=int(0.006 * size * size), stamps=stamps)
    kw = dict(stampsx=stamps, stampsy=stamps, threshHigh=info["threshHigh"], hSStampWidth=hss)
    res = []
    for fused in (1, 0):
        ctx = xbach.Context(xbach.default_params(mode=xbach.XB_MODE_MIXED, **kw), trace=True)
        ctx.set_option("fill_gram", fused)
        ctx.init(T, S)
        ctx.sss()
        ctx.cmv()
        res.append({k: ctx.array(k, dt) for k, dt in ARRAYS.items()})
        assert ctx.scalar("nstamps0") > 0
        ctx.cd()
        ctx.ksc()
        res[-1].update(sol=ctx.solution(), cur=ctx.array("cur", np.int32))
        ctx.close()
    for k, a in res[0].items():
        assert a.size > 0 and np.array_equal(a.view(np.uint8), res[1][k].view(np.uint8)), k
