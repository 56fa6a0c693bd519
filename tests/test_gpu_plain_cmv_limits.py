"""The plain path's cmv with more basis and background products per stamp than
its fits take (csrc/xb_fit.cu: 1024): the substamp matrices are made and equal the
oracle's bit for bit, and cd refuses the fit.  With 1024 or fewer both pass."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

XB_ERR_UNSUPPORTED = 10


@pytest.mark.parametrize("dg,bgorder,fits", [
    ([6, 4, 3, 2], 4, False),    # 59 functions: 58 * 15 + 15 + 225 = 1110
    ([6, 4, 2], 4, True)])       # 49 functions: 48 * 15 + 15 + 225 = 960
def test_cmv_beyond_the_fits(oracle, dg, bgorder, fits):
    import xbach
    from xbach.synth import make_pair
    T, S, info = make_pair(1, frame=2)
    sigma = [0.6, 1.2, 2.4, 4.8]
    kw = dict(stampsx=info["stamps"], stampsy=info["stamps"], threshHigh=info["threshHigh"],
              nGauss=len(dg), dg=dg + [0] * (8 - len(dg)),
              bg=[1 / (2 * s * s) for s in sigma[:len(dg)]] + [0.0] * (8 - len(dg)),
              kernelOrder=1, backgroundOrder=bgorder)
    ref = oracle.run(oracle.default_params(**kw), T.astype(np.float64), S.astype(np.float64))
    ctx = xbach.Context(xbach.default_params(**kw), trace=True)
    ctx.init(T, S)
    ctx.sss()
    ctx.cmv()
    for k in ("Q0", "Q1", "B0", "B1"):
        a, b = ctx.array(k, np.float64), ref.array(k, np.float64)
        assert np.array_equal(a.view(np.uint64), b.view(np.uint64)), k
    if fits:
        assert ctx.cd() == ref.scalar("convTemplate")
    else:
        with pytest.raises(xbach.XbError) as e:
            ctx.cd()
        assert e.value.code == XB_ERR_UNSUPPORTED
    ctx.close()
