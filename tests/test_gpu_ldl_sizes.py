"""The cluster LDL^T solve of the mixed path at system sizes around its panel
width of 16: fewer unknowns than one panel, whole panels, a remainder, many
panels.  The difference image is held to the mixed path's acceptance, 1e-3 of
the per-pixel noise of the plain FP64 result, and an 8-CTA cluster gives the
bits of the 16-CTA one."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dg,korder,bgorder,n", [
    ([1], 0, 0, 4), ([3, 1], 0, 1, 16), ([3, 1], 0, 2, 19), ([4, 2], 1, 1, 64),
    ([6, 4, 2], 1, 1, 148), ([6, 4, 2], 3, 1, 484)])
def test_system_sizes(dg, korder, bgorder, n):
    import xbach
    from xbach.accuracy import diff_error
    from xbach.synth import make_pair
    T, S, info = make_pair(1)
    sigma = [0.7, 1.5, 3.0]
    kw = dict(stampsx=info["stamps"], stampsy=info["stamps"], threshHigh=info["threshHigh"],
              nGauss=len(dg), dg=dg + [0] * (8 - len(dg)),
              bg=[1 / (2 * s * s) for s in sigma[:len(dg)]] + [0.0] * (8 - len(dg)),
              kernelOrder=korder, backgroundOrder=bgorder)
    out = {}
    for name, mode, cluster in (("plain", xbach.XB_MODE_PLAIN, 16),
                                ("mixed", xbach.XB_MODE_MIXED, 16),
                                ("mixed8", xbach.XB_MODE_MIXED, 8)):
        if cluster == 8 and n > 300:
            continue
        ctx = xbach.Context(xbach.default_params(mode=mode, **kw))
        ctx.set_option("ldl_cluster", cluster)
        ctx.run_all(T, S)
        out[name] = dict(sol=ctx.solution(), diff=ctx.image(xbach.XB_IMG_DIFF),
                         conv=ctx.image(xbach.XB_IMG_CONV), ct=ctx.scalar("convTemplate"))
    a, b = out["plain"], out["mixed"]
    assert len(a["sol"]) > n and a["ct"] == b["ct"]
    target = S if a["ct"] else T
    assert diff_error(b["diff"], a["diff"], a["conv"], target)["max_sigma"] <= 1e-3
    if "mixed8" in out:
        assert np.array_equal(b["sol"], out["mixed8"]["sol"])
        assert np.array_equal(b["diff"], out["mixed8"]["diff"])
