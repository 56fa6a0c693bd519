"""Fits whose matrix has zero rows: a basis with a Gaussian so narrow that its odd
functions vanish, and one of two equal Gaussians.  The pivot is zero, so the mixed
path's cluster LDL^T (csrc/xb_ldl.cu) hands both of cd's fits and ksc's to the
pivoted LU, which reports the singular matrix as the plain path and the reference
do; staged on 16- and 8-CTA clusters, and captured and replayed as a frame graph."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dg,bg,korder", [([2, 1], [1 / (2 * 1.5 ** 2), 1e4], 0),
                                          ([2, 0], [1 / (2 * 1.5 ** 2)] * 2, 1)])
def test_zero_rows_end_as_in_the_oracle(oracle, dg, bg, korder):
    import xbach
    from xbach.synth import make_pair
    T, S, info = make_pair(1, frame=2)
    kw = dict(stampsx=info["stamps"], stampsy=info["stamps"], threshHigh=info["threshHigh"],
              nGauss=2, dg=dg + [0] * 6, bg=bg + [0.0] * 6, kernelOrder=korder, backgroundOrder=1)
    ref = oracle.run(oracle.default_params(**kw), T.astype(np.float64), S.astype(np.float64))
    assert ref.scalar("singular") == 1 and np.isnan(ref.scalar("kernSum"))
    for mode, cluster, graph in ((xbach.XB_MODE_PLAIN, 16, 0), (xbach.XB_MODE_MIXED, 16, 0),
                                 (xbach.XB_MODE_MIXED, 8, 0), (xbach.XB_MODE_MIXED, 16, 1)):
        ctx = xbach.Context(xbach.default_params(mode=mode, **kw))
        ctx.set_option("ldl_cluster", cluster)
        ctx.set_option("graph", graph)
        for _ in range(2 if graph else 1):
            if graph:
                ctx.run(T, S)
            else:
                ctx.run_all(T, S)
            for k in ("singular", "merit0", "merit1", "convTemplate", "ksc_iterations"):
                assert ctx.scalar(k) == ref.scalar(k), (mode, cluster, graph, k)
            assert np.isnan(ctx.scalar("kernSum"))
        ctx.close()
