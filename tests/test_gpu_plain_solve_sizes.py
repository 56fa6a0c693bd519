"""The plain path's global LU and back-substitution at system sizes around the
cluster's column split (16 CTAs) and the 32-term steps of the ordered
differences: every solution, kernel sum and decision equals the FP64 oracle's
bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dg,korder,bgorder", [
    ([1], 0, 0),          # n = 4
    ([3, 1], 0, 1),       # 16
    ([3, 1], 0, 2),       # 19
    ([4, 2], 1, 0),       # 62
    ([6, 4, 2], 1, 2)])   # 151
def test_solutions_equal_the_oracle(oracle, dg, korder, bgorder):
    import xbach
    from xbach.synth import make_pair
    T, S, info = make_pair(1, frame=2)
    sigma = [0.7, 1.5, 3.0]
    kw = dict(stampsx=info["stamps"], stampsy=info["stamps"], threshHigh=info["threshHigh"],
              nGauss=len(dg), dg=dg + [0] * (8 - len(dg)),
              bg=[1 / (2 * s * s) for s in sigma[:len(dg)]] + [0.0] * (8 - len(dg)),
              kernelOrder=korder, backgroundOrder=bgorder)
    ctx = xbach.Context(xbach.default_params(**kw), trace=True)
    ctx.run_all(T, S)
    p = oracle.default_params()
    for k, v in kw.items():
        if k in ("dg", "bg"):
            arr = getattr(p, k)
            for j, x in enumerate(v):
                arr[j] = x
        else:
            setattr(p, k, v)
    ref = oracle.run(p, T.astype(np.float64), S.astype(np.float64))
    assert ref.status == 0
    for k in ("convTemplate", "ksc_iterations", "nstamps0", "nstamps1", "merit0", "merit1"):
        assert ctx.scalar(k) == ref.scalar(k), k
    for k in ("cd_solution0", "cd_solution1", "solution"):
        a, b = ctx.array(k, np.float64), ref.array(k, np.float64)
        n = min(len(a), len(b))
        assert np.array_equal(a[:n].view(np.uint64), b[:n].view(np.uint64)), k
    assert ctx.scalar("kernSum") == ref.scalar("kernSum")
