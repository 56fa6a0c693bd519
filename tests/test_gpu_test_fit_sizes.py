"""The mixed per-stamp test fit (csrc/xb_fit.cu) over numbers of unknowns (from
one, through the lanes of a warp, to 60) and stamp counts: the kernel sum of
each stamp of both sets against the solve of its own Q and B.

Elimination of a positive definite system of n unknowns is backward stable, so
each solution lies within about n^2 2^-53 cond(Q) |x| of the exact one."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dg,stamps", [([0], 5), ([1], 2), ([2, 0], 12), ([6, 1], 7), ([7], 3),
                                       ([6, 4, 2], 9), ([7, 4, 2, 0], 6), ([6, 4, 3, 2], 4)])
def test_kernel_sums_solve_their_systems(dg, stamps):
    import xbach
    from xbach.synth import make_pair
    size = max(64 * stamps, 400)
    T, S, info = make_pair(2, frame=size, size=size, n_src=int(0.006 * size * size), stamps=stamps)
    ctx = xbach.Context(xbach.default_params(mode=xbach.XB_MODE_MIXED, stampsx=stamps, stampsy=stamps,
                                             threshHigh=info["threshHigh"], nGauss=len(dg),
                                             dg=dg + [0] * (8 - len(dg)),
                                             bg=[1.4, 0.35, 0.09, 0.02][:len(dg)]), trace=True)
    ctx.init(T, S)
    ctx.sss()
    ctx.cmv()
    Qs, Bs = ([ctx.array(k + im, np.float64) for im in "01"] for k in "QB")
    ctx.cd()
    for si in range(2):
        ks = ctx.array("kernel_sums%d" % si, np.float64)
        n = ks.size
        assert n > 0
        qc = Bs[si].size // n
        Q, B = Qs[si].reshape(n, qc, qc)[:, 1:, 1:], Bs[si].reshape(n, qc)[:, 1:]
        for s in range(n):
            A = np.tril(Q[s]) + np.tril(Q[s], -1).T
            d = 1 / np.sqrt(np.diag(A))  # elimination is invariant under the scaling
            x = d * np.linalg.solve(A * d[:, None] * d, B[s] * d)
            tol = qc ** 2 * 2.0 ** -53 * np.linalg.cond(A * d[:, None] * d) * np.linalg.norm(x / d) * d[0]
            assert abs(ks[s] - x[0]) <= tol, (si, s)
    ctx.close()
