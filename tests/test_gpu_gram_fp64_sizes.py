"""The FP64 Gram kernel of the mixed path against the sums of its own W rows
over stamp counts (a few stamps, spread over many CTAs, and full lists), pixel
tiles (25 to 961 pixels, a last tile of 1 to 32) and row counts (three, more
than the tensor-core kernel's 64, and too many to stage in shared memory).

Each entry is one chain of K fused multiply-adds of the exact hi + lo, so it
lies within K 2^-53 of the sum of the magnitudes; the NumPy sum has the same
bound."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

THREE = dict(nGauss=1, dg=[1], bg=[0.4])
WIDE = dict(nGauss=4, dg=[6, 4, 3, 2], bg=[1.4, 0.35, 0.09, 0.02])


@pytest.mark.parametrize("stamps,hss,basis,order", [
    (2, 2, {}, 1), (2, 15, {}, 1), (12, 2, {}, 1), (12, 7, {}, 2), (10, 15, WIDE, 2), (2, 12, WIDE, 2),
    (3, 7, THREE, 0), (12, 8, THREE, 0), (2, 7, {}, 23)])
def test_gram_entries_are_the_sums_of_products(stamps, hss, basis, order):
    import xbach
    from xbach.synth import make_pair
    size = max(64 * stamps, 400)
    T, S, info = make_pair(2, frame=size, size=size, n_src=int(0.006 * size * size), stamps=stamps)
    ctx = xbach.Context(xbach.default_params(mode=xbach.XB_MODE_MIXED, stampsx=stamps, stampsy=stamps,
                                             threshHigh=info["threshHigh"], hSStampWidth=hss,
                                             backgroundOrder=order, **basis), trace=True)
    ctx.set_option("gram_fp64", 1)
    ctx.init(T, S)
    ctx.sss()
    ctx.cmv()
    K = (2 * hss + 1) ** 2
    ld = (K + 31) // 32 * 32
    for im in "01":
        n = int(ctx.scalar("nstamps" + im))
        assert n > 0
        W = ctx.array("Wf" + im, np.float32).astype(np.float64) + ctx.array("Wlo" + im, np.float32)
        W = W.reshape(n, -1, ld)[:, :, :K]
        Q = ctx.array("Q" + im, np.float64).reshape(n, -1)
        qc = int(round(Q.shape[1] ** 0.5))
        Q = Q.reshape(n, qc, qc)[:, 1:, 1:]
        V = W[:, :qc - 1]
        for s in range(n):
            ref = V[s] @ V[s].T
            tol = 2 * K * 2.0 ** -53 * (np.abs(V[s]) @ np.abs(V[s]).T)
            low = np.tril_indices(qc - 1)
            assert np.all(np.abs(Q[s] - ref)[low] <= tol[low]), (im, s)
    ctx.close()
