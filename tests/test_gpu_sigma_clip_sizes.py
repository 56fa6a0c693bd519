"""The sigma clip of cd (csrc/xb_device.cuh, up to 1024 values in shared memory)
against the reference's loop in NumPy over stamp counts around its 32-value chunks
and around that limit: the same stamps are kept for the test fit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def clip(x, alpha, iters):
    live = np.ones(x.size, bool)
    prev, curr, mean, std = x.size, 0, 0.0, 1e10
    for _ in range(iters):
        if curr == prev:
            break
        if prev <= 1:
            mean, std = 0.0, 1e10
            break
        curr = prev
        s = s2 = 0.0
        for c in range(0, x.size, 32):
            a = a2 = 0.0
            for v, on in zip(x[c:c + 32], live[c:c + 32]):
                d = float(v) if on else 0.0
                a += d
                a2 += d * d
            s += a
            s2 += a2
        mean = s / curr
        std = float(np.sqrt((s2 - curr * mean * mean) / (curr - 1)))
        inv = 1.0 / std
        live &= ~(np.abs(x - mean) * inv > alpha)
        prev = int(live.sum())
    return mean, std


@pytest.mark.parametrize("nx,ny", [(1, 1), (2, 1), (31, 1), (8, 4), (11, 3), (32, 32), (33, 32)])
def test_kept_stamps_follow_the_reference_loop(nx, ny):
    import xbach
    from xbach.synth import make_pair
    size = 48 * max(nx, ny, 4)
    T, S, info = make_pair(2, frame=size, size=size, n_src=int(0.006 * size * size), stamps=max(nx, ny))
    ctx = xbach.Context(xbach.default_params(mode=xbach.XB_MODE_MIXED, stampsx=nx, stampsy=ny, hSStampWidth=3,
                                             nGauss=1, dg=[1], bg=[0.4], backgroundOrder=0,
                                             threshHigh=info["threshHigh"]), trace=True)
    p = ctx.params
    ctx.init(T, S)
    ctx.sss()
    ctx.cmv()
    ctx.cd()
    for si in range(2):
        ks = ctx.array("kernel_sums%d" % si, np.float64)
        mean, std = clip(ks, p.sigClipAlpha, 10)
        with np.errstate(all="ignore"):
            kept = np.flatnonzero(np.abs((ks - mean) / std) < p.sigKernFit)
        try:
            got = ctx.array("cd_test%d" % si, np.int32)
        except KeyError:
            got = np.zeros(0, np.int32)
        assert np.array_equal(got, kept), (si, ks.size)
    ctx.close()
