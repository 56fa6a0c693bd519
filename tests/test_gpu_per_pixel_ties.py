"""The 0.99 |kernel| rule of the mixed per-pixel convolution (csrc/xb_mixed.cu) at
pixels whose ratio is close to 0.99: the taps' FP32 values summed one after the
other, rows then columns as in conv.cl:54-70, decide.  One fit, random input masks,
and the rule restated in NumPy from the fit's solution for every pixel whose ratio
is within 2e-3."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FK, HK, NK = 21, 10, 441
BAD_INPUT, BAD_CONV, OK_CONV = 1 << 7, 1 << 4, 1 << 6


def _fma(a, b, c):
    """FP32 fused multiply-add (the product is exact in FP64)."""
    return (a.astype(np.float64) * b + c).astype(np.float32)


def _rule(img, mask, sol, vec, tL, tH, order=2):
    """Pixels (y, x) near the tie and whether each is below 0.99."""
    h, w = img.shape
    n_psf, pows = len(vec), [(i, j) for i in range(order + 1) for j in range(order + 1 - i)]
    c = sol[2:2 + (n_psf - 1) * len(pows)].reshape(n_psf - 1, len(pows))
    Kt = np.tensordot(c.T, vec[1:], axes=1).reshape(len(pows), NK)
    Kt[0] += sol[1] * vec[0].ravel()
    Kt = Kt[:, ::-1]          # window order: tap (20 - ii, 20 - jj) at jj * 21 + ii
    ktf = Kt.astype(np.float32)
    bad = (img == 0) | (img >= tH) | (img <= tL) | (mask != 0)
    hx, hy = 0.5 * w, 0.5 * h
    out = []
    for y0 in range(0, h - 2 * HK, FK):
        for x0 in range(0, w - 2 * HK, FK):
            ny, nx = min(FK, h - 2 * HK - y0), min(FK, w - 2 * HK - x0)
            tile = bad[y0:y0 + ny + 2 * HK, x0:x0 + nx + 2 * HK]
            if not tile.any():
                continue
            win = np.lib.stride_tricks.sliding_window_view(tile, (FK, FK)).reshape(ny * nx, NK)
            xc, yc = (x0 + 2 * HK - hx) / hx, (y0 + 2 * HK - hy) / hy
            poly = [xc ** i * yc ** j for i, j in pows]
            kern = (np.array(poly) @ Kt).astype(np.float32)
            part = win @ np.abs(kern) / np.abs(kern).sum()
            at = np.flatnonzero(win.any(1) & (np.abs(part - 0.01) < 4e-3))
            if not len(at):
                continue
            ys, xs = y0 + HK + at // nx, x0 + HK + at % nx
            xf, yf = (xs - hx) / hx, (ys - hy) / hy
            kv = np.broadcast_to(kern, (len(at), NK)).copy()
            for t, (i, j) in enumerate(pows):
                if t:
                    dp = (xf ** i * yf ** j - poly[t]).astype(np.float32)
                    kv = _fma(np.broadcast_to(dp[:, None], kv.shape), ktf[t], kv)
            kv = np.abs(kv)
            aks = np.add.accumulate(kv, axis=1, dtype=np.float32)[:, -1]
            uks = np.add.accumulate(np.where(win[at], np.float32(0), kv), axis=1, dtype=np.float32)[:, -1]
            r = uks / aks
            near = np.abs(r - 0.99) < 2e-3
            out += [(y, x, v < np.float32(0.99), v) for y, x, v in zip(ys[near], xs[near], r[near])]
    return out


def test_near_ties_are_decided_in_tap_order(oracle, test01_oracle):
    import xbach
    from xbach.synth import make_pair
    T, S, info = make_pair(1)
    h, w = T.shape
    vec = test01_oracle.array("basis", np.float64)[:49 * NK].reshape(49, FK, FK)
    ctx = xbach.Context(xbach.default_params(mode=xbach.XB_MODE_MIXED, convPerPixel=1, stampsx=info["stamps"],
                                             stampsy=info["stamps"], threshHigh=info["threshHigh"]))
    ctx.init(T, S)
    ctx.sss()
    ctx.cmv()
    img = T if ctx.cd() else S
    ctx.ksc()
    rng = np.random.default_rng(5)
    seen, close, wrong = 0, 0, []
    for _ in range(24):
        m = (rng.uniform(size=(h, w)) < 0.02).astype(np.uint8)
        ctx.set_input_mask(m)
        ctx.conv()
        got = ctx.mask().reshape(h, w)
        for y, x, below, r in _rule(img, m, ctx.solution(), vec, ctx.params.threshLow, ctx.params.threshHigh):
            assert got[y, x] & (BAD_CONV | OK_CONV)
            seen += 1
            close += abs(float(r) - 0.99) < 2e-6
            if bool(got[y, x] & BAD_CONV) != below:
                wrong.append((x, y, float(r) - 0.99))
    ctx.close()
    assert seen > 10000 and close > 20
    assert not wrong, wrong[:10]
