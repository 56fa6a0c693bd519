"""Ranker forward, gradient and batch mean at batch sizes around the kernels'
work split (four samples per CTA in the forward pass, 16 sample groups in the
reduction, more samples than one wave), against the NumPy FP64 restatement.
Inputs are O(1) and sums run over at most ~200 FP32 products, so 1e-4 of the
largest value, the tolerance of the fixed-size test, bounds the rounding."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 3, 5, 15, 17, 131])
def test_batch_sizes(n):
    import torch
    import xbach
    from ranker_ref import bf16, forward, grad
    from xbach import ranker
    L = xbach.lib()
    rng = np.random.default_rng(n)
    w = ranker.init_weights(3)
    st = rng.normal(size=(n, 16)).astype(np.float32)
    px = rng.uniform(-1, 1, size=(n, 2, 31, 31)).astype(np.float32)
    y = (rng.random(n) > 0.3).astype(np.float32)
    z = ranker.logits(w, st, px)
    dev = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (w, st, px, y)]
    per = torch.full((n, w.size), float("nan"), device="cuda")
    g = torch.empty(w.size, device="cuda")
    loss = torch.empty(n, device="cuda")
    assert L.xb_ranker_grad(dev[0].data_ptr(), dev[1].data_ptr(), dev[2].data_ptr(),
                            dev[3].data_ptr(), None, n, per.data_ptr(), g.data_ptr(),
                            loss.data_ptr(), torch.cuda.current_stream().cuda_stream) == 0
    wb = bf16(w)
    per, mean = per.cpu().numpy(), 0.0
    for i in range(n):
        zr = forward(wb, st[i], px[i])[0]
        lr, gr = grad(wb, st[i], px[i], y[i])
        assert abs(z[i] - zr) <= 1e-4 * (1 + abs(zr)), i
        assert abs(float(loss[i]) - lr) <= 1e-4 * (1 + abs(lr)), i
        assert np.max(np.abs(per[i] - gr)) <= 1e-4 * np.max(np.abs(gr)) + 1e-6, i
        mean = mean + gr / n
    assert np.max(np.abs(g.cpu().numpy() - mean)) <= 1e-4 * np.max(np.abs(mean)) + 1e-6


def test_forward_more_samples_than_one_wave_and_unaligned_windows():
    """Every sample of a batch larger than the grid's slots gets the logit it
    has alone, from windows at an address that is only 4-byte aligned."""
    import torch
    import xbach
    from xbach import ranker
    L = xbach.lib()
    n = 4001
    gen = torch.Generator(device="cuda").manual_seed(1)
    st = torch.randn(n, 16, generator=gen, device="cuda")
    flat = torch.randn(n * 1922 + 1, generator=gen, device="cuda")
    W = torch.from_numpy(ranker.init_weights(4)).cuda()
    out, one = torch.empty(n, device="cuda"), torch.empty(1, device="cuda")
    stream = torch.cuda.current_stream().cuda_stream
    px = flat.data_ptr() + 4
    assert L.xb_ranker_forward(W.data_ptr(), st.data_ptr(), px, n, out.data_ptr(), stream) == 0
    for i in (0, 1, 1823, 1824, 2000, n - 1):
        assert L.xb_ranker_forward(W.data_ptr(), st[i].data_ptr(), px + i * 1922 * 4, 1,
                                   one.data_ptr(), stream) == 0
        assert float(one) == float(out[i]), i
