"""The gradients of the filter network that are plain sums over the samples are no further from
their 64-bit values, taken from the kernel's own activations, than plain FP32 addition."""
import numpy as np
import pytest

import canu_gb300 as oic

torch = pytest.importorskip("torch")

from test_gpu_filter import _forward, _params, _x   # noqa: E402

pytestmark = pytest.mark.gpu


def plain_fp32(g, block=1024):
    """Sum over the rows, one row after another in blocks of 1,024, then block after block."""
    total = np.zeros(g.shape[1], np.float32)
    for i in range(0, len(g), block):
        s = np.zeros(g.shape[1], np.float32)
        for row in g[i:i + block].astype(np.float32):
            s += row
        total += s
    return total.astype(np.float64)


@pytest.mark.parametrize("n", [64, 1000, 4097, 32768])
def test_bias_gradients_are_fp32_sums(n):
    mine, plain = [], []
    for seed in range(3):
        p16, x16 = _params(seed + 31), _x(n, n + seed)
        r = np.random.default_rng(n + seed)
        dy = torch.from_numpy((r.random(n) < 0.2).astype(np.float32)).cuda()
        dw = torch.from_numpy(r.uniform(0.05, 4.0, n).astype(np.float32)).cuda()
        dp, dx, logit, h1, h2 = _forward(p16, x16)
        grad, loss = torch.zeros(oic.FILTER_NPARAM, device="cuda"), torch.zeros(1, device="cuda")
        g1, g2 = (torch.empty((n, 128), dtype=torch.float16, device="cuda") for _ in range(2))
        oic.mlp_backward(dp.data_ptr(), dx.data_ptr(), h1.data_ptr(), h2.data_ptr(), logit.data_ptr(), dy.data_ptr(),
                         dw.data_ptr(), n, grad.data_ptr(), g1.data_ptr(), g2.data_ptr(), loss.data_ptr())
        torch.cuda.synchronize()
        for name, g in (("b1", g1), ("b2", g2)):
            g = g.cpu().numpy()
            at = oic.FILTER_OFFSETS[name][0]
            want, size = g.astype(np.float64).sum(0), np.abs(g.astype(np.float64)).sum(0)
            ok = size > 0
            mine.append(((grad[at:at + 128].cpu().numpy().astype(np.float64) - want)[ok] / size[ok]))
            plain.append((plain_fp32(g) - want)[ok] / size[ok])
    rms = [float(np.sqrt(np.mean(np.concatenate(v) ** 2))) for v in (mine, plain)]
    print(n, rms)
    assert rms[0] <= rms[1]


@pytest.mark.parametrize("n", [32768, 60000])
def test_output_weight_gradients_are_fp32_sums(n):
    """grad w3 = sum of (dloss / dlogit) * h2, against FP32 sums of 512 samples at a time."""
    mine, plain = [], []
    for seed in range(3):
        p16, x16 = _params(seed + 31), _x(n, n + seed)
        r = np.random.default_rng(n + seed)
        y = (r.random(n) < 0.2).astype(np.float32)
        w = r.uniform(0.05, 4.0, n).astype(np.float32)
        dy, dw = torch.from_numpy(y).cuda(), torch.from_numpy(w).cuda()
        dp, dx, logit, h1, h2 = _forward(p16, x16)
        grad, loss = torch.zeros(oic.FILTER_NPARAM, device="cuda"), torch.zeros(1, device="cuda")
        g1, g2 = (torch.empty((n, 128), dtype=torch.float16, device="cuda") for _ in range(2))
        oic.mlp_backward(dp.data_ptr(), dx.data_ptr(), h1.data_ptr(), h2.data_ptr(), logit.data_ptr(), dy.data_ptr(),
                         dw.data_ptr(), n, grad.data_ptr(), g1.data_ptr(), g2.data_ptr(), loss.data_ptr())
        torch.cuda.synchronize()
        z, h = logit.cpu().numpy().astype(np.float64), h2.cpu().numpy().view(np.float16).astype(np.float64)
        d = w.astype(np.float64) * (1 / (1 + np.exp(-z)) - y)
        want, size = d @ h, np.abs(d) @ h
        ok = size > 0
        at = oic.FILTER_OFFSETS["w3"][0]
        mine.append(((grad[at:at + 128].cpu().numpy().astype(np.float64) - want)[ok] / size[ok]))
        plain.append((plain_fp32(d.astype(np.float32)[:, None] * h.astype(np.float32), 512) - want)[ok] / size[ok])
    rms = [float(np.sqrt(np.mean(np.concatenate(v) ** 2))) for v in (mine, plain)]
    print(n, rms)
    assert rms[0] <= rms[1]
