"""A training step of the closure network at batch sizes around its block of 64
samples, against torch in FP64 on the same BF16-rounded weights. An FP32 sum of
n terms in blocks of 64 is off by at most about (64 + n / 512 + 8) 2^-24 of the
terms' absolute sum; the gradients, the layers' FP32 rounding included, are
held to 2e-5 of their largest entry."""
import ctypes as C

import numpy as np
import pytest

from rpgo_gb300 import capi

pytestmark = pytest.mark.gpu


def _exact(p, x, y):
    import torch

    r = lambda t: t.float().bfloat16().double()
    W1, b1, W2, b2 = r(p[32:1056]).view(64, 16), p[1056:1120], r(p[1120:5216]).view(64, 64), p[5216:5280]
    W3, b3 = r(p[5280:5344]), p[5344]
    xn = (x - p[:16]) * p[16:32]
    h1 = (xn @ W1.T + b1).clamp(min=0)
    h2 = (h1 @ W2.T + b2).clamp(min=0)
    z = h2 @ W3 + b3
    dz = (torch.sigmoid(z) - y) / len(y)
    d2 = torch.outer(dz, W3) * (h2 > 0)
    d1 = (d2 @ W2) * (h1 > 0)
    g = torch.cat([torch.zeros(32, dtype=p.dtype), (d1.T @ xn).reshape(-1), d1.sum(0), (d2.T @ h1).reshape(-1),
                   d2.sum(0), h2.T @ dz, dz.sum().reshape(1)])
    return g, float((z.clamp(min=0) - z * y + torch.log1p(torch.exp(-z.abs()))).mean())


@pytest.mark.parametrize("n", [1, 3, 63, 64, 65, 200, 513, 8191])
def test_gradients_and_adam(n):
    import torch

    rng = np.random.default_rng(n)
    f = lambda *s: torch.from_numpy(rng.standard_normal(s).astype(np.float32))
    x, y = f(n, 16) * 2 + 1, (f(n) > -1).float()
    p = torch.cat([torch.ones(16), torch.full((16,), 0.5), 0.3 * f(1024), 0.1 * f(64), 0.15 * f(4096), 0.1 * f(64),
                   0.2 * f(64), 0.1 * f(1)])
    want, loss = _exact(p.double(), x.double(), y.double())
    P, X, Y = p.cuda(), x.cuda(), y.cuda()
    m, v, g, out = torch.zeros_like(P), torch.zeros_like(P), torch.full_like(P, 7.0), C.c_double()
    assert capi.load().rpgo_mlp_train_step_dev(P.data_ptr(), m.data_ptr(), v.data_ptr(), 1, 1e-3, n, X.data_ptr(),
                                               Y.data_ptr(), g.data_ptr(), C.byref(out), None) == 0
    got = g.cpu().double()
    assert (got - want).abs().max() <= 2e-5 * want.abs().max()
    assert got[:32].abs().max() == 0 and abs(out.value - loss) <= 1e-5 * max(1.0, loss)
    # Adam's first step: g / (|g| + eps) times the rate
    step = (p.double() - P.cpu().double())[32:]
    assert (step - 1e-3 * got[32:] / (got[32:].abs() + 1e-8)).abs().max() <= 1e-6
    assert torch.equal(P.cpu()[:32], p[:32])
