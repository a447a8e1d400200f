"""Jagged softmax, forward and both backward forms, at the lengths where the kernels
change their way: the lanes that share a list, lists that go one by one, tiles whose
elements no longer fit, ragged last rounds, elements outside the lists.

Against long double.  With u the unit roundoff, v the largest |x - max| and n the
longest list, an exponential is within e = (2 + 1.173 v) ulp (float: the stated
bound of __expf) or 1 ulp (double), plus v u for the difference; a sum of n terms
adds n u and the few remaining operations 4 u: y is within r = 2 (2 u ulps + v u) +
(n + 4) u of the exact value, relatively, and each gradient within
(3 r + (n + 4) u) y (|g| + sum |g y|), absolutely.
"""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

LENGTHS = [
    [8] * 33, [9] * 40, [16] * 32, [17] * 31, [24] * 70, [25, 1, 0, 3] * 20, [32] * 32, [33] * 5,
    [48] * 64, [49] * 3, [96] * 40, [97, 2] * 30, [192] * 33, [193] + [1] * 64, [0, 0, 0], [5],
    [64] * 15 + [65] * 17, [1024], [1025, 7, 0, 2], [3, 5000, 2] * 3, [16] * 63 + [17], [12] * 129,
]


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("lengths", LENGTHS, ids=lambda s: f"{len(s)}x{max(s)}")
def test_softmax_lengths(lengths, dtype):
    from awkward_gb300 import autograd

    L = np.array(lengths)
    start = 3
    off = np.concatenate([[0], np.cumsum(L)]).astype(np.int64) + start
    total = int(off[-1]) + 5
    gen = torch.Generator().manual_seed(len(lengths))
    x = torch.randn(total, generator=gen, dtype=dtype)
    g = torch.randn(total, generator=gen, dtype=dtype)
    xl, gl = x.numpy().astype(np.longdouble), g.numpy().astype(np.longdouble)
    y, gx = np.zeros_like(xl), np.zeros_like(xl)
    scale = np.zeros_like(xl)
    v = 0.0
    for a, b in zip(off[:-1], off[1:]):
        if a == b:
            continue
        e = np.exp(xl[a:b] - xl[a:b].max())
        v = max(v, float(xl[a:b].max() - xl[a:b].min()))
        y[a:b] = e / e.sum()
        gx[a:b] = y[a:b] * (gl[a:b] - (gl[a:b] * y[a:b]).sum())
        scale[a:b] = y[a:b] * (abs(gl[a:b]) + abs(gl[a:b] * y[a:b]).sum())
    u = np.finfo(x.numpy().dtype).eps / 2
    ulps = 2 + 1.173 * v if dtype == torch.float32 else 1
    n = max(lengths)
    r = 2 * (2 * u * ulps + v * u) + (n + 4) * u
    for budget in (1 << 30, 0):  # y kept, y computed again
        xd = x.cuda().requires_grad_()
        out = autograd.jagged_softmax(xd, torch.from_numpy(off).cuda(), budget)
        out.backward(g.cuda())
        got, grad = out.detach().cpu().numpy(), xd.grad.cpu().numpy()
        assert (abs(got - y) <= r * y).all()
        assert (abs(grad - gx) <= (3 * r + (n + 4) * u) * scale).all()
