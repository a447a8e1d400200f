"""Reducers over lists whose offsets straddle 2^31 and 2^32: the walk keeps the low words
of the offsets, whose differences have to hold across the sign and the wrap."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("edge", [1 << 31, 1 << 32])
@pytest.mark.parametrize("dtype", ["float32", "int32"])
def test_lists_across_the_edge(edge, dtype):
    import torch

    import awkward_gb300

    be = awkward_gb300.backend()
    rng = np.random.default_rng(3)
    L = np.concatenate([rng.poisson(8, 4000), rng.poisson(40, 600), rng.poisson(130, 300), [900, 5000]])
    L = L[rng.permutation(L.size)]
    total = int(L.sum())
    start = edge - total // 2
    off = start + np.concatenate([[0], np.cumsum(L)])
    values = rng.integers(-1000, 1000, total)
    x = torch.empty(edge + total, dtype=getattr(torch, dtype), device="cuda")
    x[start:start + total] = torch.from_numpy(values).cuda()
    d_off, n, t = torch.from_numpy(off).cuda(), L.size, np.dtype(dtype).type
    total_of = torch.empty(n, dtype=torch.int64 if dtype == "int32" else x.dtype, device="cuda")
    out, arg = torch.empty(n, dtype=x.dtype, device="cuda"), torch.empty(n, dtype=torch.int64, device="cuda")
    be["awkward_reduce_sum", np.int64 if dtype == "int32" else t, t, np.int64](total_of, x, d_off, n)
    be["awkward_reduce_max", t, t, np.int64](
        out, x, d_off, n, -np.inf if dtype == "float32" else np.iinfo(np.int32).min)
    be["awkward_reduce_argmax", np.int64, t, np.int64, np.int64](arg, x, d_off, d_off[:-1], n)
    be.synchronize()
    got = total_of.cpu().numpy(), out.cpu().numpy(), arg.cpu().numpy()
    for i, (a, b) in enumerate(zip(off - start, off[1:] - start)):
        if a == b:
            assert got[2][i] == -1 and got[0][i] == 0
            continue
        part = values[a:b]  # (sums of these are exact in float32)
        assert got[0][i] == part.sum() and got[1][i] == part.max()
        assert got[2][i] == start + a + part.argmax()
