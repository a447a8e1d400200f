"""preparenext by column counts against the C oracle, bit for bit, at the edges
of its row tiles (256 rows of one bin), of its 32-column steps and of the rule
that hands a call to the radix sort (1024 columns)."""

import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu

S = 777
NAME = "awkward_ListOffsetArray_reduce_nonlocal_preparenext_64"


@pytest.mark.parametrize("rows,longest,shift", [
    ([1], 1, 0), ([255], 9, 3), ([256], 31, 0), ([257], 32, 0), ([513], 33, 5),
    ([0, 0, 300, 0, 1, 256, 255, 257, 700, 0], 40, 11), ([3] * 2000, 6, 0),
    ([600, 2, 0], 1024, 0), ([600, 2, 0], 1025, 2)])
def test_preparenext_columns(rows, longest, shift):
    import torch

    import awkward_gb300
    from awkward_gb300._signatures import SIGNATURES

    rng = np.random.default_rng(sum(rows) + longest)
    outer = np.concatenate([[0], np.cumsum(rows)]).astype(np.int64)
    L = rng.integers(0, min(longest, 12) + 1, int(outer[-1])).astype(np.int64)
    L[len(L) // 2] = longest
    off = (shift + np.concatenate([[0], np.cumsum(L)])).astype(np.int64)
    E, nb = int(off[-1] - off[0]), len(rows) * longest
    kw = {"nextcarry": np.full(E, S, np.int64), "nextoffsets": np.full(nb + 1, S, np.int64),
          "nextlen": E, "maxnextparents": np.full(1, S, np.int64),
          "distincts": np.full(nb, S, np.int64), "distinctslen": nb,
          "offsetscopy": np.full(len(off), S, np.int64), "offsets": off, "length": len(L),
          "outer_offsets": outer, "outlength": len(rows), "maxcount": longest}
    exp = {k: (v.copy() if isinstance(v, np.ndarray) else v) for k, v in kw.items()}
    oracle.call(oracle.load(), NAME, **exp)
    be = awkward_gb300.backend()
    dev = {k: torch.from_numpy(v).cuda() if isinstance(v, np.ndarray) else v for k, v in kw.items()}
    be.by_name(NAME)(*[dev[a[0]] for a in SIGNATURES[NAME]["args"]])
    be.synchronize()
    for o in ("nextcarry", "nextoffsets", "maxnextparents", "distincts"):
        np.testing.assert_array_equal(dev[o].cpu().numpy(), exp[o], err_msg=o)
