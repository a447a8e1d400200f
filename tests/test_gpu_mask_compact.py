"""array[mask] by the bitmap of the whole mask against numpy, at the edges of its
words, chunks and tiles and of the rule that chooses it.  Bytes are compared.
"""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

MIN = 1 << 20  # elements from which any array goes by the bitmap

CASES = [
    # the rule for lists of mean 16: more elements than a tile's own bitmap holds
    (16384, 16, 3, np.float64, 0.4),
    (16385, 1024, 3, np.float64, 0.4),
    (16399, 1024, 0, np.uint8, 0.4),
    (16400, 1024, 1, np.int16, 0.4),
    (32768 - 15, 1, 15, np.float32, 0.6),
    (32768 - 14, 1, 15, np.float32, 0.6),
    # elements, lists, element offset of the content's start, dtype, kept share
    (MIN - 1, 70000, 0, np.float64, 0.4),
    (MIN, 70000, 0, np.float64, 0.4),
    (MIN + 32 * 1024 - 16, 70000, 1, np.float64, 0.4),
    (MIN + 32 * 1024 - 15, 70000, 15, np.float32, 0.4),
    (MIN + 31, 3, 7, np.int16, 0.9),
    (MIN + 1023, 1, 3, np.uint8, 0.01),
    (MIN + 5000, 2_000_000, 5, np.int64, 0.5),
    (MIN + 1, 1000, 0, np.float64, 0.0),
    (MIN + 1, 1000, 2, np.float64, 1.0),
    (3_000_017, 400_000, 9, np.float32, 0.3),
]


@pytest.mark.parametrize("n,nlists,start,dtype,share", CASES)
@pytest.mark.parametrize("with_carry", [False, True])
def test_mask_select_bitmap(n, nlists, start, dtype, share, with_carry):
    from awkward_gb300 import jagged

    rng = np.random.default_rng(n + nlists)
    ends = np.sort(rng.integers(0, n + 1, nlists - 1))
    offsets = np.concatenate([[0], ends, [n]]).astype(np.int64) + start
    # some entries past the lists: neither the mask's nor the content's count
    mask = rng.random(start + n + 11) < share
    content = rng.integers(0, 100, start + n + 11).astype(dtype)
    to, out, *carry = jagged.mask_select(
        torch.from_numpy(offsets).cuda(), torch.from_numpy(content).cuda(),
        torch.from_numpy(mask).cuda(), with_carry=with_carry)
    picked = np.flatnonzero(mask[start:start + n]) + start
    ranks = np.concatenate([[0], np.cumsum(mask[start:start + n])])
    assert np.array_equal(to.cpu().numpy(), ranks[offsets - start])
    assert np.array_equal(out.cpu().numpy(), content[picked])
    if with_carry:
        assert np.array_equal(carry[0].cpu().numpy(), picked)


def test_batched_select_bitmap():
    """Arrays of a batch, each with its own tiles in one sequence, with and without
    a list, against the same arrays one by one."""
    from awkward_gb300 import batch, jagged

    gen = torch.Generator(device="cuda").manual_seed(5)
    arrays = []
    for nlists, n in ((3, 40_000), (5000, 30_000), (0, 0), (7, 0), (1, 32_753), (2000, 70_001)):
        cuts = torch.randint(0, n + 1, (max(nlists - 1, 0),), device="cuda", generator=gen)
        off = torch.cat([torch.zeros(1, dtype=torch.int64, device="cuda"), cuts.sort().values,
                         torch.full((min(nlists, 1),), n, dtype=torch.int64, device="cuda")])
        x = torch.randn(n, dtype=torch.float64, device="cuda", generator=gen)
        arrays.append((off, x, torch.rand(n, device="cuda", generator=gen) < 0.4))
    b = batch.Batch(arrays)
    plan = b.plan(batch.PLAN_VARIANTS[0])
    for _ in range(2):
        b.run(plan)
    torch.cuda.synchronize()
    b.check_errors()
    for (off, x, m), got in zip(arrays, b.outputs()):
        to, out = jagged.mask_select(off, x, m)
        count, sel_offsets, sel_content = got[3:]
        assert torch.equal(sel_offsets, to)
        assert torch.equal(sel_content, out)
        assert torch.equal(count, off[1:] - off[:-1])
    b.close()
