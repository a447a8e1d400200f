"""array[..., start:stop:step] in one kernel against awkward's own steps (carry,
then take), bit for bit: empty lists, tiles past the slot map's 16384 slots,
every item size, shifted offsets, and a list that reaches past the content;
and the index selection at the same sizes."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LENGTHS = {"none": [], "empty": [0] * 5, "one": [7], "tile": [3, 0, 1, 9] * 256,
           "tile+1": [3, 0, 1, 9] * 256 + [2], "map": [16] * 1024, "map+1": [16] * 1023 + [17],
           "long": [40_000, 0, 5, 1]}
SLICES = [(1, None, None), (None, 2, None), (-2, None, None), (None, None, 2), (None, None, -1),
          (5, 1, -3), (3, 3, None)]


def _lists(name, shift, dtype):
    import torch

    off = torch.from_numpy(shift + np.concatenate([[0], np.cumsum(LENGTHS[name])]).astype(np.int64))
    x = torch.from_numpy(np.random.default_rng(3).integers(0, 100, int(off[-1]) + 2).astype(dtype))
    return off.cuda(), x.cuda()


@pytest.mark.parametrize("name", list(LENGTHS))
@pytest.mark.parametrize("dtype", [np.int8, np.int16, np.float32, np.float64])
def test_range_select_is_the_carry_and_take(name, dtype):
    import torch

    from awkward_gb300 import jagged

    off, x = _lists(name, 4, dtype)
    for b in SLICES:
        nextoffsets, out = jagged.range_select(off, x, *b)
        if off.numel() == 1:
            assert nextoffsets.tolist() == [0] and out.numel() == 0
            continue
        want, carry = jagged.inner_range(off, *b)
        k = int(want[-1])
        assert torch.equal(nextoffsets, want) and torch.equal(out, jagged.take(x, carry[:k]))


def test_range_past_the_content_and_overlapping_lists():
    import torch

    from awkward_gb300 import jagged

    x = torch.arange(10, dtype=torch.float64, device="cuda")
    off = torch.tensor([0, 4, 12], dtype=torch.int64, device="cuda")
    with pytest.raises(ValueError, match="index out of range"):
        jagged.range_select(off, x, None, None, -1)
    off = torch.tensor([0, 10, 0, 10], dtype=torch.int64, device="cuda")  # 20 elements of 10
    nextoffsets, out = jagged.range_select(off, x)
    assert nextoffsets.tolist() == [0, 10, 10, 20] and out.tolist() == 2 * list(range(10))


@pytest.mark.parametrize("name", list(LENGTHS))
def test_index_select_at_the_same_sizes(name):
    import torch

    from awkward_gb300 import jagged

    off, x = _lists(name, 4, np.float64)
    n = off.numel() - 1
    if n == 0:
        return
    rng = np.random.default_rng(5)
    L = np.array(LENGTHS[name])
    K = np.where(L > 0, np.where(L > 16_384, L, 16), 0)  # full tiles hold 16384 slots too
    idx = np.concatenate([rng.integers(-l, l, k) for l, k in zip(L, K)] + [[]]).astype(np.int64)
    ioff = np.concatenate([[0], np.cumsum(K)]).astype(np.int64)
    o = off.cpu().numpy()
    at = idx + np.repeat(o[:-1], K) + np.where(idx < 0, np.repeat(L, K), 0)
    got_off, got, carry = jagged.index_select(off, x, torch.from_numpy(ioff).cuda(),
                                              torch.from_numpy(idx).cuda(), with_carry=True)
    np.testing.assert_array_equal(got_off.cpu().numpy(), ioff)
    np.testing.assert_array_equal(carry.cpu().numpy(), at)
    np.testing.assert_array_equal(got.cpu().numpy(), x.cpu().numpy()[at])
