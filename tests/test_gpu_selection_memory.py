"""What the selections allocate: for a few lists of a large array by the lists' span,
not by the array, while they run and in what they return; and a range slice that has
no room for a buffer of the content's length counts first."""

import pytest

pytestmark = pytest.mark.gpu

LISTS, LENGTH = 1000, 10


def _few_lists(n):
    import torch

    off = n // 2 + LENGTH * torch.arange(LISTS + 1, dtype=torch.int64, device="cuda")
    return off, torch.arange(n, dtype=torch.float64, device="cuda")


def _peak(call):
    import torch

    call()
    torch.cuda.synchronize()
    torch.cuda.reset_peak_memory_stats()
    before = torch.cuda.memory_allocated()
    out = call()
    return torch.cuda.max_memory_allocated() - before, out


def test_range_of_a_few_lists():
    from awkward_gb300 import jagged

    n = 1 << 24
    off, x = _few_lists(n)
    peak, (nextoffsets, out) = _peak(lambda: jagged.range_select(off, x, 1))
    assert peak < 1 << 20
    assert out.tolist() == [n // 2 + LENGTH * i + j for i in range(LISTS) for j in range(1, LENGTH)]
    assert int(nextoffsets[-1]) == out.numel()


@pytest.mark.parametrize("with_carry", [False, True])
def test_mask_of_a_few_lists(with_carry):
    import torch

    from awkward_gb300 import jagged

    n = 1 << 22
    off, x = _few_lists(n)
    m = torch.arange(n, device="cuda") % 3 == 0
    peak, (to, out, *carry) = _peak(lambda: jagged.mask_select(off, x, m, with_carry=with_carry))
    lo, hi = int(off[0]), int(off[-1])
    want = torch.nonzero(m[lo:hi]).flatten() + lo
    assert peak < 1 << 20
    assert torch.equal(out, want.double()) and int(to[-1]) == out.numel()
    assert out.untyped_storage().nbytes() < 1 << 20
    assert not with_carry or torch.equal(carry[0], want)
    peak, (to, index) = _peak(lambda: jagged.jagged_mask_to_index(off, m))
    assert peak < 1 << 20 and index.untyped_storage().nbytes() < 1 << 20


def test_no_room_for_the_whole_content(monkeypatch):
    import torch

    from awkward_gb300 import jagged

    off = torch.tensor([0, 40, 40, 100], dtype=torch.int64, device="cuda")
    x = torch.arange(100, dtype=torch.float32, device="cuda")
    empty = torch.empty

    def no_room(*size, **kw):
        if size[0] == 100:
            raise torch.cuda.OutOfMemoryError("no room")
        return empty(*size, **kw)

    monkeypatch.setattr(torch, "empty", no_room)
    nextoffsets, out = jagged.range_select(off, x, -2)
    assert nextoffsets.tolist() == [0, 2, 2, 4] and out.tolist() == [38, 39, 98, 99]
