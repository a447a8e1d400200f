"""The selections' argument checks: offsets of another type or another device are
refused (TypeError, as the kernel table refuses them) and strided offsets give what
their contiguous copy gives, whether or not the selection is counted first."""

import pytest


def test_arguments_must_be_cuda_tensors():
    import torch

    from awkward_gb300 import jagged

    off, x = torch.tensor([0, 2, 3]), torch.arange(3.0)
    with pytest.raises(TypeError, match="inner_offsets must be a CUDA tensor"):
        jagged.range_select(off, x)
    with pytest.raises(TypeError, match="inner_offsets must be a CUDA tensor"):
        jagged.getitem_inner_range(off, [0, 2, 3], x)


@pytest.mark.gpu
@pytest.mark.parametrize("limit", [0, 1 << 30])
def test_range_select_offsets(monkeypatch, limit):
    import torch

    from awkward_gb300 import jagged

    monkeypatch.setattr(jagged, "_WHOLE_CONTENT", limit)
    base = torch.tensor([0, 9, 4, 9, 4, 9, 10, 9, 12, 9], dtype=torch.int64, device="cuda")
    x = torch.arange(12, dtype=torch.float32, device="cuda")
    with pytest.raises(TypeError, match="inner_offsets must have dtype torch.int64"):
        jagged.getitem_inner_range(base, base.to(torch.int32), x, 1)
    with pytest.raises(TypeError, match="content must be a CUDA tensor"):
        jagged.getitem_inner_range(base, base, x.cpu(), 1)
    _, nextoffsets, out = jagged.getitem_inner_range(base, base[::2], x, 1)
    assert nextoffsets.tolist() == [0, 3, 3, 8, 9]
    assert out.tolist() == [1, 2, 3, 5, 6, 7, 8, 9, 11]
    wide = torch.stack([x, -x], 1)[:, 0]
    assert jagged.getitem_inner_range(base, base[::2], wide, 1)[2].tolist() == out.tolist()


@pytest.mark.gpu
def test_mask_arguments():
    import torch

    from awkward_gb300 import jagged

    off = torch.tensor([0, 9, 2, 9, 2, 9, 5, 9], dtype=torch.int64, device="cuda")
    x = torch.arange(5, dtype=torch.float64, device="cuda")
    m = torch.tensor([1, 0, 0, 1, 0, 0, 0, 0, 1, 1], dtype=torch.bool, device="cuda")
    for select in (jagged.mask_select, lambda o, _, mask: jagged.jagged_mask_to_index(o, mask)):
        with pytest.raises(TypeError, match="offsets must have dtype torch.int64"):
            select(off.to(torch.int32), x, m)
        with pytest.raises(TypeError, match="mask must be a CUDA tensor"):
            select(off, x, m.cpu())
        with pytest.raises(TypeError, match="mask must have entries of one byte"):
            select(off, x, m.to(torch.int64))
    to, out = jagged.mask_select(off[::2], x, m[::2])
    assert to.tolist() == [0, 1, 1, 2] and out.tolist() == [0.0, 4.0]
    to, index = jagged.jagged_mask_to_index(off[::2], m[::2])
    assert to.tolist() == [0, 1, 1, 2] and index.tolist() == [0, 2]


# below and above the size from which a mask goes by its bitmap, lists of few and of
# many elements (a tile's bitmap holds 16384)
@pytest.mark.gpu
@pytest.mark.parametrize("n,lists", [(5, 2), (16_000, 1024), (40_000, 3000), (40_000, 2),
                                     ((1 << 20) + 77, 70_000)])
def test_short_masks_raise(n, lists):
    import torch

    from awkward_gb300 import jagged

    off = torch.linspace(0, n, lists + 1, device="cuda", dtype=torch.float64).round().to(torch.int64)
    x = torch.arange(n, dtype=torch.float32, device="cuda")
    m = torch.ones(n, dtype=torch.bool, device="cuda")
    for short in (n - 1, n // 2, 0):
        for cut in (m[:short], m[:short].clone()):
            with pytest.raises(ValueError, match="index out of range.*jagged_mask_select"):
                jagged.mask_select(off, x, cut, with_carry=True)
            with pytest.raises(ValueError, match="index out of range.*jagged_mask_to_index"):
                jagged.jagged_mask_to_index(off, cut)
    with pytest.raises(ValueError, match="index out of range"):
        jagged.mask_select(off - 1, x, m)
    to, out = jagged.mask_select(off, x, m)
    assert torch.equal(to, off) and torch.equal(out, x)
    assert torch.equal(jagged.jagged_mask_to_index(off, m)[0], off)


@pytest.mark.gpu
@pytest.mark.parametrize("n,lists", [(4_000, 1024), (40_000, 3000), (40_000, 2),
                                     ((1 << 20) + 77, 70_000)])
def test_nothing_is_written_past_a_short_masks_result(n, lists):
    """The lists reach past the mask into true bytes of the same buffer: the results end
    where the mask does."""
    import torch

    from awkward_gb300 import _abi
    from awkward_gb300.kernel_table import raw_stream

    short = n - n // 3
    off = torch.linspace(0, n, lists + 1, device="cuda", dtype=torch.float64).round().to(torch.int64)
    m = torch.ones(n, dtype=torch.uint8, device="cuda")
    x = torch.arange(n, dtype=torch.int64, device="cuda")
    to = torch.empty(lists + 1, dtype=torch.int64, device="cuda")
    out, carry, index = (torch.full((n,), -7, dtype=torch.int64, device="cuda") for _ in range(3))
    err = torch.full((1,), -1, dtype=torch.int64, device="cuda")
    stream = raw_stream(0)
    assert _abi.ext_cfunc("awkward_gb300_jagged_mask_select_within")(
        to.data_ptr(), out.data_ptr(), carry.data_ptr(), m.data_ptr(), short, off.data_ptr(),
        x.data_ptr(), 8, lists, n, err.data_ptr(), stream) == 0
    assert err.item() == 0 and int(to[-1]) == short
    for a in (out, carry):
        assert torch.equal(a[:short], x[:short]) and bool((a[short:] == -7).all())
    err.fill_(-1)
    assert _abi.ext_cfunc("awkward_gb300_jagged_mask_to_index_within")(
        to.data_ptr(), index.data_ptr(), m.data_ptr(), short, off.data_ptr(), lists,
        err.data_ptr(), stream) == 0
    assert err.item() == 0 and int(to[-1]) == short and bool((index[short:] == -7).all())


@pytest.mark.gpu
def test_range_of_wide_items():
    """Items of 16 bytes are not gathered; a selection without any needs no gather."""
    import torch

    from awkward_gb300 import jagged

    off = torch.tensor([0, 3, 3, 5], dtype=torch.int64, device="cuda")
    x = torch.zeros(5, dtype=torch.complex128, device="cuda")
    _, nextoffsets, out = jagged.getitem_inner_range(off, off, x, 3)
    assert nextoffsets.tolist() == [0, 0, 0, 0] and out.numel() == 0 and out.dtype == x.dtype
    with pytest.raises(RuntimeError, match="cudaError 1$"):
        jagged.getitem_inner_range(off, off, x, 1)


@pytest.mark.gpu
def test_index_arguments():
    import torch

    from awkward_gb300 import jagged

    off = torch.tensor([0, 9, 3, 9, 5, 9], dtype=torch.int64, device="cuda")
    ioff = torch.tensor([0, 9, 1, 9, 3, 9], dtype=torch.int64, device="cuda")
    idx = torch.tensor([2, 9, -1, 9, 0, 9], dtype=torch.int64, device="cuda")
    x = torch.arange(5, dtype=torch.float32, device="cuda")
    for k, name in enumerate(("offsets", "index_offsets", "index")):
        args = [off[::2], x, ioff[::2], idx[::2]]
        at = (0, 2, 3)[k]
        args[at] = args[at].to(torch.int32)
        with pytest.raises(TypeError, match=f"^{name} must have dtype torch.int64"):
            jagged.index_select(*args)
    to, out, carry = jagged.index_select(off[::2], x, ioff[::2], idx[::2], with_carry=True)
    assert to.tolist() == [0, 1, 3] and out.tolist() == [2.0, 4.0, 3.0] and carry.tolist() == [2, 4, 3]
