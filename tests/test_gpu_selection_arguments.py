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
