"""The number of history splits a caller may ask for."""
import pytest
import torch

from nanokv_b200 import ops


@pytest.mark.parametrize("splits", [0, -1, 17])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_splits_out_of_range_are_refused(monkeypatch, splits, dtype):
    """Before any launch; 0 is the C entry's own choice and no value of this call."""
    monkeypatch.setattr(ops, "_require_cuda", lambda *tensors: torch.device("cpu"))
    monkeypatch.setattr(ops, "status_word", lambda device: torch.zeros(1, dtype=torch.int32))
    monkeypatch.setattr(ops._lib, "library", lambda: pytest.fail("reached the library"))

    class OnDevice(torch.Tensor):
        is_cuda = True

    q = torch.zeros(8, 2, 64, dtype=dtype).as_subclass(OnDevice)
    weight, bias = torch.zeros(2, 64, 64, dtype=dtype), torch.zeros(2, 64)
    with pytest.raises(ValueError, match="splits"):
        ops.attn_codec(q, None, None, weight, bias, weight, bias, scale=1.0, splits=splits)
