"""Columns past a map's width are zero for inputs of every kind."""
import pytest
import torch

from nanokv_b200 import ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("din,dout,pad", [(16, 8, 32), (128, 24, 128), (48, 40, 64), (32, 72, 128), (128, 32, 64), (20, 12, 16)])
@pytest.mark.parametrize("value", [float("inf"), float("-inf"), float("nan")])
def test_padding_of_rows_that_are_not_finite(din, dout, pad, value):
    gen = torch.Generator(device="cuda").manual_seed(din)
    x = torch.randn(200, 2, 128, generator=gen, device="cuda").to(torch.bfloat16)
    w = torch.randn(2, din, dout, generator=gen, device="cuda").abs().add(0.1).to(torch.bfloat16)
    clean = ops.head_linear(x, w, din=din, pad_to=pad)
    x[7, 0, 3] = value
    got = ops.head_linear(x, w, din=din, pad_to=pad)
    assert not bool(got[..., dout:].any())
    assert bool((got[7, 0, :dout] == value).all()) or bool(torch.isnan(got[7, 0, :dout]).all())
    got[7, 0], clean[7, 0] = 0, 0
    assert torch.equal(got, clean)
