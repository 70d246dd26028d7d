"""Per-head maps on the tensor cores against float64, at the edges of their tiles."""
import pytest
import torch

from nanokv_b200 import ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [1, 31, 127, 128, 129, 700])
@pytest.mark.parametrize("din,dout,pad", [(16, 8, 8), (128, 32, 64), (128, 64, 64), (32, 128, 128), (64, 128, 128),
                                          (128, 128, 128), (48, 40, 64), (128, 24, 128), (20, 12, 16), (128, 36, 64)])
def test_head_linear(rows, din, dout, pad):
    gen = torch.Generator(device="cuda").manual_seed(rows)
    heads = torch.tensor([3, 0, 4], dtype=torch.int32, device="cuda")
    x = torch.randn(rows, 5, 128, generator=gen, device="cuda").to(torch.bfloat16)
    w = torch.randn(3, din, dout, generator=gen, device="cuda").to(torch.bfloat16)
    got = ops.head_linear(x, w, heads=heads, din=din, pad_to=pad).double()
    assert got.shape == (rows, 3, pad) and not bool(got[..., dout:].any())
    picked = x[:, heads.long(), :din].double()
    want = torch.einsum("ngd,gde->nge", picked, w.double())
    magnitude = torch.einsum("ngd,gde->nge", picked.abs(), w.double().abs())
    # din exact products summed in fp32, one rounding to bf16
    assert bool(((got[..., :dout] - want).abs() <= 2.0 ** -8 * want.abs() + din * 2.0 ** -24 * magnitude).all())
