"""Long projections to 512 columns per block keep token rows and encoder rows in rings of their own: the rows of a call are
those of short calls, which take narrower tiles, and the float64 product's."""
import pytest
import torch

from nanokv_b200 import ops

pytestmark = pytest.mark.gpu


# chunks of 64 columns: fewer than the rings are deep, as many, one and several more
@pytest.mark.parametrize("chunks", [1, 2, 3, 4, 5, 6, 7, 8, 9, 16, 33])
@pytest.mark.parametrize("tokens,rank", [(9473, 512), (12480, 512), (18901, 512), (9473, 1024), (4737, 1024), (12480, 960)])
def test_rows_are_those_of_short_calls(tokens, rank, chunks):
    joint = 64 * chunks
    gen = torch.Generator(device="cuda").manual_seed(tokens + rank + chunks)
    centers = torch.randn(16, joint, generator=gen, device="cuda").to(torch.bfloat16)
    ids = torch.randint(0, 16, (tokens,), generator=gen, device="cuda").to(torch.uint8)
    x = (centers[ids.long()].float() + 0.3 * torch.randn(tokens, joint, generator=gen, device="cuda")).to(torch.bfloat16)
    mean = 0.1 * torch.randn(joint, generator=gen, device="cuda")
    encoder = (torch.randn(rank, joint, generator=gen, device="cuda") / joint ** 0.5).to(torch.bfloat16)
    whole = ops.project(x, centers, ids, mean, encoder)
    step = 900
    parts = [ops.project(x[i:i + step], centers, ids[i:i + step], mean, encoder) for i in range(0, tokens, step)]
    assert torch.equal(whole, torch.cat(parts))
    residual = ((x.float() - centers[ids.long()].float()) - mean).to(torch.bfloat16).double()
    exact = residual @ encoder.double().T
    # one rounding to bf16 and `joint` fp32 additions of terms that are at most the row's sum of magnitudes
    bound = 2.0 ** -8 * exact.abs() + joint * 2.0 ** -23 * (residual.abs() @ encoder.double().abs().T)
    assert ((whole.double() - exact).abs() <= bound).all()
    for group, dtype in ((rank, torch.bfloat16), (32, torch.float16)):
        codes, scales = ops.project_quant(x, centers, ids, mean, encoder, group=group, scale_dtype=dtype)
        want_codes, want_scales = ops.quant_pack(whole, group=group, scale_dtype=dtype)
        assert torch.equal(codes, want_codes) and torch.equal(scales, want_scales)
