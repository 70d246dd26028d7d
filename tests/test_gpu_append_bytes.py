"""What a history stores for a row does not depend on the length of the chunk it came in."""
import pytest
import torch

from nanokv_b200 import ops
from nanokv_b200.cache import CompressedHistory
from nanokv_b200.codec import GROUP32_FP16, Operator, QuantSpec, encode_append

pytestmark = pytest.mark.gpu


def _data(S, J, C, r):
    """Centres in near-identical pairs (one column one bf16 step apart): the distances of a pair differ by less
    than the rounding of their sums, so an id shows the order in which they were added."""
    gen = torch.Generator(device="cuda").manual_seed(J + r)
    centers = torch.randn(C, J, generator=gen, device="cuda").to(torch.bfloat16)
    twin = centers[0::2].clone()
    twin.view(torch.int16)[:, 0] += 1
    centers[1::2] = twin
    pick = torch.randint(0, C, (S,), generator=gen, device="cuda")
    rows = (centers[pick].float() + 0.3 * torch.randn(S, J, generator=gen, device="cuda")).to(torch.bfloat16)
    op = Operator(mean=0.1 * torch.randn(J, generator=gen, device="cuda"),
                  encoder=(torch.randn(r, J, generator=gen, device="cuda") / J ** 0.5).to(torch.bfloat16),
                  decoder=torch.zeros(J, r, dtype=torch.bfloat16, device="cuda"))
    return rows, centers, op


@pytest.mark.parametrize("quant", [QuantSpec(), GROUP32_FP16], ids=["token-scale", "group32"])
@pytest.mark.parametrize("J,C,r", [(1536, 256, 192), (3072, 64, 384), (5120, 512, 640)])
def test_chunks_of_any_length_store_the_same_bytes(J, C, r, quant):
    rows, centers, op = _data(3000, J, C, r)
    ids = ops.assign(rows, centers)
    codes, scales = ops.project_quant(rows, centers, ids, op.mean, op.encoder, group=quant.group,
                                      scale_dtype=quant.scale_dtype)
    for cuts in ((0, 3000), (0, 64, 500, 1700, 3000), (0, 880, 2440, 3000)):
        hist = CompressedHistory(joint=J, rank=r, capacity=3000, max_segments=len(cuts), group=quant.group,
                                 centers_per_segment=C, scale_dtype=quant.scale_dtype)
        for a, b in zip(cuts, cuts[1:]):
            encode_append(hist, rows[a:b], op, quant, centers=centers)
            assert torch.equal(ops.assign(rows[a:b], centers), ids[a:b])
        assert torch.equal(hist.ids, ids)
        assert torch.equal(hist.codes, codes)
        assert torch.equal(hist.scales.view(torch.int16), scales.view(torch.int16))
