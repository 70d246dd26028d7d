"""fp16 rows: every value is an fp32 value, so the encoder gives what it gives for the same rows in fp32."""
import pytest
import torch

from nanokv_b200 import ops
from nanokv_b200.cache import CompressedHistory
from nanokv_b200.codec import Operator, encode_append

pytestmark = pytest.mark.gpu


def _rows(S, J, C):
    gen = torch.Generator(device="cuda").manual_seed(S + J)
    centers = 3.0 * torch.randn(C, J, generator=gen, device="cuda")
    pick = torch.randint(0, C, (S,), generator=gen, device="cuda")
    pick[:C] = torch.arange(C, device="cuda")
    return (centers[pick] + 0.3 * torch.randn(S, J, generator=gen, device="cuda")).half()


@pytest.mark.parametrize("S,J,C", [(64, 64, 4), (700, 130, 16), (700, 63, 16), (9000, 256, 8)])
@pytest.mark.parametrize("iters", [0, 1, 2])
def test_kmeans(S, J, C, iters):
    rows = _rows(S, J, C)
    got, want = (ops.kmeans(x, C, iters, torch.arange(C)) for x in (rows, rows.float()))
    assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])
    mean = torch.stack([rows[got[1].long() == c].double().mean(0) for c in range(C)])
    if iters:    # rows of well separated centres: the stored centres are their members' means, rounded to bf16
        assert float((got[0].double() - mean).abs().max()) <= 2.0 ** -8 * float(mean.abs().max())


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_online_append(dtype):
    S, J, C, r = 500, 192, 16, 64
    rows = _rows(S, J, C)
    op = Operator(mean=torch.randn(J, device="cuda"), encoder=(torch.randn(r, J, device="cuda") / J ** 0.5).to(dtype),
                  decoder=torch.zeros(J, r, dtype=dtype, device="cuda"))
    stored = []
    for x in (rows, rows.float()):
        hist = CompressedHistory(joint=J, rank=r, capacity=S, max_segments=1, centers_per_segment=C)
        encode_append(hist, x, op, clusters=C)
        stored.append([hist.ids, hist.centers, hist.codes, hist.scales.view(torch.int16)])
    assert all(torch.equal(a, b) for a, b in zip(*stored))
