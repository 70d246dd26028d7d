"""The fp32 GEMMs and the fp32 read against float64."""
import pytest
import torch

from nanokv_b200 import ops
from test_gpu_decode_rows import random_history

pytestmark = pytest.mark.gpu


def _rows64(hist, decoder, mean):
    """Rows of a one-segment history in float64."""
    packed = hist.codes.long()
    codes = torch.stack((packed & 15, packed >> 4), dim=2).flatten(1).double() - 7
    scales = hist.scales.double().repeat_interleave(hist.group, dim=1)
    return (codes * scales) @ decoder.double().T + mean.double() + hist.centers[hist.ids.long()].double()


@pytest.mark.parametrize("tokens", [1, 63, 64, 65, 700])
@pytest.mark.parametrize("joint,rank,group", [(64, 6, None), (96, 64, 32), (200, 192, None), (1536, 192, 64)])
def test_decode_rows(tokens, joint, rank, group):
    hist = random_history(tokens, joint, rank, group=group)
    decoder = torch.randn(joint, rank, device="cuda") / rank ** 0.5
    mean = torch.randn(joint, device="cuda")
    got = ops.decode_rows(hist.view(), decoder, mean)
    want = _rows64(hist, decoder, mean)
    # rank products summed in fp32 (magnitudes below 1.05 * |decoder|), two additions
    bound = rank * 2.0 ** -23 * (want.abs().max() + 8.0)
    assert float((got.double() - want).abs().max()) <= bound


@pytest.mark.parametrize("tokens,queries,heads", [(1, 1, 1), (64, 64, 2), (129, 65, 3), (2048, 256, 12), (1000, 3, 1)])
@pytest.mark.parametrize("D", [16, 64, 128])
def test_read(tokens, queries, heads, D):
    joint, rank = heads * D, 32
    views, weights, rows = [], [], []
    for seed in (1, 2):
        hist = random_history(tokens, joint, rank, seed=seed)
        decoder = torch.randn(joint, rank, device="cuda") / rank ** 0.5
        mean = 0.1 * torch.randn(joint, device="cuda")
        views.append(hist.view())
        weights += [decoder.view(heads, D, rank), mean.view(heads, D)]
        rows.append(_rows64(hist, decoder, mean).view(tokens, heads, D))
    q = torch.randn(queries, 2, heads, D, device="cuda")[:, 1]       # strided over the tokens
    out, lse = ops.attn_codec(q, *views, *weights, scale=D ** -0.5)
    score = torch.einsum("qhd,nhd->qhn", q.double(), rows[0]) * D ** -0.5
    want = torch.einsum("qhn,nhd->qhd", score.softmax(-1), rows[1])
    # fp32 sums of `tokens` weights and of D products: errors of a few 2^-24 per term in the exponent
    assert float((out.double() - want).norm() / want.norm()) < 1e-5
    assert float((lse.double() - score.logsumexp(-1)).abs().max()) < 1e-4


@pytest.mark.parametrize("S,J,C", [(1, 8, 1), (65, 20, 7), (700, 258, 65), (2048, 1536, 16), (300, 31, 200)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_assignment_and_projection(S, J, C, dtype):
    gen = torch.Generator(device="cuda").manual_seed(J)
    centers = torch.randn(C, J, generator=gen, device="cuda") * 4
    pick = torch.randint(0, C, (S,), generator=gen, device="cuda")
    rows = (centers[pick] + 0.3 * torch.randn(S, J, generator=gen, device="cuda")).to(dtype)
    assert torch.equal(ops.assign(rows, centers).long() & 0xFFFF, pick)
    r = 70
    encoder = torch.randn(r, J, generator=gen, device="cuda") / J ** 0.5
    mean = torch.randn(J, generator=gen, device="cuda")
    stored, ids = centers.to(torch.bfloat16), pick.to(torch.uint8)
    got = ops.project(rows, stored, ids, mean, encoder)
    residual = rows.double() - stored[pick].double() - mean.double()
    want = residual @ encoder.double().T
    bound = (J + 4) * 2.0 ** -24 * (residual.abs() @ encoder.double().abs().T) + 2.0 ** -22 * 16
    assert bool(((got.double() - want).abs() <= bound).all())


@pytest.mark.parametrize("tokens", [1, 31, 64, 65, 193])
@pytest.mark.parametrize("joint,rank,group", [(4, 16, None), (64, 48, 16), (100, 64, 32), (132, 80, 80), (196, 192, 48)])
@pytest.mark.parametrize("scale_dtype", [torch.bfloat16, torch.float16])
def test_vector_form_gives_the_general_forms_bits(tokens, joint, rank, group, scale_dtype):
    """A decoder four bytes off a vector's start is read element by element; both sum in the same order."""
    hist = random_history(tokens, joint, rank, group=group, scale_dtype=scale_dtype, segments=min(3, tokens))
    decoder = torch.randn(joint, rank, device="cuda") / rank ** 0.5
    shifted = torch.empty(joint * rank + 1, device="cuda")[1:].view(joint, rank).copy_(decoder)
    mean = torch.randn(joint, device="cuda")
    listed = torch.tensor([tokens - 1, 0, tokens // 2] * 25, dtype=torch.int32, device="cuda")
    for rows in (None, listed):
        got, want = (ops.decode_rows(hist.view(), d, mean, rows=rows) for d in (decoder, shifted))
        assert torch.equal(got, want)
    listed[1], listed[2] = -1, tokens           # rows that are not there leave the others alone
    got = ops.decode_rows(hist.view(), decoder, mean, rows=listed)
    keep = torch.ones(75, dtype=torch.bool, device="cuda")
    keep[1:3] = False
    assert torch.equal(got[keep], want[keep])


@pytest.mark.parametrize("S", [1, 15, 16, 17, 333])
@pytest.mark.parametrize("C", [1, 16, 17, 32, 33, 64])
@pytest.mark.parametrize("J", [64, 320, 448])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_few_centres_give_the_ids_of_the_general_form(S, C, J, dtype):
    """Rows four bytes off a vector's start take the general form; both sum in the same order, ties and non-finite rows
    included."""
    x = torch.randn(S, J, device="cuda")
    centers = torch.randn(C, J, device="cuda").to(dtype)
    centers[C // 2] = centers[C - 1]                          # equal distances: the lower index
    x[S // 2] = centers[C - 1].float()
    if S > 4:
        x[1, 3], x[2, J - 1], x[3] = float("nan"), float("inf"), 3e38
    shifted = torch.empty(S * J + 1, device="cuda")[1:].view(S, J).copy_(x)
    assert torch.equal(ops.assign(x, centers), ops.assign(shifted, centers))


@pytest.mark.parametrize("S", [1, 15, 17, 48, 49, 700, 3000])
@pytest.mark.parametrize("J,r", [(32, 2), (64, 64), (96, 66), (224, 192)])
def test_projection_of_aligned_rows_gives_the_general_forms_bits(S, J, r):
    """Rows four bytes off a vector's start take the general form; both sum in the same order."""
    x = torch.randn(S, J, device="cuda")
    centers = torch.randn(16, J, device="cuda").bfloat16()
    ids = torch.randint(0, 16, (S,), device="cuda").to(torch.uint8)
    mean, encoder = torch.randn(J, device="cuda"), torch.randn(r, J, device="cuda")
    shifted = torch.empty(S * J + 1, device="cuda")[1:].view(S, J).copy_(x)
    got, want = (ops.project(rows, centers, ids, mean, encoder) for rows in (x, shifted))
    assert torch.equal(got, want)
