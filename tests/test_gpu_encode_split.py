"""Encoder GEMMs and the C-means update at the sizes where their tiles and column parts change."""
import pytest
import torch

from nanokv_b200 import ops

pytestmark = pytest.mark.gpu


def _data(S, J, C, r, seed=0):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    centers = torch.randn(C, J, generator=gen, device="cuda").to(torch.bfloat16)
    pick = torch.randint(0, C, (S,), generator=gen, device="cuda")
    rows = (centers[pick].float() + 0.3 * torch.randn(S, J, generator=gen, device="cuda")).to(torch.bfloat16)
    encoder = (torch.randn(r, J, generator=gen, device="cuda") / J ** 0.5).to(torch.bfloat16)
    mean = 0.1 * torch.randn(J, generator=gen, device="cuda")
    return rows, centers, pick, encoder, mean


@pytest.mark.parametrize("S", [1, 63, 64, 65, 333, 880, 1560, 4680, 9400])
@pytest.mark.parametrize("J,C", [(64, 16), (256, 48), (1536, 256), (3072, 512), (5120, 64)])
def test_assignment_finds_the_centre_of_every_row(S, J, C):
    """Rows sit 0.3 sqrt(J) from their centre and sqrt(2 J) from any other: no distance comes near a tie."""
    rows, centers, pick, _, _ = _data(S, J, C, 64)
    assert torch.equal(ops.assign(rows, centers).long() & 0xFFFF, pick)


@pytest.mark.parametrize("S", [1, 64, 129, 880, 1560, 4680])
@pytest.mark.parametrize("J,r", [(128, 64), (1536, 192), (3072, 384), (2048, 512), (5120, 640), (1024, 1024)])
def test_projection_and_its_quantising_form(S, J, r):
    C = 32
    rows, centers, pick, encoder, mean = _data(S, J, C, r, seed=1)
    ids = pick.to(torch.uint8)
    coeff = ops.project(rows, centers, ids, mean, encoder)
    residual = (rows.float() - centers[pick].float() - mean).to(torch.bfloat16)
    want = residual.double() @ encoder.double().T
    # J products summed in fp32 (J * 2^-24 of their magnitudes), one rounding to bf16
    magnitude = residual.double().abs() @ encoder.double().abs().T
    assert bool(((coeff.double() - want).abs() <= 2.0 ** -8 * want.abs() + J * 2.0 ** -24 * magnitude + 1e-30).all())
    for in_coeff_dtype in (False, True):
        two = ops.quant_pack(coeff, in_coeff_dtype=in_coeff_dtype)
        one = ops.project_quant(rows, centers, ids, mean, encoder, in_coeff_dtype=in_coeff_dtype)
        assert torch.equal(one[0], two[0])
        assert torch.equal(one[1].view(torch.int16), two[1].view(torch.int16))


@pytest.mark.parametrize("S,J", [(8192, 64), (8193, 130), (9000, 63), (700, 512), (20000, 576)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_update_sums_members_in_token_order(S, J, dtype):
    """One Lloyd step: centres are the fp32 means of their members added one by one in token order."""
    gen = torch.Generator().manual_seed(S)
    C = 4
    base = 4.0 * torch.randn(C, J, generator=gen)
    pick = torch.randint(0, C, (S,), generator=gen)
    pick[:C] = torch.arange(C)
    rows = (base[pick] + 0.3 * torch.randn(S, J, generator=gen)).to(dtype)
    centers, ids = ops.kmeans(rows.cuda(), C, 1, torch.arange(C))
    assert torch.equal(ids.cpu().long(), pick)
    for c in range(C):
        member = rows[pick == c].float()
        total = torch.zeros(J)
        for row in member:
            total += row
        assert torch.equal(centers[c].cpu(), (total / member.shape[0]).to(torch.bfloat16))


@pytest.mark.parametrize("J,r", [(1536, 192), (3072, 384), (5120, 640)])
def test_rows_encode_to_the_same_bytes_in_a_chunk_of_any_size(J, r):
    """The projection entry points never cut K: a row's coefficients do not depend on its neighbours."""
    rows, centers, pick, encoder, mean = _data(3000, J, 16, r, seed=2)
    ids = pick.to(torch.uint8)
    whole = ops.project(rows, centers, ids, mean, encoder)
    codes, scales = ops.project_quant(rows, centers, ids, mean, encoder)
    for a, b in ((0, 64), (64, 500), (500, 1700), (1700, 3000)):
        assert torch.equal(ops.project(rows[a:b], centers, ids[a:b], mean, encoder), whole[a:b])
        part = ops.project_quant(rows[a:b], centers, ids[a:b], mean, encoder)
        assert torch.equal(part[0], codes[a:b]) and torch.equal(part[1].view(torch.int16), scales[a:b].view(torch.int16))
