"""Encoder kernels where a call's tiles, column parts and clusters change: the bytes must not."""
import pytest
import torch

from nanokv_b200 import ops

pytestmark = pytest.mark.gpu


def _data(S, J, C, r, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    centers = torch.randn(C, J, generator=gen, device="cuda").to(torch.bfloat16)
    # every second centre is a near copy of the one before: distances agree to a few parts in 1e4
    centers[1::2] = (centers[::2].float() + 2e-3 * torch.randn(C // 2, J, generator=gen, device="cuda")).to(torch.bfloat16)
    pick = torch.randint(0, C, (S,), generator=gen, device="cuda")
    rows = (centers[pick].float() + 0.3 * torch.randn(S, J, generator=gen, device="cuda")).to(torch.bfloat16)
    encoder = (torch.randn(r, J, generator=gen, device="cuda") / J ** 0.5).to(torch.bfloat16)
    return rows, centers, encoder, 0.1 * torch.randn(J, generator=gen, device="cuda")


@pytest.mark.parametrize("J,C", [(64, 16), (192, 48), (320, 256), (1536, 64), (512, 320), (1024, 512)])
def test_ids_do_not_depend_on_the_tiling(J, C):
    """Calls of 8 to 9,472 rows take tiles of 16 to 64 rows, one to eight parts of the centres, pairs of tiles."""
    rows, centers, _, _ = _data(9472, J, C, 64, seed=J + C)
    whole = ops.assign(rows, centers).view(torch.uint8)
    for a, b in ((0, 8), (8, 72), (64, 977), (976, 3000), (3000, 9472)):
        assert torch.equal(ops.assign(rows[a:b], centers).view(torch.uint8), whole.view(9472, -1)[a:b].flatten())
    # against float64: only where the two nearest are as close as fp32 sums of J squares can tell apart
    exact = torch.cdist(rows.double(), centers.double()) ** 2
    near = exact.gather(1, ops.assign(rows, centers).long()[:, None] & 0xFFFF)[:, 0]
    assert bool((near - exact.min(dim=1).values <= J * 2.0 ** -22 * 3 * J).all())


@pytest.mark.parametrize("S", [9473, 12480])
def test_long_calls_assign_every_row(S):
    """Tiles of an odd number of rows, an odd number of tiles in pairs."""
    gen = torch.Generator(device="cuda").manual_seed(S)
    for C in (64, 512):
        centers = torch.randn(C, 256, generator=gen, device="cuda").to(torch.bfloat16)
        pick = torch.randint(0, C, (S,), generator=gen, device="cuda")
        rows = (centers[pick].float() + 0.3 * torch.randn(S, 256, generator=gen, device="cuda")).to(torch.bfloat16)
        assert torch.equal(ops.assign(rows, centers).long() & 0xFFFF, pick)


@pytest.mark.parametrize("S", [1, 31, 65, 400, 3000])
@pytest.mark.parametrize("J,r", [(64, 32), (192, 96), (1536, 160), (448, 640), (8256, 64)])
def test_groups_of_32_are_quantised_in_place(S, J, r):
    rows, centers, encoder, mean = _data(S, J, 16, r, seed=S)
    ids = ops.assign(rows, centers)
    coeff = ops.project(rows, centers, ids, mean, encoder)
    for in_coeff_dtype in (False, True):
        for scale_dtype in (torch.float16, torch.bfloat16):
            form = dict(group=32, in_coeff_dtype=in_coeff_dtype, scale_dtype=scale_dtype)
            one, two = ops.project_quant(rows, centers, ids, mean, encoder, **form), ops.quant_pack(coeff, **form)
            assert torch.equal(one[0], two[0]) and torch.equal(one[1].view(torch.int16), two[1].view(torch.int16))


def test_rows_that_are_not_finite_leave_their_neighbours_alone():
    rows, centers, encoder, mean = _data(300, 1536, 16, 192, seed=5)
    ids = ops.assign(rows, centers)
    clean = {g: ops.project_quant(rows, centers, ids, mean, encoder, group=g) for g in (192, 32)}
    bad = rows.clone()
    bad[7, 3], bad[64, 1000], bad[299, 0] = float("inf"), float("nan"), -float("inf")
    keep = torch.ones(300, dtype=torch.bool, device="cuda")
    keep[[7, 64, 299]] = False
    for group, want in clean.items():
        codes, scales = ops.project_quant(bad, centers, ids, mean, encoder, group=group)
        assert torch.equal(codes[keep], want[0][keep]) and torch.equal(scales[keep], want[1][keep])
        assert bool(((codes & 15) <= 14).all() and ((codes >> 4) <= 14).all())


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("S,J", [(40, 64), (1000, 320), (9000, 66)])
@pytest.mark.parametrize("iters", [0, 1])
def test_means_of_separated_clusters(S, J, iters, dtype):
    """Rows within 0.3 sqrt(J) of one of eight centres; the second eight start rows double the first, so their clusters
    stay empty and keep them.  One fp32 addition per row in token order, one rounding to bf16."""
    gen = torch.Generator().manual_seed(S + J)
    base = 4.0 * torch.randn(8, J, generator=gen)
    pick = torch.cat([torch.arange(8), torch.randint(0, 8, (S - 8,), generator=gen)])
    rows = (base[pick] + 0.3 * torch.randn(S, J, generator=gen)).to(dtype)
    init = torch.cat([torch.arange(8), torch.arange(8)])
    centers, ids = ops.kmeans(rows.cuda(), 16, iters, init)
    assert torch.equal(ids.cpu().long(), pick if iters else torch.zeros(S, dtype=torch.long))
    for c in range(16):
        want = rows[init[c]].float()
        if iters and c < 8:
            want = torch.zeros(J)
            for row in rows[pick == c].float():
                want += row
            want /= int((pick == c).sum())
        assert torch.equal(centers[c].cpu(), want.to(torch.bfloat16))
