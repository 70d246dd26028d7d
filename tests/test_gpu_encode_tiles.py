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
