"""Nearest-centre ids: the same whatever the length of the call that a row comes in, and those of float64 wherever fp32
sums can tell two centres apart."""
import pytest
import torch

from nanokv_b200 import ops

pytestmark = pytest.mark.gpu


def _data(S, J, C, distance, seed):
    """Rows around centres of which every second is a near copy of the one before."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    centers = torch.randn(C, J, generator=gen, device="cuda").to(torch.bfloat16)
    centers[1::2] = (centers[::2].float() + distance * torch.randn(C // 2, J, generator=gen, device="cuda")).to(torch.bfloat16)
    pick = torch.randint(0, C, (S,), generator=gen, device="cuda")
    return (centers[pick].float() + 0.3 * torch.randn(S, J, generator=gen, device="cuda")).to(torch.bfloat16), centers


@pytest.mark.parametrize("S", [9473, 9600, 12480, 18945, 25000])
@pytest.mark.parametrize("J,C", [(1536, 64), (320, 256), (512, 512)])
def test_ids_of_long_calls_are_those_of_short_ones(S, J, C):
    """Above 9,472 rows a tile takes as many rows as fill whole rounds of 148 SMs.  It starts at a multiple of eight tokens
    there too: a row's place modulo eight decides the order of its norm's sum, and that near ties."""
    rows, centers = _data(S, J, C, 2e-3, seed=S + J)
    whole = ops.assign(rows, centers)
    for a, b in ((0, 104), (104, 4784), (4784, 9464), (9464, S)):
        assert torch.equal(ops.assign(rows[a:b], centers), whole[a:b])


@pytest.mark.parametrize("S", [9473, 12480])
def test_first_ids_of_a_long_c_means_are_those_of_a_short_one(S):
    """One iteration: the ids depend on the start rows only, which both calls have."""
    rows, centers = _data(S, 1536, 64, 2e-3, seed=S)
    rows[:64] = centers
    init = torch.arange(64, dtype=torch.int32)
    _, whole = ops.kmeans(rows, 64, 1, init)
    _, part = ops.kmeans(rows[:4680], 64, 1, init)
    assert torch.equal(part, whole[:4680])


@pytest.mark.parametrize("S", [200, 4680, 12480])
@pytest.mark.parametrize("J,C", [(192, 48), (1536, 64), (512, 320), (3072, 256)])
def test_ids_against_float64(S, J, C):
    """The distance of two centres to a row is off by what its sums round: a squared norm of J terms in chains of at most
    4 J / 64 + 9 additions, a product sum of at most J additions of which sixteen are exact at a time, and the last
    three operations.  Beyond that margin the id is float64's, and nearly every row lies beyond it."""
    rows, centers = _data(S, J, C, 2e-2, seed=S + J + C)
    ids = ops.assign(rows, centers).long() & 0xFFFF
    x, c = rows.double(), centers.double()
    norm_x, norm_c = (x * x).sum(1, keepdim=True), (c * c).sum(1)
    exact = norm_x + norm_c - 2.0 * (x @ c.T)
    error = 2.0 ** -24 * ((4 * J / 64 + 9) * norm_c + 3 * (norm_x + norm_c)) + 2.0 * 2.0 ** -23 * J / 16 * (x.abs() @ c.abs().T)
    best, nearest = exact.min(1, keepdim=True)
    margin = exact - best - error - error.gather(1, nearest)
    margin.scatter_(1, nearest, float("inf"))
    clear = margin.min(1).values > 0
    assert float(clear.double().mean()) > 0.9
    assert torch.equal(ids[clear], nearest[clear, 0])
    chosen = exact.gather(1, ids[:, None]) - best
    assert bool((chosen <= error.gather(1, ids[:, None]) + error.gather(1, nearest)).all())
