"""Rows without a finite distance to any centre get an id that exists."""
import pytest
import torch

from nanokv_b200 import ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("value", [float("nan"), float("inf"), float("-inf"), 3e38])
@pytest.mark.parametrize("J,C", [(128, 16), (64, 512), (128, 20)])      # 20 centres: the CUDA-core kernel
def test_ids_stay_below_the_number_of_centres(J, C, value):
    gen = torch.Generator(device="cuda").manual_seed(C)
    centers = torch.randn(C, J, generator=gen, device="cuda").to(torch.bfloat16)
    pick = torch.randint(0, C, (300,), generator=gen, device="cuda")
    rows = (centers[pick].float() + 0.1 * torch.randn(300, J, generator=gen, device="cuda")).to(torch.bfloat16)
    bad = torch.tensor([0, 130, 299], device="cuda")
    rows[bad, 5] = value
    ids = ops.assign(rows, centers).long() & 0xFFFF
    assert int(ids.max()) < C
    keep = torch.ones(300, dtype=torch.bool, device="cuda").index_fill_(0, bad, False)
    assert torch.equal(ids[keep], pick[keep])
    init = torch.arange(C, dtype=torch.int32) % 100 + 1 if C < 100 else torch.randperm(298)[:min(C, 298)] + 1
    _, ids = ops.kmeans(rows, init.numel(), 2, init)
    assert int((ids.long() & 0xFFFF).max()) < init.numel()
