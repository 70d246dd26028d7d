"""Host tables go to the device without a wait, so nothing may be read from memory that the caller can write to afterwards."""
import pytest
import torch

from nanokv_b200 import ops

pytestmark = pytest.mark.gpu

BUSY_CYCLES = 100_000_000        # some 50 ms: the copy cannot run before the host goes on


@pytest.mark.parametrize("side", [False, True])
@pytest.mark.parametrize("pinned", [False, True])
def test_table_is_the_one_at_the_call(pinned, side):
    stream = torch.cuda.Stream() if side else torch.cuda.current_stream()
    want = torch.arange(1, 5001, dtype=torch.int32)
    values = want.pin_memory() if pinned else want.clone()
    torch.zeros(1, device="cuda")
    torch.cuda.synchronize()
    with torch.cuda.stream(stream):
        torch.cuda._sleep(BUSY_CYCLES)
        got = ops.upload(values, "cuda")
        values.zero_()
    torch.cuda.synchronize()
    assert torch.equal(got.cpu(), want)


@pytest.mark.parametrize("side", [False, True])
def test_start_rows_are_those_at_the_call(side):
    gen = torch.Generator().manual_seed(5)
    x = torch.randn(300, 128, generator=gen).to(torch.bfloat16).cuda()
    rows = torch.randperm(300, generator=gen)[:16].to(torch.int32)
    centers, ids = ops.kmeans(x, 16, 0, rows)
    stream = torch.cuda.Stream() if side else torch.cuda.current_stream()
    torch.cuda.synchronize()
    pinned = rows.pin_memory()
    with torch.cuda.stream(stream):
        torch.cuda._sleep(BUSY_CYCLES)
        got, got_ids = ops.kmeans(x, 16, 0, pinned)
        pinned.zero_()
    torch.cuda.synchronize()
    assert torch.equal(centers, x[rows.long().cuda()])
    assert torch.equal(got, centers) and torch.equal(got_ids, ids)
