"""Segments stacked into a history: one launch gives the arrays that copies one by one give."""
import pytest
import torch

from nanokv_b200 import codec
from nanokv_b200.cache import CompressedHistory

pytestmark = pytest.mark.gpu

ARRAYS = ("codes", "scales", "ids", "seg_start", "seg_center_row")


def _parts(counts, clusters, rank, joint, seed=0):
    gen = torch.Generator().manual_seed(seed)
    return [(torch.randint(0, 256, (n, rank // 2), generator=gen).to(torch.uint8), torch.randn(n, 1, generator=gen).to(torch.bfloat16),
             torch.randint(0, c, (n,), generator=gen).to(torch.uint8), torch.randn(c, joint, generator=gen).to(torch.bfloat16))
            for n, c in zip(counts, clusters)]


@pytest.mark.parametrize("counts", [[1], [1, 3, 2], [16, 160], [4680, 1, 1560], list(range(1, 38))])
@pytest.mark.parametrize("rank,joint", [(2, 8), (6, 24), (192, 1536)])
def test_one_launch_equals_copies(counts, rank, joint):
    clusters = [1 + 7 * i % 5 for i in range(len(counts))]
    parts = _parts(counts, clusters, rank, joint)
    copied = CompressedHistory.stacked(parts, joint=joint, rank=rank, device="cuda")        # from the host: one by one
    stacked = CompressedHistory.stacked([tuple(t.cuda() for t in p) for p in parts], joint=joint, rank=rank, device="cuda")
    assert stacked.tokens == sum(counts) and stacked.segments == len(counts)
    used = sum(clusters)
    for name in ARRAYS:
        assert torch.equal(getattr(stacked, name), getattr(copied, name)), name
    assert torch.equal(stacked.centers[:used], copied.centers[:used])
    assert torch.equal(stacked.codes.cpu(), torch.cat([p[0] for p in parts]))
    # misaligned sources
    shifted = [tuple(torch.cat([t.flatten()[:1], t.flatten()]).cuda()[1:].view(t.shape) for t in p) for p in parts]
    again = CompressedHistory.stacked(shifted, joint=joint, rank=rank, device="cuda")
    for name in ARRAYS:
        assert torch.equal(getattr(again, name), getattr(copied, name)), name


def test_parts_that_do_not_agree_are_refused():
    part = _parts([8], [4], 8, 16)[0]
    for bad in ((part[0][:7], *part[1:]), (*part[:2], part[2][:0], part[3]), (*part[:3], part[3][:, :12])):
        for move in (lambda t: t, lambda t: t.cuda()):
            with pytest.raises((ValueError, RuntimeError)):
                CompressedHistory.stacked([tuple(map(move, part)), tuple(map(move, bad))], joint=16, rank=8, device="cuda")


@pytest.mark.parametrize("shared", [False, True])
@pytest.mark.parametrize("form", ["ready", "fp32", "host", "strided"])
def test_given_centres_land_in_the_table(shared, form):
    gen = torch.Generator().manual_seed(3)
    op = codec.Operator(mean=torch.zeros(256).cuda(), encoder=torch.randn(64, 256, generator=gen).to(torch.bfloat16).cuda(),
                        decoder=torch.randn(256, 64, generator=gen).to(torch.bfloat16).cuda())
    hist = CompressedHistory(joint=256, rank=64, capacity=100, max_segments=3, centers_per_segment=16, shared_centers=shared)
    for step in range(3):
        table = torch.randn(16, 256, generator=gen).to(torch.bfloat16)
        given = {"ready": table.cuda(), "fp32": table.float().cuda(), "host": table,
                 "strided": torch.stack([table, table], dim=1).cuda()[:, 0]}[form]
        rows = (table[torch.randint(0, 16, (33,), generator=gen)].float()
                + 0.1 * torch.randn(33, 256, generator=gen)).to(torch.bfloat16).cuda()
        offset = codec.encode_append(hist, rows, op, centers=given)
        first = 0 if shared else 16 * step
        assert offset == 33 * step and torch.equal(hist.centers[first:first + 16].cpu(), table)
        assert hist.seg_start[:step + 2].tolist() == [33 * i for i in range(step + 2)]
        assert hist.seg_center_row[:step + 1].tolist() == [0 if shared else 16 * i for i in range(step + 1)]
