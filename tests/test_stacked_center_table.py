"""Segments with different numbers of centres stacked into one history: the table's rows that no segment owns are zero,
whatever the memory held before, because sums over the whole table read them."""
import pytest
import torch

from nanokv_b200 import attention
from nanokv_b200.cache import CompressedHistory

JOINT, RANK, HEAD_DIM = 128, 64, 32


@pytest.fixture
def used_memory(monkeypatch):
    """Memory handed out without being cleared holds NaN, or the largest whole number."""
    real = torch.empty

    def empty(*size, **kwargs):
        array = real(*size, **kwargs)
        return array.fill_(float("nan") if array.is_floating_point() else torch.iinfo(array.dtype).max)

    monkeypatch.setattr(torch, "empty", empty)


def _parts(counts, clusters, device):
    gen = torch.Generator().manual_seed(11)
    parts = [(torch.randint(0, 256, (n, RANK // 2), generator=gen).to(torch.uint8),
              torch.rand(n, 1, generator=gen).to(torch.bfloat16), torch.randint(0, c, (n,), generator=gen).to(torch.uint8),
              torch.randn(c, JOINT, generator=gen).to(torch.bfloat16)) for n, c in zip(counts, clusters)]
    return [tuple(t.to(device) for t in part) for part in parts]


def _check_table(hist, parts, clusters):
    used = sum(clusters)
    assert hist.centers.shape[0] == len(clusters) * max(clusters)
    assert torch.equal(hist.centers[:used].cpu(), torch.cat([p[3] for p in parts]).cpu())
    assert not hist.centers[used:].any()
    counts = torch.zeros(hist.centers.shape[0], device=hist.centers.device)
    counts[:used] = 1.0
    assert torch.isfinite(counts @ hist.centers.float()).all()


@pytest.mark.parametrize("clusters", [(32, 4), (4, 32), (1, 16, 3), (8, 8), (5,)])
def test_rows_of_no_segment_are_zero_on_the_host(clusters, used_memory):
    parts = _parts([40] * len(clusters), clusters, "cpu")
    _check_table(CompressedHistory.stacked(parts, joint=JOINT, rank=RANK, device="cpu"), parts, clusters)


@pytest.mark.gpu
@pytest.mark.parametrize("source", ["cuda", "cpu"])         # one launch; copies one by one
@pytest.mark.parametrize("clusters", [(32, 4), (4, 32), (1, 16, 3), (8, 8), (5,)])
def test_rows_of_no_segment_are_zero(clusters, source, used_memory):
    parts = _parts([40] * len(clusters), clusters, source)
    _check_table(CompressedHistory.stacked(parts, joint=JOINT, rank=RANK, device="cuda"), parts, clusters)


@pytest.mark.gpu
def test_value_mean_residual_over_segments_of_different_centre_counts(used_memory):
    """The mixed-width read with its mean correction, against the same segments appended to a cleared history."""
    heads, width, clusters = JOINT // HEAD_DIM, 16, (32, 4)
    parts = _parts([70, 30], clusters, "cuda")
    gen = torch.Generator().manual_seed(12)
    index = torch.arange(width).expand(heads, width).contiguous()
    select = torch.zeros(heads, HEAD_DIM, width).scatter_(1, index[:, None, :], 1.0)
    read = torch.randn(heads, width, RANK, generator=gen) / RANK ** 0.5
    payload = dict(heads=heads, native_dim=HEAD_DIM, rank=RANK, groups=[dict(
        heads=torch.arange(heads), indices=index, q_reduce=select, k_read=read, v_read=read, k_affine=select,
        v_affine=select, lift=select.transpose(1, 2).contiguous())])
    mean = 0.1 * torch.randn(JOINT, generator=gen).cuda()
    decoder = (torch.randn(JOINT, RANK, generator=gen) / RANK ** 0.5).to(torch.bfloat16).cuda()
    q = torch.randn(24, heads, HEAD_DIM, generator=gen).to(torch.bfloat16).cuda()

    def appended():
        hist = CompressedHistory(joint=JOINT, rank=RANK, capacity=100, max_segments=2, centers_per_segment=max(clusters))
        for codes, scales, ids, centers in parts:
            offset, rows = hist.reserve_segment(ids.shape[0], centers.shape[0])
            rows.copy_(centers)
            for array, part in ((hist.codes, codes), (hist.scales, scales), (hist.ids, ids)):
                array[offset:offset + part.shape[0]].copy_(part)
        return hist

    def read_of(hist):
        low = dict(k=hist, v=hist, k_mean=mean, v_mean=mean, v_decoder=decoder)
        reader = attention.Reader(payload, dtype=torch.bfloat16)
        return attention.hybrid_attention(q, q, [], [low], reader, value_mean_residual=True)

    got, want = read_of(CompressedHistory.stacked(parts, joint=JOINT, rank=RANK, device="cuda")), read_of(appended())
    assert torch.isfinite(want).all() and torch.equal(got, want)
