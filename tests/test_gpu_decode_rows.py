"""Rows rebuilt on the tensor cores against the CUDA-core kernel with the same rounding points."""
import pytest
import torch

from nanokv_b200 import ops
from nanokv_b200.cache import CompressedHistory

pytestmark = pytest.mark.gpu


def random_history(tokens, joint, rank, *, group=None, scale_dtype=torch.bfloat16, clusters=16, segments=1, seed=0):
    """A history of random codes, scales, ids and centres (nothing here depends on how it was encoded)."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    hist = CompressedHistory(joint=joint, rank=rank, capacity=tokens, max_segments=segments,
                             centers_per_segment=clusters, group=group, scale_dtype=scale_dtype)
    cuts = [tokens * s // segments for s in range(segments + 1)]
    for a, b in zip(cuts, cuts[1:]):
        _, table = hist.reserve_segment(b - a, clusters)
        table.copy_(torch.randn(clusters, joint, generator=gen, device="cuda"))
    low, high = (torch.randint(0, 15, hist.codes.shape, generator=gen, device="cuda") for _ in range(2))
    hist.codes.copy_((low | (high << 4)).to(torch.uint8))
    hist.scales.copy_(0.05 + 0.1 * torch.rand(hist.scales.shape, generator=gen, device="cuda"))
    hist.ids.copy_(torch.randint(0, clusters, hist.ids.shape, generator=gen, device="cuda"))
    return hist


def operator(joint, rank, seed=1):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    decoder = (torch.randn(joint, rank, generator=gen, device="cuda") / rank ** 0.5).to(torch.bfloat16)
    return decoder, 0.1 * torch.randn(joint, generator=gen, device="cuda")


def both_paths(view, decoder, mean, rows=None):
    got = ops.decode_rows(view, decoder, mean, rows=rows)
    ops.force_simt(True)
    try:
        want = ops.decode_rows(view, decoder, mean, rows=rows)
    finally:
        ops.force_simt(False)
    return got.float(), want.float()


def check(got, want, rank):
    """Both kernels sum the same bf16 products in fp32 in different orders: the sums differ by at most
    rank * 2^-24 of the sum of magnitudes (below 2^-12 of a unit here), which moves a value only across a
    bf16 rounding boundary -- one step of the first rounding (|first| <= 8) and one of the second."""
    step = 2.0 ** -8 * (want.abs() + 8.0)
    assert bool(((got - want).abs() <= 2 * step).all())
    assert float((got != want).float().mean()) <= 4 * rank * 2.0 ** -15, "share of values that moved"


@pytest.mark.parametrize("tokens", [1, 127, 128, 129, 256, 257, 1000])
@pytest.mark.parametrize("joint,rank", [(64, 64), (192, 128), (1536, 192), (2048, 512), (5120, 640)])
def test_tile_edges(tokens, joint, rank):
    hist = random_history(tokens, joint, rank, segments=min(3, tokens))
    got, want = both_paths(hist.view(), *operator(joint, rank))
    check(got, want, rank)


@pytest.mark.parametrize("group,scale_dtype,clusters", [(32, torch.float16, 300), (64, torch.bfloat16, 16),
                                                        (None, torch.float16, 256)])
def test_quantiser_forms(group, scale_dtype, clusters):
    hist = random_history(700, 1280, 320 if group != 64 else 384, group=group, scale_dtype=scale_dtype,
                          clusters=clusters, segments=2)
    got, want = both_paths(hist.view(), *operator(1280, hist.rank))
    check(got, want, hist.rank)


def test_listed_rows_of_a_cut_history():
    hist = random_history(5000, 3072, 384, segments=7)
    decoder, mean = operator(3072, 384)
    gen = torch.Generator(device="cuda").manual_seed(5)
    rows = torch.randint(0, 3000, (1500,), generator=gen, device="cuda", dtype=torch.int32)
    got, want = both_paths(hist.view_tokens(777, 4001), decoder, mean, rows)
    check(got, want, 384)


def test_many_column_tiles_per_pair():
    """More (token tile, column tile) pairs than CTA pairs: runs that cross token tiles."""
    hist = random_history(9000, 5120, 640, clusters=64, segments=2)
    got, want = both_paths(hist.view(), *operator(5120, 640))
    check(got, want, 640)
