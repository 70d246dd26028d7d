"""Scratch of the reads: sized by what a launch uses, and not needed where memory is short."""
import pytest
import torch

from nanokv_b200 import _lib, ops
from test_gpu_decode_rows import operator, random_history

MB = 1 << 20


@pytest.mark.parametrize("dtype", [_lib.NKV_BF16, _lib.NKV_F32])
@pytest.mark.parametrize("heads,tokens,queries", [(148, 128, 256), (12, 2048, 256), (40, 1500, 1100), (40, 99840, 4680)])
@pytest.mark.parametrize("splits", [0, 4])
def test_workspace_holds_rows_and_used_partials_only(dtype, heads, tokens, queries, splits):
    D, size = 128, 4 if dtype == _lib.NKV_F32 else 2
    need = _lib.library().nkv_attn_codec_rows_workspace_bytes(dtype, queries, heads, D, D, tokens, 192, 192, splits)
    rows = 2 * tokens * heads * D * size
    bound = min(rows, 512 * MB) + 8192
    if dtype == _lib.NKV_F32:
        bound += 16 * queries * heads * (D + 4) * 4          # at most 16 splits
    elif splits:
        bound += splits * queries * heads * (2 * D + 4)
    elif heads != 148:                                       # 148 units of 256 queries fill one round: nothing is cut
        bound += 2 * 148 * 256 * (D + 1) * 4
    assert need <= bound
    if not splits and dtype == _lib.NKV_BF16:
        plain = _lib.library().nkv_attention_lse_workspace_bytes(queries, heads, D, tokens)
        assert plain <= (8192 if heads == 148 else 2 * 148 * 256 * (D + 1) * 4 + 8192)


@pytest.fixture
def no_scratch(monkeypatch):
    """Allocations of more than 64 KB of bytes fail, as they do on a device that is nearly full."""
    refused = []
    real = torch.empty

    def empty(*size, **kwargs):
        if kwargs.get("dtype") is torch.uint8 and len(size) == 1 and isinstance(size[0], int) and size[0] > 65536:
            refused.append(size[0])
            raise torch.OutOfMemoryError("out of memory")
        return real(*size, **kwargs)

    monkeypatch.setattr(torch, "empty", empty)
    yield refused
    assert refused, "nothing was asked for"


def _read_inputs(dtype, heads=3, D=128, rank=192, tokens=1500, queries=300):
    joint = heads * D
    views, weights = [], []
    for seed in (1, 2):
        views.append(random_history(tokens, joint, rank, seed=seed).view())
        decoder, mean = operator(joint, rank, seed)
        weights += [decoder.to(dtype).view(heads, D, rank), mean.to(torch.bfloat16).float().view(heads, D)]
    q = torch.randn(queries, heads, D, generator=torch.Generator(device="cuda").manual_seed(3), device="cuda").to(dtype)
    return q, views, weights


@pytest.mark.gpu
@pytest.mark.parametrize("dtype,bound", [(torch.bfloat16, 2.0 ** -7), (torch.float32, 1e-5)])
@pytest.mark.parametrize("splits", [None, 1])
def test_a_read_without_scratch(dtype, bound, splits, request):
    q, views, weights = _read_inputs(dtype)
    want, want_lse = ops.attn_codec(q, *views, *weights, scale=0.1, splits=splits)
    request.getfixturevalue("no_scratch")
    got, got_lse = ops.attn_codec(q, *views, *weights, scale=0.1, splits=splits)
    # bf16: weights and rows rounded to bf16 (2^-9 each) on both sides; fp32: the order of the sums
    assert float((got.double() - want.double()).norm() / want.double().norm()) < bound
    assert float((got_lse - want_lse).abs().max()) < 2 * bound


@pytest.mark.gpu
def test_plain_attention_without_scratch(request):
    gen = torch.Generator(device="cuda").manual_seed(4)
    q, k, v = (torch.randn(n, 3, 128, generator=gen, device="cuda").to(torch.bfloat16) for n in (300, 1500, 1500))
    want, want_lse = ops.attention_lse(q, k, v, scale=0.1)
    request.getfixturevalue("no_scratch")
    got, got_lse = ops.attention_lse(q, k, v, scale=0.1)
    assert float((got.float() - want.float()).norm() / want.float().norm()) < 2.0 ** -7
    assert float((got_lse - want_lse).abs().max()) < 2.0 ** -9
