"""The read that rebuilds rows first against the fused kernel, over every form both accept."""
import ctypes

import pytest
import torch

from nanokv_b200 import _lib, attention, ops
from test_gpu_decode_rows import operator, random_history

pytestmark = pytest.mark.gpu


def _read(entry, q, hk, hv, wk, bk, wv, bv, *, prepared, splits, rope=None, camera_k=None, camera_v=None):
    lib = _lib.library()
    Q, H, D = q.shape
    out = torch.full((Q, H, D), float("nan"), dtype=q.dtype, device="cuda")
    lse = torch.full((Q, H), float("nan"), device="cuda")
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    if entry == "nkv_attn_codec_rows":
        nbytes = lib.nkv_attn_codec_rows_workspace_bytes(_lib.NKV_BF16, Q, H, D, D, hk.tokens, hk.rank, hk.group, splits)
        assert nbytes > 0
    else:
        nbytes = lib.nkv_attn_codec_workspace_bytes(Q, H, D, splits)
    workspace = torch.empty(max(nbytes, 1), dtype=torch.uint8, device="cuda")
    pointer = lambda t: ctypes.c_void_p(t.data_ptr())
    sk, sv = hk.struct(), hv.struct()
    extra = [None if item is None else ctypes.byref(item.struct()) for item in (rope, camera_k, camera_v)]
    _lib.check(getattr(lib, entry)(
        pointer(q), _lib.NKV_BF16, q.stride(0), q.stride(1), Q, H, D, D, ctypes.byref(sk), ctypes.byref(sv),
        pointer(wk), pointer(bk), pointer(wv), pointer(bv), 1 if prepared else 0, *extra, D ** -0.5, pointer(out),
        pointer(lse), pointer(status), splits, pointer(workspace), nbytes,
        ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
    assert int(status.item()) == 0
    return out.float(), lse


def compare(heads, D, rank, tokens, queries, *, rope=False, selected=False, camera=False, prepared=True, splits=1,
            **form):
    joint = heads * D
    hk = random_history(tokens, joint, rank, seed=3, **form).view()
    hv = random_history(tokens, joint, rank, seed=4, **form).view()
    gen = torch.Generator(device="cuda").manual_seed(5)
    weights = []
    for seed in (6, 7):
        w, mean = operator(joint, rank, seed)
        weights += [ops.prepare_decoder(w) if prepared else w, mean.to(torch.bfloat16).float()]
    # a strided view: the queries of every other row of a wider tensor
    q = torch.randn(queries, 2, heads, D, generator=gen, device="cuda").to(torch.bfloat16)[:, 1]
    extra = {}
    if rope or selected:
        half = D if selected else D // 2      # pairs of a native row; selected readers keep a subset
        angles = torch.rand(96, half, generator=gen, device="cuda").double() * 6.0
        table = attention.RopeTable(torch.polar(torch.ones_like(angles), angles), frame_seqlen=48, width=8)
        pairs = (torch.randint(0, half, (heads, D // 2), generator=gen, device="cuda", dtype=torch.int32)
                 if selected else None)
        extra["rope"] = table.view(torch.arange(tokens, device="cuda") * 3 % 4000, pairs)
    if camera:
        for name in ("camera_k", "camera_v"):
            extra[name] = ops.CameraView(torch.randn(5, 4, 4, 4, generator=gen, device="cuda"),
                                         torch.randint(0, 4, (heads, D // 8), generator=gen, device="cuda",
                                                       dtype=torch.int32), -(-tokens // 5))
    got, got_lse = _read("nkv_attn_codec_rows", q, hk, hv, *weights, prepared=prepared, splits=splits, **extra)
    want, want_lse = _read("nkv_attn_codec_pos", q, hk, hv, *weights, prepared=prepared, splits=max(splits, 1), **extra)
    # Both attend the same bf16 rows with bf16 weights (2^-9 each) and round O, and a split's partial O, to
    # bf16; a rebuilt value may sit one bf16 step apart where fp32 sums meet a rounding boundary.
    assert float((got - want).norm() / want.norm()) < 2.0 ** -7
    assert float((got_lse - want_lse).abs().max()) < 2.0 ** -6
    return got


@pytest.mark.parametrize("tokens,queries", [(1, 1), (127, 128), (129, 129), (1000, 300), (4100, 513)])
@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("splits", [0, 1, 5])
def test_sizes(tokens, queries, D, splits):
    compare(3, D, 192, tokens, queries, splits=splits, segments=min(2, tokens))


@pytest.mark.parametrize("prepared", [True, False])
@pytest.mark.parametrize("form", [dict(group=32, scale_dtype=torch.float16, clusters=300), dict(group=64),
                                  dict(scale_dtype=torch.float16, segments=3)])
def test_quantiser_forms(form, prepared):
    compare(4, 128, 320 if form.get("group") != 64 else 640, 777, 200, prepared=prepared, **form)


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("position", [dict(rope=True), dict(selected=True), dict(camera=True),
                                      dict(rope=True, camera=True)])
def test_positional_forms(D, position):
    compare(5, D, 128, 900, 260, **position)


@pytest.mark.parametrize("heads,D,tokens,queries", [(12, 128, 2048, 256), (3, 128, 5000, 700), (8, 64, 3000, 5000),
                                                    (40, 128, 1500, 1100), (1, 128, 20000, 64), (149, 64, 640, 100)])
def test_left_over_units_are_cut(heads, D, tokens, queries):
    """Units that do not fill a round of the SMs: none whole, one cut many ways, whole rounds and a tail."""
    compare(heads, D, 64, tokens, queries, splits=0)


def test_head_batches():
    """Rows of all heads exceed the scratch bound: the read goes through the heads in batches."""
    compare(40, 128, 64, 30000, 64, rope=True, splits=0)


def test_reads_on_two_streams_do_not_share_state():
    joint, rank, heads = 1024, 128, 8
    views = [random_history(6000, joint, rank, seed=s).view() for s in (1, 2)]
    w, mean = operator(joint, rank)
    bias = mean.to(torch.bfloat16).float().view(heads, 128)
    q = torch.randn(700, heads, 128, device="cuda").to(torch.bfloat16)
    read = lambda v: ops.attn_codec(q, v, v, w.view(heads, 128, rank), bias, w.view(heads, 128, rank), bias, scale=0.1)[0]
    want = [read(v) for v in views]
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in views]
    got = []
    for _ in range(4):
        for stream, view in zip(streams, views):
            with torch.cuda.stream(stream):
                got.append(read(view))
    torch.cuda.synchronize()
    assert all(torch.equal(out, want[i % 2]) for i, out in enumerate(got))


@pytest.mark.parametrize("N,Q,H,D", [(1, 1, 1, 64), (128, 256, 2, 128), (129, 257, 3, 128), (5000, 100, 2, 64)])
def test_plain_rows_against_the_cuda_core_kernel(N, Q, H, D):
    gen = torch.Generator(device="cuda").manual_seed(N)
    q, k, v = (torch.randn(n, H, D, generator=gen, device="cuda").to(torch.bfloat16) for n in (Q, N, N))
    got, got_lse = ops.attention_lse(q, k, v, scale=D ** -0.5)
    ops.force_simt(True)
    try:
        want, want_lse = ops.attention_lse(q, k, v, scale=D ** -0.5)
    finally:
        ops.force_simt(False)
    # weights go to bf16 (2^-9) before the sum, results and split partials are rounded to bf16
    assert float((got.float() - want.float()).norm() / want.float().norm()) < 2.0 ** -7
    assert float((got_lse - want_lse).abs().max()) < 2.0 ** -9


@pytest.mark.parametrize("heads,rank,queries,tokens,by_rows", [
    (16, 512, 1024, 1500, 0), (16, 512, 1024, 2561, 1), (24, 384, 512, 1000, 0), (24, 384, 1024, 1000, 1),
    (24, 384, 2048, 1000, 0), (16, 512, 256, 1000, 1), (12, 192, 1024, 1000, 1), (40, 640, 1024, 1000, 1)])
def test_which_form_reads(heads, rank, queries, tokens, by_rows):
    """The rule on 148 SMs, and the same result from either side of it through the public call."""
    lib = _lib.library()
    faster = lib.nkv_attn_codec_rows_is_faster(_lib.NKV_BF16, queries, heads, 128, 128, tokens, rank, rank, 0)
    if torch.cuda.get_device_properties(0).multi_processor_count == 148:
        assert faster == by_rows
    assert lib.nkv_attn_codec_rows_is_faster(_lib.NKV_BF16, queries, heads, 128, 128, tokens, rank, rank, 1) == 1
    compare(heads, 128, rank, tokens, queries, splits=0)
