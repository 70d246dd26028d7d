"""What a decode whose waits give up leaves behind: a status, NaN rows, and NaN LSEs of the read over them.

The self-test entries run the row decode with nobody loading its decoder rows and a wait budget of a tenth of a
millisecond: the waits for those rows run out, nothing is in flight, and the context stays usable."""
import ctypes

import pytest
import torch

from nanokv_b200 import _lib, ops
from test_gpu_decode_rows import operator, random_history

BUDGET = 1 << 18


def _pointer(tensor):
    return ctypes.c_void_p(tensor.data_ptr())


def _stream():
    return ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)


@pytest.mark.gpu
@pytest.mark.parametrize("tokens,joint,rank,listed", [(1, 64, 64, False), (700, 1536, 192, False), (700, 1536, 192, True),
                                                      (9000, 5120, 640, False)])
def test_rows_that_were_not_finished_are_nan(tokens, joint, rank, listed):
    view = random_history(tokens, joint, rank, segments=min(2, tokens)).view()
    decoder, mean = operator(joint, rank)
    rows = torch.arange(0, tokens, 3, dtype=torch.int32, device="cuda") if listed else None
    if listed:
        rows[5] = -1                      # not a token: its row stays as it was
    n = tokens if rows is None else rows.numel()
    out = torch.zeros(n, joint, dtype=torch.bfloat16, device="cuda")
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    struct = view.struct()
    _lib.check(_lib.library().nkv_selftest_decode_gives_up(
        ctypes.byref(struct), None if rows is None else _pointer(rows), n, _pointer(decoder), _pointer(mean), joint,
        _pointer(out), _pointer(status), BUDGET, _stream()))
    assert 700 <= int(status.item()) < 760
    with pytest.raises(RuntimeError, match="device-side wait"):
        _lib.check_device_status(int(status.item()))
    unfinished = torch.isnan(out).all(dim=1)
    if listed:
        assert not bool(out[5].any()) and int(unfinished.sum()) == n - 1
    else:
        assert bool(unfinished.all())
    ops.check_status()                    # the device's own word was not involved
    assert not bool(torch.isnan(ops.decode_rows(view, decoder, mean, rows=None)).any())
    ops.check_status()


@pytest.mark.gpu
@pytest.mark.parametrize("D", [64, 128])
# whole units, units cut many ways, whole units and a cut tail; history splits
@pytest.mark.parametrize("heads,tokens,queries,splits", [(149, 300, 100, 0), (3, 2048, 256, 0), (40, 1500, 1100, 0),
                                                         (3, 2048, 300, 4)])
def test_a_read_over_rows_that_were_not_finished_has_nan_lse(D, heads, tokens, queries, splits):
    joint, rank = heads * D, 64
    hk, hv = (random_history(tokens, joint, rank, seed=s).view() for s in (1, 2))
    decoder, mean = operator(joint, rank)
    q = torch.randn(queries, heads, D, device="cuda").to(torch.bfloat16)
    lib = _lib.library()
    nbytes = lib.nkv_attn_codec_rows_workspace_bytes(_lib.NKV_BF16, queries, heads, D, D, tokens, rank, rank, splits)
    workspace = torch.zeros(nbytes, dtype=torch.uint8, device="cuda")
    out = torch.zeros(queries, heads, D, dtype=torch.bfloat16, device="cuda")
    lse = torch.zeros(queries, heads, device="cuda")
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    sk, sv = hk.struct(), hv.struct()
    _lib.check(lib.nkv_selftest_read_gives_up(
        _pointer(q), q.stride(0), q.stride(1), queries, heads, D, ctypes.byref(sk), ctypes.byref(sv), _pointer(decoder),
        _pointer(mean), _pointer(decoder), _pointer(mean), D ** -0.5, _pointer(out), _pointer(lse), _pointer(status), splits,
        _pointer(workspace), nbytes, BUDGET, _stream()))
    assert 700 <= int(status.item()) < 760
    assert bool(torch.isnan(lse).all())
    # the next read through the same memory is not affected
    status.zero_()
    _lib.check(lib.nkv_attn_codec_rows(
        _pointer(q), _lib.NKV_BF16, q.stride(0), q.stride(1), queries, heads, D, D, ctypes.byref(sk), ctypes.byref(sv),
        _pointer(decoder), _pointer(mean), _pointer(decoder), _pointer(mean), 0, None, None, None, D ** -0.5, _pointer(out),
        _pointer(lse), _pointer(status), splits, _pointer(workspace), nbytes, _stream()))
    assert int(status.item()) == 0
    assert not bool(torch.isnan(lse).any()) and not bool(torch.isnan(out).any())


def test_bad_arguments_are_refused():
    lib = _lib.library()
    history = _lib.History()
    for budget in (0, 1 << 40):
        assert lib.nkv_selftest_decode_gives_up(ctypes.byref(history), None, 0, None, None, 64, None, ctypes.c_void_p(16),
                                                budget, None) == _lib.NKV_ERR_INVALID
    assert lib.nkv_selftest_decode_gives_up(ctypes.byref(history), None, 0, None, None, 64, None, None, 1000,
                                            None) == _lib.NKV_ERR_INVALID


@pytest.mark.gpu
def test_a_captured_decode_makes_no_status_word(monkeypatch):
    """A word made inside a capture would lie in the graph's pool and be cleared by every replay."""
    view = random_history(300, 256, 64).view()
    decoder, mean = operator(256, 64)
    want = ops.decode_rows(view, decoder, mean)
    torch.cuda.synchronize()
    monkeypatch.setattr(ops, "_STATUS_WORDS", {})
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = ops.decode_rows(view, decoder, mean)
    assert not ops._STATUS_WORDS
    got.zero_()
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(got, want)
