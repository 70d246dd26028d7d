"""nkv_attn_codec_rows and nkv_attention_lse_bf16 refuse what their kernels cannot take, before any CUDA call."""
import ctypes

import pytest

from nanokv_b200 import _lib

TOKENS, HEADS, D, RANK = 64, 2, 64, 64


def _history():
    """Addresses that are never read: every call below is refused on the host."""
    at = 1 << 20
    return _lib.History(at, at, at, at, at, at, TOKENS, 1, RANK, RANK, _lib.NKV_BF16, 1, 16, HEADS * D)


def _read(dtype, out, workspace, nbytes, splits=0):
    lib = _lib.library()
    history = _history()
    at = ctypes.c_void_p(1 << 20)
    return lib.nkv_attn_codec_rows(
        at, dtype, HEADS * D, D, 8, HEADS, D, D, ctypes.byref(history), ctypes.byref(history), at, at, at, at, 0, None, None,
        None, 0.1, ctypes.c_void_p(out), at, None, splits, workspace, nbytes, None)


@pytest.mark.parametrize("dtype", [_lib.NKV_BF16, _lib.NKV_F32])
def test_misaligned_results(dtype):
    for offset in (4, 8, 2):
        assert _read(dtype, (1 << 20) + offset, ctypes.c_void_p(1 << 20), 1 << 40) == _lib.NKV_ERR_INVALID
        assert b"results must be 16-byte aligned" in _lib.library().nkv_last_error()


@pytest.mark.parametrize("dtype", [_lib.NKV_BF16, _lib.NKV_F32])
@pytest.mark.parametrize("splits", [0, 1, 4])
def test_too_small_a_workspace(dtype, splits):
    need = _lib.library().nkv_attn_codec_rows_workspace_bytes(dtype, 8, HEADS, D, D, TOKENS, RANK, RANK, splits)
    assert need > 0
    for workspace, nbytes in ((ctypes.c_void_p(1 << 20), need - 1), (ctypes.c_void_p(1 << 20), 0), (None, need)):
        assert _read(dtype, 1 << 20, workspace, nbytes, splits) == _lib.NKV_ERR_INVALID
        assert b"too small" in _lib.library().nkv_last_error()


def test_plain_attention():
    lib = _lib.library()
    at = ctypes.c_void_p(1 << 20)
    need = lib.nkv_attention_lse_workspace_bytes(8, HEADS, D, TOKENS)
    for out, workspace, nbytes, message in (((1 << 20) + 8, at, need, b"results must be"), (1 << 20, at, need - 1, b"too small")):
        assert lib.nkv_attention_lse_bf16(at, at, at, HEADS * D, D, HEADS * D, D, 8, TOKENS, HEADS, D, D, 0.1,
                                          ctypes.c_void_p(out), at, None, workspace, nbytes, None) == _lib.NKV_ERR_INVALID
        assert message in lib.nkv_last_error()
