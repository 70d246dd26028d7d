"""The C-means takes its scratch wherever it starts: a caller's arena may hand out any address."""
import ctypes

import pytest
import torch

from nanokv_b200 import _lib, ops

pytestmark = pytest.mark.gpu

GUARD = 512


def _kmeans(x, clusters, iters, init, shift):
    """nkv_kmeans with scratch that starts ``shift`` bytes past a multiple of 256; what lies around it is left alone."""
    lib = _lib.library()
    S, J = x.shape
    need = lib.nkv_kmeans_workspace_bytes(S, J, clusters)
    arena = torch.full((need + 2 * GUARD,), 0xA5, dtype=torch.uint8, device="cuda")
    assert arena.data_ptr() % 256 == 0
    first = 256 + shift
    centers = torch.empty(clusters, J, dtype=torch.bfloat16, device="cuda")
    ids = torch.empty(S, dtype=torch.uint8, device="cuda")
    pointer = lambda t, offset=0: ctypes.c_void_p(t.data_ptr() + offset)
    _lib.check(lib.nkv_kmeans(
        pointer(x), ops.dtype_code(x.dtype), S, J, clusters, iters, pointer(init), pointer(centers), pointer(ids), 1,
        pointer(arena, first), need, ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
    assert bool((arena[:first] == 0xA5).all()) and bool((arena[first + need:] == 0xA5).all())
    return centers, ids


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("S,J,C", [(1, 64, 1), (300, 320, 16), (777, 192, 48), (130, 50, 7)])
def test_scratch_may_start_anywhere(S, J, C, dtype):
    gen = torch.Generator(device="cuda").manual_seed(S + J)
    x = torch.randn(S, J, generator=gen, device="cuda").to(dtype)
    init = torch.randperm(S, generator=torch.Generator().manual_seed(C))[:C].to(torch.int32).cuda()
    for iters in (0, 2):
        want_centers, want_ids = _kmeans(x, C, iters, init, 0)
        for shift in (1, 2, 4, 8, 12, 16, 255):
            centers, ids = _kmeans(x, C, iters, init, shift)
            assert torch.equal(centers.view(torch.int16), want_centers.view(torch.int16)) and torch.equal(ids, want_ids)
