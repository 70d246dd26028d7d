"""Projection and quantiser in one call: the library says whether it takes scratch, and a call is made once."""
import pytest
import torch

from nanokv_b200 import _lib, ops

BF16, F32 = _lib.NKV_BF16, _lib.NKV_F32


@pytest.mark.parametrize("r,group,one", [(64, 64, True), (640, 640, True), (1024, 1024, True), (96, 32, True), (640, 32, True),
                                         (32, 32, False), (608, 32, False), (96, 96, False), (1088, 1088, False),
                                         (64, 16, False), (192, 64, False)])
def test_scratch_of_ranks_and_groups(r, group, one):
    need = _lib.library().nkv_project_quant_workspace_bytes
    assert need(BF16, BF16, 100, 128, r, group, 256) == (0 if one else 100 * r * 2)
    assert need(BF16, BF16, 100, 96, r, group, 256) == 100 * r * 2                 # rows that are not whole chunks
    assert need(BF16, BF16, 100, 128, r, group, 264) == 100 * r * 2                # codes off 16 bytes
    assert need(F32, BF16, 100, 128, r, group, 256) == 100 * r * 2
    assert need(F32, F32, 100, 128, r, group, 256) == 100 * r * 4
    assert need(BF16, BF16, 0, 128, r, group, 256) == 0


def _counted(monkeypatch):
    """Counts the calls that reach the library."""
    calls, library = [], _lib.library()

    class Counting:
        def __getattr__(self, name):
            function = getattr(library, name)
            if name != "nkv_project_quant":
                return function
            return lambda *arguments: (calls.append(name), function(*arguments))[1]

    monkeypatch.setattr(_lib, "library", lambda: Counting())
    return calls


def _operands(S, J, r):
    gen = torch.Generator(device="cuda").manual_seed(r)
    centers = torch.randn(8, J, generator=gen, device="cuda").to(torch.bfloat16)
    ids = torch.randint(0, 8, (S,), generator=gen, device="cuda").to(torch.uint8)
    rows = (centers[ids.long()].float() + 0.3 * torch.randn(S, J, generator=gen, device="cuda")).to(torch.bfloat16)
    encoder = (torch.randn(r, J, generator=gen, device="cuda") / J ** 0.5).to(torch.bfloat16)
    return rows, centers, ids, 0.1 * torch.randn(J, generator=gen, device="cuda"), encoder


@pytest.mark.gpu
@pytest.mark.parametrize("r,group", [(64, 64), (32, 32), (608, 32), (96, 32), (640, 32), (96, 96), (1088, 1088), (192, 64)])
def test_one_call_per_chunk(r, group, monkeypatch):
    operands = _operands(77, 128, r)
    form = dict(group=group, scale_dtype=torch.float16)
    want = ops.quant_pack(ops.project(*operands), **form)
    calls = _counted(monkeypatch)
    got = ops.project_quant(*operands, **form)
    assert len(calls) == 1
    assert torch.equal(got[0], want[0]) and torch.equal(got[1].view(torch.int16), want[1].view(torch.int16))


@pytest.mark.gpu
def test_a_refused_call_is_not_repeated(monkeypatch):
    rows, *rest = _operands(77, 128, 64)
    shifted = torch.empty(77 * 128 + 1, dtype=torch.bfloat16, device="cuda")[1:].view(77, 128).copy_(rows)
    calls = _counted(monkeypatch)
    with pytest.raises(ValueError, match="aligned"):
        ops.project_quant(shifted, *rest)
    assert len(calls) == 1
