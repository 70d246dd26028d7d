"""Plain attention: rows that do not agree are refused on the host, before any launch."""
import pytest
import torch

from nanokv_b200 import ops


@pytest.mark.parametrize("k_shape,v_shape,message", [
    ((64, 3, 128), (63, 3, 128), "tokens"), ((64, 3, 128), (0, 3, 128), "tokens"), ((64, 3, 128), (65, 3, 128), "tokens"),
    ((64, 2, 128), (64, 3, 128), "heads"), ((64, 3, 128), (64, 2, 128), "heads"),
    ((64, 3, 64), (64, 3, 128), "wide")])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_rows_that_do_not_agree_are_refused(monkeypatch, k_shape, v_shape, message, dtype):
    monkeypatch.setattr(ops, "_require_cuda", lambda *tensors: tensors[0].device)
    monkeypatch.setattr(ops._lib, "library", lambda: pytest.fail("reached the library"))
    q = torch.zeros(8, 3, 128, dtype=dtype)
    with pytest.raises(ValueError, match=message):
        ops.attention_lse(q, torch.zeros(k_shape, dtype=dtype), torch.zeros(v_shape, dtype=dtype), scale=1.0)


def test_mixed_dtypes_are_refused(monkeypatch):
    monkeypatch.setattr(ops, "_require_cuda", lambda *tensors: tensors[0].device)
    monkeypatch.setattr(ops._lib, "library", lambda: pytest.fail("reached the library"))
    rows = torch.zeros(8, 3, 128)
    with pytest.raises(ValueError, match="dtype"):
        ops.attention_lse(rows, rows.to(torch.bfloat16), rows.to(torch.bfloat16), scale=1.0)


@pytest.mark.gpu
@pytest.mark.parametrize("k_heads,v_heads", [(3, 5), (4, 3), (5, 5)])
@pytest.mark.parametrize("D", [64, 128])
def test_rows_with_more_heads_than_the_queries(k_heads, v_heads, D):
    gen = torch.Generator(device="cuda").manual_seed(k_heads)
    q, k, v = (torch.randn(n, h, D, generator=gen, device="cuda").to(torch.bfloat16)
               for n, h in ((200, 3), (333, k_heads), (333, v_heads)))
    got = ops.attention_lse(q, k, v, scale=D ** -0.5)
    want = ops.attention_lse(q, k[:, :3].contiguous(), v[:, :3].contiguous(), scale=D ** -0.5)
    assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])


@pytest.mark.gpu
def test_rows_that_start_off_a_16_byte_boundary_are_refused():
    flat = torch.randn(3, 64 * 2 * 128 + 8, device="cuda").to(torch.bfloat16)
    aligned = [row[:64 * 2 * 128].view(64, 2, 128) for row in flat]
    for which in range(3):
        rows = list(aligned)
        rows[which] = flat[which][4:4 + 64 * 2 * 128].view(64, 2, 128)
        with pytest.raises(ValueError, match="aligned"):
            ops.attention_lse(*rows, scale=0.1)
