"""Rows whose scores are not finite: a cut unit hands back what a whole one does."""
import pytest
import torch

from nanokv_b200 import ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("heads,tokens,queries", [(1, 100, 64), (148, 256, 256),          # whole units
                                                  (12, 2048, 256), (40, 1500, 1100)])     # cut ones
@pytest.mark.parametrize("D", [64, 128])
def test_no_weight_at_all(heads, tokens, queries, D):
    """Every key is NaN, so no part of a unit has a weight: (NaN, -inf), merged or not."""
    gen = torch.Generator(device="cuda").manual_seed(heads)
    q, v = (torch.randn(n, heads, D, generator=gen, device="cuda").to(torch.bfloat16) for n in (queries, tokens))
    k = torch.full_like(v, float("nan"))
    out, lse = ops.attention_lse(q, k, v, scale=0.1)
    assert bool(torch.isnan(out).all())
    assert bool((lse == float("-inf")).all())
    ops.check_status()
