"""The fp32 read cut into history splits is as close to float64 as an undivided one."""
import pytest
import torch

from nanokv_b200 import ops
from test_gpu_decode_rows import random_history
from test_gpu_f32_read import _rows64

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tokens,queries", [(300, 300), (771, 50), (3102, 73), (4096, 33)])
@pytest.mark.parametrize("D,heads", [(128, 12), (64, 12)])
def test_lse_rounds_once(tokens, queries, D, heads):
    joint, rank = heads * D, 192
    views, weights, rows = [], [], []
    for seed in (1, 2):
        hist = random_history(tokens, joint, rank, seed=seed)
        hist.scales.mul_(0.4)                                  # scores of a few units, LSEs of 6 to 10
        decoder = torch.randn(joint, rank, generator=torch.Generator("cuda").manual_seed(seed), device="cuda") / rank ** 0.5
        mean = torch.zeros(joint, device="cuda")
        views.append(hist.view())
        weights += [decoder.view(heads, D, rank), mean.view(heads, D)]
        rows.append(_rows64(hist, decoder, mean).view(tokens, heads, D))
    q = torch.randn(queries, heads, D, generator=torch.Generator("cuda").manual_seed(3), device="cuda")
    out, lse = ops.attn_codec(q, *views, *weights, scale=D ** -0.5)
    score = torch.einsum("qhd,nhd->qhn", q.double(), rows[0]) * D ** -0.5
    want = torch.einsum("qhn,nhd->qhd", score.softmax(-1), rows[1])
    exact = score.logsumexp(-1)
    assert float((out.double() - want).norm() / want.norm()) < 2e-6
    # in steps of the LSE's own rounding: 0.29 rms from the last rounding, as much again from the parts' LSEs
    # averaged over the parts, the rest from scores and sums; a fold over 16 parts has 0.5 and more
    step = torch.exp2(torch.floor(torch.log2(exact.abs())) - 23)
    assert float(((lse.double() - exact) / step).square().mean().sqrt()) < 0.44
