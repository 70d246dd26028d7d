"""fp32 assignment and projection: every sum is one chain of fused multiply-adds in the order of K, so that what is
stored (ids, codes) does not depend on how a kernel cuts its work."""
import numpy as np
import pytest
import torch

from nanokv_b200 import ops

pytestmark = pytest.mark.gpu


def _chain(a, b):
    """[n,K] x [m,K] in float32: acc = fma(a_k, b_k, acc) for k = 0, 1, 2 ...; the 64-bit significand of an extended
    number holds the exact product and rounds the sum far below a float32 step."""
    acc = np.zeros((a.shape[0], b.shape[0]), dtype=np.float32)
    a, b = a.astype(np.longdouble), b.astype(np.longdouble)
    for k in range(a.shape[1]):
        acc = (a[:, k:k + 1] * b[None, :, k] + acc).astype(np.float32)
    return acc


def _squares(x):
    """Four interleaved chains, added in pairs."""
    parts = [np.zeros(x.shape[0], dtype=np.float32) for _ in range(4)]
    wide = x.astype(np.longdouble)
    for k in range(x.shape[1]):
        parts[k % 4] = (wide[:, k] * wide[:, k] + parts[k % 4]).astype(np.float32)
    return (parts[0] + parts[1]) + (parts[2] + parts[3])


def _data(S, J, C):
    gen = torch.Generator().manual_seed(S + J)
    centers = torch.randn(C, J, generator=gen).to(torch.bfloat16).float()
    twin = centers[0::2][:C // 2].clone()
    twin[:, 0] += 2.0 ** -9          # distances of a pair of centres differ by less than the rounding of their sums
    centers[1::2] = twin
    pick = torch.randint(0, C, (S,), generator=gen)
    return centers[pick] + 0.3 * torch.randn(S, J, generator=gen), centers, gen


@pytest.mark.parametrize("S,J,r", [(1, 8, 1), (65, 31, 70), (300, 200, 192), (1000, 258, 65), (5000, 64, 192)])
def test_projection(S, J, r):
    rows, centers, gen = _data(S, J, 16)
    stored = centers.to(torch.bfloat16)
    ids = torch.randint(0, 16, (S,), generator=gen).to(torch.uint8)
    mean, encoder = torch.randn(J, generator=gen), torch.randn(r, J, generator=gen) / J ** 0.5
    got = ops.project(rows.cuda(), stored.cuda(), ids.cuda(), mean.cuda(), encoder.cuda()).cpu()
    residual = (rows - stored.float()[ids.long()]) - mean
    assert np.array_equal(got.numpy(), _chain(residual.numpy(), encoder.numpy()))


@pytest.mark.parametrize("S,J,C", [(1, 8, 2), (65, 31, 20), (700, 200, 16), (300, 258, 130), (10000, 64, 64)])
def test_assignment(S, J, C):
    rows, centers, _ = _data(S, J, C)
    got = ops.assign(rows.cuda(), centers.cuda()).cpu().long() & 0xFFFF
    dist = (_squares(rows.numpy())[:, None] + _squares(centers.numpy())[None]) - np.float32(2) * _chain(rows.numpy(), centers.numpy())
    assert np.array_equal(got.numpy(), dist.argmin(axis=1))     # the first of equal distances
