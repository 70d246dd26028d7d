"""Scales whose reciprocal is not a finite number (a caller's own small ``eps``, rows of zeros or of tiny coefficients)."""
import pytest
import torch

from nanokv_b200 import ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("eps", [1e-38, 1e-39, 7e-40])
@pytest.mark.parametrize("S,r", [(5, 64), (130, 192), (40, 640)])
def test_rows_of_zeros_get_the_code_of_zero(S, r, eps):
    """Matrix-Game's rule takes the IEEE quotient, 0 / scale = 0 for any scale above zero."""
    gen = torch.Generator(device="cuda").manual_seed(r)
    centers = torch.randn(4, 128, generator=gen, device="cuda").to(torch.bfloat16)
    ids = torch.randint(0, 4, (S,), generator=gen, device="cuda").to(torch.uint8)
    rows = centers[ids.long()].contiguous()                       # residual zero
    rows[::3] += 1.0                                              # ordinary rows between them
    encoder = (torch.randn(r, 128, generator=gen, device="cuda") / 128 ** 0.5).to(torch.bfloat16)
    mean = torch.zeros(128, device="cuda")
    codes, scales = ops.project_quant(rows, centers, ids, mean, encoder, eps=eps, in_coeff_dtype=True)
    usual, usual_scales = ops.project_quant(rows, centers, ids, mean, encoder, in_coeff_dtype=True)
    zero = torch.ones(S, dtype=torch.bool, device="cuda")
    zero[::3] = False
    assert bool((codes[zero] == 0x77).all()) and bool((scales[zero].view(torch.int16) > 0).all())
    assert torch.equal(codes[~zero], usual[~zero]) and torch.equal(scales[~zero], usual_scales[~zero])


@pytest.mark.parametrize("in_coeff_dtype", [False, True])
@pytest.mark.parametrize("group", [64, 32])
def test_codes_stay_in_range_without_any_scale(group, in_coeff_dtype):
    """eps = 0 and a group of zeros: 0 / 0 has no code, but what is stored decodes to 0 and is one of -7 .. 7."""
    centers = torch.randn(2, 64, generator=torch.Generator().manual_seed(1)).to(torch.bfloat16).cuda()
    ids = torch.tensor([0, 1, 1], dtype=torch.uint8, device="cuda")
    encoder = torch.randn(64, 64, generator=torch.Generator().manual_seed(2)).to(torch.bfloat16).cuda()
    codes, scales = ops.project_quant(centers[ids.long()].contiguous(), centers, ids, torch.zeros(64, device="cuda"), encoder,
                                      group=group, eps=0.0, in_coeff_dtype=in_coeff_dtype)
    assert bool(((codes & 15) <= 14).all()) and bool(((codes >> 4) <= 14).all()) and not scales.any()
