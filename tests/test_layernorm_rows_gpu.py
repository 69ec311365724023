"""LayerNorm forward of bf16 rows with all loads first, at the edges of its widths and of a block's rows, against float64 PyTorch."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [1, 7, 8, 9, 4097])
@pytest.mark.parametrize("D", [8, 248, 256, 264, 512, 520, 768, 776, 1024])
@pytest.mark.parametrize("residual", [False, True])
def test_rows(rows, D, residual):
    from cme213_final_project_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(rows * 2000 + D)
    x, res = (torch.randn(rows, D, generator=g, device="cuda").to(torch.bfloat16) for _ in range(2))
    gamma, beta = (torch.randn(D, generator=g, device="cuda").to(torch.bfloat16) for _ in range(2))
    y, mean, rstd, summed = ops.layernorm_fwd(x, gamma, beta, 1e-5, residual=res if residual else None, save_sum=residual)
    z = x.double() + (res.double() if residual else 0)
    mu, var = z.mean(1), z.var(1, unbiased=False)
    scale = 1 / torch.sqrt(var + 1e-5)
    want = (z - mu[:, None]) * scale[:, None] * gamma.double() + beta.double()
    # sums of at most 1024 elements up to 8 in fp32, a square root and a few products
    tol = 1024 * 2.0 ** -24
    assert (mean.double() - mu).abs().max().item() < 8 * tol
    assert ((rstd.double() - scale).abs() / scale).max().item() < 8 * tol
    size = (z - mu[:, None]).abs() * scale[:, None] * gamma.double().abs() + beta.double().abs()
    assert ((y.double() - want).abs() <= want.abs() * 2.0 ** -8 + size * 16 * tol).all()      # rounded once to 8 bits
    if residual:
        assert torch.equal(summed, z.to(torch.bfloat16))       # one fp32 addition, rounded once
