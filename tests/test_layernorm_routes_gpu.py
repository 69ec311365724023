"""LayerNorm forward on both sides of the sizes at which its kernel changes, and with operands off a 16-byte boundary."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _inputs(rows, D, dtype, seed, offset=0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    out = []
    for n in (rows * D, rows * D, D, D):
        t = torch.empty(n + offset, device="cuda", dtype=dtype)[offset:]
        t.copy_(torch.randn(n, generator=g, device="cuda"))
        out.append(t.view(rows, D) if n > D else t)
    return out


def _reference(x, res, gamma, beta):
    v = x.double() + res.double() if res is not None else x.double()
    mu = v.mean(-1, keepdim=True)
    rs = ((v - mu).square().mean(-1, keepdim=True) + 1e-5).rsqrt()
    return (v - mu) * rs * gamma.double() + beta.double(), mu[:, 0], rs[:, 0]


# bf16: one rounding, 2^-9 relative at most in each element; fp32: a few roundings of 2^-24 around values of size 1
def _close(got, want, dtype):
    return ((got.double() - want).norm() / want.norm()).item() < (2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -20)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("residual", [False, True])
@pytest.mark.parametrize("rows,D", [(8191, 264), (8192, 8), (8192, 264), (8193, 512), (20001, 40), (60000, 384), (70000, 256)])
def test_rows_around_the_switch(dtype, residual, rows, D):
    from cme213_final_project_b200 import ops
    x, res, gamma, beta = _inputs(rows, D, dtype, 1)
    y, mean, rstd, summed = ops.layernorm_fwd(x, gamma, beta, residual=res if residual else None, save_sum=residual)
    want, mu, rs = _reference(x, res if residual else None, gamma, beta)
    assert _close(y, want, dtype) and _close(rstd, rs, torch.float32)
    assert ((mean.double() - mu).abs() <= 2.0 ** -18).all()
    assert not residual or torch.equal(summed, (x.float() + res.float()).to(dtype))
    # the same rows in a call small enough for the other kernel: the same bits
    for i in (0, rows - 300):
        part = ops.layernorm_fwd(x[i:i + 300].contiguous(), gamma, beta, residual=res[i:i + 300].contiguous() if residual else None)
        assert torch.equal(part[0], y[i:i + 300]) and torch.equal(part[1], mean[i:i + 300]) and torch.equal(part[2], rstd[i:i + 300])


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("rows,D", [(77, 256), (9000, 64)])
def test_operands_off_a_vector_boundary(dtype, rows, D):
    """Contiguous tensors that begin one element into a buffer: forward and backward."""
    from cme213_final_project_b200 import ops
    x, res, gamma, beta = _inputs(rows, D, dtype, 2, offset=1)
    assert x.data_ptr() % 16 and gamma.data_ptr() % 16
    y, mean, rstd, _ = ops.layernorm_fwd(x, gamma, beta, residual=res)
    want, mu, rs = _reference(x, res, gamma, beta)
    assert _close(y, want, dtype) and _close(rstd, rs, torch.float32)
    dx, dg, db = ops.layernorm_bwd(y, x, gamma, mean, rstd, dres=res)
    a = [t.clone() for t in (y, x, gamma, res)]
    want_dx, want_dg, want_db = ops.layernorm_bwd(a[0], a[1], a[2], mean, rstd, dres=a[3])
    assert _close(dx, want_dx.double(), dtype) and _close(dg, want_dg.double(), dtype) and _close(db, want_db.double(), dtype)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("rows,D", [(300, 64), (300, 520), (300, 768), (8193, 768), (20001, 384)])
def test_order_of_a_row_sum(dtype, rows, D):
    """The mean bit for bit: a lane adds the elements of its 16-byte vectors (lane, lane + 32, ...) one after the other, then the
    32 lanes are added in pairs at distances 16, 8, 4, 2, 1.  A whole model's later bits hang on this order."""
    from cme213_final_project_b200 import ops
    if D % (16 // dtype.itemsize) or D > 32 * 4 * (16 // dtype.itemsize):
        pytest.skip("rows that the vector kernels do not take")
    x, _, gamma, beta = _inputs(rows, D, dtype, 3)
    _, mean, _, _ = ops.layernorm_fwd(x, gamma, beta)
    w = 16 // dtype.itemsize
    n = -(-D // (32 * w))
    v = torch.zeros(rows, n * 32 * w, device="cuda")
    v[:, :D] = x.float()                                    # (adding zeros changes nothing)
    v = v.view(rows, n, 32, w)
    lanes = torch.zeros(rows, 32, device="cuda")
    for i in range(n):
        for j in range(w):
            lanes = lanes + v[:, i, :, j]
    at = torch.arange(32, device="cuda")
    for distance in (16, 8, 4, 2, 1):
        lanes = lanes + lanes[:, at ^ distance]
    assert torch.equal(mean, lanes[:, 0] / torch.full_like(mean, D))       # (by a number, torch multiplies by its reciprocal)
