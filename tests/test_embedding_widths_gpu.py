"""Embedding gather and position-table gradient at the row widths and batch sizes where the work is divided differently."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("D", [4, 8, 12, 16, 24, 40, 64, 72, 128, 136, 256, 264, 1032])
def test_gather_of_every_width(dtype, D):
    from cme213_final_project_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(2)
    V, T, B = 91, 37, 5
    tok, pos = (torch.randn(n, D, generator=g, device="cuda").to(dtype) for n in (V, T))
    tokens = torch.randint(0, V, (B * T,), generator=g, device="cuda", dtype=torch.int32)
    big = torch.full((B * T + 64, D), 7.0, device="cuda", dtype=dtype)
    ops._check(ops.lib().cme_embedding_fwd(ops._dt(tok), ops._p(tokens), ops._p(tok), ops._p(pos), ops._p(big), B * T, T, D, V, ops._stream()))
    assert torch.equal(big[:B * T], (tok.float()[tokens.long()] + pos.float().repeat(B, 1)).to(dtype))
    assert (big[B * T:] == 7).all()


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("B", [1, 2, 8, 16, 17, 33])
@pytest.mark.parametrize("T,D", [(1, 8), (33, 72), (64, 256), (1024, 768), (301, 1024), (592, 1024)])
def test_position_gradient_of_few_and_many_rows(dtype, B, T, D):
    from cme213_final_project_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(3)
    dout, base = torch.randn(B * T, D, generator=g, device="cuda").to(dtype), torch.randn(T, D, generator=g, device="cuda").to(dtype)
    tokens = torch.zeros(B * T, dtype=torch.int32, device="cuda")
    want = dout.double().reshape(B, T, D).sum(0)
    for accumulate in (0, 1):
        out = torch.full((T + 8, D), 7.0, device="cuda", dtype=dtype)
        out[:T] = base
        ops._check(ops.lib().cme_embedding_bwd(ops._dt(dout), ops._p(tokens), ops._p(dout), None, ops._p(out), B * T, T, D, 1, accumulate,
                                               ops._stream()))
        ref = want + base.double() * accumulate
        # B + 1 fp32 sums of terms up to 5, the result rounded once
        tol = ref.abs() * (2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -24) + (B + 1) ** 2 * 5 * 2.0 ** -24
        assert ((out[:T].double() - ref).abs() <= tol).all()
        assert (out[T:] == 7).all()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("V,D,n", [(50304, 264, 18000), (50304, 264, 24001), (20000, 768, 33000), (9000, 136, 39001), (9000, 136, 40500), (70, 1032, 30001)])
def test_token_gradient_of_long_lists(dtype, V, D, n):
    """Lists around the lengths at which one block per SM fits instead of two, and none."""
    from cme213_final_project_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(4)
    tokens = (torch.rand(n, generator=g, device="cuda").pow(3) * V).to(torch.int32)          # crowded towards the first ids
    dout = torch.randn(n, D, generator=g, device="cuda").to(dtype)
    out = torch.full((V + 1, D), 7.0, device="cuda", dtype=dtype)
    ops._check(ops.lib().cme_embedding_bwd(ops._dt(dout), ops._p(tokens), ops._p(dout), ops._p(out), None, n, 1, D, V, 0, ops._stream()))
    want = torch.zeros(V, D, dtype=torch.float64, device="cuda").index_add_(0, tokens.long(), dout.double())
    # fp32 sums rounded once; the atomics round 16-bit sums once per token, some thousand of them in the first rows
    tol = 1e-5 if dtype == torch.float32 else 2.0 ** -8 if n < 39500 else 0.1
    assert ((out[:V].double() - want).norm() / want.norm()).item() < tol
    assert (out[V] == 7).all()
