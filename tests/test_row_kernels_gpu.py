"""Row-wise kernels at the edges of their register and shared-memory tiles, against float64 PyTorch.

bf16 results are rounded once: at most 2^-8 relative, for a single value as for the 2-norm."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DTYPES = [torch.float32, torch.bfloat16]


def _ops():
    from cme213_final_project_b200 import ops
    return ops


def _rand(shape, dtype, seed, scale=1.0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return (torch.randn(*shape, generator=g, device="cuda") * scale).to(dtype)


def _rel(got, want):
    return ((got.double() - want).norm() / want.norm().clamp_min(1e-30)).item()


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("rows,V", [(1, 1), (9, 31), (300, 64), (300, 65), (64, 128), (64, 129), (33, 512), (33, 1024),
                                    (17, 1025), (17, 2049), (5, 4095), (5, 4097)])
def test_cross_entropy_short_rows(dtype, rows, V):
    ops = _ops()
    logits = _rand((rows, V), dtype, 6, 3.0)
    if 2 < V <= 4096:
        logits[0, 0] = float("-inf")                       # a masked symbol
        logits[rows - 1, 1] = torch.finfo(dtype).min
    g = torch.Generator(device="cuda").manual_seed(7)
    targets = torch.randint(2 if V > 2 else 0, V, (rows,), generator=g, device="cuda", dtype=torch.int32)
    x = logits.double().requires_grad_(True)
    losses = -torch.log_softmax(x, -1).gather(1, targets.long()[:, None])[:, 0]
    want = torch.autograd.grad(losses.mean(), x)[0]
    for inplace in (False, True):
        src = logits.clone()
        loss, grad, per_row = ops.cross_entropy(src, targets, inplace=inplace)
        # __expf: 2^-21 relative, the sum of V of them, one rounding of the gradient
        assert (per_row.double() - losses.detach()).abs().max().item() < 2e-5
        assert abs(loss.item() - losses.mean().item()) < 2e-5
        assert (grad.double() - want).abs().max().item() < (2.0 ** -8 if dtype == torch.bfloat16 else 4e-6) / rows
        assert inplace or torch.equal(src, logits)


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("residual", [False, True])
@pytest.mark.parametrize("rows,D", [(1, 8), (7, 256), (20000, 264), (9001, 768), (5000, 1024), (4096, 512), (13, 516)])
def test_layernorm_rows_through_the_ring(dtype, residual, rows, D):
    """One row to several rounds of the persistent grid (the ring wraps), one to four vectors per lane."""
    ops = _ops()
    x, res, dy = (_rand((rows, D), dtype, s) for s in (1, 2, 3))
    gamma, beta = _rand((D,), dtype, 4, 0.1) + 1, _rand((D,), dtype, 5, 0.1)
    y, mean, rstd, summed = ops.layernorm_fwd(x, gamma, beta, residual=res if residual else None, save_sum=residual)
    xin = x.double() + res.double() if residual else x.double()
    mu = xin.mean(-1, keepdim=True)
    rs = ((xin - mu).square().mean(-1, keepdim=True) + 1e-5).rsqrt()
    tol = 2.0 ** -8 if dtype == torch.bfloat16 else 4e-6
    assert _rel(y, (xin - mu) * rs * gamma.double() + beta.double()) < tol
    assert _rel(rstd, rs[:, 0]) < (tol if D % (8 if dtype == torch.bfloat16 else 4) else 4e-6)
    src = summed if residual else x
    leaves = [src.double().requires_grad_(True), gamma.double().requires_grad_(True), beta.double().requires_grad_(True)]
    m = leaves[0].mean(-1, keepdim=True)
    r = ((leaves[0] - m).square().mean(-1, keepdim=True) + 1e-5).rsqrt()
    want = torch.autograd.grad((leaves[0] - m) * r * leaves[1] + leaves[2], leaves, dy.double())
    mean2, rstd2 = m.detach()[:, 0].float(), r.detach()[:, 0].float()
    dx, dg, db = ops.layernorm_bwd(dy, src, gamma, mean2, rstd2, dres=res if residual else None)
    assert _rel(dx, want[0] + res.double() if residual else want[0]) < tol
    assert _rel(dg, want[1]) < max(tol, 2e-5) and _rel(db, want[2]) < max(tol, 2e-5)


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("n", [1, 3, 4, 1027, 2_500_002])
def test_optimizer_tails_and_ranges(dtype, n):
    """Counts that are not whole vectors, no-decay ranges that begin and end inside a group of four."""
    ops = _ops()
    master, m = _rand((n,), torch.float32, 14, 0.02), _rand((n,), torch.float32, 15, 1e-4)
    v, grads = _rand((n,), torch.float32, 16, 1e-3).square_(), _rand((n,), dtype, 17, 1e-3)
    nd = [r for r in [[0, 1], [5, 11], [601, 1001], [n - 2, n]] if 0 <= r[0] < r[1] <= n]
    nd = [r for i, r in enumerate(nd) if i == 0 or r[0] >= nd[i - 1][1]]
    nodecay = torch.tensor(nd, dtype=torch.int64, device="cuda").reshape(-1, 2)
    normsq = ops.grad_normsq(grads)
    assert abs(normsq.item() / grads.double().square().sum().item() - 1) < 1e-5
    keep = torch.ones(n, device="cuda", dtype=torch.float64)
    for a, b in nd:
        keep[a:b] = 0
    g = grads.double() * min(1.0, 0.01 / float(normsq.sqrt()))
    m2, v2 = 0.9 * m.double() + 0.1 * g, 0.95 * v.double() + 0.05 * g * g
    want = master.double() * (1 - 3e-4 * 0.1 * keep) - 3e-4 * (m2 / (1 - 0.9 ** 5)) / ((v2 / (1 - 0.95 ** 5)).sqrt() + 1e-8)
    step, lr = torch.full((1,), 5, dtype=torch.int32, device="cuda"), torch.full((1,), 3e-4, device="cuda")
    comp = torch.empty(n, dtype=torch.bfloat16, device="cuda")
    ops.adam_step(master, grads, m, v, step, lr, compute=comp, normsq=normsq, beta2=0.95, weight_decay=0.1, clip_norm=0.01,
                  nodecay=nodecay)
    assert (master.double() - want).abs().max().item() < 1e-7
    assert _rel(m, m2) < 1e-5 and _rel(v, v2) < 1e-5
    assert torch.equal(comp, master.to(torch.bfloat16))


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("V,D,B,T,ids", [(7, 8, 2, 4, "uniform"), (65, 384, 16, 64, "uniform"), (50304, 264, 2, 512, "uniform"),
                                         (3000, 768, 4, 512, "one"), (3000, 136, 4, 512, "few"), (1, 16, 3, 40, "one"),
                                         (50304, 64, 32, 1023, "few"), (65, 64, 63, 1024, "few"), (300, 100, 4, 33, "few")])
def test_token_table_gradient_by_stripes(dtype, V, D, B, T, ids):
    """Rows without a token, rows with one, rows that many tokens share (summed by the whole block), ids outside the
    table; twice the same bits; accumulation on top of what is there."""
    ops = _ops()
    n = B * T
    g = torch.Generator(device="cuda").manual_seed(8)
    tokens = torch.randint(0, V, (n,), generator=g, device="cuda", dtype=torch.int32)
    if ids == "one":
        tokens.fill_(V - 1)
    elif ids == "few":
        tokens = tokens % min(V, 5)
        tokens[::7] = V - 1
        tokens[3], tokens[11] = -1, V                      # no row: ignored
    dout = _rand((n, D), dtype, 9)
    ok = (tokens >= 0) & (tokens < V)
    want = torch.zeros(V, D, dtype=torch.float64, device="cuda").index_add_(0, tokens[ok].long(), dout[ok].double())
    want_pos = dout.double().reshape(B, T, D).sum(0)
    dtok, dpos = ops.embedding_bwd(tokens, dout, V, T)
    again, _ = ops.embedding_bwd(tokens, dout, V, T)
    if D % 8 == 0 and (dtype == torch.bfloat16 or V * n <= 1 << 22):
        assert torch.equal(dtok, again)
        # fp32 sums of up to n terms, rounded once
        tol = 2.0 ** -8 if dtype == torch.bfloat16 else 1e-5
    else:
        tol = 3e-2 if dtype == torch.bfloat16 else 1e-5    # atomics round once per token
    assert _rel(dtok, want) < tol
    assert _rel(dpos, want_pos) < (2.0 ** -8 if dtype == torch.bfloat16 else 1e-6)
    base, base_pos = _rand((V, D), dtype, 10), _rand((T, D), dtype, 11)
    got, got_pos = base.clone(), base_pos.clone()
    ops.embedding_bwd(tokens, dout, V, T, dtok=got, dpos=got_pos, accumulate=True)
    assert _rel(got, want + base.double()) < tol
    assert _rel(got_pos, want_pos + base_pos.double()) < (2.0 ** -8 if dtype == torch.bfloat16 else 1e-6)
    untouched = torch.ones(V, dtype=torch.bool, device="cuda")
    untouched[tokens[ok].long()] = False
    assert torch.equal(got[untouched], base[untouched])


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("D,T", [(768, 100), (100, 7)])
def test_embedding_gather_rows(dtype, D, T):
    ops = _ops()
    tok, pos = _rand((500, D), dtype, 12), _rand((T, D), dtype, 13)
    tokens = torch.randint(0, 500, (3 * T,), device="cuda", dtype=torch.int32)
    tokens[0], tokens[1] = -3, 900                         # clamped to the table
    want = (tok.float()[tokens.long().clamp(0, 499)] + pos.float().repeat(3, 1)).to(dtype)
    assert torch.equal(ops.embedding_fwd(tokens, tok, pos), want)
