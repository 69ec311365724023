"""The attention kernels other than the flash kernel at the edges of their tiles, against float64 PyTorch."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _reference(q, k, v, do, B, H, T, layout, causal):
    def heads(t):
        t = t.double()
        if layout == "flat":
            return t.reshape(B * H, T, -1)
        return t.reshape(B, T, H, -1).transpose(1, 2).reshape(B * H, T, -1)

    def back(t):
        if layout == "split":
            t = t.reshape(B, H, T, -1).transpose(1, 2)
        return t.reshape(B * T, -1)

    leaves = [heads(t).requires_grad_(True) for t in (q, k, v)]
    s = leaves[0] @ leaves[1].transpose(1, 2) / leaves[0].shape[-1] ** 0.5
    if causal:
        s = s.masked_fill(torch.ones(T, T, dtype=torch.bool, device=s.device).triu(1), float("-inf"))
    out = torch.softmax(s, -1) @ leaves[2]
    grads = torch.autograd.grad(out, leaves, heads(do))
    return back(out.detach()), torch.logsumexp(s, -1).detach().reshape(-1), [back(g) for g in grads]


def _inputs(B, H, T, HD, dtype, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return [torch.randn(B * T, H * HD, generator=g, device="cuda").to(dtype) for _ in range(4)]


def _rel(got, want):
    return ((got.double() - want).norm() / want.norm()).item()


# bf16: P and dS are rounded to 8 bits once and so is each result (2^-8 relative at most, well below half of that in the
# 2-norm); the bound is two full roundings
BF16_REL = 2 * 2.0 ** -8


@pytest.mark.parametrize("B,H,T,HD,layout,causal", [
    (2, 4, 64, 32, "flat", False), (2, 4, 64, 128, "flat", False), (3, 2, 56, 40, "flat", True), (1, 2, 8, 8, "flat", False),
    (2, 3, 64, 64, "split", True), (2, 3, 63, 64, "split", False), (1, 2, 17, 64, "split", True), (1, 1, 1, 64, "split", True),
    (1, 4, 64, 120, "flat", True)])
def test_short_sequences_in_one_launch(B, H, T, HD, layout, causal):
    from cme213_final_project_b200 import ops
    q, k, v, do = _inputs(B, H, T, HD, torch.bfloat16, 3)
    before = ops.launch_count()
    out, lse = ops.attention_fwd(q, k, v, B, H, T, layout, causal)
    grads = ops.attention_bwd(q, k, v, out, lse, do, B, H, T, layout, causal)
    assert ops.launch_count() - before == 2
    ref, ref_lse, ref_grads = _reference(q, k, v, do, B, H, T, layout, causal)
    assert _rel(out, ref) < BF16_REL
    assert (lse.double() - ref_lse).abs().max().item() < 1e-4
    for got, want in zip(grads, ref_grads):
        # one visible key: dS = P (dP - delta) cancels to rounding noise of the bf16 output, compare with dO's size
        if T == 1:
            assert (got.double() - want).abs().max().item() < 2.0 ** -6
        else:
            assert _rel(got, want) < 2 * BF16_REL
    again = ops.attention_bwd(q, k, v, out, lse, do, B, H, T, layout, causal)
    assert all(torch.equal(a, b) for a, b in zip(grads, again))


def test_short_sequences_write_nothing_outside_their_rows():
    """A ragged fused [tokens, 3D] projection: rows beyond T and columns beyond the head stay as they were."""
    import ctypes
    from cme213_final_project_b200 import ops
    B, H, T, HD = 2, 2, 40, 64
    D = H * HD
    g = torch.Generator(device="cuda").manual_seed(5)
    qkv = torch.randn(B * T + 8, 3 * D, generator=g, device="cuda").to(torch.bfloat16)
    q, k, v = (qkv[:B * T, i * D:(i + 1) * D].contiguous() for i in range(3))
    do = torch.randn(B * T, D, generator=g, device="cuda").to(torch.bfloat16)
    want, lse_want = ops.attention_fwd(q, k, v, B, H, T, "split", True)
    grads = ops.attention_bwd(q, k, v, want, lse_want, do, B, H, T, "split", True)
    out = torch.full((B * T + 8, D), 7.0, device="cuda", dtype=torch.bfloat16)
    dqkv = torch.full_like(qkv, 7.0)
    lse, delta = torch.zeros(2, B * H * T, device="cuda")
    acc = torch.zeros(B * T * D, device="cuda")
    a = ops._attn_desc(q, B, H, T, "split", True)
    a.sb, a.st = T * 3 * D, 3 * D
    base, dbase = qkv.data_ptr(), dqkv.data_ptr()
    a.q, a.k, a.v, a.o, a.lse = base, base + 2 * D, base + 4 * D, out.data_ptr(), lse.data_ptr()
    ops._check(ops.lib().cme_attention_fwd(ctypes.byref(a), 0, ops._stream()))
    a.d_o, a.dq, a.dk, a.dv = do.data_ptr(), dbase, dbase + 2 * D, dbase + 4 * D
    a.delta, a.dq_accum = delta.data_ptr(), acc.data_ptr()
    ops._check(ops.lib().cme_attention_bwd(ctypes.byref(a), 0, ops._stream()))
    assert torch.equal(out[:B * T], want) and torch.equal(lse, lse_want)
    assert torch.equal(dqkv[:B * T], torch.cat(grads, 1))
    assert (out[B * T:] == 7).all() and (dqkv[B * T:] == 7).all()


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("B,H,T,HD,layout,causal", [
    (2, 4, 64, 128, "flat", False), (2, 2, 65, 32, "split", True), (1, 3, 130, 96, "split", False), (1, 2, 33, 100, "split", True),
    (1, 2, 70, 33, "flat", True), (1, 1, 1, 7, "split", False), (40, 4, 64, 64, "split", True)])
def test_cuda_core_kernel_at_tile_edges(dtype, B, H, T, HD, layout, causal):
    from cme213_final_project_b200 import ops
    q, k, v, do = _inputs(B, H, T, HD, dtype, 4)
    out, lse = ops.attention_fwd(q, k, v, B, H, T, layout, causal, backend="simt")
    grads = ops.attention_bwd(q, k, v, out, lse, do, B, H, T, layout, causal, backend="simt")
    ref, ref_lse, ref_grads = _reference(q, k, v, do, B, H, T, layout, causal)
    # fp32: a chain of HD + T sums, each rounded to 2^-24, in quantities of the size of the results; __expf adds 2^-21
    bound = (HD + T + 8) * 2.0 ** -24 + 2.0 ** -20 if dtype == torch.float32 else BF16_REL
    assert _rel(out, ref) < bound
    assert (lse.double() - ref_lse).abs().max().item() < 1e-4
    for got, want in zip(grads, ref_grads):
        if T == 1:
            assert (got.double() - want).abs().max().item() < (1e-4 if dtype == torch.float32 else 2.0 ** -5)
        else:
            assert _rel(got, want) < 2 * bound
