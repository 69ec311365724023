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
