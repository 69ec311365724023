"""The CUDA-core attention backward at the edges of its forms: one block for a head (up to 64 tokens) and the split form beyond,
every padded head width, rows of whole 16-byte words and others; against float64 PyTorch."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T", [1, 31, 64, 65, 128, 130])
@pytest.mark.parametrize("HD", [5, 32, 48, 64, 70, 96, 128])
@pytest.mark.parametrize("dtype,causal", [(torch.float32, False), (torch.float32, True), (torch.bfloat16, True)])
def test_gradients(T, HD, dtype, causal):
    from cme213_final_project_b200 import ops
    B, H = 2, 3
    g = torch.Generator(device="cuda").manual_seed(T * 1000 + HD)
    q, k, v, do = (torch.randn(B * T, H * HD, generator=g, device="cuda").to(dtype) for _ in range(4))
    out, lse = ops.attention_fwd(q, k, v, B, H, T, "split", causal, backend="simt")
    got = ops.attention_bwd(q, k, v, out, lse, do, B, H, T, "split", causal, backend="simt")
    leaves = [t.double().view(B, T, H, HD).transpose(1, 2).requires_grad_(True) for t in (q, k, v)]
    s = leaves[0] @ leaves[1].transpose(-1, -2) / HD ** 0.5
    if causal:
        s = s.masked_fill(torch.ones(T, T, dtype=torch.bool, device="cuda").triu(1), float("-inf"))
    # the kernel's delta comes from the stored output: the reference's does too
    p = torch.softmax(s, -1)
    d_o, o = (t.double().view(B, T, H, HD).transpose(1, 2) for t in (do, out))
    dp = d_o @ leaves[2].transpose(-1, -2)
    ds = (p * (dp - (d_o * o).sum(-1, keepdim=True))).detach() / HD ** 0.5
    want = [ds @ leaves[1], ds.transpose(-1, -2) @ leaves[0], p.transpose(-1, -2) @ d_o]
    # three chained sums of at most T or HD terms in fp32, relative to the size of what enters; bf16 results are rounded once more
    bound = 3 * (T + HD) * 2.0 ** -24 + (2.0 ** -8 if dtype == torch.bfloat16 else 0.0)
    for name, a, b, size in zip("qkv", got, want, (d_o.norm(), d_o.norm(), d_o.norm())):
        b = b.detach().transpose(1, 2).reshape(B * T, H * HD)
        assert torch.isfinite(a).all()
        assert (a.double() - b).norm() <= bound * max(b.norm(), size), name
