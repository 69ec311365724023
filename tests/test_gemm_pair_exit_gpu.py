"""CTA pairs at their end: the accumulators' last hand-backs reach the leader's barriers before it exits, launch after launch, with
none, one and several tiles before them; the bits are those of single CTAs."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("force_bn", [384, 512])
@pytest.mark.parametrize("M", [256, 300, 256 * 74, 256 * 75, 256 * 160])          # 1, 2, 74, 75 and 160 tiles for 74 pairs at most
@pytest.mark.parametrize("kind", ["no TMA stores", "fp32", "bias", "plain", "gelu"])
def test_back_to_back_launches(force_bn, M, kind):
    from cme213_final_project_b200 import ops
    N, K = (181 if kind == "no TMA stores" else 184), 64
    g = torch.Generator(device="cuda").manual_seed(M)
    a, b = (torch.randn(s, generator=g, device="cuda").to(torch.bfloat16) for s in ((M, K), (N, K)))
    bias, aux = torch.randn(N, generator=g, device="cuda").to(torch.bfloat16), torch.empty(M, N, dtype=torch.bfloat16, device="cuda")
    kw = {"no TMA stores": {"bias": bias, "act": "relu"}, "fp32": {"out_dtype": torch.float32}, "bias": {"bias": bias}, "plain": {},
          "gelu": {"bias": bias, "act": "gelu", "aux_out": aux, "aux_deriv": True}}[kind]
    want = ops.gemm(a, b, b_trans=True, backend="tcgen05", force_bn=128, **kw)
    got = [torch.zeros_like(want) for _ in range(24)]
    for out in got:
        ops.gemm(a, b, b_trans=True, backend="tcgen05", force_bn=force_bn, out=out, **kw)
    torch.cuda.synchronize()
    assert ops.gemm_check_status() == 0
    assert all(torch.equal(out, want) for out in got)
