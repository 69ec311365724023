"""Three products into one bf16 result, rounded after each, as one launch: the bits of three products that accumulate."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N,K,one_launch", [(2048, 128, 128, True), (64, 64, 64, True), (200, 72, 136, True), (4096, 512, 512, True),
                                              (130, 8, 8, True), (20000, 256, 64, None), (16384, 768, 768, None), (96, 65, 64, False)])
@pytest.mark.parametrize("a_trans,b_trans", [(0, 1), (0, 0), (1, 0)])
def test_same_bits_as_three_products(M, N, K, one_launch, a_trans, b_trans):
    from cme213_final_project_b200 import ops
    if N % 8 and not b_trans or (a_trans and M % 8):
        pytest.skip("an operand's rows are not 16-byte addressable")
    g = torch.Generator(device="cuda").manual_seed(1)
    a = torch.randn((3, K, M) if a_trans else (3, M, K), generator=g, device="cuda").to(torch.bfloat16)
    b = torch.randn((3, N, K) if b_trans else (3, K, N), generator=g, device="cuda").to(torch.bfloat16)
    want = torch.empty(M, N, dtype=torch.bfloat16, device="cuda")
    for i in range(3):        # no splits: their sums have another order
        ops.gemm(a[i], b[i], a_trans=bool(a_trans), b_trans=bool(b_trans), out=want, accumulate=i > 0, force_splits=1)
    out = torch.empty(M, N, dtype=torch.bfloat16, device="cuda")
    d = ops.CmeGemm(M, N, K, 3, a.data_ptr(), a.shape[2], M * K, a_trans, b.data_ptr(), b.shape[2], N * K, b_trans,
                    out.data_ptr(), N, 0, 1, 1)
    lib = ops.lib()
    if one_launch is not None:
        assert bool(lib.cme_gemm_sum3_planned(ctypes.byref(d))) == one_launch
    assert lib.cme_gemm_sum3(ctypes.byref(d), 0, ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
    torch.cuda.synchronize()
    assert ops.gemm_check_status() == 0
    assert torch.equal(out, want)


@pytest.mark.parametrize("M,N,K", [(256, 192, 512), (200, 72, 1032)])
@pytest.mark.parametrize("kind,splits,allow_tf32", [("bf16", 4, 0), ("bf16", 1, 0), ("fp32", 0, 0), ("fp32", 0, 2), ("fp32", 3, 2)])
@pytest.mark.parametrize("accumulate", [False, True])
def test_products_that_go_one_by_one(M, N, K, kind, splits, allow_tf32, accumulate):
    """What one launch does not make -- split reductions, fp32 storage exact and as tf32, a sum on top of C -- is made by three."""
    from cme213_final_project_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(2)
    dt = torch.bfloat16 if kind == "bf16" else torch.float32
    a, b, c = (torch.randn(s, generator=g, device="cuda").to(dt) for s in ((3, M, K), (3, N, K), (M, N)))
    kw = {"b_trans": True, "force_splits": splits, "allow_tf32": allow_tf32}
    want, out = c.clone(), c.clone()
    for i in range(3):
        ops.gemm(a[i], b[i], out=want, accumulate=accumulate or i > 0, **kw)
    ws = torch.empty(16 << 20, device="cuda")
    d = ops.CmeGemm(M, N, K, 3, a.data_ptr(), K, M * K, 0, b.data_ptr(), K, N * K, 1, out.data_ptr(), N, 0, ops._dt(out), ops._dt(a))
    d.accumulate, d.force_splits, d.allow_tf32, d.workspace, d.workspace_bytes = int(accumulate), splits, allow_tf32, ws.data_ptr(), 64 << 20
    assert not ops.lib().cme_gemm_sum3_planned(ctypes.byref(d)) or (kind, splits, accumulate) == ("bf16", 1, False)
    assert ops.lib().cme_gemm_sum3(ctypes.byref(d), 0, ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
    torch.cuda.synchronize()
    assert ops.gemm_check_status() == 0
    assert torch.equal(out, want)
