"""Products whose reduction is split over CTAs with partial rows that are not whole 16-byte words, against float64."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu


def _mk(shape, seed, dtype):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randn(*shape, generator=g, device="cuda").to(dtype)


@pytest.mark.parametrize("out_dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("M,N,K,splits", [(128, 65, 2048, 8), (65, 66, 1024, 3), (256, 67, 4096, 2), (130, 264, 2048, 4)])
def test_split_reduction_with_odd_rows(M, N, K, splits, out_dtype):
    """Weight gradient of an output head: both operands stored along the reduction, the rows of the result not whole words
    (padded partial rows), with and without adding to what is there."""
    from cme213_final_project_b200 import ops
    pitch = (N + 7) // 8 * 8
    a, b = _mk((K, (M + 7) // 8 * 8), 4, torch.bfloat16), _mk((K, pitch), 5, torch.bfloat16)
    ws = ops.workspace()
    want = a[:, :M].double().t() @ b[:, :N].double()
    for accumulate in (False, True):
        buf = _mk((M * N + 64,), 6, out_dtype)
        before = buf.clone()
        g = ops.CmeGemm()
        g.M, g.N, g.K, g.batch = M, N, K, 1
        g.A, g.lda, g.a_trans, g.B, g.ldb = a.data_ptr(), a.shape[1], 1, b.data_ptr(), pitch
        g.C, g.ldc, g.c_dtype, g.ab_dtype = buf.data_ptr(), N, ops._dt(buf), ops.BF16
        g.accumulate, g.force_splits = int(accumulate), splits
        g.workspace, g.workspace_bytes = ws.data_ptr(), ws.numel() * 4
        ops._check(ops.lib().cme_gemm(ctypes.byref(g), 1, ops._stream()))
        ref = want + before[:M * N].view(M, N).double() if accumulate else want
        got = buf[:M * N].view(M, N).double()
        assert ((got - ref).norm() / ref.norm()).item() < (2.0 ** -8 if out_dtype == torch.bfloat16 else 1e-5)
        assert torch.equal(buf[M * N:], before[M * N:])
