"""fp32 products with an operand stored along M or N: which of them run as tf32, and what the tf32 kernel makes of them."""
import ctypes

import pytest
import torch

from cme213_final_project_b200 import ops

F32 = torch.float32


def _native_answer(M, N, K, a_trans, b_trans, batch=1, workspace_bytes=64 << 20, allow=1):
    """What the tensor-core kernel says to a product, without a device: 2 (shape not supported), or 1 once it looks for one."""
    lib = ops.host_lib()
    if lib is None or torch.cuda.is_available():
        pytest.skip("asks the native library without a device")
    g = ops.CmeGemm(M, N, K, batch, 1 << 20, M if a_trans else K, M * K if batch > 1 else 0, a_trans,
                    1 << 21, K if b_trans else N, N * K if batch > 1 else 0, b_trans, 1 << 22, N, M * N, ops.F32, ops.F32,
                    0, 0, N, 0, 0, N, 0, 0, 0, 1 << 23 if workspace_bytes else 0, workspace_bytes, 0, 0, 0, 0, None, allow)
    return lib.cme_gemm(ctypes.byref(g), 1, None)


@pytest.mark.parametrize("M,N,K,a_trans,b_trans,batch,ws,tf32", [
    (128, 256, 32, 1, 0, 1, 64 << 20, True), (128, 256, 33, 1, 0, 1, 64 << 20, False), (128, 256, 1001, 1, 0, 1, 64 << 20, False),
    (512, 2048, 4095, 1, 0, 1, 64 << 20, False), (512, 2048, 2048, 1, 0, 1, 64 << 20, True),
    (512, 2048, 3276, 1, 0, 1, 64 << 20, True), (512, 2048, 3280, 1, 0, 1, 64 << 20, False), (512, 2048, 8192, 1, 0, 1, 64 << 20, False),
    (16384, 512, 2048, 0, 0, 1, 64 << 20, True), (16384, 2048, 4096, 0, 0, 1, 64 << 20, False), (64, 64, 64, 1, 0, 1, 0, False),
    (64, 64, 64, 0, 1, 1, 0, True), (128, 128, 128, 1, 0, 200, 64 << 20, True), (128, 128, 128, 1, 0, 300, 64 << 20, False)])
def test_which_products_are_taken(M, N, K, a_trans, b_trans, batch, ws, tf32):
    assert _native_answer(M, N, K, a_trans, b_trans, batch, ws) == (1 if tf32 else 2)
    assert _native_answer(M, N, K, a_trans, b_trans, batch, ws, allow=2) == 1
    assert _native_answer(M, N, K, a_trans, b_trans, batch, ws, allow=0) == 2


@pytest.mark.parametrize("M,N,K,pair", [(8192, 768, 2304, True), (16384, 768, 768, True), (8192, 2048, 512, True), (16384, 3072, 768, True),
                                        (2048, 512, 512, False), (1000, 384, 384, False), (128, 4096, 4096, False)])
def test_operands_along_k_use_pairs_that_fill_the_machine(M, N, K, pair):
    """Shapes on which pair tiles measured 8 to 15 % faster than single CTAs, and small ones on which they do not pay."""
    lib = ops.host_lib()
    if lib is None:
        pytest.skip("native library not built")
    out = (ctypes.c_int * 3)()
    assert lib.cme_gemm_plan_tf32(M, N, K, 0, ctypes.c_longlong(64 << 20), 148, 74, out) == 0
    assert bool(out[1]) == pair


def _rand(shape, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randn(*shape, generator=g, device="cuda")


def _rel(got, want):
    return ((got.double() - want).norm() / want.norm()).item()


@pytest.mark.gpu
@pytest.mark.parametrize("M,N,K", [(128, 256, 33), (132, 260, 1001), (64, 512, 4095), (512, 2048, 3280)])
def test_other_products_keep_all_bits_of_their_inputs(M, N, K):
    """Weight gradients over a token count that is not a multiple of four, or over operands beyond 32 MB."""
    x, dy = _rand((K, M), 1), _rand((K, N), 2)
    # a chain of at most K sums, each rounded to 2^-24; the errors of a random sum grow with its square root
    assert _rel(ops.gemm(x, dy, a_trans=True), x.double().t() @ dy.double()) < 4 * K ** 0.5 * 2.0 ** -24
    with pytest.raises(ops.NativeError):
        ops.gemm(x, dy, a_trans=True, backend="tcgen05")
    assert 2.0 ** -13 < _rel(ops.gemm(x, dy, a_trans=True, allow_tf32=2), x.double().t() @ dy.double()) < TF32_REL


# tf32 keeps 11 bits of each input (10 stored), rounded or cut: 2^-10 relative each, independent over the sum
TF32_REL = 2.0 ** -10


@pytest.mark.gpu
@pytest.mark.parametrize("a_trans,b_trans", [(True, False), (False, False), (True, True)])
@pytest.mark.parametrize("bn,splits", [(0, 0), (64, 1), (128, 2), (256, 3), (512, 1)])
@pytest.mark.parametrize("M,N,K", [(256, 264, 33), (256, 264, 36), (388, 516, 1001), (300, 192, 4095)])
def test_ragged_operands_along_m_or_n(M, N, K, bn, splits, a_trans, b_trans):
    """K that does not fill a 32-deep block, every tile width, split and accumulating, nothing written beside the result."""
    if splits > max(1, -(-K // 32) // 4):
        pytest.skip("too short to split")
    if K % 4 and (b_trans or not a_trans):
        pytest.skip("rows along K that are not whole 16-byte words")
    a, b = _rand((K, M) if a_trans else (M, K), 3), _rand((N, K) if b_trans else (K, N), 4)
    want = (a.double().t() if a_trans else a.double()) @ (b.double().t() if b_trans else b.double())
    big = torch.full((M * N + 2048,), 7.0, device="cuda")
    out = big[1024:1024 + M * N].view(M, N)
    kw = dict(a_trans=a_trans, b_trans=b_trans, backend="tcgen05", force_bn=bn, force_splits=splits, allow_tf32=2)
    ops.gemm(a, b, out=out, **kw)
    assert ops.gemm_check_status() == 0
    assert _rel(out, want) < TF32_REL
    base = _rand((M, N), 5)
    out.copy_(base)
    ops.gemm(a, b, out=out, accumulate=True, **kw)
    assert _rel(out, want + base.double()) < TF32_REL
    assert (big[:1024] == 7).all() and (big[-1024:] == 7).all()


@pytest.mark.gpu
@pytest.mark.parametrize("shared", ["none", "a", "b"])
@pytest.mark.parametrize("a_trans,b_trans", [(True, False), (False, False), (True, True)])
@pytest.mark.parametrize("M,N,K", [(136, 72, 40), (260, 256, 100)])
def test_batched_operands_along_m_or_n(M, N, K, a_trans, b_trans, shared):
    """Batches of both operands, or of one with the other shared by all."""
    batch = 3
    a, b = _rand((batch,) * (shared != "a") + ((K, M) if a_trans else (M, K)), 6), _rand((batch,) * (shared != "b") + ((N, K) if b_trans else (K, N)), 7)
    A, B = (a.transpose(-1, -2) if a_trans else a).double(), (b.transpose(-1, -2) if b_trans else b).double()
    got = ops.gemm(a, b, a_trans=a_trans, b_trans=b_trans, backend="tcgen05")
    assert ops.gemm_check_status() == 0
    assert got.shape == (batch, M, N) and _rel(got, torch.matmul(A, B)) < TF32_REL
