"""The compiled wrappers refuse what the Python statements before them refused, and give the same objects back."""
import numpy as np
import pytest
import torch

from cme213_final_project_b200 import ops

CALLS = {
    "cross_entropy": lambda x, i: ops.cross_entropy(x, i),
    "attention_fwd": lambda x, i: ops.attention_fwd(x, x, x, 1, 1, 8),
    "attention_bwd": lambda x, i: ops.attention_bwd(x, x, x, x, x, x, 1, 1, 8),
    "layernorm_fwd": lambda x, i: ops.layernorm_fwd(x, x[0], x[0]),
    "layernorm_bwd": lambda x, i: ops.layernorm_bwd(x, x, x[0], x[0], x[0]),
    "bias_act_residual": lambda x, i: ops.bias_act_residual(x),
    "dact_colsum": lambda x, i: ops.dact_colsum(x),
    "embedding_fwd": lambda x, i: ops.embedding_fwd(i, x, x),
    "embedding_bwd": lambda x, i: ops.embedding_bwd(i, x, 8, 8),
}


@pytest.mark.parametrize("name", CALLS)
def test_tensors_of_the_host_are_refused(name):
    with pytest.raises(ops.NativeError, match="contiguous CUDA tensors"):
        CALLS[name](torch.zeros(8, 64), torch.zeros(8, dtype=torch.int32))


def test_unknown_options_are_refused_before_anything_else():
    x = torch.zeros(8, 64)
    for call in (lambda: ops.attention_fwd(x, x, x, 1, 1, 8, backend="?"), lambda: ops.bias_act_residual(x, act="?"),
                 lambda: ops.dact_colsum(x, act="?")):
        with pytest.raises(KeyError):
            call()


@pytest.mark.gpu
@pytest.mark.parametrize("name", CALLS)
def test_strides_types_and_shapes_that_are_refused(name):
    i = torch.zeros(8, dtype=torch.int32, device="cuda")
    with pytest.raises(ops.NativeError, match="contiguous CUDA tensors"):
        CALLS[name](torch.zeros(64, 64, device="cuda")[:8, ::2], i)
    with pytest.raises(ops.NativeError, match="unsupported dtype torch.float16"):
        CALLS[name](torch.zeros(8, 64, device="cuda", dtype=torch.float16), i)


@pytest.mark.gpu
def test_objects_that_the_caller_passed_come_back():
    x = torch.randn(8, 64, device="cuda")
    i = torch.zeros(8, dtype=torch.int32, device="cuda")
    assert ops.cross_entropy(x.clone(), i)[1] is not x
    y = x.clone()
    assert ops.cross_entropy(y, i, inplace=True)[1] is y
    g, b = torch.zeros(2, 64, device="cuda").unbind(0)
    _, mean, rstd, none = ops.layernorm_fwd(x, g, b)
    assert none is None
    out = ops.layernorm_bwd(x, x, g, mean, rstd, dgamma=g, dbeta=b, accumulate=True)
    assert out[1] is g and out[2] is b
    assert ops.dact_colsum(x)[0] is None and ops.bias_act_residual(x)[1] is None
    with pytest.raises(ops.NativeError, match="status"):
        ops.embedding_bwd(i, x, 4, 3)                       # 8 tokens are not whole sequences of 3


@pytest.fixture
def poisoned():
    """Every tensor that torch allocates starts as NaN, the largest number where it holds whole ones (torch's own debugging aid)."""
    torch.use_deterministic_algorithms(True)
    assert torch.empty(1000, device="cuda").isnan().all() and (torch.empty(1000, dtype=torch.uint8, device="cuda") == 255).all()
    yield
    torch.use_deterministic_algorithms(False)


@pytest.mark.gpu
@pytest.mark.parametrize("T,HD,layout,dtype", [(64, 64, "split", torch.bfloat16), (64, 128, "flat", torch.bfloat16), (96, 64, "split", torch.bfloat16),
                                               (96, 128, "flat", torch.bfloat16), (64, 128, "split", torch.bfloat16), (64, 64, "flat", torch.float32)])
def test_each_attention_path_gets_its_scratch(poisoned, T, HD, layout, dtype):
    """Every path of the dispatch and every way to complete dQ, with results and scratch in memory full of NaN: what a kernel reads
    it, or the wrapper, has written."""
    B, H = 2, 4
    g = torch.Generator(device="cuda").manual_seed(1)
    q, k, v, do = (torch.randn(B * T, H * HD, generator=g, device="cuda").to(dtype) for _ in range(4))
    want = ops.attention_fwd(q, k, v, B, H, T, layout, True, backend="simt")
    want_grads = ops.attention_bwd(q, k, v, *want, do, B, H, T, layout, True, backend="simt")
    for mode in (0, 1, 2):
        out, lse = ops.attention_fwd(q, k, v, B, H, T, layout, True)
        grads = ops.attention_bwd(q, k, v, out, lse, do, B, H, T, layout, True, dq_mode=mode)
        # bf16: P, dS and the results rounded to 8 bits on either side
        tol = 2.0 ** -6 if dtype == torch.bfloat16 else 1e-5
        for a, b in zip((out, lse) + tuple(grads), want + tuple(want_grads)):
            assert ((a.float() - b.float()).norm() / b.float().norm()).item() < tol
    scratch = torch.empty(q.numel(), device="cuda"), torch.empty(B * H * ((T + 127) // 128), dtype=torch.int32, device="cuda")
    grads = ops.attention_bwd(q, k, v, out, lse, do, B, H, T, layout, True, scratch=scratch)
    assert all(t.isfinite().all() for t in grads)           # (mode 0 clears the accumulator that it is given)


@pytest.mark.gpu
@pytest.mark.parametrize("yes,no", [(np.bool_(True), np.bool_(False)), (1.0, 0.0), (np.int64(1), 0)])
def test_flags_are_what_counts_as_true(yes, no):
    g = torch.Generator(device="cuda").manual_seed(2)
    q, k, v, do = (torch.randn(40, 64, generator=g, device="cuda").to(torch.bfloat16) for _ in range(4))
    for flag, plain in ((yes, True), (no, False)):
        out, lse = ops.attention_fwd(q, k, v, 1, 1, 40, causal=flag)
        want, want_lse = ops.attention_fwd(q, k, v, 1, 1, 40, causal=plain)
        assert torch.equal(out, want) and torch.equal(lse, want_lse)
        for a, b in zip(ops.attention_bwd(q, k, v, out, lse, do, 1, 1, 40, causal=flag),
                        ops.attention_bwd(q, k, v, out, lse, do, 1, 1, 40, causal=plain)):
            assert torch.equal(a, b)
        sums = [torch.ones(64, device="cuda", dtype=torch.bfloat16) for _ in range(2)]
        ops.dact_colsum(do, dbias=sums[0], accumulate=flag)
        ops.dact_colsum(do, dbias=sums[1], accumulate=plain)
        assert torch.equal(*sums)
        assert (ops.bias_act_residual(q, save_pre=flag)[1] is None) == (not plain)
