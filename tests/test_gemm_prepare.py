"""What ops.gemm hands to the native call for the operands that it accepts, and which it refuses."""
import pytest
import torch

from cme213_final_project_b200 import ops


@pytest.fixture
def seen(monkeypatch):
    calls = []

    class Lib:
        @staticmethod
        def cme_gemm(desc, backend, stream):
            calls.append(desc._obj)
            return 0

    monkeypatch.setattr(ops, "lib", lambda: Lib)
    monkeypatch.setattr(ops, "_cuda", lambda *t: None)
    monkeypatch.setattr(ops, "_st", lambda: 0)
    return calls


@pytest.mark.parametrize("sa,sb,at,bt,shape,strides", [
    ((5, 7), (7, 3), 0, 0, (5, 3), (0, 0)), ((7, 5), (3, 7), 1, 1, (5, 3), (0, 0)), ((4, 5, 7), (7, 3), 0, 0, (4, 5, 3), (35, 0)),
    ((5, 7), (4, 3, 7), 0, 1, (4, 5, 3), (0, 21)), ((4, 7, 5), (4, 7, 3), 1, 0, (4, 5, 3), (35, 21)), ((1, 5, 7), (2, 7, 3), 0, 0, (2, 5, 3), (0, 21)),
    ((3, 7, 5), (1, 3, 7), 1, 1, (3, 5, 3), (35, 0)), ((1, 5, 7), (1, 7, 3), 0, 0, (1, 5, 3), (35, 21))])
def test_shapes_and_strides(seen, sa, sb, at, bt, shape, strides):
    a, b = torch.zeros(sa), torch.zeros(sb, dtype=torch.float32)
    out = ops.gemm(a, b, a_trans=at, b_trans=bt, out_dtype=torch.bfloat16)
    g = seen[0]
    assert tuple(out.shape) == shape and out.dtype == torch.bfloat16
    assert (g.M, g.N, g.K, g.batch) == (5, 3, 7, shape[0] if len(shape) == 3 else 1)
    assert (g.lda, g.ldb, g.ldc, g.strideA, g.strideB, g.strideC) == (sa[-1], sb[-1], 3, *strides, 15)
    assert (g.A, g.B, g.C) == (a.data_ptr(), b.data_ptr(), out.data_ptr()) and (g.ab_dtype, g.c_dtype) == (ops.F32, ops.BF16)


def test_optional_operands_and_choices(seen):
    a, b, r, x = (torch.zeros(8, 8) for _ in range(4))
    v, out = torch.zeros(8), torch.ones(8, 8)
    assert ops.gemm(a, b, out=out, bias=v, act="gelu", aux_out=x, residual=r, accumulate=True, aux_deriv=True, backend="tcgen05",
                    force_bn=128, force_splits=3, allow_tf32=2) is out
    ops.gemm(a, b, dact="relu", aux_in=x, allow_tf32=False)
    g, h = seen
    assert (g.bias, g.residual, g.aux_out, g.aux_in, g.act, g.dact) == (v.data_ptr(), r.data_ptr(), x.data_ptr(), None, 2, 0)
    assert (g.accumulate, g.aux_deriv, g.force_bn, g.force_splits, g.allow_tf32, g.ldres, g.ldaux) == (1, 1, 128, 3, 2, 8, 8)
    assert (h.bias, h.residual, h.aux_out, h.aux_in, h.act, h.dact, h.accumulate, h.allow_tf32) == (None, None, None, x.data_ptr(), 0, 1, 0, 0)
    assert g.workspace and g.workspace_bytes == 64 << 20 and not g.colsum and not g.colsum_slabs


def test_refusals(seen):
    a = torch.zeros(8, 8)
    with pytest.raises(ops.NativeError, match=r"gemm: inner dimensions differ \(8 vs 4\)"):
        ops.gemm(a, torch.zeros(4, 8))
    with pytest.raises(IndexError):
        ops.gemm(a, torch.zeros(8))
    with pytest.raises(KeyError):
        ops.gemm(a, a, act="?")
    with pytest.raises(ops.NativeError, match="unsupported dtype torch.float16"):
        ops.gemm(a.half(), a.half())
    assert not seen


@pytest.mark.parametrize("sa,sb", [((2, 5, 7), (3, 7, 3)), ((3, 5, 7), (2, 7, 3)), ((0, 5, 7), (2, 7, 3)), ((2, 5, 7), (0, 7, 3))])
def test_batches_that_do_not_match(seen, sa, sb):
    """A descriptor has one number of matrices: entries beyond an operand's own lie outside its memory."""
    with pytest.raises(ops.NativeError, match=f"operands of {sa[0]} and {sb[0]} matrices"):
        ops.gemm(torch.zeros(sa), torch.zeros(sb))
    assert not seen


@pytest.mark.parametrize("kw,what", [
    ({"out": torch.zeros(7, 8)}, "out has 56 of 64"), ({"bias": torch.zeros(7)}, "bias has 7 of 8"),
    ({"residual": torch.zeros(8, 7)}, "residual has 56 of 64"), ({"aux_out": torch.zeros(8)}, "aux_out has 8 of 64"),
    ({"dact": "relu", "aux_in": torch.zeros(8)}, "aux_in has 8 of 64"), ({"dact": "relu"}, "dact needs aux_in"),
    ({"bias": torch.zeros(8).bfloat16()}, "bias has to have the type of a"),
    ({"residual": torch.zeros(8, 8).bfloat16()}, "residual has to have the type of out"),
    ({"out_dtype": torch.bfloat16, "aux_out": torch.zeros(8, 8)}, "aux_out has to have the type of out"),
    ({"out": torch.zeros(8, 8).bfloat16(), "dact": "relu", "aux_in": torch.zeros(8, 8)}, "aux_in has to have the type of out"),
    ({"b": torch.zeros(8, 8).bfloat16()}, "b has to have the type of a"), ({"dbias": torch.zeros(7)}, "dbias has 7 of 8"),
    ({"dbias": torch.zeros(8).half()}, "unsupported dtype")])
def test_operands_that_the_kernels_would_leave(seen, kw, what):
    with pytest.raises(ops.NativeError, match=what):
        ops.gemm(torch.zeros(8, 8), **{"b": torch.zeros(8, 8), **kw})
    assert not seen


def test_operands_of_other_shapes(seen):
    """What holds enough elements is taken as before, whatever its shape; an auxiliary input without use is not looked at."""
    a, b = torch.zeros(2, 4, 8), torch.zeros(8, 8)
    out = torch.zeros(100)
    assert ops.gemm(a, b, out=out, bias=torch.zeros(1, 9), residual=torch.zeros(64), aux_in=torch.zeros(1)) is out
    assert ops.gemm(b, b.clone(), out_dtype=torch.bfloat16, bias=torch.zeros(8), residual=torch.zeros(8, 8).bfloat16()).shape == (8, 8)
    assert len(seen) == 2


@pytest.mark.gpu
@pytest.mark.parametrize("backend", ["tcgen05", "simt"])
@pytest.mark.parametrize("na,nb", [(1, 3), (3, 1), (3, 3)])
def test_one_matrix_is_shared(na, nb, backend):
    g = torch.Generator(device="cuda").manual_seed(1)
    a, b = (torch.randn(s, generator=g, device="cuda").to(torch.bfloat16) for s in ((na, 72, 64), (nb, 64, 40)))
    got = ops.gemm(a, b, backend=backend)
    want = torch.stack([ops.gemm(a[i % na].contiguous(), b[i % nb].contiguous(), backend=backend) for i in range(3)])
    assert torch.equal(got, want)


@pytest.mark.gpu
@pytest.mark.parametrize("backend", ["auto", "simt"])              # with column sums from the epilogue, and from a pass of their own
@pytest.mark.parametrize("out_dtype,sum_dtype", [(torch.bfloat16, torch.float32), (torch.float32, torch.bfloat16), (torch.bfloat16, torch.bfloat16)])
def test_column_sums_of_another_type(out_dtype, sum_dtype, backend):
    g = torch.Generator(device="cuda").manual_seed(1)
    a, b, x = (torch.randn(s, generator=g, device="cuda") for s in ((96, 64), (64, 40), (96, 40)))
    around = torch.full((3 * 40,), 7.0, dtype=sum_dtype, device="cuda")
    kw = {"dact": "relu", "aux_in": x.to(out_dtype)} if out_dtype == torch.bfloat16 else {}
    room = torch.full((100, 40), 9.0, dtype=out_dtype, device="cuda")           # more than the product fills
    ops.gemm(a.bfloat16(), b.bfloat16(), out=room, dbias=around[40:80], backend=backend, **kw)
    assert (room[96:] == 9).all()
    out = room[:96]
    want, size = out.double().sum(0), out.double().abs().sum(0)
    # sums of 96 in fp32 (of the epilogue's unrounded values, a bf16 result's are 2^-8 off each), rounded once
    bound = size * (96 * 2.0 ** -24 + (2.0 ** -8 if out_dtype == torch.bfloat16 else 0)) + want.abs() * (2.0 ** -8 if sum_dtype == torch.bfloat16 else 0)
    assert ((around[40:80].double() - want).abs() <= bound).all()
    assert (around[:40] == 7).all() and (around[80:] == 7).all()
