"""The 256 x 192 tile of the CTA pair against the 256 x 256 one: an output element is the same sum in the same order whatever the
tile's width, so every epilogue has to give the same bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _mk(shape, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randn(*shape, generator=g, device="cuda").to(torch.bfloat16)


def _both(a, b, **kw):
    from cme213_final_project_b200 import ops
    new = {k: v() if callable(v) else v for k, v in kw.items()}, {k: v() if callable(v) else v for k, v in kw.items()}
    out = [ops.gemm(a, b, backend="tcgen05", force_bn=bn, **n) for bn, n in zip((384, 512), new)]
    torch.cuda.synchronize()
    assert ops.gemm_check_status() == 0
    return out, new


@pytest.mark.parametrize("a_trans,b_trans", [(False, False), (False, True), (True, False), (True, True)])
@pytest.mark.parametrize("M,N,K", [(256, 192, 64), (257, 96, 72), (1000, 200, 328), (640, 384, 1536), (2304, 1160, 192), (24, 8, 64),
                                   (40000, 576, 64)])
def test_layouts_and_edges(M, N, K, a_trans, b_trans):
    a, b = _mk(((K, (M + 7) // 8 * 8) if a_trans else (M, K)), 1), _mk((N, K) if b_trans else (K, N), 2)
    (got, want), _ = _both(a, b, a_trans=a_trans, b_trans=b_trans)
    assert torch.equal(got, want)
    ref = (a.float().t() if a_trans else a.float()) @ (b.float().t() if b_trans else b.float())
    assert (got.float() - ref).abs().max().item() <= 2 ** -8 * ref.abs().max().item()       # half a unit of bf16, and its sums


@pytest.mark.parametrize("M,N,K", [(1024, 1536, 192), (1000, 520, 328), (40000, 384, 64)])
def test_epilogues(M, N, K):
    a, b, bias, res = _mk((M, K), 3), _mk((K, N), 4), _mk((N,), 5), _mk((M, N), 6)
    aux = lambda: torch.empty(M, N, dtype=torch.bfloat16, device="cuda")      # noqa: E731
    sums = lambda: torch.empty(N, dtype=torch.bfloat16, device="cuda")        # noqa: E731
    for kw in ({"bias": bias}, {"bias": bias, "act": "relu"}, {"residual": res}, {"bias": bias, "residual": res},
               {"bias": bias, "act": "gelu", "aux_out": aux}, {"bias": bias, "act": "gelu", "aux_out": aux, "aux_deriv": True},
               {"dact": "gelu", "aux_in": res}, {"dact": "relu", "aux_in": res}, {"dact": "gelu", "aux_in": res, "aux_deriv": True},
               {"dact": "gelu", "aux_in": res, "aux_deriv": True, "dbias": sums}, {"dact": "relu", "aux_in": res, "dbias": sums},
               {"out": res.clone, "accumulate": True}, {"out_dtype": torch.float32}):
        (got, want), (x, y) = _both(a, b, **kw)
        assert torch.equal(got, want), kw.keys()
        for k in ("aux_out", "dbias"):
            assert k not in x or torch.equal(x[k], y[k]), kw.keys()


@pytest.mark.parametrize("splits", [2, 5])
def test_splits(splits):
    a, b = _mk((2048, 512), 7), _mk((2048, 400), 8)
    (got, want), _ = _both(a, b, a_trans=True, force_splits=splits)
    assert torch.equal(got, want)


@pytest.mark.parametrize("sa,sb", [((3, 520, 72), (3, 72, 200)), ((3, 520, 72), (72, 200)), ((520, 72), (3, 72, 200))])
def test_batches(sa, sb):
    """Several matrices, and one operand for all of them; plain, and with epilogue operands that arrive by TMA."""
    a, b, x = _mk(sa, 9), _mk(sb, 10), _mk((3, 520, 200), 11)
    for kw in ({}, {"residual": x}, {"dact": "gelu", "aux_in": x}, {"dact": "relu", "aux_in": x}, {"out": x.clone, "accumulate": True},
               {"act": "gelu", "aux_out": lambda: torch.empty_like(x)}, {"out_dtype": torch.float32}):
        (got, want), (u, v) = _both(a, b, **kw)
        assert torch.equal(got, want), kw.keys()
        assert "aux_out" not in u or torch.equal(u["aux_out"], v["aux_out"])
        if not kw:
            ref = a.float() @ b.float()
            assert (got.float() - ref).abs().max().item() <= 2 ** -8 * ref.abs().max().item()
