"""Flags of the wrappers may be anything that counts as a whole number, as numpy's truth values do."""
import numpy as np
import pytest
import torch

from cme213_final_project_b200 import ops


@pytest.mark.parametrize("yes,no", [(True, False), (np.bool_(True), np.bool_(False)), (np.int64(1), np.int64(0)), (1.0, 0.0)])
def test_product_flags(monkeypatch, yes, no):
    seen = []

    class Lib:
        @staticmethod
        def cme_gemm(desc, backend, stream):
            g = desc._obj
            seen.append((g.a_trans, g.b_trans, g.accumulate, g.aux_deriv, g.allow_tf32))
            return 0

    monkeypatch.setattr(ops, "lib", lambda: Lib)
    monkeypatch.setattr(ops, "_cuda", lambda *t: None)
    monkeypatch.setattr(ops, "_st", lambda: 0)
    a, b = torch.zeros(32, 16), torch.zeros(24, 32)
    ops.gemm(a, b, a_trans=yes, b_trans=yes, out=torch.zeros(16, 24), accumulate=yes, aux_deriv=yes, allow_tf32=no)
    ops.gemm(a.t(), b.t(), a_trans=no, b_trans=no, allow_tf32=yes)
    assert seen == [(1, 1, 1, 1, 0), (0, 0, 0, 0, 1)]


@pytest.mark.parametrize("causal,want", [(np.bool_(True), 1), (np.bool_(False), 0), (1.0, 1), (0, 0)])
def test_attention_flag(monkeypatch, causal, want):
    seen = []

    class Native:
        @staticmethod
        def attention_fwd(*args):
            seen.append(args[3:])
            return None, None

        @staticmethod
        def attention_bwd(*args):
            seen.append(args[6:])
            return None, None, None

    monkeypatch.setattr(ops, "_native", lambda: Native)
    x = torch.zeros(8, 64)
    ops.attention_fwd(x, x, x, 1, 1, 8, "split", causal)
    ops.attention_bwd(x, x, x, x, x, x, 1, 1, 8, "flat", causal, ordered_dq=True)
    # B, H, T, flat, causal, backend and, backward, the way dQ is completed and the caller's scratch
    assert seen == [(1, 1, 8, False, want, 0), (1, 1, 8, True, want, 0, 1, None, None)]
    assert all(type(args[4]) is int for args in seen)
