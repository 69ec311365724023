"""The kernel that adds up partial column sums, at the row counts and widths where the number of its row groups changes."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("rows,cols", [(1, 1), (1, 300), (3, 33), (16, 257), (17, 257), (31, 65), (96, 100), (97, 100), (130, 31), (2049, 64),
                                       (1, 50304), (200, 32768), (200, 32769), (513, 32800), (128, 40), (513, 40)])
def test_partial_rows_are_added_up(dtype, rows, cols):
    from cme213_final_project_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(1)
    part = torch.randn(rows, cols, generator=g, device="cuda")
    base = torch.randn(cols, generator=g, device="cuda").to(dtype)
    want = part.double().sum(0)
    for accumulate in (0, 1):
        out = torch.full((cols + 64,), 7.0, device="cuda", dtype=dtype)
        out[:cols] = base
        ops._check(ops.lib().cme_colsum_slabs_finalize(ops._dt(out), ops._p(part), rows, cols, ops._p(out), accumulate, ops._stream()))
        ref = want + base.double() * accumulate
        # a chain of `rows` fp32 sums of terms up to 5, the result rounded once
        tol = ref.abs() * (2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -23) + (rows + 1) * 2.0 ** -24 * part.double().abs().sum(0)
        assert ((out[:cols].double() - ref).abs() <= tol + 1e-7).all()
        assert (out[cols:] == 7).all()
