"""Cross-entropy of bf16 rows held in registers, at both edges of each width's range, against float64 PyTorch."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("V", [2048, 2056, 4096, 4104, 6144, 6152, 8192, 8200, 12288, 12296, 16384, 16392, 20480, 20488, 26624, 26632,
                               32768, 32776, 40960, 40968, 53248])
@pytest.mark.parametrize("inplace", [False, True])
def test_row_widths(V, inplace):
    from cme213_final_project_b200 import ops
    rows = 5
    g = torch.Generator(device="cuda").manual_seed(V)
    x = (torch.randn(rows, V, generator=g, device="cuda") * 3).to(torch.bfloat16)
    x[3] = -float("inf")
    x[3, V - 1] = 2.0
    targets = torch.tensor([0, V - 1, V // 2, V - 1, 2047], dtype=torch.int32, device="cuda")
    ref = x.double()
    lse = torch.logsumexp(ref, 1)
    pick = torch.arange(rows, device="cuda")
    want = torch.softmax(ref, 1)
    want[pick, targets.long()] -= 1
    src = x.clone()
    loss, grad, losses = ops.cross_entropy(src, targets, inplace=inplace)
    assert inplace == (grad.data_ptr() == src.data_ptr())
    # logarithm and exponentials to 2^-20 of arguments up to 20
    assert (losses.double() - (lse - ref[pick, targets.long()])).abs().max().item() < 20 * 2.0 ** -19
    assert abs(loss.item() - losses.mean().item()) < 1e-5
    # half a unit of bf16 (8 significant bits: 2^-8), before it half a unit of fp16 (2^-11; 2^-25 where an exponential is below
    # 2^-14) and 2^-16 for the exponential, the sum and the products; the target's element is p - 1 with the error of p <= 1
    err = (grad.double() * rows - want).abs()
    bound = want.abs() * (2.0 ** -8 + 2.0 ** -11 + 2.0 ** -16) + 2.0 ** -24
    bound[pick, targets.long()] += 2.0 ** -11
    assert (err <= bound).all()
