"""Cross-entropy of rows held in registers, at both edges of each width's range, against float64 PyTorch."""
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


@pytest.mark.parametrize("V", [512, 513, 640, 641, 768, 769, 1023, 1025, 1280, 1281, 1536, 1537, 2047, 2049, 2559, 2561, 3071, 3073, 4095])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("rows", [11, 297])        # eight warps share a row of more than 1024 up to two rows per SM, fewer beyond
def test_short_row_widths(V, dtype, rows):
    from cme213_final_project_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(V)
    x = (torch.randn(rows, V, generator=g, device="cuda") * 3).to(dtype)
    targets = torch.randint(0, V, (rows,), generator=g, device="cuda", dtype=torch.int32)
    targets[0], targets[1] = 0, V - 1
    ref, pick = x.double(), torch.arange(rows, device="cuda")
    want = torch.softmax(ref, 1)
    want[pick, targets.long()] -= 1
    _, grad, losses = ops.cross_entropy(x.clone(), targets, inplace=True)
    assert (losses.double() - (torch.logsumexp(ref, 1) - ref[pick, targets.long()])).abs().max().item() < 20 * 2.0 ** -19
    # exponential, sum and products to 2^-16; a bf16 result rounded once; the target's element is p - 1 with the error of p <= 1
    bound = want.abs() * (2.0 ** -16 + (2.0 ** -8 if dtype == torch.bfloat16 else 0.0))
    bound[pick, targets.long()] += 2.0 ** -16
    assert ((grad.double() * rows - want).abs() <= bound).all()
