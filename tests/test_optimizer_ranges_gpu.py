"""The optimizer over many ranges without weight decay: in a small arena each thread starts deep in the list, in a large one
it walks on from there."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,count,length", [(40_000, 150, 64), (40_000, 1, 1), (4096, 512, 3), (4096, 513, 3), (4096, 600, 3), (6_000_002, 150, 3072), (6_000_002, 3, 5)])
def test_many_ranges(n, count, length):
    from cme213_final_project_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(3)
    master, m, grads = (torch.randn(n, generator=g, device="cuda") * s for s in (0.02, 1e-4, 1e-3))
    v = torch.randn(n, generator=g, device="cuda").mul_(1e-3).square_()
    starts = torch.arange(count, device="cuda") * (n // count) + (n // count - length if count > 1 else n // 2)
    nodecay = torch.stack([starts, starts + length], 1).to(torch.int64).contiguous()
    keep = torch.ones(n, dtype=torch.float64, device="cuda")
    for a, b in nodecay.tolist():
        keep[a:b] = 0
    gd = grads.double()
    m2, v2 = 0.9 * m.double() + 0.1 * gd, 0.95 * v.double() + 0.05 * gd * gd
    per_m = 0.05 / (1 - 0.9 ** 5) / ((v2 / (1 - 0.95 ** 5)).sqrt() + 1e-8)          # the update is m2 times this
    start = master.double()
    want = start * (1 - 0.05 * 0.1 * keep) - per_m * m2
    # fp32: each factor is right to 2^-24 of its size, and m2 to 2^-24 of the size of its two terms; eight roundings in a row
    # stay below 2^-20.  A decay applied or left out wrongly is 5e-3 of the weight.
    bound = 2.0 ** -20 * (start.abs() + per_m * (0.9 * m.double().abs() + 0.1 * gd.abs()))
    ops.adam_step(master, grads, m, v, torch.full((1,), 5, dtype=torch.int32, device="cuda"), torch.full((1,), 0.05, device="cuda"),
                  beta2=0.95, weight_decay=0.1, nodecay=nodecay)
    assert ((master.double() - want).abs() <= bound).all()


@pytest.mark.parametrize("n", [1_000_000, 1_000_001, 1_000_002])
def test_moments_are_rounded_once(n):
    """Whole groups of four or not.  The sum's rounding is 2^-24 / sqrt(3) of the value's power of two, 2.4e-8 relative in the
    2-norm over the mantissas; that of the smaller term adds a little.  A second rounding of the larger term makes it 3.8e-8."""
    from cme213_final_project_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(4)
    master, m, grads = (torch.randn(n, generator=g, device="cuda") * s for s in (0.02, 1e-4, 1e-3))
    v = torch.randn(n, generator=g, device="cuda").mul_(1e-3).square_()
    b1, b2 = (torch.tensor(b, dtype=torch.float32).double().item() for b in (0.9, 0.95))
    m2, v2 = (b * x.double() + (1 - b) * y for b, x, y in ((b1, m, grads.double()), (b2, v, grads.double().square())))
    ops.adam_step(master, grads, m, v, torch.full((1,), 5, dtype=torch.int32, device="cuda"), torch.full((1,), 1e-4, device="cuda"),
                  beta2=0.95)
    assert ((v.double() - v2).norm() / v2.norm()).item() < 3.2e-8
    assert ((m.double() - m2).norm() / m2.norm()).item() < 4.5e-8           # its two terms are of one size
