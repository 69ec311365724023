"""The optimizer where the rounds per block change (multiples of 757 760 elements up to four), and where the last block and round are
not full."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("clip,ranges", [(0.0, False), (0.01, True)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("n", [4, 1023, 1024, 1029, 454_655, 454_656, 454_661, 757_760, 757_761, 1_515_520, 1_515_525, 1_818_624,
                               1_818_629, 1_820_676, 2_273_284, 3_031_040, 3_031_041, 4_000_003])
def test_every_element_is_updated_once(n, dtype, clip, ranges):
    from cme213_final_project_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(1)
    master, m, grads = (torch.randn(n, generator=g, device="cuda") * s for s in (0.02, 1e-4, 1e-3))
    v = torch.randn(n, generator=g, device="cuda").mul_(1e-3).square_()
    grads = grads.to(dtype)
    comp = torch.empty(n, device="cuda", dtype=torch.bfloat16)
    norm = grads.double().square().sum().float()[None]
    scale = min(1.0, clip / norm.sqrt().item()) if clip else 1.0
    keep = torch.ones(n, dtype=torch.float64, device="cuda")
    spans = [[n // 3, n // 3 + 1], [n // 2, n // 2 + n // 8 + 1]] if ranges else [[0, 0]]
    for a, b in spans:
        keep[a:b] = 0
    gd = grads.double() * scale
    m2, v2 = 0.9 * m.double() + 0.1 * gd, 0.95 * v.double() + 0.05 * gd * gd
    per_m = 0.05 / (1 - 0.9 ** 5) / ((v2 / (1 - 0.95 ** 5)).sqrt() + 1e-8)
    want = master.double() * (1 - 0.05 * 0.1 * keep) - per_m * m2
    # as in test_optimizer_ranges_gpu: eight fp32 roundings in a row, each of 2^-24, and as many more in the clipped scale
    bound = 2.0 ** -19 * (master.double().abs() + per_m * (0.9 * m.double().abs() + 0.1 * gd.abs()))
    ops.adam_step(master, grads, m, v, torch.full((1,), 5, dtype=torch.int32, device="cuda"), torch.full((1,), 0.05, device="cuda"),
                  compute=comp, normsq=norm if clip else None, clip_norm=clip, beta2=0.95, weight_decay=0.1,
                  nodecay=torch.tensor(spans, dtype=torch.int64, device="cuda"))
    assert ((master.double() - want).abs() <= bound).all()
    assert torch.equal(comp, master.to(torch.bfloat16))
