"""The launches that a step was left with: the update that adds up the norm's partial sums itself, and the staged batch."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("n,skew", [(1, 0), (7, 1), (1024, 0), (5003, 0), (300001, 1), (2000003, 0)])
def test_update_from_partial_norms_equals_the_one_from_the_norm(n, skew, dtype):
    from cme213_final_project_b200 import ops
    lib = ops.lib()
    gen = torch.Generator(device="cuda").manual_seed(n)
    base = torch.randn(n + skew, generator=gen, device="cuda").to(dtype)
    grads = base[skew:]                                     # skew: not 16-byte aligned, the scalar kernels
    runs = []
    for fused in (False, True):
        master, m, v = torch.ones(n, device="cuda"), torch.zeros(n, device="cuda"), torch.zeros(n, device="cuda")
        step, lr = torch.full((1,), 4, dtype=torch.int32, device="cuda"), torch.full((1,), 1e-2, device="cuda")
        partial, norm = torch.empty(1024, device="cuda"), torch.zeros(1, device="cuda")
        if fused:
            ops._check(lib.cme_grad_normsq_partials(ops._dt(grads), ops._p(grads), ctypes.c_longlong(n), ops._p(partial), ops._p(step),
                                                    ops._stream()))
            ops._check(lib.cme_adam_partials(
                ops._dt(grads), ops._p(master), None, ops._p(grads), ops._p(m), ops._p(v), ctypes.c_longlong(n), ops._p(step), ops._p(lr),
                ops._p(partial), *map(ctypes.c_float, (0.9, 0.999, 1e-8, 0.0, 1.0, 0.5)), None, 0, 1024, ops._p(norm), ops._stream()))
        else:
            ops._check(lib.cme_step_inc(ops._p(step), ops._stream()))
            norm = ops.grad_normsq(grads)
            ops.adam_step(master, grads, m, v, step, lr, normsq=norm, clip_norm=0.5)
        assert step.item() == 5
        runs.append((master, m, v, norm))
    assert abs(runs[1][3].item() / grads.double().square().sum().item() - 1) < 1e-5
    for a, b in zip(*runs):                                 # the totals are added in another order: a few units of 2^-24
        assert ((a - b).abs() <= 1e-6 * b.abs() + 1e-9).all()


@pytest.mark.parametrize("n", [1, 255, 4096, 400001])
def test_staged_batch(n):
    from cme213_final_project_b200 import ops
    x, y = torch.randint(0, 1 << 30, (2, n), dtype=torch.int32, device="cuda").unbind(0)
    dx, dy = torch.full((2, n + 1), 7, dtype=torch.int32, device="cuda").unbind(0)
    ops._check(ops.lib().cme_copy_pair_i32(ops._a(dx), ops._a(x), ops._a(dy), ops._a(y), n, ops._st()))
    assert torch.equal(dx[:n], x) and torch.equal(dy[:n], y) and dx[n] == 7 and dy[n] == 7
