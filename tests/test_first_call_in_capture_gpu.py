"""Operators that need no state on the device may be captured into a graph by the first call of a process."""
import os
import subprocess
import sys

import pytest
import torch

pytestmark = pytest.mark.gpu

PROGRAM = """
import torch
from cme213_final_project_b200 import ops
g = torch.Generator(device="cuda").manual_seed(1)
x, res, dy = (torch.randn(300, 256, generator=g, device="cuda").to(torch.bfloat16) for _ in range(3))
gamma, beta = (torch.randn(256, generator=g, device="cuda").to(torch.bfloat16) for _ in range(2))
tokens = torch.randint(0, 9000, (300,), generator=g, device="cuda", dtype=torch.int32)
targets = tokens % 256

def work():
    y, mean, rstd, r = ops.layernorm_fwd(x, gamma, beta, residual=res, save_sum=True)
    out = [y, mean, rstd, r, *ops.layernorm_bwd(dy, r, gamma, mean, rstd, dres=res)]
    out += [*ops.embedding_bwd(tokens, dy, 9000, 100), *ops.embedding_bwd(targets, dy, 256, 100)]
    out += [*ops.cross_entropy(y, targets), ops.grad_normsq(dy), *ops.dact_colsum(dy, x, "gelu")]
    q, k, v, d = (t.view(1200, 64) for t in (x, res, dy, y))
    o, lse = ops.attention_fwd(q, k, v, 20, 1, 60, "split", True)
    return out + [o, lse, *ops.attention_bwd(q, k, v, o, lse, d, 20, 1, 60, "split", True)]

torch.cuda.synchronize()
graph = torch.cuda.CUDAGraph()
with torch.cuda.graph(graph):
    captured = work()
graph.replay()
torch.cuda.synchronize()
eager = work()
assert all(torch.equal(a, b) for a, b in zip(captured, eager)), [i for i, (a, b) in enumerate(zip(captured, eager)) if not torch.equal(a, b)]
print("the same")
"""


def test_first_calls_under_capture():
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", PROGRAM], cwd=root, env=dict(os.environ, PYTHONPATH=root), capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "the same" in r.stdout, r.stderr[-2000:]
