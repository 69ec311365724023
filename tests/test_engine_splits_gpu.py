"""The weight gradients of a training step have the K splits that keep the order of their sums, in either model family."""
import ctypes
import os
import re
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu

STEP = """
import torch
from cme213_final_project_b200.config import ModelConfig, OptimConfig, RunConfig
from cme213_final_project_b200.models.engine import NativeEngine
from cme213_final_project_b200.parallel.dist import DistributedContext
gpt = {gpt}
cfg = ModelConfig(mode="gpt" if gpt else "parity", vocab_size=64, seq_len=64, hidden=512, heads=8, ff=2048, layers=1, batch_size=40,
                  activation="gelu" if gpt else "relu", causal=gpt, head_layout="split" if gpt else "flat", tied_embeddings=gpt,
                  final_layernorm=gpt, init="normal")
ctx = DistributedContext().init(backend="auto", device="cuda")
model = NativeEngine(cfg, OptimConfig(lr=1e-4), RunConfig(synthetic=True), ctx, seed=1)
tokens = torch.zeros(cfg.batch_size * cfg.seq_len, dtype=torch.int32, device="cuda")
model.forward(tokens, tokens)
model.backward()
torch.cuda.synchronize()
"""


@pytest.mark.parametrize("gpt", [False, True])
def test_weight_gradients(gpt):
    from cme213_final_project_b200 import ops
    out = subprocess.run([sys.executable, "-c", STEP.format(gpt=gpt)], env={**os.environ, "CME213_GEMM_TRACE": "1"}, timeout=300,
                         cwd=Path(__file__).resolve().parents[1], capture_output=True, text=True)
    assert out.returncode == 0, out.stderr[-2000:]
    found = [tuple(map(int, m)) for m in re.findall(r"\[gemm\] M=(\d+) N=(\d+) K=(\d+) batch=(\d+) at=1 .* splits=(\d+)", out.stderr)]
    assert len(found) >= 4
    for M, N, K, batch, splits in found:
        assert splits == ops.lib().cme_gemm_kept_splits(M, N, K, batch, 1, ctypes.c_longlong(64 << 20), 148, 74), (M, N, K)
