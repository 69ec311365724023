"""K splits of the engine's bf16 products: the order of a training step's sums stays as it was, whatever the planner learns."""
import ctypes

import pytest

from cme213_final_project_b200 import ops


@pytest.mark.parametrize("M,N,K,batch,plain,ws,splits", [
    (128, 512, 1024, 1, 1, 64 << 20, 4), (256, 256, 2560, 3, 1, 64 << 20, 10), (512, 512, 2048, 1, 1, 64 << 20, 8),
    (1600, 512, 2048, 1, 1, 64 << 20, 5), (512, 512, 3840, 3, 1, 64 << 20, 6), (2048, 512, 3584, 1, 1, 64 << 20, 4),
    (512, 512, 2048, 1, 0, 64 << 20, 1), (512, 512, 2048, 1, 1, 3 << 20, 3), (512, 128, 192, 1, 1, 64 << 20, 1),
    (2048, 128, 128, 1, 1, 64 << 20, 1), (384, 1152, 16384, 1, 1, 64 << 20, 9), (768, 2304, 16384, 1, 1, 64 << 20, 5)])
def test_splits_stay(M, N, K, batch, plain, ws, splits):
    lib = ops.host_lib()
    if lib is None:
        pytest.skip("native library not built")
    assert lib.cme_gemm_kept_splits(M, N, K, batch, plain, ctypes.c_longlong(ws), 148, 74) == splits
    # the planner takes them as they are: only the tile is its own
    out = (ctypes.c_int * 3)()
    assert lib.cme_gemm_plan(M, N, K, batch, plain, ctypes.c_longlong(ws), 148, 74, 0, splits, out) == 0
    assert out[2] == splits
