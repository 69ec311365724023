"""Which of the flash attention's kernels a call takes, by how its 128-row tiles fill 148 SMs (True: 128 x 128 blocks)."""
import pytest

from cme213_final_project_b200 import ops


@pytest.mark.parametrize("heads,T,causal,forward,backward", [
    (1, 1, False, True, True), (24, 582, False, True, True), (16, 1024, True, True, True),      # fewer tiles than SMs
    (148, 128, True, True, True), (149, 128, True, True, False),
    (74, 192, True, True, True), (75, 192, True, False, False), (148, 129, False, False, False),
    (148, 256, True, True, False), (149, 256, True, False, False),                              # two tiles an SM
    (24, 1024, True, True, True), (24, 1024, False, True, False), (48, 449, True, True, True), (48, 448, True, True, False),
    (48, 1024, True, True, False), (48, 1024, False, True, True), (64, 582, False, True, True),   # three
    (64, 582, True, True, False), (80, 582, True, False, False), (64, 768, True, True, False), (192, 256, False, False, True),
    (192, 192, False, False, False), (64, 1024, False, True, False), (64, 1024, True, False, False),
    (96, 1024, False, True, False), (80, 1024, False, True, True), (160, 512, False, False, False), (128, 582, False, True, True),
    (128, 1024, False, False, False), (160, 1024, False, True, False), (148, 1024, False, False, False), (160, 1024, True, False, False),
    (192, 1024, True, False, False), (384, 256, True, False, False), (65536, 1024, False, False, False)])
def test_rule(heads, T, causal, forward, backward):
    lib = ops.host_lib()
    if lib is None:
        pytest.skip("native library not built")
    assert [bool(lib.cme_attention_tc_wide(heads, T, int(causal), b, 148)) for b in (0, 1)] == [forward, backward]
