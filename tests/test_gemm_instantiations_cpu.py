"""Every fused epilogue with a kernel of its own on the 256-column tile of the CTA pair has one on the 192-column tile: the plan
chooses between the two by size alone."""
import re
from pathlib import Path

import cme213_final_project_b200


def test_pair_tiles_have_the_same_epilogues():
    text = (Path(cme213_final_project_b200.__file__).parent / "ops/csrc/gemm_tc_inst_list.h").read_text()
    found = {(int(bn), spec) for bn, pair, spec in re.findall(r"^CME_GEMM_TC_EXTERN\((\d+), \w+, (\w+), ([-\w]+)\)", text, re.M)
             if pair == "true"}
    wide = {spec for bn, spec in found if bn == 256} - {"SPEC_TF32"}          # the 192-column tile is for bf16 only
    assert wide and wide <= {spec for bn, spec in found if bn == 192}
