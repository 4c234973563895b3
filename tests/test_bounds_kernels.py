"""The debug build's index checks, kernel by kernel where a file has several: each of these indexes global memory by hand."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "linearnexus_b200" / "csrc"


def body(src, name):
    """The kernel's definition: from its name to the next brace in the first column."""
    at = re.search(r"__global__[^;{]*\b%s\(" % name, src).end()
    return src[at:src.index("\n}", at)]


@pytest.mark.parametrize("file,name,checks", [("dr_kda_sm100.cuh", "intra_kernel", 6), ("dr_kda_sm100.cuh", "intra_trans_kernel", 7),
                                              ("dr_kda_sm100.cuh", "trans_state_kernel", 3), ("dr_bwd_pre_kda.cuh", "pre_sm100_kda_kernel", 6),
                                              ("dr_bwd_local_kda.cuh", "local_sm100_kda_kernel", 3), ("dr_bwd_local_sm100.cuh", "local_sm100_kernel", 2)])
def test_kernels_ask_before_plain_accesses(file, name, checks):
    assert len(re.findall(r"\bin_bounds(_run)?\(", body((CSRC / file).read_text(), name))) >= checks
