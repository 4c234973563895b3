"""Kernels whose bounded waits can give up (DR_DEV_TIMEOUT), read as source: a CTA lets the copies and products that it has started finish before it ends
or frees its tensor memory."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "linearnexus_b200" / "csrc"
FILES = sorted(f.name for f in CSRC.glob("*.cuh") if f.name != "dr_sm100_common.cuh" and re.search(r"wait_(inline|more)\(", f.read_text()))


def test_the_kernels_are_found():
    assert {"dr_bwd_chunk.cuh", "dr_bwd_local_kda.cuh", "dr_bwd_local_sm100.cuh", "dr_bwd_pre_kda.cuh", "dr_chunk_sm100.cuh", "dr_kda_sm100.cuh",
            "dr_ssd_sm100.cuh"} <= set(FILES)


@pytest.mark.parametrize("name", FILES)
def test_a_cta_settles_before_it_ends(name):
    lines = (CSRC / name).read_text().splitlines()
    kernels = [i for i, x in enumerate(lines) if re.search(r"bool|auto wait_\w+ = \[&\]", x) and "wait_" in x and "= [&]" in x and "bar" in x and
               any(re.search(r"wait_(inline|more)\(", y) for y in lines[i:i + 5])]
    ends = [i for i, x in enumerate(lines) if "settle(ctl.abort);" in x]
    assert len(kernels) == len(ends) > 0   # once per kernel: in front of the tensor memory's end, or where the copying warp leaves
    for i, x in enumerate(lines):
        if "tc::tmem_dealloc(" in x:
            assert "settle(ctl.abort);" in lines[i - 1]
