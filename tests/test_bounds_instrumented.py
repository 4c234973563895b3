"""Every source file with kernels either asks in_bounds() before its plain accesses to global memory, or is one of the files named
here: what the debug build with index checks covers is a decision, not an oversight."""
from pathlib import Path

CSRC = Path(__file__).resolve().parents[1] / "linearnexus_b200" / "csrc"
# decode, backward, block operators, the test kernels of the tcgen05 wrappers and of the waits
UNCHECKED = {"dr_step.cuh", "dr_step_stream.cuh", "dr_bwd.cuh", "dr_bwd_chunk.cuh", "dr_block_ops.cuh", "dr_umma_selftest.cuh",
             "dr_sm100_common.cuh"}


def test_files_with_kernels_are_instrumented_or_named():
    kernels = {f.name for f in CSRC.iterdir() if f.suffix in (".cu", ".cuh") and "__global__" in f.read_text()}
    checked = {f for f in kernels if "in_bounds" in (CSRC / f).read_text()}
    assert kernels - checked == UNCHECKED
