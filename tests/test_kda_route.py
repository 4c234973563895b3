"""The KDA backward's choice between its kernels, as its source has it: what the tcgen05 ones cannot take leaves every chunk to the others, and no call is refused."""
import re
from pathlib import Path

SRC = (Path(__file__).resolve().parents[1] / "linearnexus_b200" / "csrc" / "dr_bwd_chunk.cuh").read_text()


def test_a_register_count_that_does_not_fit_changes_the_route_alone():
    """local_sm100_kda_kernel's register split waits for good when the block was launched with fewer registers than it counts on."""
    assert "cudaErrorInvalidConfiguration" not in SRC
    few = re.search(r"p\.few = (.*);", SRC).group(1)
    assert "fits" in few and "tma_base(g)" in few
    # whoever launches the tcgen05 kernels has asked
    for kernel in ("local_sm100_kda_kernel", "pre_sm100_kda_kernel"):
        at = SRC.index(f"launch_pdl({kernel}")
        assert "p.few" in SRC[SRC.rindex("inline cudaError_t launch_", 0, at):at]
