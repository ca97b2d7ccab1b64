"""Properties of the kernels that no run shows."""
import os
import re

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_offsets_of_an_overlapped_launch_are_not_read_as_constant_data():
    """Decode blocks start while the launch that writes their group offsets still runs, so these loads may not take the
    path for data that does not change during the kernel."""
    text = open(os.path.join(ROOT, "cachegen_b200", "csrc", "cg_decode.cu")).read()
    kernels = text[:text.index("// ---- launch helpers")]
    assert not re.search(r"__ldg\([^;]*group_off", kernels)
    reads = list(re.finditer(r"written_offset\((p|job)\.group_off", kernels))
    assert len(reads) == len(re.findall(r"(p|job)\.group_off \+", kernels)) == 4
    for read in reads:  # the wait stands in front of the load, in the same kernel
        before = kernels[:read.start()]
        assert before.rindex("wait_for_launch_before();") > before.rindex("__global__")
