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


def test_symbols_of_an_overlapped_launch_are_not_read_as_constant_data():
    """The coder's blocks may start while the quantiser still writes the words of symbols: the same for them, and for what else
    a launch in front writes.  What the coder takes with __ldg are the caller's inputs."""
    text = open(os.path.join(ROOT, "cachegen_b200", "csrc", "cg_store.cu")).read()
    coder = text[text.index("static __device__ __noinline__ uint32_t encode_again("):text.index("// the tail of the separate calls")]
    inputs = {"p.out.bins + row", "p.out.table_row_off + row"}
    assert set(re.findall(r"__ldg\(([^)]*)\)", coder)) == inputs
    reads = list(re.finditer(r"written_symbols\(", coder))
    assert len(reads) == len(re.findall(r"\b(?:sp|q)\b(?:\[s\])? \+ |\(q\)", coder)) == 5
    kernel = coder.index("__global__")
    for read in reads:
        if read.start() > kernel:  # the others are in what the kernel calls once it has read its symbols
            assert "wait_for_launch_before();" in coder[kernel:read.start()]
    # the columns of ready tables are read with __ldg: the kernel that writes them has to have ended
    assert re.search(r"early = alone && z\.nsub == 1;", text)
    assert re.search(r"launch\(packed_tables_kernel, [^;]*, false, st, table_jobs", text)


def test_borrowed_columns_are_read_behind_a_barrier():
    """Lanes behind the last channel decode from columns that the last active lane of their warp has staged.  A barrier that every
    lane meets whatever the table's size stands between the two, in each kernel that lends columns."""
    text = open(os.path.join(ROOT, "cachegen_b200", "csrc", "cg_decode.cu")).read()
    kernels = [k for k in re.split(r"(?=__global__)", text[:text.index("// ---- launch helpers")]) if "borrow_stream(start[i]" in k]
    assert len(kernels) == 2
    for k in kernels:
        between = k[k.rindex("stage_table_column"):k.index("borrow_stream(start[i]")]
        assert re.search(r"^    __sync(warp|threads)\(\);", between, re.M)  # a statement of the kernel's body itself, in no branch
