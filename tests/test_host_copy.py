"""The host memory primitives of the byte-string copies, as this processor builds them and in the portable form that any
other processor gets, at the edges of the wide copy: its 4,096 byte start, runs of 128, every alignment."""
import ctypes
import os
import re
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.parametrize("portable", [False, True])
def test_copies_and_touches(tmp_path, portable):
    so = str(tmp_path / "hostcopy.so")
    subprocess.check_call(["g++", "-O2", "-std=c++17", "-Wall", "-Werror", "-fPIC", "-shared", "-o", so] +
                          (["-DCG_PORTABLE_HOST"] if portable else []) +
                          [os.path.join(ROOT, "tests", "host_model", "hostcopy_host.cpp")])
    lib = ctypes.CDLL(so)
    lib.hc_copy.argtypes, lib.hc_copy.restype = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_int64], None
    lib.hc_touch.argtypes, lib.hc_touch.restype = [ctypes.c_void_p, ctypes.c_int64], None
    assert not (portable and lib.hc_uses_x86())
    rng = np.random.default_rng(1)
    src = rng.integers(0, 256, 20000, dtype=np.uint8)
    for n in (0, 1, 31, 127, 4095, 4096, 4097, 4127, 4223, 4224, 4225, 8192, 12345):
        for to, at in ((0, 0), (1, 0), (31, 7), (32, 1), (17, 33)):
            dst = rng.integers(0, 256, 20000, dtype=np.uint8)
            want = dst.copy()
            want[to:to + n] = src[at:at + n]
            lib.hc_copy(dst.ctypes.data + to, src.ctypes.data + at, n)
            assert (dst == want).all(), (n, to, at)
    lib.hc_pause()
    kept = src.copy()
    lib.hc_touch(src.ctypes.data, src.size)
    assert (src == kept).all()


def test_processor_instructions_stand_behind_the_guard():
    """Outside cg_hostcopy.h no source names an x86 header, intrinsic, target or instruction."""
    csrc = os.path.join(ROOT, "cachegen_b200", "csrc")
    for name in os.listdir(csrc):
        if name.endswith((".cu", ".cuh", ".h")) and name != "cg_hostcopy.h":
            text = open(os.path.join(csrc, name)).read()
            assert not re.search(r"immintrin|_mm\d*_|__m(128|256|512)|target\(\"|\"lock|__builtin_cpu", text), name


OUT_OF_MEMORY = """
import ctypes, resource, sys
sys.path.insert(0, {root!r})
from cachegen_b200 import _lib
lib, here = _lib.lib(), ctypes.create_string_buffer(4096)
at, n = ctypes.addressof(here), 1 << 40  # 2^40 bytes are 2^23 pieces, whose list takes more than is left
used = 4096 * int(open("/proc/self/statm").read().split()[0])
resource.setrlimit(resource.RLIMIT_AS, (used + (64 << 20), used + (64 << 20)))
handle = ctypes.c_void_p()
seg = (_lib.HostSegment * 1)((at, at, n))
print(lib.cg_host_stage(at, n, at, n, ctypes.byref(handle)), lib.cg_host_upload(seg, 1, at, n, None), handle.value)
"""


def test_no_exception_leaves_an_entry():
    """Host memory that is not there is an error code, not the end of the process."""
    import sys
    run = subprocess.run([sys.executable, "-c", OUT_OF_MEMORY.format(root=ROOT)], capture_output=True, text=True)
    assert run.returncode == 0 and run.stdout.split() == ["-6", "-6", "None"], run.stdout + run.stderr
