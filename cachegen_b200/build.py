"""Builds libcachegen_b200.so in-tree with nvcc for sm_100a (no torch headers: a few seconds per file), and _calls.*.so, the
host side of the calls on torch's tensors, with the host compiler.  The library needs neither torch nor Python's headers;
where those are not there it is built without _calls.*.so.

    python -m cachegen_b200.build [--force] [--verbose]
"""
import os
import subprocess
import sys
import sysconfig
from concurrent.futures import ThreadPoolExecutor

PKG = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(PKG, "csrc")
LIB = os.path.join(PKG, "libcachegen_b200.so")
SOURCES = ["cg_api.cu", "cg_quant.cu", "cg_tables.cu", "cg_encode.cu", "cg_store.cu", "cg_decode.cu", "cg_host.cu"]
HEADERS = [os.path.join(CSRC, "cg_common.cuh"), os.path.join(CSRC, "cg_coder.cuh"), os.path.join(CSRC, "cg_hostcopy.h"),
           os.path.join(PKG, "..", "include", "cachegen_b200.h")]
CALLS = os.path.join(PKG, "_calls" + sysconfig.get_config_var("EXT_SUFFIX"))
CALLS_SOURCE = os.path.join(CSRC, "cg_calls.cpp")
NVCC_FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
              "-Xcompiler", "-fPIC,-pthread"]


def _nvcc():
    home = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    return os.path.join(home, "bin", "nvcc")


def needs_build():
    if not os.path.exists(LIB):
        return True
    t = os.path.getmtime(LIB)
    deps = [os.path.join(CSRC, s) for s in SOURCES] + HEADERS
    return any(os.path.getmtime(d) > t for d in deps)


def calls_built_for():
    """What the host module is compiled against: inlined code of another torch's headers would read its objects wrongly."""
    import torch
    return f"torch {torch.__version__} {torch.version.git_version} abi {int(torch._C._GLIBCXX_USE_CXX11_ABI)}"


def calls_need_build():
    if not os.path.exists(CALLS) or any(os.path.getmtime(d) > os.path.getmtime(CALLS) for d in (CALLS_SOURCE, HEADERS[-1])):
        return True
    try:
        mark = calls_built_for().encode()
    except ImportError:
        return True
    with open(CALLS, "rb") as f:
        return mark not in f.read()


def build_calls():
    import torch
    base = os.path.dirname(torch.__file__)
    include = [os.path.join(base, "include"), os.path.join(base, "include", "torch", "csrc", "api", "include"),
               os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include"), sysconfig.get_paths()["include"]]
    made = f"{CALLS}.{os.getpid()}"  # a process that imports the module meanwhile finds the old one or the new one
    cmd = [os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden", "-o", made, CALLS_SOURCE,
           f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}", f'-DCG_BUILT_FOR="{calls_built_for()}"'] + [
           f"-I{d}" for d in include] + ["-L" + os.path.join(base, "lib")] + [
           "-l" + n for n in ("torch_python", "torch", "torch_cpu", "torch_cuda", "c10", "c10_cuda")]
    try:
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError(f"{cmd[0]} failed on cg_calls.cpp:\n{r.stdout}\n{r.stderr}")
        os.replace(made, CALLS)
    finally:
        if os.path.exists(made):
            os.remove(made)


def build(force=False, verbose=False, extra_flags=(), out=None):
    """Compiles the library and returns its path.  `out` builds a second copy elsewhere (with
    `extra_flags`, e.g. -D switches) without touching the in-tree one; CACHEGEN_B200_LIB selects it."""
    target = out or LIB
    if out or force or needs_build():
        build_library(target, out, verbose, extra_flags)
    if not out and (force or calls_need_build()):
        try:
            build_calls()
        except (ImportError, OSError, RuntimeError) as e:
            print(f"{CALLS} was not built; the library does not need it, calls of the Python classes take longer: {e}", file=sys.stderr)
    return target


def build_library(target, out, verbose, extra_flags):
    flags = NVCC_FLAGS + list(extra_flags)
    if verbose:
        flags = flags + ["-Xptxas", "-v"]
    obj_prefix = (out + ".") if out else (CSRC + os.sep)

    def one(src):
        obj = obj_prefix + src.replace(".cu", ".o")
        cmd = [_nvcc(), "-c", os.path.join(CSRC, src), "-o", obj] + flags
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError(f"nvcc failed on {src}:\n{r.stdout}\n{r.stderr}")
        if verbose:
            sys.stderr.write(r.stderr)
        return obj

    with ThreadPoolExecutor(max_workers=len(SOURCES)) as ex:
        objs = list(ex.map(one, SOURCES))
    cmd = [_nvcc(), "-shared", "-o", target] + objs + ["-gencode", "arch=compute_100a,code=sm_100a", "-lcudart"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"link failed:\n{r.stdout}\n{r.stderr}")


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="--verbose" in sys.argv))
