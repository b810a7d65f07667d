"""Build libfda_sm100.so in-tree with nvcc, for sm_100a only, and beside it _fda_torch.so, the C++ host path of the
Python functions, against the torch that runs this script.

    python build_lib.py            # incremental
    python build_lib.py --force    # rebuild everything

Environment (same names as the reference's setup.py:5-13 where they make sense here):
  FDA_LINEINFO=0        drop -lineinfo (on by default)
  FDA_RESOURCE_USAGE=1  print registers / spills / shared memory per kernel (ptxas -v)
  NVCC_THREADS, MAX_JOBS  parallelism
"""

import os
import subprocess
import sys
from concurrent.futures import ThreadPoolExecutor

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
OBJ = os.path.join(HERE, "build")
LIB = os.path.join(HERE, "fast_diffusion_attention", "libfda_sm100.so")
TORCH_SRC = os.path.join(CSRC, "torch_binding.cpp")
TORCH_EXT = os.path.join(HERE, "fast_diffusion_attention", "_fda_torch.so")
TORCH_STAMP = os.path.join(OBJ, "_fda_torch.txt")   # what TORCH_EXT was built with
SOURCES = ["abi.cu", "fwd_sm100.cu", "bwd_sm100.cu", "bwd_fused_sm100.cu", "selftest_sm100.cu", "varlen_list.cu"]


def _nvcc():
    cand = os.path.join(_cuda_home(), "bin", "nvcc")
    return cand if os.path.exists(cand) else "nvcc"


def _headers():
    out = [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith((".h", ".cuh"))]
    out.append(os.path.join(HERE, "..", "include", "fda.h"))
    return out


def _cuda_home():
    return os.environ.get("CUDA_HOME", "/usr/local/cuda")


def _torch_command():
    """g++ line of the host path. The torch libraries are already loaded when the module is imported, so it carries no
    run path."""
    import sysconfig

    import torch
    root = os.path.dirname(torch.__file__)
    inc = [os.path.join(root, "include"), os.path.join(root, "include", "torch", "csrc", "api", "include"),
           os.path.join(_cuda_home(), "include"), sysconfig.get_paths()["include"]]
    libs = ["-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch_cuda", "-ltorch", "-ltorch_python",
            # the shared C++ runtime that torch uses: some toolchains carry only a static one, and a second copy of the
            # stream classes in one process crashes on the first exception text that goes through both
            "-nostdlib++", "-l:libstdc++.so.6", "-lm"]
    return ([os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden",
             f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}"] + ["-I" + i for i in inc] +
            [TORCH_SRC, "-o", TORCH_EXT, "-L" + os.path.join(root, "lib")] + libs)


def _stale(target, deps):
    if not os.path.exists(target):
        return True
    t = os.path.getmtime(target)
    return any(os.path.getmtime(d) > t for d in deps)


def _torch_stamp(command):
    import torch
    return " ".join([torch.__version__] + command)


def _torch_ext_stale(command):
    """The host path is bound to the torch it was built against, whose headers no time stamp here covers: another version,
    another place or other flags rebuild it."""
    if _stale(TORCH_EXT, [TORCH_SRC, os.path.join(HERE, "..", "include", "fda.h")]) or not os.path.exists(TORCH_STAMP):
        return True
    with open(TORCH_STAMP) as f:
        return f.read() != _torch_stamp(command)


def build(force=False, verbose=False):
    os.makedirs(OBJ, exist_ok=True)
    flags = ["-std=c++17", "-O3", "-gencode", "arch=compute_100a,code=sm_100a", "-Xcompiler", "-fPIC",
             "--expt-relaxed-constexpr", "-Xcudafe", "--diag_suppress=177"]
    if os.environ.get("FDA_LINEINFO", "1") == "1":
        flags.append("-lineinfo")
    if os.environ.get("FDA_RESOURCE_USAGE", "0") == "1":
        flags += ["-Xptxas", "-v"]
    flags += ["--threads", os.environ.get("NVCC_THREADS", "2")]
    headers = _headers()
    jobs = []
    objs = []
    for src in SOURCES:
        s = os.path.join(CSRC, src)
        o = os.path.join(OBJ, src.replace(".cu", ".o"))
        objs.append(o)
        if force or _stale(o, [s] + headers):
            jobs.append([_nvcc(), "-c", s, "-o", o] + flags)

    def run(cmd):
        r = subprocess.run(cmd, capture_output=True, text=True)
        if verbose or r.returncode != 0 or os.environ.get("FDA_RESOURCE_USAGE", "0") == "1":
            sys.stderr.write(" ".join(cmd) + "\n" + r.stdout + r.stderr)
        if r.returncode != 0:
            raise RuntimeError("compilation failed: " + " ".join(cmd))

    links = list(jobs)
    torch_command = _torch_command()
    torch_stale = force or _torch_ext_stale(torch_command)
    if torch_stale:
        jobs.append(torch_command)
    with ThreadPoolExecutor(max_workers=int(os.environ.get("MAX_JOBS", "4"))) as ex:
        list(ex.map(run, jobs))
    if torch_stale:
        with open(TORCH_STAMP, "w") as f:
            f.write(_torch_stamp(torch_command))
    if force or links or _stale(LIB, objs):
        run([_nvcc(), "-shared", "-o", LIB] + objs + ["-cudart", "static"])
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
