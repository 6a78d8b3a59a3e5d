"""Builds libizb200.so (the CUDA library behind include/izb200.h) in-tree with nvcc for sm_100a.

    python -m arcinferzero_b200.build [--verbose]

nvcc cross-compiles without a GPU.  Objects are cached under arcinferzero_b200/csrc/build/ and rebuilt when a source
or header is newer.
"""
from __future__ import annotations

import os
import subprocess
import sys
from concurrent.futures import ThreadPoolExecutor

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
OUT = os.path.join(HERE, "libizb200.so")
PY_OUT = os.path.join(HERE, "_izb_py.so")  # the Python binding's native side (csrc/izb_py.cpp)
NVCC = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17", "-Xcompiler", "-fPIC", "-Xcompiler", "-fopenmp",
         "-ccbin", "/usr/bin/g++"]


def sources():
    return sorted(f for f in os.listdir(CSRC) if f.endswith(".cu"))


def python_module_for() -> str:
    """What a built binding belongs to: it uses internals of torch and CPython, so another version of either wants another build."""
    import sysconfig

    import torch
    return f"{sysconfig.get_config_var('SOABI')} torch {torch.__version__} cxx11abi {int(torch.compiled_with_cxx11_abi())}"


def build_python_module() -> None:
    """_izb_py.so: plain C++ against the CPython and torch headers (no CUDA code of its own)."""
    import sysconfig

    import torch
    src, hdr = os.path.join(CSRC, "izb_py.cpp"), os.path.join(os.path.dirname(HERE), "include", "izb200.h")
    stamp, made_for = PY_OUT + ".build", python_module_for()
    if os.path.exists(PY_OUT) and os.path.getmtime(PY_OUT) >= max(os.path.getmtime(src), os.path.getmtime(hdr)) and os.path.exists(stamp):
        with open(stamp) as f:
            if f.read() == made_for:
                return
    t = os.path.dirname(torch.__file__)
    cmd = ["/usr/bin/g++", "-O2", "-std=c++17", "-fPIC", "-shared", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch.compiled_with_cxx11_abi())}",
           "-I" + sysconfig.get_paths()["include"], "-isystem", os.path.join(t, "include"), "-isystem", os.path.join(t, "include/torch/csrc/api/include"),
           "-isystem", os.path.join(os.path.dirname(os.path.dirname(NVCC)), "include"), src, "-o", PY_OUT, "-L" + os.path.join(t, "lib"), "-ltorch_python",
           "-ltorch_cuda", "-ltorch_cpu", "-ltorch", "-lc10_cuda", "-lc10"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError("g++ failed:\n" + " ".join(cmd) + "\n" + r.stdout + r.stderr)
    with open(stamp, "w") as f:
        f.write(made_for)


def build(verbose: bool = False) -> str:
    os.makedirs(os.path.join(CSRC, "build"), exist_ok=True)
    hdrs = [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith(".cuh")] + [
        os.path.join(os.path.dirname(HERE), "include", "izb200.h")]
    newest_hdr = max(os.path.getmtime(h) for h in hdrs)
    objs, jobs = [], []
    for s in sources():
        src, obj = os.path.join(CSRC, s), os.path.join(CSRC, "build", s[:-3] + ".o")
        objs.append(obj)
        if not os.path.exists(obj) or os.path.getmtime(obj) < max(os.path.getmtime(src), newest_hdr):
            jobs.append([NVCC, *FLAGS, *(["-Xptxas", "-v"] if verbose else []), "-c", src, "-o", obj])

    def run(cmd):
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError("nvcc failed:\n" + " ".join(cmd) + "\n" + r.stdout + r.stderr)
        return r.stderr

    with ThreadPoolExecutor(max_workers=min(8, 1 + len(jobs))) as ex:
        py = ex.submit(build_python_module)
        for log in ex.map(run, jobs):
            if verbose and log:
                print(log)
    if jobs or not os.path.exists(OUT):
        run([NVCC, "-shared", "-o", OUT, *objs, "-lcudart", "-ldl", "-lgomp", "-ccbin", "/usr/bin/g++"])
    py.result()  # (last: the library needs neither torch nor Python headers, and is there for C hosts when the binding cannot be built)
    return OUT


if __name__ == "__main__":
    print(build(verbose="--verbose" in sys.argv))
