"""Build ``libdaisy_b200.so`` in-tree with nvcc for sm_100a, and ``_C.so``, its torch binding, with g++.

    python -m daisy_b200.build [--force] [--verbose]

One object per ``csrc/*.cu`` (rebuilt when the source or a header is newer), linked into
``daisy_b200/libdaisy_b200.so`` with the static CUDA runtime, so the library has no
load-time dependency on libcuda and can be opened on a machine without a GPU.  ``_C.so`` (``csrc/torch_bind.cpp``) links
against it (found next to it through its run path) and against the installed torch.
"""
from __future__ import annotations

import os
import shutil
import subprocess
import sys
from concurrent.futures import ThreadPoolExecutor

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
BUILD = os.path.join(CSRC, "build")
LIB = os.path.join(HERE, "libdaisy_b200.so")
EXT = os.path.join(HERE, "_C.so")
NVCC_FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-lineinfo",
              "-Xcompiler", "-fPIC", "--expt-relaxed-constexpr"]


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and os.path.exists(cand):
            return cand
    raise RuntimeError("nvcc not found (set NVCC)")


def _newest_header() -> float:
    hs = [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith((".cuh", ".h"))]
    hs.append(os.path.join(os.path.dirname(HERE), "include", "daisy_b200.h"))
    return max(os.path.getmtime(h) for h in hs)


def _ext_cmds():
    """-> (compile command, link command, object) of the torch binding."""
    import sysconfig
    import torch
    tdir = os.path.dirname(torch.__file__)
    cuda = os.path.dirname(os.path.dirname(_nvcc()))
    src, obj = os.path.join(CSRC, "torch_bind.cpp"), os.path.join(BUILD, "torch_bind.o")
    inc = [os.path.join(tdir, "include"), os.path.join(tdir, "include", "torch", "csrc", "api", "include"),
           os.path.join(cuda, "include"), sysconfig.get_paths()["include"]]
    comp = [shutil.which("g++") or "g++", "-O2", "-std=c++17", "-fPIC", "-fvisibility=hidden", "-DTORCH_EXTENSION_NAME=_C", "-DTORCH_API_INCLUDE_EXTENSION_H",
            f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}", *[f"-isystem{i}" for i in inc], "-c", src, "-o", obj]
    link = [comp[0], "-shared", obj, "-o", EXT, "-L" + HERE, "-ldaisy_b200", "-L" + os.path.join(tdir, "lib"), "-lc10", "-ltorch_cpu",
            "-ltorch", "-ltorch_python", "-lc10_cuda", "-ltorch_cuda", "-Wl,-rpath,$ORIGIN"]
    return comp, link, obj


def build(force: bool = False, verbose: bool = False) -> str:
    os.makedirs(BUILD, exist_ok=True)
    nvcc = _nvcc()
    srcs = sorted(f for f in os.listdir(CSRC) if f.endswith(".cu"))
    hdr_t = _newest_header()
    jobs, objs = [], []
    for s in srcs:
        src, obj = os.path.join(CSRC, s), os.path.join(BUILD, s[:-3] + ".o")
        objs.append(obj)
        if force or not os.path.exists(obj) or os.path.getmtime(obj) < max(os.path.getmtime(src), hdr_t):
            cmd = [nvcc, *NVCC_FLAGS, "-c", src, "-o", obj]
            if verbose:
                cmd.insert(1, "-Xptxas=-v")
            jobs.append(cmd)
    ext_comp, ext_link, ext_obj = _ext_cmds()
    ext_src = os.path.join(CSRC, "torch_bind.cpp")
    if force or not os.path.exists(ext_obj) or os.path.getmtime(ext_obj) < max(os.path.getmtime(ext_src), hdr_t):
        jobs.insert(0, ext_comp)

    def run(cmd):
        r = subprocess.run(cmd, capture_output=True, text=True)
        return cmd, r

    with ThreadPoolExecutor(max_workers=max(1, min(len(jobs), os.cpu_count() or 1))) as ex:
        for cmd, r in ex.map(run, jobs):
            if verbose or r.returncode != 0:
                sys.stderr.write(" ".join(cmd) + "\n" + r.stdout + r.stderr)
            if r.returncode != 0:
                raise RuntimeError(f"{os.path.basename(cmd[0])} failed on {cmd[-3]}")
    if jobs or not os.path.exists(LIB) or not os.path.exists(EXT):
        for cmd in ([nvcc, "-shared", "-o", LIB, *objs, "-cudart", "static"], ext_link):
            r = subprocess.run(cmd, capture_output=True, text=True)
            if r.returncode != 0:
                sys.stderr.write(r.stdout + r.stderr)
                raise RuntimeError("link failed")
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="--verbose" in sys.argv))
