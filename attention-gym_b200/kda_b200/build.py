"""Ahead-of-time build of libkda_b200.so (sm_100a only) with nvcc.

One shared library, built in-tree next to this file; no JIT, no autotuning, no alternative
back end.  ``python -m kda_b200.build`` rebuilds it.
"""

from __future__ import annotations

import os
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "csrc")
LIB_PATH = os.path.join(HERE, "libkda_b200.so")
TORCH_LIB_PATH = os.path.join(HERE, "libkda_b200_torch.so")      # operators in C++ on top of it
TORCH_SOURCE = "kda_torch.cpp"
OBJ = os.path.join(HERE, "_obj")
STAMP_PATH = os.path.join(OBJ, "torch_build")       # the torch that the operator library was built against
SOURCES = [
    "kda_cabi.cu",
    "kda_recurrent.cu",
    "kda_stream.cu",
    "kda_preops.cu",
    "kda_conv.cu",
    "kda_chunk_fwd.cu",
    "kda_prepare_tc.cu",
    "kda_decode_prep.cu",
    "kda_epilogue.cu",
    "kda_state_tc.cu",
    "kda_chunk_bwd.cu",
    "kda_bwd_chunk_tc.cu",
    "kda_cp.cu",
]
NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC",
]


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), "/usr/local/cuda/bin/nvcc", "nvcc"):
        if cand and (os.path.isabs(cand) and os.path.exists(cand) or not os.path.isabs(cand)):
            return cand
    return "nvcc"


def _torch_build() -> str:
    """What the operator library's C++ ABI hangs on."""
    import torch

    return f"{torch.__version__} cxx11={int(torch._C._GLIBCXX_USE_CXX11_ABI)}"


def _built_for() -> str:
    try:
        with open(STAMP_PATH) as f:
            return f.read()
    except OSError:
        return ""


def needs_build() -> bool:
    if not os.path.exists(LIB_PATH) or not os.path.exists(TORCH_LIB_PATH) or _built_for() != _torch_build():
        return True
    built = min(os.path.getmtime(LIB_PATH), os.path.getmtime(TORCH_LIB_PATH))
    deps = [os.path.join(CSRC, f) for f in os.listdir(CSRC)]
    deps.append(os.path.join(os.path.dirname(os.path.dirname(HERE)), "include", "kda_b200.h"))
    return any(os.path.getmtime(d) > built for d in deps if os.path.exists(d))


def build(force: bool = False, verbose: bool = False) -> str:
    """Compile every kernel for sm_100a into one shared library, and the C++ operators into a second one; returns the
    path of the first.  Both are linked aside and put in place together, so that a failed build leaves the old ones.  A process that
    already runs the old code cannot take up the new one and is told so."""
    from . import _cabi

    if not force and not needs_build():
        return LIB_PATH
    objs = []
    procs = []
    linked = os.path.join(OBJ, "linked")
    os.makedirs(linked, exist_ok=True)
    for src in SOURCES:
        path = os.path.join(CSRC, src)
        if not os.path.exists(path):
            raise FileNotFoundError(path)
        obj = os.path.join(OBJ, src.replace(".cu", ".o"))
        objs.append(obj)
        cmd = [_nvcc(), *NVCC_FLAGS, "-c", path, "-o", obj]
        if verbose:
            cmd.insert(1, "-Xptxas=-v")
        procs.append((src, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT)))
    for src, proc in procs:
        out, _ = proc.communicate()
        if verbose or proc.returncode:
            sys.stderr.write(out.decode())
        if proc.returncode:
            raise RuntimeError(f"nvcc failed on {src}")
    new, new_torch = (os.path.join(linked, os.path.basename(p)) for p in (LIB_PATH, TORCH_LIB_PATH))
    subprocess.check_call([_nvcc(), "-shared", "-o", new, *objs, "-lcudart", "-ldl"])
    _build_torch(linked, new_torch)
    os.replace(new, LIB_PATH)
    os.replace(new_torch, TORCH_LIB_PATH)
    with open(STAMP_PATH, "w") as f:
        f.write(_torch_build())
    if _cabi.mapped():
        raise RuntimeError("the libraries were rebuilt, but this process runs the old ones: restart it")
    return LIB_PATH


def _cxx_runtime() -> list:
    """The C++ runtime that torch runs in this process.  Named before the compiler's own: a compiler that finds only a static one
    would give the library a second runtime, and formatting a number into an error message then crashes the process."""
    with open("/proc/self/maps") as f:
        return sorted({line.split()[-1] for line in f if "/libstdc++.so" in line})[:1]


def _build_torch(linked: str, path: str) -> None:
    """The operators, against the library of the same name in `linked`."""
    import torch

    root = os.path.dirname(torch.__file__)
    lib = os.path.join(root, "lib")
    cuda = os.path.dirname(os.path.dirname(_nvcc())) if os.path.isabs(_nvcc()) else "/usr/local/cuda"
    includes = [os.path.join(root, "include"), os.path.join(root, "include", "torch", "csrc", "api", "include"),
                os.path.join(cuda, "include")]
    subprocess.check_call([
        os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-fPIC", "-shared",
        f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}", *(f"-I{i}" for i in includes),
        os.path.join(CSRC, TORCH_SOURCE), "-o", path, f"-L{linked}", "-l:libkda_b200.so", f"-L{lib}", "-ltorch",
        "-ltorch_cpu", "-lc10", "-lc10_cuda", *_cxx_runtime(), "-Wl,-rpath,$ORIGIN"])


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
