"""Builds ``libacct_b200.so`` (the C-ABI library) from ``csrc/*.cu`` with nvcc for sm_100a.

Beside it, ``_torch_host.so`` (the native host path of the Python layers) is compiled from ``csrc/torch_host.cpp`` with
the host compiler against the installed torch; without torch, only the library is built.

The library is built in-tree, next to this file, so that it travels with the source tree.
``python -m acctransformer_b200.build`` rebuilds it; ``build()`` is also what
``__graft_entry__.build()`` calls.
"""
from __future__ import annotations

import os
import shutil
import subprocess
import sys
from concurrent.futures import ThreadPoolExecutor

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
OBJ_DIR = os.path.join(HERE, "build")
LIB_PATH = os.path.join(HERE, "libacct_b200.so")

SOURCES = ["api.cu", "fa_fwd.cu", "fa_bwd.cu", "fa_bwd_pair.cu", "fa_bwd_wide.cu", "fa_bwd_mid.cu", "mask_plan.cu", "decode.cu", "decode_gqa.cu", "decode_static.cu", "ms_aot.cu"]
NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-lineinfo",
    "-Xcompiler", "-fPIC", "-Xcompiler", "-fvisibility=hidden", "--expt-relaxed-constexpr",
]
HOST_SOURCE = "torch_host.cpp"
HOST_PATH = os.path.join(HERE, "_torch_host.so")
HOST_STAMP = os.path.join(OBJ_DIR, "_torch_host.built_for")


def host_built_for():
    """What the host module is compiled against and only good for: torch's C++ classes and the interpreter."""
    import torch
    python = ".".join(map(str, sys.version_info[:2]))
    return f"torch {torch.__version__}, C++ ABI {int(torch._C._GLIBCXX_USE_CXX11_ABI)}, Python {python}"


def host_is_stale():
    sources = [os.path.join(CSRC, HOST_SOURCE), os.path.join(os.path.dirname(HERE), "include", "acct_b200.h")]
    if _stale(HOST_PATH, sources) or not os.path.exists(HOST_STAMP):
        return True
    with open(HOST_STAMP) as f:
        return f.read() != host_built_for()


def _host_command(src, out):
    """Compiles the CPython module; torch's own libraries are in the process before it is imported."""
    import sysconfig

    import torch
    inc = os.path.join(os.path.dirname(torch.__file__), "include")
    cuda = os.path.dirname(os.path.dirname(_nvcc()))
    lib = os.path.join(os.path.dirname(torch.__file__), "lib")
    return ["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden", "-Wno-attributes",
            f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}", f'-DACCT_BUILT_FOR="{host_built_for()}"',
            "-I" + inc, "-I" + os.path.join(inc, "torch", "csrc", "api", "include"), "-I" + sysconfig.get_paths()["include"],
            "-I" + os.path.join(cuda, "include"), src, "-o", out,
            "-L" + lib, "-ltorch_python", "-ltorch_cuda", "-ltorch_cpu", "-ltorch", "-lc10_cuda", "-lc10", "-ldl"]


def _nvcc():
    exe = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(exe):
        raise RuntimeError("nvcc not found: cannot build libacct_b200.so")
    return exe


def _stale(target, deps):
    if not os.path.exists(target):
        return True
    t = os.path.getmtime(target)
    return any(os.path.getmtime(d) > t for d in deps)


def build(force=False, verbose=False):
    """Compile every CUDA source and the host module, and link the shared library.  Returns the library's path."""
    os.makedirs(OBJ_DIR, exist_ok=True)
    headers = [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith((".cuh", ".h"))]
    headers.append(os.path.join(os.path.dirname(HERE), "include", "acct_b200.h"))
    nvcc = _nvcc()
    jobs = []
    objs = []
    for src in SOURCES:
        s = os.path.join(CSRC, src)
        o = os.path.join(OBJ_DIR, src.replace(".cu", ".o"))
        objs.append(o)
        if force or _stale(o, [s] + headers):
            cmd = [nvcc] + NVCC_FLAGS + (["-Xptxas", "-v"] if verbose else []) + ["-c", s, "-o", o]
            jobs.append(cmd)

    def run(cmd):
        r = subprocess.run(cmd, capture_output=True, text=True)
        if verbose or r.returncode != 0:
            sys.stderr.write(r.stdout + r.stderr)
        if r.returncode != 0:
            raise RuntimeError("compiling failed: " + " ".join(cmd))

    try:
        host_built_for()
        host = force or host_is_stale()
    except ImportError:      # the C ABI (MindSpore and other callers) needs no torch
        sys.stderr.write("no torch here: _torch_host is not built (the Python layers need it, the library does not)\n")
        host = False
    if host:
        jobs.append(_host_command(os.path.join(CSRC, HOST_SOURCE), HOST_PATH))
    device_jobs = any(cmd[0] == nvcc for cmd in jobs)

    with ThreadPoolExecutor(max_workers=4) as ex:
        list(ex.map(run, jobs))
    if host:
        with open(HOST_STAMP, "w") as f:
            f.write(host_built_for())
    if force or device_jobs or _stale(LIB_PATH, objs):
        run([nvcc, "-shared", "-o", LIB_PATH] + objs + ["-lcudart"])
    return LIB_PATH


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
