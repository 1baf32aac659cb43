"""Build ``libqmm.so`` (the C-ABI kernel library) in-tree with nvcc for sm_100a, and ``_calls.so`` (the torch-facing calls).

    python -m jax_metallib_b200.build [--force]

nvcc cross-compiles without a GPU.  Objects go to ``csrc/build/``; the shared
library is written next to this file so that it travels with the source tree.
``_calls.so`` needs a torch with CUDA to build against; without one it is left
out, and ``ops`` and ``quantized`` make their calls in Python.
"""

from __future__ import annotations

import os
import shutil
import subprocess
import sys
from concurrent.futures import ThreadPoolExecutor

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
OBJ = os.path.join(CSRC, "build")
LIB = os.path.join(HERE, "libqmm.so")
CALLS_SRC = os.path.join(HERE, "binding", "calls.cc")
CALLS = os.path.join(HERE, "_calls.so")
CALLS_KEY = os.path.join(OBJ, "calls.key")   # what _calls.so was built from

GXX_FLAGS = ["-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden"]
NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC", "-Xcompiler", "-fvisibility=hidden",
]


def _nvcc() -> str:
    exe = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(exe):
        raise RuntimeError("nvcc not found; libqmm.so cannot be built")
    return exe


def sources() -> list[str]:
    out = []
    for root, _dirs, files in os.walk(CSRC):
        if os.path.basename(root) == "build":
            continue
        for f in sorted(files):
            if f.endswith((".cu", ".cc")):
                out.append(os.path.join(root, f))
    return sorted(out)


def _headers_mtime() -> float:
    latest = 0.0
    for root, _dirs, files in os.walk(CSRC):
        for f in files:
            if f.endswith((".cuh", ".h", ".hpp")):
                latest = max(latest, os.path.getmtime(os.path.join(root, f)))
    inc = os.path.join(os.path.dirname(HERE), "include")
    for f in os.listdir(inc):
        latest = max(latest, os.path.getmtime(os.path.join(inc, f)))
    return latest


def calls_key(torch_version: str, cuda_version: str, abi: int) -> str:
    """What a binary of calls.cc depends on: the sources, and the C++ of this Python and of this torch, whose layouts change
    from version to version."""
    import hashlib
    import sysconfig

    header = os.path.join(os.path.dirname(HERE), "include", "qmm.h")
    digest = hashlib.sha256(b"".join(open(path, "rb").read() for path in (CALLS_SRC, header))).hexdigest()
    return "\n".join((digest, torch_version, cuda_version, str(abi), str(sysconfig.get_config_var("SOABI")), " ".join(GXX_FLAGS)))


def build_calls(force: bool = False) -> str | None:
    """The extension module of ops.py and quantized.py: C++ against the headers of the torch that is installed.  None, and no
    module, where there is no torch with CUDA."""
    try:
        import torch
    except ImportError:
        torch = None
    if torch is None or not torch.version.cuda:
        for path in (CALLS, CALLS_KEY):   # one for another torch is of no use
            if os.path.exists(path):
                os.remove(path)
        print("no torch with CUDA: _calls.so is not built, calls are made in Python", file=sys.stderr)
        return None
    abi = int(torch._C._GLIBCXX_USE_CXX11_ABI)
    key = calls_key(torch.__version__, torch.version.cuda, abi)
    if not force and os.path.exists(CALLS) and os.path.exists(CALLS_KEY) and open(CALLS_KEY).read() == key:
        return CALLS
    import sysconfig

    root = os.path.dirname(torch.__file__)
    cuda = os.path.dirname(os.path.dirname(os.path.realpath(_nvcc())))
    include = [os.path.join(root, "include"), os.path.join(root, "include", "torch", "csrc", "api", "include"),
               sysconfig.get_paths()["include"], os.path.join(cuda, "include")]
    cmd = ["g++", *GXX_FLAGS, f"-D_GLIBCXX_USE_CXX11_ABI={abi}", f'-DQMM_TORCH_VERSION="{torch.__version__}"',
           *[f"-isystem{d}" for d in include], CALLS_SRC, "-o", CALLS, f"-L{os.path.join(root, 'lib')}",
           "-ltorch_python", "-ltorch_cpu", "-lc10", "-lc10_cuda"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError("g++ failed:\n" + " ".join(cmd) + "\n" + r.stdout + r.stderr)
    os.makedirs(os.path.dirname(CALLS_KEY), exist_ok=True)
    with open(CALLS_KEY, "w") as f:
        f.write(key)
    return CALLS


def build(force: bool = False, verbose: bool = False) -> str:
    os.makedirs(OBJ, exist_ok=True)
    nvcc = _nvcc()
    hdr = _headers_mtime()
    jobs = []
    objs = []
    for src in sources():
        rel = os.path.relpath(src, CSRC).replace(os.sep, "_")
        obj = os.path.join(OBJ, os.path.splitext(rel)[0] + ".o")
        objs.append(obj)
        stale = force or not os.path.exists(obj) or os.path.getmtime(obj) < max(os.path.getmtime(src), hdr)
        if stale:
            cmd = [nvcc, *NVCC_FLAGS, *os.environ.get("QMM_EXTRA_NVCC_FLAGS", "").split(), "-x", "cu", "-c", src, "-o", obj]
            if verbose:
                cmd.insert(1, "-Xptxas=-v")
            jobs.append(cmd)

    def run(cmd):
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError("nvcc failed:\n" + " ".join(cmd) + "\n" + r.stdout + r.stderr)
        return r.stderr

    if jobs:
        with ThreadPoolExecutor(max_workers=min(8, len(jobs))) as ex:
            for log in ex.map(run, jobs):
                if verbose and log:
                    print(log)
    if jobs or not os.path.exists(LIB) or force:
        cmd = [nvcc, "-shared", "-o", LIB, *objs, "-Xcompiler", "-fPIC", "-lcudart_static", "-ldl", "-lpthread", "-lrt"]
        run(cmd)
    build_calls(force)
    return LIB


if __name__ == "__main__":
    path = build(force="--force" in sys.argv, verbose="-v" in sys.argv)
    print(path)
