"""Build the CUDA library in-tree: ``python -m blockgtq_b200.build``.

Compiles every ``csrc/*.cu`` for sm_100a with nvcc and links one shared
library, ``blockgtq_b200/libbgtq.so``, exporting the C ABI of ``include/bgtq.h``.
nvcc cross-compiles without a GPU.  The library links only the CUDA runtime.
``csrc/bgtq_native.cpp``, the host side of the frequent calls, becomes the extension
module ``blockgtq_b200/_native.so`` (g++ against torch and Python).
"""
from __future__ import annotations

import glob
import os
import shutil
import subprocess
import sys

PKG = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(PKG, "csrc")
LIB = os.environ.get("BGTQ_LIB") or os.path.join(PKG, "libbgtq.so")
NATIVE_SRC = os.path.join(CSRC, "bgtq_native.cpp")
NATIVE = os.path.join(PKG, "_native.so")
NATIVE_STAMP = os.path.join(PKG, "build", "native.abi")         # the versions it was built for
NVCC_FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
              "--use_fast_math=false", "-Xcompiler", "-fPIC", "-Xcompiler", "-fvisibility=hidden"]


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and os.path.exists(cand):
            return cand
    raise RuntimeError("nvcc not found (set NVCC=/path/to/nvcc)")


def sources() -> list:
    return sorted(glob.glob(os.path.join(CSRC, "*.cu")))


def native_abi() -> str:
    """What the extension module is bound to beyond its sources: torch's internal C++ API and the Python ABI."""
    import sysconfig

    import torch
    return f"torch {torch.__version__}, {sysconfig.get_config_var('SOABI')}"


def needs_build() -> bool:
    if not os.path.exists(LIB) or not os.path.exists(NATIVE):
        return True
    try:
        with open(NATIVE_STAMP) as f:
            if f.read() != native_abi():
                return True
    except OSError:
        pass            # (the module says it itself when it is loaded)
    header = os.path.join(os.path.dirname(PKG), "include", "bgtq.h")
    if os.path.getmtime(NATIVE) < max(os.path.getmtime(NATIVE_SRC), os.path.getmtime(header)):
        return True
    t = os.path.getmtime(LIB)
    deps = sources() + glob.glob(os.path.join(CSRC, "*.h")) + glob.glob(os.path.join(CSRC, "*.cuh")) + \
        [header]
    return any(os.path.getmtime(d) > t for d in deps)


JIT_SOURCES = ["bgtq_common.cuh", "bgtq_plan.h", "bgtq_decode_params.cuh", "bgtq_decode_cluster.cuh", "bgtq_decode_kernel.cuh"]


def _embed_jit_sources(objdir: str) -> str:
    """The decode kernel is also compiled at run time from its own text: write each source file it consists of
    as a C++ raw string literal (``<name>.str``) for csrc/bgtq_decode_jit.cu to include."""
    out = os.path.join(objdir, "jit_src")
    os.makedirs(out, exist_ok=True)
    for name in JIT_SOURCES:
        text = open(os.path.join(CSRC, name)).read()
        lines = [ln for ln in text.splitlines()
                 if not ln.startswith("#pragma once") and not ln.startswith('#include "')]
        body = "\n".join(lines)
        assert ')BGTQSRC"' not in body
        with open(os.path.join(out, name + ".str"), "w") as f:
            f.write('R"BGTQSRC(' + body + '\n)BGTQSRC"\n')
    return out


def _native_cmd(out: str) -> list:
    import sysconfig

    import torch
    base = os.path.dirname(torch.__file__)
    cuda = os.path.dirname(os.path.dirname(os.path.realpath(_nvcc())))
    cxx = os.environ.get("CXX") or shutil.which("g++") or "g++"
    inc = [os.path.join(base, "include"), os.path.join(base, "include", "torch", "csrc", "api", "include"),
           os.path.join(cuda, "include"), sysconfig.get_paths()["include"]]
    return [cxx, "-shared", "-fPIC", "-O2", "-std=c++17", "-fvisibility=hidden", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
            f'-DBGTQ_NATIVE_ABI="{native_abi()}"',
            *[x for d in inc for x in ("-isystem", d)], NATIVE_SRC, "-o", out, "-L", os.path.join(base, "lib"),
            "-ltorch_python", "-ltorch", "-ltorch_cpu", "-ltorch_cuda", "-lc10", "-lc10_cuda"]


def build(force: bool = False, verbose: bool = False) -> str:
    if not force and not needs_build():
        return LIB
    nvcc = _nvcc()
    native_cmd = _native_cmd(NATIVE + ".tmp")
    native = subprocess.Popen(native_cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT)
    objdir = os.path.join(PKG, "build")
    os.makedirs(objdir, exist_ok=True)
    jit_inc = _embed_jit_sources(objdir)
    procs = []
    for src in sources():
        obj = os.path.join(objdir, os.path.basename(src)[:-3] + ".o")
        cmd = [nvcc] + [f for f in NVCC_FLAGS if f != "--use_fast_math=false"] + \
            (["-Xptxas", "-v"] if verbose else []) + os.environ.get("BGTQ_NVCC_EXTRA", "").split() + \
            ["-I", jit_inc, "-c", src, "-o", obj]
        procs.append((obj, cmd, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT)))
    objs = []
    for obj, cmd, p in procs:
        out = p.communicate()[0].decode()
        if p.returncode != 0:
            raise RuntimeError("nvcc failed: " + " ".join(cmd) + "\n" + out)
        if verbose:
            sys.stderr.write(out)
        objs.append(obj)
    tmp = LIB + ".tmp"
    cmd = [nvcc, "-shared", "-o", tmp] + objs + ["-cudart", "shared", "-ldl"]
    r = subprocess.run(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT)
    if r.returncode != 0:
        raise RuntimeError("link failed: " + r.stdout.decode())
    os.replace(tmp, LIB)
    out = native.communicate()[0].decode()
    if native.returncode != 0:
        raise RuntimeError("building the host extension failed: " + " ".join(native_cmd) + "\n" + out)
    os.replace(NATIVE + ".tmp", NATIVE)
    with open(NATIVE_STAMP, "w") as f:
        f.write(native_abi())
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
