"""Builds ``libvfkv.so`` in-tree with nvcc for sm_100a.

Run as ``python -m vulkanforge_b200.build`` (add ``--verbose`` for ptxas
register / shared-memory reports).  The shared object lands beside this file so
that it travels with the source tree.
"""
from __future__ import annotations

import os
import shutil
import subprocess
import sys
import sysconfig

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
OUT = os.path.join(HERE, "libvfkv.so")
CALLS = os.path.join(HERE, "_native.so")        # Python bindings of the per-layer calls (csrc/py_calls.cpp), linked to OUT
SOURCES = ["api.cu", "append.cu", "attn_generic.cu", "attn_mma.cu", "attn_mma_host.cu", "attn_wide.cu", "attn_merge.cu", "exchange.cu", "attn_prefill.cu", "attn_prefill_f32.cu", "attn_prefill_tc5.cu", "attn_prefill_tc5s.cu", "rope_append.cu", "routes.cpp", "noalloc.cu", "kv_cache.cpp"]
ARCH = ["-gencode", "arch=compute_100a,code=sm_100a"]


def _nvcc() -> str:
    for cand in (shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and os.path.exists(cand):
            return cand
    raise RuntimeError("nvcc not found; libvfkv.so cannot be built")


def _stale() -> bool:
    if not (os.path.exists(OUT) and os.path.exists(CALLS)):
        return True
    t = min(os.path.getmtime(OUT), os.path.getmtime(CALLS))
    deps = [os.path.join(CSRC, f) for f in os.listdir(CSRC)]
    deps.append(os.path.join(HERE, "..", "include", "vfkv.h"))
    deps.append(os.path.join(HERE, "..", "include", "vfkv_next.h"))
    deps.append(os.path.abspath(__file__))
    return any(os.path.getmtime(d) > t for d in deps)


def build(force: bool = False, verbose: bool = False) -> str:
    if not force and not _stale():
        return OUT
    objdir = os.path.join(HERE, "build")
    os.makedirs(objdir, exist_ok=True)
    common = ["-O3", "-std=c++17", "-lineinfo", "-Xcompiler", "-fPIC", "-ccbin", "/usr/bin/g++"] + ARCH
    if verbose:
        common += ["-Xptxas", "-v"]
    procs = []
    objs = []
    for src in SOURCES:
        obj = os.path.join(objdir, src.rsplit(".", 1)[0] + ".o")
        objs.append(obj)
        cmd = [_nvcc(), "-c", os.path.join(CSRC, src), "-o", obj] + common
        procs.append((src, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
    failed = False
    for src, p in procs:
        out, _ = p.communicate()
        if p.returncode != 0 or verbose:
            sys.stderr.write(f"---- {src} ----\n{out}\n")
        failed |= p.returncode != 0
    if failed:
        raise RuntimeError("nvcc failed; see messages above")
    link(objs)
    build_calls()
    return OUT


def link(objs) -> None:
    # the soname is what the bindings ask for, and find beside themselves wherever the package lies; without one they
    # would ask for the path that it was built at
    subprocess.run([_nvcc(), "-shared", "-o", OUT] + objs + ARCH + ["-ccbin", "/usr/bin/g++", "-Xlinker",
                    "-soname=" + os.path.basename(OUT)], check=True)


def build_calls() -> str:
    subprocess.run(["/usr/bin/g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-I" + sysconfig.get_paths()["include"],
                    os.path.join(CSRC, "py_calls.cpp"), "-o", CALLS, OUT, "-Wl,-rpath,$ORIGIN"], check=True)
    return CALLS


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="--verbose" in sys.argv))
