"""Builds the gtd shared library (libgtd.so) for sm_103a, in-tree.

Every translation unit under csrc/ is compiled by nvcc in parallel with
``-gencode arch=compute_103a,code=sm_103a`` and linked into
``gisbdw_gb300/_build/libgtd.so`` (cudart linked statically, so the library
only needs the driver at run time). gtd_pack.c, the batch packer over Python
edge lists, becomes a library of its own next to it, for the interpreter that
builds it; without a C compiler or the Python headers the package does without.
"""
from __future__ import annotations

import glob
import os
import subprocess
import sys
import sysconfig
from concurrent.futures import ThreadPoolExecutor
from typing import Optional

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
OUT_DIR = os.path.join(HERE, "_build")
LIB = os.path.join(OUT_DIR, "libgtd.so")
# edge lists to masks: reads CPython's objects, so one file per interpreter
PACK_LIB = os.path.join(OUT_DIR, "libgtdpack" + (sysconfig.get_config_var("EXT_SUFFIX") or ".so"))
PACK_SRC = os.path.join(CSRC, "gtd_pack.c")
INCLUDE = os.path.join(os.path.dirname(HERE), "include")

ARCH = ["-gencode", "arch=compute_103a,code=sm_103a"]
NVCC_FLAGS = ["-std=c++17", "-O3", "-lineinfo", "-Xcompiler", "-fPIC,-O2,-ffp-contract=off",
              "--expt-relaxed-constexpr", "-I" + INCLUDE, "-I" + CSRC] + ARCH


def nvcc() -> str:
    for c in (os.environ.get("NVCC"), "/usr/local/cuda/bin/nvcc", "nvcc"):
        if c and (os.path.sep not in c or os.path.exists(c)):
            return c
    return "nvcc"


def _compile(src: str, verbose: bool) -> str:
    obj = os.path.join(OUT_DIR, os.path.basename(src) + ".o")
    cmd = [nvcc()] + NVCC_FLAGS + ["-c", src, "-o", obj]
    if verbose:
        cmd.insert(1, "-Xptxas=-v")
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"nvcc failed on {src}:\n{r.stderr}")
    if verbose and r.stderr:
        sys.stderr.write(r.stderr)
    return obj


def _compile_pack() -> bool:
    tmp = PACK_LIB + ".tmp"
    cmd = ["gcc", "-O2", "-fPIC", "-shared", "-I" + sysconfig.get_paths()["include"], PACK_SRC, "-o", tmp]
    try:
        done = subprocess.run(cmd, capture_output=True, text=True).returncode == 0
    except OSError:
        done = False
    if done:
        os.replace(tmp, PACK_LIB)
    elif os.path.exists(PACK_LIB):
        os.remove(PACK_LIB)  # of an older source
    return done


def pack_library() -> Optional[str]:
    """The batch packer's library, compiled when it is missing or stale; None
    where it cannot be."""
    if not _newer(PACK_LIB, [PACK_SRC, __file__]) and not _compile_pack():
        return None
    return PACK_LIB


def sources():
    return sorted(glob.glob(os.path.join(CSRC, "*.cu")))


def _newer(lib: str, deps) -> bool:
    return os.path.exists(lib) and all(os.path.getmtime(d) <= os.path.getmtime(lib) for d in deps)


def up_to_date() -> bool:
    deps = sources() + glob.glob(os.path.join(CSRC, "*.h")) + glob.glob(os.path.join(CSRC, "*.cuh"))
    return _newer(LIB, deps + glob.glob(os.path.join(INCLUDE, "*.h")) + [__file__])


def build(force: bool = False, verbose: bool = False) -> str:
    if not force and up_to_date():
        return LIB
    os.makedirs(OUT_DIR, exist_ok=True)
    srcs = sources()
    with ThreadPoolExecutor(max_workers=max(1, min(len(srcs), os.cpu_count() or 4))) as ex:
        pack = ex.submit(_compile_pack)
        objs = list(ex.map(lambda s: _compile(s, verbose), srcs))
        if not pack.result():
            sys.stderr.write("gtd_pack.c not compiled (gcc or Python headers missing): batches are packed in Python\n")
    tmp = LIB + ".tmp"
    cmd = [nvcc()] + ARCH + ["-shared", "-o", tmp] + objs + ["-lpthread", "-ldl", "-lrt"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"link failed:\n{r.stderr}")
    os.replace(tmp, LIB)
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
