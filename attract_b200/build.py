"""Build ``libattract_b200.so`` in-tree with nvcc for sm_100a.

    python -m attract_b200.build [--force] [--checked]

``--checked`` builds ``libattract_b200_checked.so`` with -DATT_BOUNDS_CHECK:
every computed grid, list and receptor index of the scoring kernels is
checked before its access; a failed check skips the access and records
(check code, index, bound) for att_kernel_debug_info.  Load it with
$ATTRACT_B200_LIB (the tests do).
"""
from __future__ import annotations

import os
import subprocess
import sys
import tempfile
from concurrent.futures import ThreadPoolExecutor

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
# (source, further flags): score.cu is compiled in four parts of a few modes
# each, in parallel (one part takes a minute, the whole would take four; one
# compilation with --split-compile spills more: 132 bytes in the 32-lane
# minimiser where a plain one spills none)
UNITS = [("score.cu", [f"-DATT_SCORE_PART={i}"]) for i in range(4)] + [
    (s, []) for s in ("launch.cu", "build.cu", "allpairs.cu", "capi.cu")]
OUT = os.path.join(HERE, "libattract_b200.so")
OUT_CHECKED = os.path.join(HERE, "libattract_b200_checked.so")
ARCH = ["-gencode", "arch=compute_100a,code=sm_100a"]
FLAGS = ["-O3", "-lineinfo", "-std=c++17", "-Xcompiler", "-fPIC", "--expt-relaxed-constexpr"]


def _inputs():
    csrc = os.path.join(HERE, "csrc")
    return sorted({os.path.join(csrc, s) for s, _ in UNITS}) + [
        os.path.join(csrc, "common.cuh"), os.path.join(csrc, "score_parts.h"),
        os.path.join(ROOT, "include", "attract_b200.h")]


def needs_build() -> bool:
    if not os.path.exists(OUT):
        return True
    t = os.path.getmtime(OUT)
    return any(os.path.getmtime(d) > t for d in _inputs())


def needs_build_checked() -> bool:
    if not os.path.exists(OUT_CHECKED):
        return True
    t = os.path.getmtime(OUT_CHECKED)
    return any(os.path.getmtime(d) > t for d in _inputs())


def build(force: bool = False, verbose: bool = False, checked: bool = False) -> str:
    """Compile the CUDA sources into the package directory; returns the .so path."""
    out = OUT_CHECKED if checked else OUT
    if not force and not (needs_build_checked() if checked else needs_build()):
        return out
    nvcc = os.environ.get("NVCC", "nvcc")
    base = [nvcc, *(["-Xptxas=-v"] if verbose else []), *ARCH, *FLAGS, *(["-DATT_BOUNDS_CHECK"] if checked else []),
            "-I", os.path.join(ROOT, "include")]
    with tempfile.TemporaryDirectory() as d:
        def compile_unit(i):
            src, flags = UNITS[i]
            obj = os.path.join(d, f"{i}.o")
            subprocess.run([*base, *flags, "-c", os.path.join(HERE, "csrc", src), "-o", obj], check=True)
            return obj

        with ThreadPoolExecutor(min(len(UNITS), os.cpu_count() or 1)) as ex:
            objs = list(ex.map(compile_unit, range(len(UNITS))))
        tmp = out + ".tmp"
        subprocess.run([nvcc, *ARCH, "-shared", *objs, "-o", tmp], check=True)
    os.replace(tmp, out)
    return out


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv, checked="--checked" in sys.argv))
