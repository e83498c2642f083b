"""Build the sm_100a shared library ``maddening_b200/liblbm_b200.so`` in-tree.

    python -m maddening_b200.build [--verbose]

The library is a plain C ABI (``include/lbm_b200.h``) compiled by nvcc with
the CUDA runtime linked statically, so it loads next to any torch build.  Its
translation units compile in parallel, then link into the one library.  A
build is skipped only when the library's recorded input digest (sources,
headers, flags, nvcc version) equals the current one, so a library built from
other sources is always rebuilt, whatever its timestamps.
"""

from __future__ import annotations

import hashlib
import os
import shutil
import subprocess
import sys
from concurrent.futures import ThreadPoolExecutor
from pathlib import Path

PKG = Path(__file__).resolve().parent
ROOT = PKG.parent
CSRC = PKG / "csrc"
LIB = PKG / "liblbm_b200.so"
DIGEST = PKG / "liblbm_b200.so.sha256"
SOURCES = ["lbm_abi.cu", "lbm_steps.cu", "lbm_batch.cu", "lbm_tiled.cu", "lbm_grad.cu",
           "lbm_pipe.cu"]
HEADERS = ["lbm_host.h", "lbm_kernels.cuh", "lbm_lattice.cuh", "lbm_adjoint.cuh",
           "lbm_staged.cuh", "lbm_tiled.cuh", "lbm_pair.cuh", "lbm_pipe.cuh",
           "lbm_multiphase.cuh", "lbm_pack.cuh"]

ARCH = ["-gencode", "arch=compute_100a,code=sm_100a"]
CFLAGS = ["-O3", "-lineinfo", "-std=c++17", "--expt-relaxed-constexpr",
          "-Xcompiler", "-fPIC,-O3", "-Xfatbin", "-compress-all"]
# Units: (source, object name, definitions).  The step kernels are compiled once
# per lattice and storage, side by side, and each unit as a whole: a split
# compile of one large unit gave code that differed from build to build, with
# the way the unit happened to be divided (builds of one k_tiled source ran a
# 256^3 update in 0.62 or 0.68 ms, and in 0.60 compiled whole).
_STORES = {"f32": "float", "f16": "__half", "bf16": "__nv_bfloat16", "f64": "double"}


def units():
    out = []
    for src, stores in (("lbm_steps.cu", _STORES), ("lbm_batch.cu", _STORES),
                        ("lbm_tiled.cu", ("f16", "bf16", "f32"))):
        for q in (19, 9):
            for st in stores:
                out.append((src, f"{Path(src).stem}_{q}_{st}",
                            [f"-DLBM_UNIT_Q={q}", f"-DLBM_UNIT_S={_STORES[st]}"]))
    return out + [(s, Path(s).stem, []) for s in ("lbm_grad.cu", "lbm_pipe.cu", "lbm_abi.cu")]


LFLAGS = ["-shared", "-cudart", "static"]


def nvcc() -> str:
    cand = os.environ.get("NVCC") or shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not Path(cand).exists():
        raise RuntimeError("nvcc not found (set NVCC or put CUDA on PATH)")
    return cand


def _inputs():
    files = [CSRC / s for s in SOURCES] + [CSRC / h for h in HEADERS]
    files.append(ROOT / "include" / "lbm_b200.h")
    files.append(Path(__file__))
    return files


def input_digest() -> str:
    h = hashlib.sha256()
    for f in _inputs():
        h.update(f.name.encode())
        h.update(f.read_bytes())
    h.update(" ".join(ARCH + CFLAGS + LFLAGS).encode())
    h.update(repr(units()).encode())
    try:
        h.update(subprocess.run([nvcc(), "--version"], capture_output=True,
                                text=True).stdout.encode())
    except (RuntimeError, OSError):
        pass
    return h.hexdigest()


def up_to_date() -> bool:
    return LIB.exists() and DIGEST.exists() and DIGEST.read_text().strip() == input_digest()


def build(verbose: bool = False, force: bool = False) -> Path:
    if not force and up_to_date():
        return LIB
    digest = input_digest()
    objdir = PKG / "_build"
    objdir.mkdir(exist_ok=True)

    def compile_unit(unit):
        src, name, defs = unit
        obj = objdir / (name + ".o")
        cmd = [nvcc(), *ARCH, *CFLAGS, *defs, "-I", str(ROOT / "include"), "-c",
               str(CSRC / src), "-o", str(obj)]
        if verbose:
            cmd.insert(1, "-Xptxas=-v")
        res = subprocess.run(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
        return obj, " ".join(cmd), res

    with ThreadPoolExecutor(max_workers=max(1, os.cpu_count() or 1)) as pool:
        done = list(pool.map(compile_unit, units()))
    failed = False
    for _obj, cmd, res in done:
        if verbose:
            print(cmd, flush=True)
        if verbose or res.returncode != 0:
            sys.stdout.write(res.stdout)
        failed |= res.returncode != 0
    if failed:
        raise RuntimeError("nvcc failed")
    cmd = [nvcc(), *ARCH, *LFLAGS, *(str(d[0]) for d in done), "-o", str(LIB) + ".tmp"]
    res = subprocess.run(cmd, capture_output=True, text=True)
    if res.returncode != 0:
        sys.stderr.write(res.stdout + res.stderr)
        raise RuntimeError(f"nvcc link failed ({res.returncode})")
    os.replace(str(LIB) + ".tmp", LIB)
    DIGEST.write_text(digest + "\n")
    return LIB


if __name__ == "__main__":
    build(verbose="--verbose" in sys.argv, force=True)
    print(LIB)
