"""Build the sm_100a shared library in-tree with nvcc.

The library is a plain C-ABI ``.so`` (no torch headers); it is compiled next to
its sources so that it travels with the source tree.  ``build()`` is idempotent:
it recompiles only when a source file is newer than the library.
"""
from __future__ import annotations

import os
import shutil
import subprocess
import tempfile
from concurrent.futures import ThreadPoolExecutor
from pathlib import Path

CSRC = Path(__file__).resolve().parent / "csrc"
LIBRARY = CSRC / "libi8muon_b200.so"
SOURCES = ("ns_api.cu", "api_float.cu", "api_int8.cu", "api_bq.cu", "api_passes.cu")
NVCC_FLAGS = (
    "-std=c++17", "-O3", "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo",
    # FP32 expressions are evaluated exactly as written; fused multiply-adds
    # appear only where the code asks for them.
    "--fmad=false", "-Xcompiler", "-fPIC",
)


def _nvcc() -> str:
    found = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not Path(found).exists():
        raise RuntimeError("nvcc not found; the sm_100a library cannot be built")
    return found


def needs_build() -> bool:
    if not LIBRARY.exists():
        return True
    built = LIBRARY.stat().st_mtime
    header = Path(__file__).resolve().parents[1] / "include" / "i8muon_b200.h"
    deps = [*CSRC.glob("*.cu"), *CSRC.glob("*.cuh"), header]
    return any(dep.stat().st_mtime > built for dep in deps)


def _compile(source: str, output: Path, verbose: bool) -> str:
    command = [_nvcc(), *NVCC_FLAGS, *(["-Xptxas=-v"] if verbose else []), "-c", "-o", str(output), str(CSRC / source)]
    result = subprocess.run(command, capture_output=True, text=True)
    if result.returncode != 0:
        raise RuntimeError(f"nvcc failed on {source}:\n{result.stdout}\n{result.stderr}")
    return " ".join(command) + "\n" + result.stderr


def build(force: bool = False, verbose: bool = False) -> Path:
    """Compile ``csrc/*.cu`` (one nvcc process per file, in parallel) into ``csrc/libi8muon_b200.so`` for sm_100a."""
    if not force and not needs_build():
        return LIBRARY
    verbose = verbose or os.environ.get("I8MUON_BUILD_VERBOSE", "0") not in ("", "0")
    with tempfile.TemporaryDirectory() as work, ThreadPoolExecutor(len(SOURCES)) as pool:
        objects = [Path(work) / (source + ".o") for source in SOURCES]
        logs = list(pool.map(_compile, SOURCES, objects, [verbose] * len(SOURCES)))
        link = [_nvcc(), *NVCC_FLAGS, "-shared", "-o", str(LIBRARY), *map(str, objects)]
        result = subprocess.run(link, capture_output=True, text=True)
    if result.returncode != 0:
        raise RuntimeError(f"linking failed:\n{result.stdout}\n{result.stderr}")
    if verbose:
        print("\n".join(logs))
    return LIBRARY


if __name__ == "__main__":
    print(build(force=True, verbose=True))
