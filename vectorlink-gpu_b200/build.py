"""Builds libvlgpu.so (the sm_100a kernels + C ABI) in-tree with nvcc.

    python vectorlink-gpu_b200/build.py [--force]

nvcc cross-compiles for sm_100a without a GPU.  The library lands beside the Python
package (vectorlink_gpu/libvlgpu.so), where the ctypes loader looks for it.
"""
from __future__ import annotations

import os
import subprocess
import sys
import tempfile
from concurrent.futures import ThreadPoolExecutor

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
INCLUDE = os.path.abspath(os.path.join(HERE, "..", "include"))
OUT = os.path.join(HERE, "vectorlink_gpu", "libvlgpu.so")
SOURCES = ["vl_api.cu", "vl_distance.cu", "vl_queue.cu", "vl_prune.cu", "vl_symmetrize.cu", "vl_components.cu", "vl_order.cu", "vl_beam.cu", "vl_beam_pair.cu", "vl_beam_solo.cu", "vl_beam_timed.cu", "vl_beam_team.cu", "vl_knn_tile.cu"]


def _stale() -> bool:
    if not os.path.exists(OUT):
        return True
    t = os.path.getmtime(OUT)
    deps = [os.path.join(CSRC, f) for f in os.listdir(CSRC)] + [os.path.join(INCLUDE, f) for f in os.listdir(INCLUDE)]
    return any(os.path.getmtime(d) > t for d in deps)


def build(force: bool = False, verbose: bool = False) -> str:
    if not force and not _stale():
        return OUT
    nvcc = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
    arch = [nvcc, "-gencode", "arch=compute_100a,code=sm_100a"]
    options = ["-lineinfo", "-O3", "-std=c++17", "-I", INCLUDE, "-Xcompiler", "-fPIC"] + (["-Xptxas", "-v"] if verbose else [])
    # one compiler per source, side by side: the beam search's files hold dozens of instantiations each
    with tempfile.TemporaryDirectory() as objects, ThreadPoolExecutor(os.cpu_count() or 1) as pool:
        def compile_one(source):
            out = os.path.join(objects, source + ".o")
            subprocess.check_call(arch + options + ["-c", "-o", out, os.path.join(CSRC, source)])
            return out

        subprocess.check_call(arch + ["-shared", "-Xcompiler", "-fPIC", "-o", OUT] + list(pool.map(compile_one, SOURCES)))
    return OUT


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
