"""Builds the CUDA libraries in place with nvcc for sm_100a: `python -m flaggems_vllm.build`.

  libdsv4_prologue.so            the operators (the product)
  _host_calls.so                 native front ends of the Python operators (CPython extension, plain C++ against torch)
  testing/libdsv4_hbm_probe.so   aids: the bandwidth probe the benchmark compares the kernels with, and the on-device
                                 check of the quantisers' division shortcut that a test runs

Cross-compiles without a GPU.  The CUDA runtime is linked statically so the libraries
load (and export their symbols) on a machine that has no driver.
"""
from __future__ import annotations

import os
import shutil
import subprocess
import sys
import sysconfig
from pathlib import Path

PKG = Path(__file__).resolve().parent
CSRC = PKG.parent / "csrc"
OUT = PKG / "libdsv4_prologue.so"
PROBE_OUT = PKG / "testing" / "libdsv4_hbm_probe.so"
HOST_OUT = PKG / "_host_calls.so"
HOST_SOURCES = ("host_calls.cpp",)
PROBE_SOURCES = ("hbm_probe.cu", "division_probe.cu")
SOURCES = ("abi.cu", "prologue_rows.cu", "prologue_bulk.cu", "gather_dequant.cu", "q_kv_rmsnorm.cu", "inv_rope_fp8_quant.cu", "indexer_k_quant.cu",
           "indexer_q_rope_quant.cu", "cp_gather_indexer.cu", "topk_indices.cu", "topk_per_row.cu", "group_quant_fp8.cu")
HEADERS = ("dsv4_common.cuh", "current_device.h", "../../include/dsv4_prologue.h", "../../include/dsv4_hbm_probe.h")


def nvcc_path() -> str:
    exe = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not Path(exe).exists():
        raise RuntimeError("nvcc not found; it is required to build libdsv4_prologue.so")
    return exe


def command(extra_flags=(), out: Path = OUT, sources=SOURCES) -> list[str]:
    return [
        nvcc_path(), "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
        "-Xcompiler", "-fPIC", "-shared", "-cudart", "static", *extra_flags,
        "-o", str(out), *[str(CSRC / s) for s in sources],
    ]


def built_for() -> str:
    """What the extension module depends on besides its sources: the interpreter and torch, whose C++ interface it calls."""
    import torch

    return f"dsv4-built-for:{sys.implementation.cache_tag}:torch-{torch.__version__};"


def host_command(out: Path = HOST_OUT) -> list[str]:
    """g++ command of the extension module: linked against the operator library beside it (found at load time through
    $ORIGIN) and against torch's libraries, which the interpreter has loaded by then."""
    import torch

    root = Path(torch.__file__).resolve().parent
    cuda = Path(nvcc_path()).resolve().parent.parent
    includes = (root / "include", root / "include/torch/csrc/api/include", cuda / "include", sysconfig.get_paths()["include"])
    return [
        shutil.which("g++") or "g++", f'-DDSV4_BUILT_FOR="{built_for()}"', "-O2", "-std=c++17", "-fPIC", "-shared", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch.compiled_with_cxx11_abi())}",
        *[f"-I{i}" for i in includes], *[str(CSRC / s) for s in HOST_SOURCES], "-o", str(out),
        f"-L{OUT.parent}", f"-l:{OUT.name}", f"-L{root / 'lib'}", "-ltorch_python", "-ltorch_cuda", "-ltorch_cpu", "-lc10_cuda", "-lc10",
        "-Wl,-rpath,$ORIGIN",
    ]


def up_to_date(out: Path = OUT, sources=SOURCES) -> bool:
    if not out.exists():
        return False
    if out == HOST_OUT and built_for().encode() not in out.read_bytes():
        return False  # built for another torch: its symbols need not be there any more
    newest = max((CSRC / f).resolve().stat().st_mtime for f in tuple(sources) + HEADERS)
    return out.stat().st_mtime >= newest


def build(force: bool = False, verbose: bool = False, extra_flags=()) -> Path:
    """Build whichever of the libraries is older than its sources; returns the operator library's path."""
    env = dict(os.environ)
    env.pop("CC", None), env.pop("CXX", None)  # let nvcc pick the system host compiler
    for out, sources in ((OUT, SOURCES), (HOST_OUT, HOST_SOURCES), (PROBE_OUT, PROBE_SOURCES)):
        if not force and up_to_date(out, sources):
            continue
        cmd = host_command(out) if out == HOST_OUT else command(extra_flags, out, sources)
        res = subprocess.run(cmd, capture_output=True, text=True, env=env)
        if verbose or res.returncode != 0:
            sys.stderr.write(" ".join(cmd) + "\n" + res.stdout + res.stderr)
        if res.returncode != 0:
            raise RuntimeError(f"{Path(cmd[0]).name} failed building {out.name}")
    return OUT


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose=True,
                extra_flags=("-Xptxas", "-v") if "--ptxas" in sys.argv else ()))
