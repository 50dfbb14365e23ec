"""Build the package's two shared objects in-tree (no JIT cache).

    python -m layer_quant_b200.build [--force]

``liblayer_quant_b200.so`` holds the kernels, compiled with nvcc for sm_100a behind a plain C ABI
(``include/layer_quant_b200.h``); it links the CUDA runtime statically and nothing else, so it loads with
``ctypes`` next to any PyTorch build.  ``_native.so`` is the Python module that reads torch tensors and calls that
library (``csrc/lq_torch.cpp``), compiled with g++ against the installed PyTorch's headers.
"""
from __future__ import annotations

import os
import shutil
import subprocess
import sys
import sysconfig
from concurrent.futures import ThreadPoolExecutor
from pathlib import Path

PKG = Path(__file__).resolve().parent
CSRC = PKG / "csrc"
LIB = PKG / "liblayer_quant_b200.so"
NATIVE = PKG / "_native.so"
NATIVE_SOURCE = CSRC / "lq_torch.cpp"
SOURCES = ["lq_api.cu", "lq_mx_state.cu", "lq_int4_kv.cu", "lq_dense_state.cu"]
NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC", "-Xcompiler", "-fvisibility=hidden",
]


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and Path(cand).exists():
            return cand
    raise RuntimeError("nvcc not found: the CUDA library cannot be built (there is no CPU fallback)")


def _sources() -> list[Path]:
    return [CSRC / s for s in SOURCES if (CSRC / s).exists()]


def needs_build() -> bool:
    if not LIB.exists():
        return True
    deps = list(CSRC.glob("*.cu")) + list(CSRC.glob("*.cuh")) + list(CSRC.glob("*.h"))
    deps.append(PKG.parent / "include" / "layer_quant_b200.h")
    return any(d.stat().st_mtime > LIB.stat().st_mtime for d in deps if d.exists())


def native_needs_build() -> bool:
    if not NATIVE.exists():
        return True
    deps = (NATIVE_SOURCE, PKG.parent / "include" / "layer_quant_b200.h")
    return any(d.stat().st_mtime > NATIVE.stat().st_mtime for d in deps)


def build_native() -> Path:
    import torch
    root = Path(torch.__file__).resolve().parent
    cuda = Path(_nvcc()).resolve().parent.parent
    tmp = NATIVE.with_suffix(".so.tmp")
    cmd = [os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden",
           f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
           "-isystem", str(root / "include"), "-isystem", str(root / "include/torch/csrc/api/include"),
           "-isystem", str(cuda / "include"), "-I", sysconfig.get_paths()["include"], str(NATIVE_SOURCE), "-o", str(tmp),
           "-L", str(root / "lib"), "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch_python", "-ldl"]
    res = subprocess.run(cmd, capture_output=True, text=True)
    if res.returncode != 0:
        raise RuntimeError(f"g++ failed for {NATIVE_SOURCE.name}:\n{res.stdout}\n{res.stderr}")
    os.replace(tmp, NATIVE)
    return NATIVE


def build(force: bool = False, verbose: bool = False) -> Path:
    if force or native_needs_build():
        build_native()
    if not force and not needs_build():
        return LIB
    nvcc = _nvcc()
    objdir = PKG / "build"
    objdir.mkdir(exist_ok=True)

    def compile_one(src: Path) -> Path:
        obj = objdir / (src.stem + ".o")
        cmd = [nvcc, *NVCC_FLAGS, "-c", str(src), "-o", str(obj)]
        if verbose:
            cmd.insert(1, "-Xptxas=-v")
        res = subprocess.run(cmd, capture_output=True, text=True)
        if res.returncode != 0:
            raise RuntimeError(f"nvcc failed for {src.name}:\n{res.stdout}\n{res.stderr}")
        if verbose:
            print(res.stderr)
        return obj

    with ThreadPoolExecutor(max_workers=4) as pool:
        objs = list(pool.map(compile_one, _sources()))
    tmp = LIB.with_suffix(".so.tmp")
    cmd = [nvcc, "-shared", "-gencode", "arch=compute_100a,code=sm_100a", "-o", str(tmp), *map(str, objs)]
    res = subprocess.run(cmd, capture_output=True, text=True)
    if res.returncode != 0:
        raise RuntimeError(f"link failed:\n{res.stdout}\n{res.stderr}")
    os.replace(tmp, LIB)
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
