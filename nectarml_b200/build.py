"""In-tree build of the CUDA library (nvcc, sm_100a only).

``python -m nectarml_b200.build`` compiles ``csrc/nml_api.cu`` (which includes the contraction
kernels) and ``csrc/nml_layers.cu`` (normalisation / optimizer kernels of the training step) into ``nectarml_b200/libnectarml_b200.so``,
``csrc/nml_torch.cpp`` (the tensor-level host path on top of that library's C ABI) into ``nectarml_b200/_native.so``, and
``csrc/nml_dropin.cpp`` (the drop-in's calls of the same ABI) into ``nectarml_b200/_dropin.so``.
nvcc cross-compiles without a GPU.
"""
from __future__ import annotations

import os
import subprocess
import sys
import sysconfig

_HERE = os.path.dirname(os.path.abspath(__file__))
SOURCES = [os.path.join(_HERE, "csrc", "nml_api.cu"), os.path.join(_HERE, "csrc", "nml_layers.cu")]
HEADERS = [os.path.join(_HERE, "csrc", n) for n in ("nml_launch.cuh", "nml_ptx.cuh", "nml_umma.cuh", "nml_prepass.cuh", "nml_gemm.cuh")] + [
    os.path.join(os.path.dirname(_HERE), "include", "nectarml_b200.h")]
OUTPUT = os.path.join(_HERE, "libnectarml_b200.so")
NATIVE_SOURCE = os.path.join(_HERE, "csrc", "nml_torch.cpp")
NATIVE_OUTPUT = os.path.join(_HERE, "_native.so")
DROPIN_SOURCE = os.path.join(_HERE, "csrc", "nml_dropin.cpp")
DROPIN_OUTPUT = os.path.join(_HERE, "_dropin.so")

NVCC_FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
              "-shared", "-Xcompiler", "-fPIC"]


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), "/usr/local/cuda/bin/nvcc", "nvcc"):
        if cand and (os.path.sep not in cand or os.path.exists(cand)):
            return cand
    raise RuntimeError("nvcc not found")


def _fresh(output: str, sources) -> bool:
    if not os.path.exists(output):
        return False
    t = os.path.getmtime(output)
    return all(os.path.getmtime(p) <= t for p in sources)


def up_to_date() -> bool:
    return (_fresh(OUTPUT, SOURCES + HEADERS) and _fresh(NATIVE_OUTPUT, [NATIVE_SOURCE, HEADERS[-1]]) and
            _fresh(DROPIN_OUTPUT, [DROPIN_SOURCE, HEADERS[-1]]))


def _native_command():
    import torch
    root = os.path.dirname(torch.__file__)
    nvcc = _nvcc()
    cuda = os.path.dirname(os.path.dirname(nvcc)) if os.path.sep in nvcc else "/usr/local/cuda"
    inc = [sysconfig.get_paths()["include"], os.path.join(root, "include"),
           os.path.join(root, "include", "torch", "csrc", "api", "include"), os.path.join(cuda, "include")]
    return ["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-fvisibility=hidden",
            f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}"] + [f"-I{d}" for d in inc] + [
        NATIVE_SOURCE, "-o", NATIVE_OUTPUT, f"-L{_HERE}", "-l:libnectarml_b200.so", "-Wl,-rpath,$ORIGIN",
        f"-L{os.path.join(root, 'lib')}", "-ltorch_python", "-ltorch_cpu", "-lc10_cuda", "-lc10"]


def _dropin_command():
    return ["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-fvisibility=hidden", f"-I{sysconfig.get_paths()['include']}", DROPIN_SOURCE,
            "-o", DROPIN_OUTPUT, f"-L{_HERE}", "-l:libnectarml_b200.so", "-Wl,-rpath,$ORIGIN"]


def _run(cmd, verbose: bool) -> None:
    res = subprocess.run(cmd, capture_output=True, text=True)
    if verbose or res.returncode != 0:
        sys.stderr.write(res.stdout + res.stderr)
    if res.returncode != 0:
        raise RuntimeError("build failed: " + " ".join(cmd))


def build(force: bool = False, verbose: bool = False) -> str:
    """Builds the library and the two modules on top of it where their sources are newer; returns the library's path."""
    if force or not _fresh(OUTPUT, SOURCES + HEADERS):
        _run([_nvcc()] + NVCC_FLAGS + (["-Xptxas", "-v"] if verbose else []) + ["-o", OUTPUT] + SOURCES, verbose)
    if force or not _fresh(NATIVE_OUTPUT, [NATIVE_SOURCE, HEADERS[-1]]):
        _run(_native_command(), verbose)
    if force or not _fresh(DROPIN_OUTPUT, [DROPIN_SOURCE, HEADERS[-1]]):
        _run(_dropin_command(), verbose)
    return OUTPUT


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
