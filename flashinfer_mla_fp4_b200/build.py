"""Build the two in-tree binaries: libmla_fp4_b200.so (nvcc, sm_100a: kernels and C ABI, no torch dependency) and
_native.so (g++: the native call path of the Python entry points, against torch's headers)."""
from __future__ import annotations

import os
import shutil
import subprocess
import sys
from pathlib import Path

PKG_DIR = Path(__file__).resolve().parent
CSRC = PKG_DIR / "csrc"
LIB_PATH = Path(os.environ.get("MLA_FP4_B200_LIB") or (PKG_DIR / "libmla_fp4_b200.so"))
SOURCES = ["abi.cu", "kernels_simt.cu", "combine.cu", "cache_write.cu", "cp_exchange.cu", "decode_sm100.cu"]
NATIVE_PATH = PKG_DIR / "_native.so"
NATIVE_SOURCE = CSRC / "py_native.cpp"
HEADERS = ["common.cuh", "decode_pair.cuh", "dequant.cuh", "launch.h", "ptx_sm100.cuh", "../../include/mla_fp4_b200.h"]


def _nvcc() -> str:
    cand = os.environ.get("NVCC") or shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not Path(cand).exists():
        raise RuntimeError("nvcc not found; set NVCC")
    return cand


def _native_command(out: Path) -> list:
    import sysconfig

    import torch

    base = Path(torch.__file__).resolve().parent
    cuda = Path(_nvcc()).resolve().parent.parent
    includes = [base / "include", base / "include/torch/csrc/api/include", cuda / "include", sysconfig.get_paths()["include"]]
    libs = ["c10", "c10_cuda", "torch_cpu", "torch_cuda", "torch_python"]
    return ([os.environ.get("CXX") or "g++", "-std=c++17", "-O2", "-fPIC", "-shared", "-fvisibility=hidden", "-DNDEBUG",
             f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}"]
            + [f"-isystem{i}" for i in includes] + [str(NATIVE_SOURCE), "-o", str(out), f"-L{base / 'lib'}"] + [f"-l{x}" for x in libs]
            + [f"-L{cuda / 'lib64'}", "-lcudart_static", "-lrt", "-ldl", "-lpthread"])


def native_needs_build() -> bool:
    deps = [NATIVE_SOURCE, PKG_DIR.parent / "include" / "mla_fp4_b200.h"]
    return not NATIVE_PATH.exists() or any(d.stat().st_mtime > NATIVE_PATH.stat().st_mtime for d in deps)


def needs_build() -> bool:
    if not LIB_PATH.exists():
        return True
    t = LIB_PATH.stat().st_mtime
    deps = [CSRC / s for s in SOURCES] + [(CSRC / h).resolve() for h in HEADERS] + [Path(__file__)]
    return any(d.stat().st_mtime > t for d in deps)


def build(force: bool = False, verbose: bool = False) -> Path:
    """Compile every CUDA source for sm_100a into one shared library next to this file, and the native call path."""
    native = None
    if force or native_needs_build():  # runs beside the CUDA compilation
        native = subprocess.Popen(_native_command(NATIVE_PATH.with_suffix(".tmp")), stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
    try:
        if force or needs_build():
            _build_library(verbose)
    finally:
        if native is not None:
            out, _ = native.communicate()
    if native is not None:
        if native.returncode != 0:
            sys.stderr.write(f"--- {NATIVE_SOURCE.name}\n{out}\n")
            raise RuntimeError("the native call path failed to compile")
        os.replace(NATIVE_PATH.with_suffix(".tmp"), NATIVE_PATH)
    return LIB_PATH


def _build_library(verbose: bool) -> None:
    objs = []
    build_dir = PKG_DIR / "build"
    build_dir.mkdir(exist_ok=True)
    common = [
        _nvcc(), "-std=c++17", "-O3", "-lineinfo",
        "-gencode", "arch=compute_100a,code=sm_100a",
        "-Xcompiler", "-fPIC", "-Xptxas", "-v" if verbose else "-O3",
        "--expt-relaxed-constexpr",
    ] + os.environ.get("MLA_FP4_NVCC_FLAGS", "").split()
    procs = []
    for s in SOURCES:
        o = build_dir / (s + ".o")
        objs.append(str(o))
        procs.append((s, subprocess.Popen(common + ["-c", str(CSRC / s), "-o", str(o)],
                                          stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
    failed = False
    for s, p in procs:
        out, _ = p.communicate()
        if verbose or p.returncode != 0:
            sys.stderr.write(f"--- nvcc {s}\n{out}\n")
        failed |= p.returncode != 0
    if failed:
        raise RuntimeError("nvcc failed")
    link = [_nvcc(), "-shared", "-o", str(LIB_PATH)] + objs + ["-cudart", "static"]
    r = subprocess.run(link, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
    if r.returncode != 0:
        sys.stderr.write(r.stdout)
        raise RuntimeError("link failed")


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
