"""Builds libflashoptim_b200.so in-tree with nvcc for sm_100a, and the host extension over it.

The step-kernel family is split into instantiation slices (optimizer x state kind x kernel)
compiled from one source with different -D switches, so the build runs in parallel.
Objects go to csrc/build/, the library to lib/.  Nothing is compiled at import time:
call build_native() and build_host() (or `python -m flashoptim_jax_b200.build`, which does both).
"""

from __future__ import annotations

import concurrent.futures
import hashlib
import os
import shutil
import subprocess
import sys
from typing import List, Tuple

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
OBJ_DIR = os.path.join(CSRC, "build")
LIB_DIR = os.path.join(HERE, "lib")
LIB_PATH = os.path.join(LIB_DIR, "libflashoptim_b200.so")
HOST_PATH = os.path.join(HERE, "_fo_host.so")  # the host side (csrc/fo_host.cc): a Python extension over torch's C++ tensors

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-lineinfo", "-O3", "-std=c++17",
    "-fmad=false",  # a*b+c never contracts; the explicit __fmaf_rn calls stay FMAs
    "--ftz=false", "--prec-div=true", "--prec-sqrt=true",
    "-Xcompiler", "-fPIC,-ffp-contract=off,-O2",
]

# (object name, source, extra defines)
_OPTS = (("adam", "FO_OPT_ADAM"), ("lion", "FO_OPT_LION"), ("sgd", "FO_OPT_SGD"))
_KINDS = (("quant", 0), ("full", 1), ("generic", 3))


# Block shape of a slice: (threads per block, resident blocks per SM).  Measured on B200: the
# Adam kernels run best as one 512-thread block per SM (all warps of an SM share one instruction
# stream and one set of tables); the kernels that also read peers' gradients keep 256-thread blocks,
# whose smaller stages leave room for a deeper copy pipeline.
# "tile": the slices that run tile_kernel (quantized moments, one feature at most), one block per SM.  The 16 elements of a lane want 150 to
# 168 registers under AdamW (2^28 elements, 24-bit masters: 564 us with 384 threads, 585 with 512; with the power cap reached
# 650 and 666; clipping 602 and 714) and 138 under SGD (65 M elements, 32-bit masters, results elsewhere: 129 us with 384 threads, 143 with 512, 132 with 256);
# Lion fits 512 (2^28 elements at the cap, 24-bit masters: bf16 445 us, 462 with 384; fp16 479 and 493).
_SHAPES = {("adam", "plain"): (512, 1), ("adam", "clip"): (512, 1), ("adam", "out"): (512, 1),
           ("adam", "delta"): (512, 1), ("adam", "all"): (384, 1), ("adam", "group8"): (512, 1), ("adam", "tile"): (384, 1),
           ("lion", "plain"): (768, 1), ("lion", "clip"): (512, 1), ("lion", "out"): (512, 1), ("lion", "all"): (512, 1), ("lion", "group8"): (512, 1),
           ("lion", "tile"): (512, 1),
           ("sgd", "clip"): (512, 1), ("sgd", "out"): (512, 1), ("sgd", "all"): (512, 1), ("sgd", "group8"): (512, 1), ("sgd", "tile"): (384, 1)}
_TILE_MODES = ("plain", "clip", "out", "group", "delta")
# Name and feature mask (fo_step.cuh) of the kernels of a slice.  Groups of 8, two to a tile's lane, go through step_kernel (one of their own: AdamW
# 4096 x 4096 49 us, through the kernel that carries all features 59; Lion 32.9 and 34.8, SGDW 31.9 and 33.3).
_MODES = (("plain", 0), ("clip", 1), ("out", 2), ("group", 4), ("group8", 4), ("delta", 8), ("all", 15), ("peer", 16), ("piece", -1))


def _has_kernel(oname: str, kname: str, mname: str) -> bool:
    """Group sizes concern quantized moments only, the parameter hand-back Adam only."""
    return not (mname.startswith("group") and kname != "quant") and not (mname == "delta" and oname != "adam")


def _units(shapes=None, ffi_dir: str | None = None) -> List[Tuple[str, str, List[str]]]:
    shapes = _SHAPES if shapes is None else shapes
    units = [(name, name + ".cu", []) for name in ("fo_api", "fo_codec", "fo_selftest", "fo_norm")]
    if ffi_dir is not None:
        units.append(("fo_ffi", "fo_ffi.cc", ["-x", "cu", f"-I{ffi_dir}"]))

    def step_unit(oname: str, omacro: str, kname: str, kind: int, mname: str, mode: int):
        suffix = f"_{mname}" if mname else ""
        flags = [f"-DFO_INST_OPT={omacro}", f"-DFO_INST_KIND={kind}", f"-DFO_INST_MODE={mode}",
                 f"-DFO_INST_NAME=lookup_{oname}_{kname}{suffix}"]
        tiles = kind == 0 and mname in _TILE_MODES
        if tiles:
            flags.append("-DFO_INST_TILES")
        shape = shapes.get((oname, "tile" if tiles else mname))
        if shape is not None and kind != 3:
            flags += [f"-DFO_THREADS={shape[0]}", f"-DFO_MIN_BLOCKS_ADAM={shape[1]}", f"-DFO_MIN_BLOCKS_MOMENTUM={shape[1]}"]
            if len(shape) > 2:
                flags.append(f"-DFO_PLAIN_STAGES={shape[2]}")
            flags.append("-DFO_SHAPE_NS=shape_" + "_".join(str(x) for x in shape))
        units.append((f"fo_step_{oname}_{kname}{suffix}", "fo_step_inst.cu", flags))

    for oname, omacro in _OPTS:
        for kname, kind in _KINDS:
            if kind == 3:
                step_unit(oname, omacro, kname, kind, "", 1)
            else:
                for mname, mode in _MODES:
                    if _has_kernel(oname, kname, mname):
                        step_unit(oname, omacro, kname, kind, mname, mode)
    for mname, mode in _MODES:
        if _has_kernel("sgd", "none", mname):
            step_unit("sgd", "FO_OPT_SGD", "none", 2, mname, mode)
    return units


def ffi_include_dir() -> str | None:
    """Directory of jaxlib's XLA FFI headers (xla/ffi/api/ffi.h), or None when jax is not installed.
    The jax.ffi shim (csrc/fo_ffi.cc) is compiled into the library only when this resolves."""
    try:
        import jax.ffi  # noqa: PLC0415

        path = jax.ffi.include_dir()
    except Exception:  # jax absent, or too old to have jax.ffi
        return None
    return path if os.path.exists(os.path.join(path, "xla", "ffi", "api", "ffi.h")) else None


def _nvcc() -> str:
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        raise RuntimeError("nvcc not found; the CUDA toolkit is required to build libflashoptim_b200.so")
    return nvcc


def _sources_digest(extra: List[str], units=None) -> str:
    h = hashlib.sha256()
    for root in (CSRC, os.path.join(os.path.dirname(HERE), "include")):
        for name in sorted(os.listdir(root)):
            if name.endswith((".cu", ".cuh", ".h", ".cc")):
                with open(os.path.join(root, name), "rb") as f:
                    h.update(name.encode())
                    h.update(f.read())
    h.update(" ".join(NVCC_FLAGS + extra).encode())
    h.update(repr(units if units is not None else _units()).encode())
    return h.hexdigest()


def build_native(force: bool = False, jobs: int | None = None, extra_flags: List[str] | None = None,
                 lib_path: str = LIB_PATH, verbose: bool = False, shapes=None) -> str:
    """Compile every CUDA source for sm_100a and link the shared object; returns its path.
    `shapes` takes the place of _SHAPES, the block shapes of the step slices; where it names none the default of fo_step.cuh holds."""
    extra = list(extra_flags or [])
    units = _units(shapes, ffi_include_dir())
    os.makedirs(OBJ_DIR, exist_ok=True)
    os.makedirs(os.path.dirname(lib_path), exist_ok=True)
    stamp = lib_path + ".digest"
    digest = _sources_digest(extra, units)
    if not force and os.path.exists(lib_path) and os.path.exists(stamp) and open(stamp).read() == digest:
        return lib_path
    nvcc = _nvcc()
    tag = hashlib.sha256((" ".join(extra) + repr(shapes)).encode()).hexdigest()[:8] if (extra or shapes is not None) else "std"

    def compile_one(unit):
        name, src, defs = unit
        obj = os.path.join(OBJ_DIR, f"{name}.{tag}.o")
        cmd = [nvcc, *NVCC_FLAGS, *extra, *defs, "-c", os.path.join(CSRC, src), "-o", obj]
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError(f"nvcc failed for {name}:\n{' '.join(cmd)}\n{r.stdout}\n{r.stderr}")
        if verbose and (r.stdout or r.stderr):
            print(f"[{name}]\n{r.stdout}{r.stderr}")
        return obj

    jobs = jobs or max(1, min(len(units), os.cpu_count() or 1))
    with concurrent.futures.ThreadPoolExecutor(max_workers=jobs) as pool:
        objs = list(pool.map(compile_one, units))
    cmd = [nvcc, "-shared", "-gencode", "arch=compute_100a,code=sm_100a", "-o", lib_path, *objs, "-lcudart"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"link failed:\n{' '.join(cmd)}\n{r.stdout}\n{r.stderr}")
    with open(stamp, "w") as f:
        f.write(digest)
    return lib_path


def build_host(force: bool = False) -> str:
    """Compile the extension module flashoptim_jax_b200._fo_host with the host compiler; returns its path."""
    import sysconfig

    import torch
    from torch.utils.cpp_extension import include_paths

    source = os.path.join(CSRC, "fo_host.cc")
    libs = os.path.join(os.path.dirname(torch.__file__), "lib")
    dirs = [*include_paths(), sysconfig.get_paths()["include"], os.path.join(os.path.dirname(os.path.dirname(_nvcc())), "include")]
    cmd = ["g++", "-O2", "-std=c++17", "-fPIC", "-shared", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
           *[f"-I{d}" for d in dirs], source, "-o", HOST_PATH, f"-L{libs}", "-ltorch_python", "-ltorch", "-ltorch_cpu", "-ltorch_cuda",
           "-lc10", "-lc10_cuda"]
    stamp = HOST_PATH + ".digest"
    digest = _sources_digest([torch.__version__, sys.version, *cmd], [])
    if not force and os.path.exists(HOST_PATH) and os.path.exists(stamp) and open(stamp).read() == digest:
        return HOST_PATH
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"host build failed:\n{' '.join(cmd)}\n{r.stdout}\n{r.stderr}")
    with open(stamp, "w") as f:
        f.write(digest)
    return HOST_PATH


if __name__ == "__main__":
    path = build_native(force="--force" in sys.argv, verbose="-v" in sys.argv)
    print(build_host(force="--force" in sys.argv))
    print(path)
