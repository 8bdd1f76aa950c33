"""Build libwave_b200.so (nvcc, sm_100a) and the host module _fast.so (g++) in-tree: `python -m wave_b200.build`."""

from __future__ import annotations

import shutil
import subprocess
import sys
from pathlib import Path

PKG = Path(__file__).resolve().parent
CSRC = PKG / "csrc"
OUT = PKG / "libwave_b200.so"
SOURCES = [CSRC / "api.cu"]
HEADERS = sorted(CSRC.glob("*.cuh")) + [PKG.parent / "include" / "wave_b200.h"]

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-O3", "-lineinfo", "-std=c++17",
    "-shared", "-Xcompiler", "-fPIC",
]


def needs_build() -> bool:
    if not OUT.exists():
        return True
    t = OUT.stat().st_mtime
    return any(p.stat().st_mtime > t for p in SOURCES + HEADERS)


TRACE_OUT = PKG / "libwave_b200_trace.so"
CHECKS_OUT = PKG / "libwave_b200_checks.so"
CEILING_OUT = PKG / "libwave_b200_mma_ceiling.so"


def _stale(out: Path) -> bool:
    return not out.exists() or any(p.stat().st_mtime > out.stat().st_mtime for p in SOURCES + HEADERS)


def build(force: bool = False, verbose: bool = False, trace: bool = False, checks: bool = False,
          mma_ceiling: bool = False) -> Path:
    """Compile the library if it is missing or older than its sources. Returns its path.
    `trace`: the measurement variant with per-CTA timeline marks in the skinny kernels (-DWB200_TRACE), written to
    libwave_b200_trace.so; load it with WAVE_B200_LIB=... (see `python -m wave_b200.perf --timeline`).
    `checks`: the debug-checked variant (-DWB200_CHECKS: index predicates in front of every copy-engine issue and
    global store, see csrc/checks.cuh), written to libwave_b200_checks.so.
    `mma_ceiling`: a measurement variant of the tile kernels (-DWB200_MMA_CEILING) that loads only the first ring of
    stages and never reads the accumulators, so that what remains is the scale-factor copies and the MMAs on
    operands resident in shared memory: the tensor pipe's ceiling for this tile shape under the GPU's power limit
    (`python -m wave_b200.perf --mma-ceiling`). Its results are wrong by construction; never load it for anything else."""
    out = TRACE_OUT if trace else CHECKS_OUT if checks else CEILING_OUT if mma_ceiling else OUT
    if not force and not _stale(out):
        return out
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    variant = ["-DWB200_TRACE"] if trace else ["-DWB200_CHECKS"] if checks else ["-DWB200_MMA_CEILING"] if mma_ceiling else []
    cmd = [nvcc, *NVCC_FLAGS, *variant, "-o", str(out), *map(str, SOURCES)]
    if verbose:
        cmd.insert(1, "-Xptxas")
        cmd.insert(2, "-v")
        print(" ".join(cmd))
    res = subprocess.run(cmd, capture_output=True, text=True)
    if res.returncode != 0:
        raise RuntimeError(f"nvcc failed ({res.returncode}):\n{res.stdout}\n{res.stderr}")
    if verbose:
        print(res.stderr)
    return out


FAST_OUT = PKG / "_fast.so"
FAST_SOURCE = CSRC / "fast_call.cpp"


def fast_target() -> str:
    """What `_fast.so` is compiled against; the module carries it."""
    import torch
    return f"torch {torch.__version__}, python {sys.version_info.major}.{sys.version_info.minor}"


def fast_stale() -> bool:
    """`_fast.so` is missing, older than its source, or was compiled against another torch or Python."""
    return not FAST_OUT.exists() or FAST_SOURCE.stat().st_mtime > FAST_OUT.stat().st_mtime or fast_target().encode() not in FAST_OUT.read_bytes()


def build_fast(force: bool = False) -> Path:
    """Compile `wave_b200._fast` (csrc/fast_call.cpp, against the installed torch) if it is not there as it should be (`fast_stale`)."""
    if not force and not fast_stale():
        return FAST_OUT
    import sysconfig

    import torch
    root = Path(torch.__file__).resolve().parent
    nvcc = Path(shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc").resolve()
    includes = [root / "include", root / "include" / "torch" / "csrc" / "api" / "include", nvcc.parent.parent / "include",
                Path(sysconfig.get_paths()["include"])]
    cmd = [shutil.which("g++") or "c++", "-O2", "-std=c++17", "-shared", "-fPIC", "-w", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
           f'-DWB200_FAST_TARGET="{fast_target()}"',
           *(f"-I{i}" for i in includes), str(FAST_SOURCE), "-o", str(FAST_OUT), f"-L{root / 'lib'}", "-lc10", "-lc10_cuda", "-ltorch_cpu",
           "-ltorch_cuda", "-ltorch_python"]
    res = subprocess.run(cmd, capture_output=True, text=True)
    if res.returncode != 0:
        raise RuntimeError(f"g++ failed ({res.returncode}):\n{res.stdout}\n{res.stderr}")
    return FAST_OUT


if __name__ == "__main__":
    print(build_fast(force="--force" in sys.argv))
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv, trace="--trace" in sys.argv, checks="--checks" in sys.argv,
                mma_ceiling="--mma-ceiling" in sys.argv))
