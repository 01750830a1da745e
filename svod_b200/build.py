"""Builds the CUDA library in-tree: `svod_b200/lib/libsvodb.so` for sm_100a.

Run as `python -m svod_b200.build` (or through `__graft_entry__.build()`).
nvcc cross-compiles without a GPU. Objects are rebuilt only when a source or
header is newer.
"""
from __future__ import annotations

import os
import subprocess
import sys
from concurrent.futures import ThreadPoolExecutor
from pathlib import Path

ROOT = Path(__file__).resolve().parent
CSRC = ROOT / "csrc"
INCLUDE = ROOT.parent / "include"
OUT_DIR = ROOT / "lib"
OBJ_DIR = OUT_DIR / "obj"
LIB = OUT_DIR / "libsvodb.so"
FAST = OUT_DIR / "_fastops.so"  # the op layer's Python call path (csrc/fastops.cpp)

NVCC = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
CXX = os.environ.get("CXX", "g++")
FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC",
    f"-I{INCLUDE}", f"-I{CSRC}",
]


def _newest_header() -> float:
    hs = list(CSRC.glob("*.h")) + list(CSRC.glob("*.cuh")) + list(INCLUDE.glob("*.h"))
    return max(h.stat().st_mtime for h in hs)


def _compile(src: Path, verbose: bool) -> Path:
    obj = OBJ_DIR / (src.stem + ".o")
    stamp = max(src.stat().st_mtime, _newest_header())
    if obj.exists() and obj.stat().st_mtime >= stamp:
        return obj
    cmd = [NVCC, *FLAGS, "-c", str(src), "-o", str(obj)]
    if verbose:
        cmd.insert(1, "-Xptxas")
        cmd.insert(2, "-v")
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"nvcc failed for {src.name}:\n{r.stdout}\n{r.stderr}")
    if verbose:
        sys.stderr.write(r.stderr)
    return obj


def _build_fast() -> None:
    """The CPython module against torch's headers; its torch symbols are those of the
    libraries `import torch` has loaded, so another torch or Python builds it anew."""
    src = CSRC / "fastops.cpp"
    stamp = max(src.stat().st_mtime, (INCLUDE / "svodb.h").stat().st_mtime)
    import sysconfig
    from importlib import metadata
    against = f"{metadata.version('torch')} {sysconfig.get_config_var('SOABI')}"
    built = FAST.with_suffix(".built")
    if FAST.exists() and FAST.stat().st_mtime >= stamp and built.exists() and built.read_text() == against:
        return

    import torch
    inc = Path(torch.__file__).resolve().parent / "include"
    cmd = [CXX, "-O2", "-std=c++17", "-fPIC", "-shared", "-w", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
           f'-DSVODB_TORCH="{torch.__version__}"',
           f"-I{INCLUDE}", f"-I{inc}", f"-I{inc}/torch/csrc/api/include", f"-I{sysconfig.get_paths()['include']}",
           f"-I{Path(NVCC).parent.parent}/include", str(src), "-o", str(FAST), f"-L{inc.parent}/lib", "-ltorch_python", "-ltorch_cpu",
           "-lc10", "-lc10_cuda"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"{CXX} failed for {src.name}:\n{r.stdout}\n{r.stderr}")
    built.write_text(against)


def _try_build_fast() -> None:
    """The library is whole without the module, and a user of the C library needs neither
    torch's headers nor Python's: what keeps it from being built is said, not raised. One
    that is there and could not be brought up to date goes, so that nothing loads it."""
    try:
        _build_fast()
    except Exception as e:
        FAST.unlink(missing_ok=True)
        print(f"svod_b200.build: without {FAST.name} (ops take the ctypes path): {e}", file=sys.stderr)


def build(verbose: bool = False) -> Path:
    OBJ_DIR.mkdir(parents=True, exist_ok=True)
    srcs = sorted(CSRC.glob("*.cu"))
    with ThreadPoolExecutor(max_workers=min(8, len(srcs) + 1)) as ex:
        fast = ex.submit(_try_build_fast)
        objs = list(ex.map(lambda s: _compile(s, verbose), srcs))
    fast.result()
    if not LIB.exists() or any(o.stat().st_mtime > LIB.stat().st_mtime for o in objs):
        cmd = [NVCC, "-shared", "-gencode", "arch=compute_100a,code=sm_100a", "-o", str(LIB), *map(str, objs)]
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError(f"link failed:\n{r.stdout}\n{r.stderr}")
    return LIB


if __name__ == "__main__":
    print(build(verbose="-v" in sys.argv))
