"""Ahead-of-time build of the C-ABI library (`libbraid_b200.so`) with nvcc.

The reference engine JIT-builds its extension on first use
(braid/kernels/loader.py:10-44: `torch.utils.cpp_extension.load`, `-O3 -lineinfo`,
no fast-math).  Here the library is built once, in-tree, for sm_100a only, and
loaded with ctypes — it has no torch or Python dependency at all.  A second, small
one (`_host.so`, g++) holds the native calls of `quant.py` and does link torch.  Flags keep
the reference's numerics contract: no `--use_fast_math`, IEEE division and
square root, no flush-to-zero.

Run `python -m braid_b200.build` to (re)build; `python -m braid_b200.build -v`
adds `-Xptxas -v` (registers, spills, shared memory per kernel).
`python -m braid_b200.build --phases` builds a second, development-only library
(`libbraid_b200_phases.so`, compiled with `-DBQ_PHASES`) whose decode-regime kernels stamp
the time of each of their phases; `BRAID_B200_LIB=<path>` makes the package load it
(`python bench.py --sweep --only phases` prints the table).  The shipped library contains
none of that code.
"""
from __future__ import annotations

import os
import shutil
import subprocess
import sys
import warnings
from importlib.machinery import EXTENSION_SUFFIXES
from pathlib import Path

PKG = Path(__file__).resolve().parent
CSRC = PKG / "csrc"
LIB = PKG / "libbraid_b200.so"
SOURCES = ("quant_act.cu", "norm_quant.cu", "gemm_w8a8.cu", "cabi.cu")
HEADERS = (CSRC / "ptx.cuh", CSRC / "gemm_wide.cuh", CSRC / "quant_device.cuh", CSRC / "grid_amax.cuh",
           PKG.parent / "include" / "braid_b200.h")


def nvcc_path() -> str:
    cand = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not Path(cand).exists():
        raise RuntimeError("nvcc not found; the CUDA toolkit is needed to build libbraid_b200.so")
    return cand


HOST_SRC = CSRC / "host_calls.cpp"
HOST = PKG / "_host.so"


HOST_MARK = b"braid_b200 native calls for "


def host_key() -> str:
    """The torch and the Python that the native calls have to be compiled against to run in this process."""
    import torch
    return (f"torch {torch.__version__} ({torch.version.git_version}), cxx11 abi {int(torch._C._GLIBCXX_USE_CXX11_ABI)}, "
            f"python{EXTENSION_SUFFIXES[0]}")


def host_problem() -> str | None:
    """Why the native calls cannot be loaded here, None if they can.  Looks at the file without loading it: the
    code reads torch's objects by the layout it was compiled with, and another torch need not refuse it."""
    if not HOST.exists():
        return f"{HOST.name} is not built"
    built = HOST.read_bytes()
    at = built.find(HOST_MARK)
    key = built[at + len(HOST_MARK):built.index(b"\0", at)].decode() if at >= 0 else "an unknown torch"
    return None if key == host_key() else f"{HOST.name} was built for {key}; this is {host_key()}"


def build_host(force: bool = False) -> Path:
    """Compile the native calls of quant.py against the torch that is installed."""
    deps = (HOST_SRC, PKG.parent / "include" / "braid_b200.h")
    if not force and host_problem() is None and all(d.stat().st_mtime <= HOST.stat().st_mtime for d in deps):
        return HOST
    import sysconfig

    import torch
    from torch.utils import cpp_extension
    torch_lib = Path(torch.__file__).resolve().parent / "lib"
    cuda = Path(nvcc_path()).resolve().parent.parent
    includes = [*cpp_extension.include_paths(), sysconfig.get_paths()["include"], str(cuda / "include")]
    cmd = ["g++", "-std=c++17", "-O2", "-shared", "-fPIC", "-fvisibility=hidden",
           f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
           f'-DBQ_HOST_KEY="{host_key()}"',
           *(arg for path in includes for arg in ("-isystem", path)),
           str(HOST_SRC), "-o", str(HOST), f"-L{torch_lib}",
           "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch_cuda", "-ltorch", "-ltorch_python"]
    proc = subprocess.run(cmd, capture_output=True, text=True)
    if proc.returncode != 0:
        raise RuntimeError("g++ failed:\n" + proc.stdout + proc.stderr)
    return HOST


def is_stale() -> bool:
    if not LIB.exists():
        return True
    built = LIB.stat().st_mtime
    deps = [CSRC / s for s in SOURCES] + list(HEADERS)
    return any(d.stat().st_mtime > built for d in deps)


PHASES_LIB = PKG / "libbraid_b200_phases.so"


def build(force: bool = False, verbose: bool = False, defines: tuple[str, ...] = (),
          out: Path | None = None) -> Path:
    """Compile the CUDA sources for sm_100a into one shared library, and the native calls beside it.  The
    package runs without those, so that they cannot be built (no g++, no headers) is a warning."""
    if out is not None or defines:
        return _compile(out if out is not None else LIB, verbose, defines)
    if force or is_stale():
        _compile(LIB, verbose)
    try:
        build_host(force)
    except Exception as e:
        warnings.warn(f"the native calls of quant.py are not built, eager calls take the Python path: {e}", stacklevel=2)
    return LIB


def _compile(lib: Path, verbose: bool = False, defines: tuple[str, ...] = ()) -> Path:
    cmd = [
        nvcc_path(), "-std=c++17", "-O3", "-lineinfo",
        "-gencode", "arch=compute_100a,code=sm_100a",
        "-shared", "-Xcompiler", "-fPIC",
        "--ftz=false", "--prec-div=true", "--prec-sqrt=true", "--fmad=true",
        "-cudart", "static",
        "-I", str(PKG.parent / "include"),
        "-o", str(lib),
    ]
    cmd += [f"-D{d}" for d in defines]
    if verbose or os.environ.get("BRAID_B200_VERBOSE") == "1":
        cmd += ["-Xptxas", "-v"]
    cmd += [str(CSRC / s) for s in SOURCES]
    proc = subprocess.run(cmd, capture_output=True, text=True)
    if proc.returncode != 0:
        raise RuntimeError("nvcc failed:\n" + proc.stdout + proc.stderr)
    if verbose:
        sys.stderr.write(proc.stdout + proc.stderr)
    return lib


if __name__ == "__main__":
    if "--phases" in sys.argv[1:]:
        print(build(force=True, verbose="-v" in sys.argv[1:], defines=("BQ_PHASES",), out=PHASES_LIB))
    else:
        print(build(force=True, verbose="-v" in sys.argv[1:]))
