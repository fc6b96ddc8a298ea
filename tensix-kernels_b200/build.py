"""build.py: compiles libtkd.so (the CUDA kernels and their C-ABI) for sm_100a and tkd_host.so (the Python layer's
native launch path over it), in the tree, with nvcc and g++.

    python tensix-kernels_b200/build.py [--verbose]

Both sit beside their sources (csrc/); the Python layer loads them and refuses to work without them. nvcc
cross-compiles: no GPU is needed to build.
"""

import shutil
import subprocess
import sys
import sysconfig
from concurrent.futures import ThreadPoolExecutor
from pathlib import Path

CSRC = Path(__file__).resolve().parent / "csrc"
SOURCES = ["tkd_api.cu", "tkd_pack.cu", "tkd_stream.cu", "tkd_stream_bfp8.cu", "tkd_stream_bfp4.cu", "tkd_stream_bf16.cu",
           "tkd_stream_int4.cu", "tkd_wide_bfp8.cu", "tkd_wide_bfp4.cu", "tkd_wide_bf16.cu", "tkd_hadamard.cu", "tkd_moe.cu",
           "tkd_topk.cu"]
LIB = CSRC / "libtkd.so"
FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-lineinfo", "-std=c++17", "-Xcompiler", "-fPIC"]
OBJ = CSRC / "build"
HOST = CSRC / "tkd_host.so"


def _older(target, deps):
    return not target.exists() or any(d.stat().st_mtime > target.stat().st_mtime for d in deps)


def stale():
    header = CSRC.parents[1] / "include" / "tkd.h"
    return _older(LIB, [*CSRC.glob("*.cu"), *CSRC.glob("*.cuh"), *CSRC.glob("*.h"), header])


def host_for():
    """What tkd_host.so is compiled against besides libtkd: another torch or Python needs another module."""
    import torch

    return f"torch {torch.__version__}, Python {sys.version_info[0]}.{sys.version_info[1]}"


def host_stale():
    return (_older(HOST, [CSRC / "tkd_host.cpp", CSRC.parents[1] / "include" / "tkd.h", LIB])
            or host_for().encode() not in HOST.read_bytes())


def build_host(verbose=False, force=False):
    """tkd_host.so, the extension module over libtkd.so (which it finds beside itself) and torch's C++ libraries."""
    if not force and not host_stale():
        return HOST
    import torch

    at = Path(torch.__file__).parent
    inc = [sysconfig.get_paths()["include"], at / "include", at / "include/torch/csrc/api/include", _cuda_include()]
    _run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
          f'-DTKD_HOST_FOR="{host_for()}"',
          *(f"-I{i}" for i in inc), "-o", str(HOST), str(CSRC / "tkd_host.cpp"), f"-L{at / 'lib'}", "-lc10", "-lc10_cuda",
          "-ltorch_cpu", "-ltorch_cuda", "-ltorch_python", f"-L{CSRC}", "-l:libtkd.so", "-Wl,-rpath,$ORIGIN"], verbose)
    return HOST


def _cuda_include():
    """The headers of the toolkit whose nvcc compiles the library."""
    nvcc = shutil.which("nvcc")
    if nvcc is None:
        raise RuntimeError("the build needs nvcc on the PATH")
    return Path(nvcc).resolve().parents[1] / "include"


def _run(cmd, verbose):
    r = subprocess.run(cmd, capture_output=True, text=True)
    if verbose or r.returncode:
        sys.stderr.write(r.stdout + r.stderr)
    if r.returncode:
        raise RuntimeError("the build failed: " + " ".join(cmd))


def build(verbose=False, force=False, defines=(), lib=LIB):
    """Compile the sources (one nvcc per file, side by side) and link them, then the host module. defines: extra -D flags
    (experiments: the library alone)."""
    if not force and not defines and not stale():
        build_host(verbose)
        return lib
    OBJ.mkdir(exist_ok=True)
    extra = [*(["-Xptxas", "-v"] if verbose else []), *[f"-D{d}" for d in defines]]
    objs = [OBJ / (Path(s).stem + "".join("_" + d.replace("=", "_") for d in defines) + ".o") for s in SOURCES]
    with ThreadPoolExecutor(len(SOURCES)) as pool:
        list(pool.map(lambda so: _run(["nvcc", *FLAGS, *extra, "-c", "-o", str(so[1]), str(CSRC / so[0])], verbose),
                      zip(SOURCES, objs)))
    _run(["nvcc", "-gencode", "arch=compute_100a,code=sm_100a", "-shared", "-o", str(lib), *map(str, objs)], verbose)
    if lib == LIB:
        build_host(verbose, force)
    return lib


if __name__ == "__main__":
    build(verbose="--verbose" in sys.argv, force=True)
    print(LIB)
