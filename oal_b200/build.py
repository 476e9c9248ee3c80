"""Build the CUDA library of oal_b200 for sm_100a with nvcc (in-tree, no JIT cache).

    python -m oal_b200.build [--force] [--verbose]

Two results: ``oal_b200/liboal_b200.so``, the kernels behind the C ABI (no torch in it), and
``oal_b200/_host.so``, the native host path of the prepared call (autograd node, allocation, status
queue), linked against the first.  nvcc cross-compiles without a GPU present.
"""

from __future__ import annotations

import argparse
import hashlib
import os
import shutil
import subprocess
import sys
from pathlib import Path

PKG = Path(__file__).resolve().parent
CSRC = PKG / "csrc"
LIB = PKG / "liboal_b200.so"
HOST = PKG / "_host.so"
HOST_SOURCE = CSRC / "oal_host.cpp"
STAMP = PKG / "csrc" / ".build_stamp"

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-O3", "-std=c++17", "-lineinfo", "-shared", "-Xcompiler", "-fPIC",
    "--expt-relaxed-constexpr",
]


def sources() -> list[Path]:
    return sorted(CSRC.glob("*.cu"))


def _digest() -> str:
    h = hashlib.sha256()
    for p in sorted([HOST_SOURCE] + list(CSRC.glob("*.cu")) + list(CSRC.glob("*.cuh")) + list(CSRC.glob("*.h"))
                    + [PKG.parent / "include" / "oal_b200.h"]):
        h.update(p.name.encode())
        h.update(p.read_bytes())
    import torch

    h.update((" ".join(NVCC_FLAGS) + torch.__version__).encode())
    return h.hexdigest()


def find_nvcc() -> str:
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        raise RuntimeError("nvcc not found: the oal_b200 CUDA library cannot be built")
    return nvcc


def _host_compile(obj: Path) -> list[str]:
    """g++ command for the host path: torch's headers, the interpreter's, CUDA's runtime API header."""
    import sysconfig

    import torch
    from torch.utils.cpp_extension import include_paths

    cuda = Path(find_nvcc()).resolve().parent.parent / "include"
    includes = [*include_paths(), sysconfig.get_paths()["include"], str(cuda)]
    return ["g++", "-O2", "-std=c++17", "-fPIC", "-fvisibility=hidden", "-DTORCH_API_INCLUDE_EXTENSION_H",
            "-DTORCH_EXTENSION_NAME=_host", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch.compiled_with_cxx11_abi())}",
            *[x for path in includes for x in ("-isystem", path)], "-c", str(HOST_SOURCE), "-o", str(obj)]


def _host_link(obj: Path) -> list[str]:
    from torch.utils.cpp_extension import library_paths

    dirs = [str(PKG), *library_paths()]
    return ["g++", "-shared", "-o", str(HOST), str(obj), *[f"-L{d}" for d in dirs], "-loal_b200", "-ltorch_python", "-ltorch",
            "-ltorch_cpu", "-lc10", "-lc10_cuda", "-Wl,-rpath,$ORIGIN"]


def build(force: bool = False, verbose: bool = False) -> Path:
    """Compile every .cu under csrc/ into one shared library (skipped when up to date)."""
    digest = _digest()
    if not force and LIB.exists() and HOST.exists() and STAMP.exists() and STAMP.read_text() == digest:
        return LIB
    objs = []
    nvcc = find_nvcc()
    build_dir = PKG / "csrc" / "_obj"
    build_dir.mkdir(exist_ok=True)
    procs = []
    for src in sources():
        obj = build_dir / (src.stem + ".o")
        cmd = [nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-lineinfo",
               "-Xcompiler", "-fPIC", "--expt-relaxed-constexpr", "-c", str(src), "-o", str(obj)]
        if verbose:
            cmd.insert(1, "-Xptxas")
            cmd.insert(2, "-v")
        procs.append((src, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
        objs.append(obj)
    host_obj = build_dir / "oal_host.o"
    procs.append((HOST_SOURCE, subprocess.Popen(_host_compile(host_obj), stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
    for src, proc in procs:
        out, _ = proc.communicate()
        if verbose or proc.returncode:
            sys.stderr.write(out)
        if proc.returncode:
            raise RuntimeError(f"nvcc failed on {src.name}")
    link = [nvcc, "-shared", "-o", str(LIB)] + [str(o) for o in objs] + ["-lcudart", "-Xlinker", "-soname=liboal_b200.so"]
    subprocess.run(link, check=True)
    subprocess.run(_host_link(host_obj), check=True)
    STAMP.write_text(digest)
    return LIB


if __name__ == "__main__":
    ap = argparse.ArgumentParser()
    ap.add_argument("--force", action="store_true")
    ap.add_argument("--verbose", action="store_true")
    a = ap.parse_args()
    print(build(force=a.force, verbose=a.verbose))
