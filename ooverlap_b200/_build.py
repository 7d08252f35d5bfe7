"""In-tree build of the native library with nvcc for sm_100a.

Every source under ``csrc/`` is compiled with
``-gencode arch=compute_100a,code=sm_100a`` into ``build/obj`` and linked into
``ooverlap_b200/lib/libooverlap_b200.so`` (plus the ``oob_topology`` CLI).  A
stamp file holding a hash of the sources and flags makes the step a no-op when
nothing changed, so a machine that receives the tree with the built library
does not rebuild it.

``_fast_ops.so``, the native Python entries of the small ops, is built with it
against the installed PyTorch and Python and has a stamp of its own.  The library
does not need it: where it cannot be built (no host compiler, no headers) the
build says so, and the Python implementations are used.

Capability parity: the reference builds with CMake (CMakeLists.txt:12-129,
src/CMakeLists.txt:169-683) for compute_90a only.
"""
from __future__ import annotations

import hashlib
import importlib.metadata
import importlib.util
import os
import shutil
import subprocess
import sys
import sysconfig
import warnings
from concurrent.futures import ThreadPoolExecutor
from pathlib import Path

ROOT = Path(__file__).resolve().parent.parent
CSRC = ROOT / "csrc"
OBJ = ROOT / "build" / "obj"
LIB_DIR = Path(__file__).resolve().parent / "lib"
LIB = LIB_DIR / "libooverlap_b200.so"
CLI = LIB_DIR / "oob_topology"
FAST = LIB_DIR / "_fast_ops.so"
STAMP = LIB_DIR / "build.stamp"
FAST_STAMP = LIB_DIR / "fast.stamp"
FAST_SRC = CSRC / "python" / "fast_ops.cpp"

ARCH_FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a"]
COMMON = ["-O3", "-std=c++17", "-lineinfo", "-Xcompiler", "-fPIC", "-Xcompiler", "-fvisibility=hidden",
          "-DOOB_BUILDING=1", "--expt-relaxed-constexpr"]


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and os.path.exists(cand):
            return cand
    raise RuntimeError("nvcc not found (set NVCC or put it on PATH)")


def _sources() -> list[Path]:
    srcs = sorted(p for p in CSRC.rglob("*") if p.suffix in (".cu", ".cpp") and not {"cli", "python"} & set(p.parts))
    return srcs


def _all_inputs() -> list[Path]:
    return sorted(p for p in CSRC.rglob("*") if p.suffix in (".cu", ".cpp", ".h", ".cuh") and "python" not in p.parts)


def source_hash() -> str:
    h = hashlib.sha256()
    h.update(" ".join(ARCH_FLAGS + COMMON).encode())
    for p in _all_inputs():
        h.update(str(p.relative_to(ROOT)).encode())
        h.update(p.read_bytes())
    return h.hexdigest()


def is_current() -> bool:
    return LIB.exists() and STAMP.exists() and STAMP.read_text().strip() == source_hash()


def fast_hash() -> str:
    h = hashlib.sha256(f"{importlib.metadata.version('torch')} {sys.implementation.cache_tag}".encode())
    for p in (FAST_SRC, *sorted((CSRC / "api").glob("*.h"))):
        h.update(p.read_bytes())
    return h.hexdigest()


def fast_is_current() -> bool:
    return FAST.exists() and FAST_STAMP.exists() and FAST_STAMP.read_text().strip() == fast_hash()


def _gxx(args: list) -> None:
    res = subprocess.run(["g++", *map(str, args)], capture_output=True, text=True)
    if res.returncode != 0:
        raise RuntimeError(f"g++ failed for {FAST_SRC}:\n{res.stdout}\n{res.stderr}")


def _torch_dir() -> Path:
    return Path(importlib.util.find_spec("torch").submodule_search_locations[0])


def _compile_fast() -> Path:
    import torch
    cuda, base = Path(_nvcc()).resolve().parent.parent, _torch_dir()
    include = [base / "include", base / "include/torch/csrc/api/include", cuda / "include", sysconfig.get_paths()["include"]]
    OBJ.mkdir(parents=True, exist_ok=True)
    obj = OBJ / "python__fast_ops.cpp.o"
    _gxx(["-O2", "-std=c++17", "-fPIC", "-fvisibility=hidden", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch.compiled_with_cxx11_abi())}",
          *(f"-I{p}" for p in include), "-c", FAST_SRC, "-o", obj])
    return obj


def _link_fast(obj: Path) -> None:
    # Into a file of its own first: another process may have the one in place loaded.
    tmp = FAST.with_name(f"_fast_ops.{os.getpid()}.tmp")
    _gxx(["-shared", obj, "-o", tmp, f"-L{_torch_dir() / 'lib'}", f"-L{LIB_DIR}", "-ltorch_python", "-ltorch", "-ltorch_cpu", "-lc10_cuda",
          "-lc10", "-looverlap_b200", "-Wl,-rpath,$ORIGIN"])
    os.replace(tmp, FAST)
    FAST_STAMP.write_text(fast_hash() + "\n")


def build_fast(compiled=None) -> bool:
    """Builds the native Python entries (``compiled``: their object file, if it is there); whether they can be used.  The library must be
    built."""
    try:
        _link_fast(compiled() if compiled is not None else _compile_fast())
        return True
    except Exception as e:
        warnings.warn(f"the native Python entries cannot be built, the Python implementations are used: {e}", RuntimeWarning, stacklevel=2)
        return False


def build(force: bool = False, verbose: bool = False, ptxas_info: bool = False) -> Path:
    """Compile and link; returns the path of the shared library."""
    if not force and is_current():
        if not fast_is_current():
            build_fast()
        return LIB
    nvcc = _nvcc()
    OBJ.mkdir(parents=True, exist_ok=True)
    LIB_DIR.mkdir(parents=True, exist_ok=True)
    srcs = _sources()
    extra = ["-Xptxas", "-v"] if ptxas_info else []

    def compile_one(src: Path) -> Path:
        obj = OBJ / (str(src.relative_to(CSRC)).replace("/", "__") + ".o")
        cmd = [nvcc, *ARCH_FLAGS, *COMMON, *extra, "-x", "cu", "-c", str(src), "-o", str(obj)]
        res = subprocess.run(cmd, capture_output=True, text=True)
        if res.returncode != 0:
            raise RuntimeError(f"nvcc failed for {src}:\n{res.stdout}\n{res.stderr}")
        if verbose or ptxas_info:
            sys.stderr.write(res.stderr)
        return obj

    with ThreadPoolExecutor(max_workers=min(8, os.cpu_count() or 2)) as ex:
        fast = ex.submit(_compile_fast)
        objs = list(ex.map(compile_one, srcs))
    link = [nvcc, *ARCH_FLAGS, "-shared", "-o", str(LIB), *map(str, objs), "-Xcompiler", "-fPIC", "-lpthread", "-ldl"]
    res = subprocess.run(link, capture_output=True, text=True)
    if res.returncode != 0:
        raise RuntimeError(f"link failed:\n{res.stdout}\n{res.stderr}")
    cli_src = CSRC / "cli" / "topology_cli.cpp"
    cli = [nvcc, "-O2", "-std=c++17", str(cli_src), "-o", str(CLI), f"-L{LIB_DIR}", "-looverlap_b200",
           "-Xlinker", "-rpath", "-Xlinker", "$ORIGIN"]
    res = subprocess.run(cli, capture_output=True, text=True)
    if res.returncode != 0:
        raise RuntimeError(f"CLI link failed:\n{res.stdout}\n{res.stderr}")
    STAMP.write_text(source_hash() + "\n")
    build_fast(fast.result)
    return LIB


if __name__ == "__main__":
    path = build(force="--force" in sys.argv, verbose=True, ptxas_info="--ptxas" in sys.argv)
    print(path)
