"""Build the sm_100a shared library in-tree: ``python -m apt_serve_b200.build``.

One ``nvcc`` invocation over ``csrc/*.cu`` producing ``lib/libaptserve_b200.so``.
(Beside it ``lib/libaptserve_b200_host.<interpreter's tag>.so`` from ``csrc/host_tables.cpp``, by the host compiler.)
The library exports the C ABI declared in ``include/aptserve_b200.h`` and links
the CUDA runtime dynamically, so that it shares the runtime PyTorch has loaded.
"""
from __future__ import annotations

import os
import shutil
import subprocess
import sys
import sysconfig
from pathlib import Path

PKG = Path(__file__).resolve().parent
CSRC = PKG / "csrc"
LIB_DIR = PKG / "lib"
LIB_PATH = LIB_DIR / "libaptserve_b200.so"
# reads Python objects: not part of the C-ABI library, and one per interpreter (as in _native.py)
HOST_LIB_PATH = LIB_DIR / ("libaptserve_b200_host" + (sysconfig.get_config_var("EXT_SUFFIX") or ".so"))
SOURCES = ["c_api.cu", "cache_ops.cu", "paged_attention.cu", "hybrid_attention.cu", "hidden_simt.cu", "metadata_ops.cu",
           "tp_comm.cu", "absorbed_attention.cu", "hidden_attention.cu", "hidden_fp32.cu", "decode_step.cu", "tensor_maps.cu",
           "prefill_attention.cu"]
NVCC_FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
              "-Xcompiler", "-fPIC", "-cudart", "shared"]


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and os.path.exists(cand):
            return cand
    raise RuntimeError("nvcc not found; set NVCC or put it on PATH")


def build_host(force: bool = False):
    """Compiles the host library; None, with a word on stderr, where there is no host compiler or no ``Python.h`` (numpy then
    packs the block tables)."""
    src = CSRC / "host_tables.cpp"
    if not force and HOST_LIB_PATH.exists() and HOST_LIB_PATH.stat().st_mtime >= src.stat().st_mtime:
        return HOST_LIB_PATH
    LIB_DIR.mkdir(exist_ok=True)
    tmp = HOST_LIB_PATH.with_name(HOST_LIB_PATH.name + ".tmp")
    cmd = [os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-fPIC", "-shared", "-I", sysconfig.get_paths()["include"],
           str(src), "-o", str(tmp)]
    try:
        r = subprocess.run(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
        failure = None if r.returncode == 0 else r.stdout
    except OSError as exc:
        failure = str(exc)
    if failure is not None:
        print(f"host library not built, {cmd[0]} failed on {src.name}:\n{failure}", file=sys.stderr)
        HOST_LIB_PATH.unlink(missing_ok=True)   # an older one may not fit its callers any more
        return None
    os.replace(tmp, HOST_LIB_PATH)
    return HOST_LIB_PATH


def needs_build() -> bool:
    if not LIB_PATH.exists():
        return True
    t = LIB_PATH.stat().st_mtime
    deps = list(CSRC.glob("*.cu")) + list(CSRC.glob("*.cuh")) + \
        [PKG.parent / "include" / "aptserve_b200.h"]
    return any(d.stat().st_mtime > t for d in deps)


def build(force: bool = False, verbose: bool = False) -> Path:
    path = build_cuda(force, verbose)
    build_host(force)
    return path


def build_cuda(force: bool = False, verbose: bool = False) -> Path:
    if not force and not needs_build():
        return LIB_PATH
    LIB_DIR.mkdir(exist_ok=True)
    objs = []
    procs = []
    obj_dir = LIB_DIR / "obj"
    obj_dir.mkdir(exist_ok=True)
    for src in SOURCES:
        obj = obj_dir / (src[:-3] + ".o")
        cmd = [_nvcc(), *NVCC_FLAGS, "-c", str(CSRC / src), "-o", str(obj)]
        if verbose:
            cmd.insert(1, "-Xptxas=-v")
        procs.append((src, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
        objs.append(str(obj))
    for src, p in procs:
        out, _ = p.communicate()
        if verbose and out:
            print(out)
        if p.returncode != 0:
            raise RuntimeError(f"nvcc failed on {src}:\n{out}")
    tmp = LIB_PATH.with_suffix(".so.tmp")
    link = [_nvcc(), "-shared", "-cudart", "shared", "-o", str(tmp), *objs, "-ldl"]
    r = subprocess.run(link, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"link failed:\n{r.stdout}")
    os.replace(tmp, LIB_PATH)
    return LIB_PATH


if __name__ == "__main__":
    path = build(force="--force" in sys.argv, verbose="-v" in sys.argv)
    print(path)
