"""Build ``liblik_b200.so`` from ``csrc/*.cu`` with nvcc for sm_100a, and the native host path ``_host.so`` from
``csrc/host/*.cpp`` (both in-tree).

Each translation unit is compiled to an object file (in parallel, only when its sources are newer) and the objects are
linked into one shared library next to this file.  The kernel library speaks plain C and sees no torch headers; the host
path is a Python extension on top of it that takes torch tensors.
"""

from __future__ import annotations

import os
import shutil
import subprocess
import sys
from concurrent.futures import ThreadPoolExecutor

PKG_DIR = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(PKG_DIR, "csrc")
INCLUDE = os.path.join(os.path.dirname(PKG_DIR), "include")
HOST_SRC = os.path.join(CSRC, "host")
LIB_PATH = os.path.join(PKG_DIR, "liblik_b200.so")
HOST_PATH = os.path.join(PKG_DIR, "_host.so")
OBJ_DIR = os.path.join(PKG_DIR, "build")

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-O3", "-lineinfo", "-std=c++17",
    "-Xcompiler", "-fPIC",
    "-I", INCLUDE, "-I", CSRC,
]


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and os.path.exists(cand):
            return cand
    raise RuntimeError("nvcc not found; cannot build liblik_b200.so")


def _sources():
    return sorted(os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith(".cu"))


def _headers():
    hs = [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith((".cuh", ".h"))]
    hs += [os.path.join(INCLUDE, f) for f in os.listdir(INCLUDE) if f.endswith(".h")]
    return hs


def _host_sources():
    return sorted(os.path.join(HOST_SRC, f) for f in os.listdir(HOST_SRC) if f.endswith(".cpp"))


def _host_headers():
    hs = [os.path.join(HOST_SRC, f) for f in os.listdir(HOST_SRC) if f.endswith(".h")]
    return hs + [os.path.join(INCLUDE, f) for f in os.listdir(INCLUDE) if f.endswith(".h")]


def _stale(target, inputs) -> bool:
    if not os.path.exists(target):
        return True
    t = os.path.getmtime(target)
    return any(os.path.getmtime(p) > t for p in inputs)


def _host_abi() -> str:
    """What a built host path is bound to besides its sources: torch's class layouts and the interpreter."""
    import sysconfig
    from importlib.metadata import version

    return f"host path for torch {version('torch')}, {sysconfig.get_config_var('SOABI')}"


def _host_fits(path) -> bool:
    """Whether the extension at ``path`` was built for this torch and this interpreter (it carries their names)."""
    with open(path, "rb") as f:
        return _host_abi().encode() + b"\0" in f.read()


def _run(cmd, what):
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"{what} failed:\n{r.stdout}\n{r.stderr}")
    return r.stderr


def _host_flags():
    import sysconfig

    from torch.utils import cpp_extension

    inc = [INCLUDE, HOST_SRC, sysconfig.get_paths()["include"], *cpp_extension.include_paths("cuda")]
    flags = ["-O2", "-std=c++17", "-fPIC", "-fvisibility=hidden", "-DTORCH_EXTENSION_NAME=_host", "-DTORCH_API_INCLUDE_EXTENSION_H", f'-DLIK_HOST_ABI="{_host_abi()}"']
    return flags + [x for p in inc for x in ("-isystem" if p not in (INCLUDE, HOST_SRC) else "-I", p)]


def build(force: bool = False, verbose: bool = False, extra_flags=()) -> str:
    """Compile what is stale and return the path of the kernel library."""
    want_lib = force or _stale(LIB_PATH, _sources() + _headers())
    other_host = os.path.exists(HOST_PATH) and not _host_fits(HOST_PATH)  # torch or the interpreter was replaced
    want_host = force or other_host or _stale(HOST_PATH, _host_sources() + _host_headers())
    if not (want_lib or want_host):
        return LIB_PATH
    os.makedirs(OBJ_DIR, exist_ok=True)
    nvcc = _nvcc() if want_lib else None
    host_flags = _host_flags() if want_host else None

    def compile_one(src):
        host = src.endswith(".cpp")
        obj = os.path.join(OBJ_DIR, os.path.splitext(os.path.basename(src))[0] + ".o")
        if not (force or (host and other_host)) and not _stale(obj, [src] + (_host_headers() if host else _headers())):
            return obj, ""
        cmd = ["g++", *host_flags, "-c", src, "-o", obj] if host else [nvcc, *NVCC_FLAGS, *extra_flags, "-c", src, "-o", obj]
        return obj, _run(cmd, f"compiling {src}")

    with ThreadPoolExecutor(max_workers=min(8, os.cpu_count() or 1)) as ex:
        lib_jobs = [ex.submit(compile_one, s) for s in (_sources() if want_lib else [])]
        host_jobs = [ex.submit(compile_one, s) for s in (_host_sources() if want_host else [])]
        lib_objs, host_objs = [j.result() for j in lib_jobs], [j.result() for j in host_jobs]
    if verbose:
        for _, log in lib_objs + host_objs:
            if log.strip():
                print(log, file=sys.stderr)
    if want_lib:
        tmp = LIB_PATH + ".tmp"
        _run([nvcc, "-shared", "-o", tmp, *[o for o, _ in lib_objs], "-Xlinker", "-soname=liblik_b200.so",
              "-gencode", "arch=compute_100a,code=sm_100a"], "linking the kernel library")
        os.replace(tmp, LIB_PATH)
    if want_host:
        from torch.utils import cpp_extension

        tmp = HOST_PATH + ".tmp"
        libs = [x for p in cpp_extension.library_paths() for x in ("-L", p)]
        _run(["g++", "-shared", "-o", tmp, *[o for o, _ in host_objs], *libs, "-L", PKG_DIR, "-l:liblik_b200.so", "-Wl,-rpath,$ORIGIN",
              "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch", "-ltorch_python"], "linking the host path")
        os.replace(tmp, HOST_PATH)
    return LIB_PATH


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose=True, extra_flags=["-Xptxas", "-v"] if "-v" in sys.argv else []))
