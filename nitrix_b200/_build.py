"""Builds the CUDA library in-tree with nvcc for sm_100a.

The shared object lands in ``nitrix_b200/_lib/`` next to the sources so that it
travels with a checkout (it is not installed into site-packages).  nvcc
cross-compiles without a GPU, so this runs on a CPU-only host as well.

Every ``csrc/*.cu`` is compiled to its own object file (in parallel, and only
when the file, a header or the flags changed since its object was made); the
objects are then linked into one shared library.  ``csrc/host/torch_ops.cpp``
(the operations as C++ autograd functions) is compiled by the host compiler
against the installed torch into a Python extension module beside it.
"""
from __future__ import annotations

import concurrent.futures
import hashlib
import os
import pathlib
import shutil
import subprocess
import sysconfig

PKG = pathlib.Path(__file__).resolve().parent
CSRC = PKG / "csrc"
INCLUDE = PKG.parent / "include"
LIBDIR = PKG / "_lib"
OBJDIR = LIBDIR / "obj"
LIBNAME = "libnitrix_b200_attention.so"

COMPILE_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-lineinfo", "-O3", "-std=c++17", "--use_fast_math",
    "-Xcompiler", "-fPIC",
    "-Xcompiler", "-fvisibility=hidden",
]
LINK_FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-shared", "-Xcompiler", "-fPIC"]


HOST_SOURCE = CSRC / "host" / "torch_ops.cpp"
HOST_MODULE = "_torch_ops"
HOST_FLAGS = ["-O2", "-std=c++17", "-shared", "-fPIC", "-fvisibility=hidden"]


def sources() -> list[pathlib.Path]:
    return sorted(CSRC.glob("*.cu"))


def _headers_digest() -> bytes:
    h = hashlib.sha256()
    for f in sorted(list(CSRC.glob("*.cuh")) + list(INCLUDE.glob("*.h"))):
        h.update(f.name.encode())
        h.update(f.read_bytes())
    h.update(" ".join(COMPILE_FLAGS).encode())
    return h.digest()


def _object_digest(src: pathlib.Path, headers: bytes) -> str:
    h = hashlib.sha256(headers)
    h.update(src.name.encode())
    h.update(src.read_bytes())
    return h.hexdigest()


def _digest() -> str:
    headers = _headers_digest()
    h = hashlib.sha256()
    for f in sources():
        h.update(_object_digest(f, headers).encode())
    h.update(" ".join(LINK_FLAGS).encode())
    return h.hexdigest()


def lib_path() -> pathlib.Path:
    return LIBDIR / LIBNAME


def host_module_path() -> pathlib.Path:
    return LIBDIR / (HOST_MODULE + ".so")


def host_runtime() -> str:
    """What the host module is built against; kept beside it, so that it can be compared before the module is loaded."""
    import torch

    return f"torch {torch.__version__}, Python {sysconfig.get_python_version()}"


def host_module_runtime() -> str:
    """:func:`host_runtime` at the time the host module was built."""
    stamp = LIBDIR / "build_host.runtime"
    return stamp.read_text().strip() if stamp.exists() else "an unknown torch"


def _host_digest() -> str:
    h = hashlib.sha256(" ".join([*HOST_FLAGS, host_runtime()]).encode())
    for f in [HOST_SOURCE, *sorted(INCLUDE.glob("*.h"))]:
        h.update(f.read_bytes())
    return h.hexdigest()


def _stamped(path: pathlib.Path, stamp: pathlib.Path, digest: str) -> bool:
    return path.exists() and stamp.exists() and stamp.read_text().strip() == digest


def is_current() -> bool:
    return (_stamped(lib_path(), LIBDIR / "build.sha256", _digest())
            and _stamped(host_module_path(), LIBDIR / "build_host.sha256", _host_digest()))


def _compile_host() -> None:
    import torch

    root = pathlib.Path(torch.__file__).parent
    cuda = pathlib.Path(_nvcc()).resolve().parent.parent
    includes = [root / "include", root / "include" / "torch" / "csrc" / "api" / "include", sysconfig.get_paths()["include"],
                cuda / "include", INCLUDE]
    tmp = LIBDIR / (HOST_MODULE + ".so.tmp")
    cmd = [os.environ.get("CXX", "g++"), *HOST_FLAGS, f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
           *(f"-I{d}" for d in includes), str(HOST_SOURCE), "-o", str(tmp), f"-L{root / 'lib'}", "-lc10", "-lc10_cuda",
           "-ltorch_cpu", "-ltorch_python"]
    res = subprocess.run(cmd, capture_output=True, text=True)
    if res.returncode != 0:
        raise RuntimeError("host compiler failed:\n" + " ".join(cmd) + "\n" + res.stdout + res.stderr)
    os.replace(tmp, host_module_path())
    (LIBDIR / "build_host.runtime").write_text(host_runtime() + "\n")
    (LIBDIR / "build_host.sha256").write_text(_host_digest() + "\n")


def _nvcc() -> str:
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        raise RuntimeError("nvcc not found; cannot build " + LIBNAME)
    return nvcc


def _compile_one(nvcc: str, src: pathlib.Path, obj: pathlib.Path, verbose: bool) -> str:
    cmd = [nvcc, *COMPILE_FLAGS, f"-I{INCLUDE}", f"-I{CSRC}", "-c", "-o", str(obj), str(src)]
    if verbose:
        cmd[1:1] = ["-Xptxas", "-v"]
    res = subprocess.run(cmd, capture_output=True, text=True)
    if res.returncode != 0:
        raise RuntimeError("nvcc failed:\n" + " ".join(cmd) + "\n" + res.stdout + res.stderr)
    return res.stderr


def build(force: bool = False, verbose: bool = False) -> pathlib.Path:
    """Compile every ``csrc/*.cu``, link one shared library and compile the host module (no-op when current)."""
    if not force and not verbose and is_current():
        return lib_path()
    nvcc = _nvcc()
    OBJDIR.mkdir(parents=True, exist_ok=True)
    headers = _headers_digest()
    jobs = []
    objs = []
    for src in sources():
        obj = OBJDIR / (src.stem + ".o")
        stamp = OBJDIR / (src.stem + ".sha256")
        want = _object_digest(src, headers)
        objs.append(obj)
        if force or verbose or not obj.exists() or not stamp.exists() or stamp.read_text().strip() != want:
            jobs.append((src, obj, stamp, want))
    with concurrent.futures.ThreadPoolExecutor(max_workers=max(1, min(len(jobs) + 1, os.cpu_count() or 1))) as pool:
        host = None
        if force or not _stamped(host_module_path(), LIBDIR / "build_host.sha256", _host_digest()):
            host = pool.submit(_compile_host)
        futures = {pool.submit(_compile_one, nvcc, src, obj, verbose): (src, stamp, want) for src, obj, stamp, want in jobs}
        for fut in concurrent.futures.as_completed(futures):
            src, stamp, want = futures[fut]
            log = fut.result()
            stamp.write_text(want + "\n")
            if verbose:
                print(f"==== {src.name}\n{log}")
    tmp = LIBDIR / (LIBNAME + ".tmp")
    cmd = [nvcc, *LINK_FLAGS, "-o", str(tmp), *map(str, objs)]
    res = subprocess.run(cmd, capture_output=True, text=True)
    if res.returncode != 0:
        raise RuntimeError("nvcc link failed:\n" + " ".join(cmd) + "\n" + res.stdout + res.stderr)
    os.replace(tmp, lib_path())
    (LIBDIR / "build.sha256").write_text(_digest() + "\n")
    if host is not None:
        host.result()   # (after the library, which does without the module)
    return lib_path()


if __name__ == "__main__":
    import sys

    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
