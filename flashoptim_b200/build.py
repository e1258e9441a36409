"""In-tree build of ``libflashoptim_b200.so`` (hand-written sm_100a CUDA, C ABI).

``python -m flashoptim_b200.build`` compiles every ``csrc/*.cu`` with nvcc for
``sm_100a`` and links one shared library next to the package.  The library has
no PyTorch dependency: Python passes raw device pointers and the current CUDA
stream through :mod:`ctypes` (see :mod:`flashoptim_b200.ops.native`).  The host
walk over a parameter group, ``csrc/fo_host.cpp``, is a CPython extension of its
own, built against the installed PyTorch (:mod:`flashoptim_b200.ops.host`).
Stamp files holding a hash of sources and flags make repeated calls free.
"""

from __future__ import annotations

import contextlib
import hashlib
import os
import shutil
import subprocess
import sys
import tempfile
from concurrent.futures import ThreadPoolExecutor
from pathlib import Path

PKG_DIR = Path(__file__).resolve().parent
SRC_DIR = PKG_DIR / "csrc"
LIB_DIR = PKG_DIR / "_lib"
LIB_PATH = LIB_DIR / "libflashoptim_b200.so"
STAMP_PATH = LIB_DIR / "build.stamp"
HOST_SOURCE = SRC_DIR / "fo_host.cpp"
HOST_PATH = LIB_DIR / "_fo_host.so"
HOST_STAMP_PATH = LIB_DIR / "host.stamp"
HOST_FLAGS = ["-O2", "-std=c++17", "-fPIC", "-shared", "-Wno-unknown-pragmas"]

NVCC_FLAGS = [
    "-gencode",
    "arch=compute_100a,code=sm_100a",
    "-lineinfo",
    "-O3",
    "-std=c++17",
    "-Xcompiler",
    "-fPIC",
]


def find_nvcc() -> str | None:
    cand = os.environ.get("NVCC") or shutil.which("nvcc")
    if cand:
        return cand
    p = Path(os.environ.get("CUDA_HOME", "/usr/local/cuda")) / "bin" / "nvcc"
    return str(p) if p.exists() else None


def _sources() -> list[Path]:
    return sorted(SRC_DIR.glob("*.cu"))


def source_hash(extra_flags: tuple[str, ...] = ()) -> str:
    h = hashlib.sha256()
    for f in sorted(SRC_DIR.iterdir()):
        if f.suffix in (".cu", ".cuh", ".h"):
            h.update(f.name.encode())
            h.update(f.read_bytes())
    h.update(" ".join(NVCC_FLAGS + list(extra_flags)).encode())
    return h.hexdigest()


def is_current(extra_flags: tuple[str, ...] = ()) -> bool:
    return (
        LIB_PATH.exists()
        and STAMP_PATH.exists()
        and STAMP_PATH.read_text().strip() == source_hash(extra_flags)
    )


@contextlib.contextmanager
def _build_lock(lock_dir: Path):
    """Exclusive inter-process lock: under torchrun every rank may find the library stale at
    the same moment, and only one of them may run nvcc into the shared object directory."""
    lock_dir.mkdir(parents=True, exist_ok=True)
    with open(lock_dir / ".build.lock", "w") as fh:
        try:
            import fcntl

            fcntl.flock(fh, fcntl.LOCK_EX)
        except ImportError:  # no fcntl: single-process builds only
            pass
        yield


def build(
    force: bool = False,
    verbose: bool = False,
    extra_flags: tuple[str, ...] = (),
    out_path: Path | None = None,
) -> Path:
    """Compile and link the library; returns its path.

    ``extra_flags`` (e.g. ``-DFO_UNROLL=4``) and ``out_path`` exist for tuning
    builds; the default build writes ``_lib/libflashoptim_b200.so``.
    """
    default_target = out_path is None
    out = LIB_PATH if default_target else Path(out_path)
    if default_target and not force and is_current(extra_flags):
        return out
    nvcc = find_nvcc()
    if nvcc is None:
        raise RuntimeError(
            "nvcc not found: cannot build libflashoptim_b200.so "
            "(set NVCC or CUDA_HOME, or ship a prebuilt _lib/)"
        )
    with _build_lock(out.parent):
        # another process may have finished the same build while this one waited
        if default_target and not force and is_current(extra_flags):
            return out
        return _build_locked(nvcc, out, default_target, verbose, extra_flags)


def _build_locked(nvcc: str, out: Path, default_target: bool, verbose: bool, extra_flags: tuple[str, ...]) -> Path:
    obj_dir = out.parent / ("obj_" + out.stem)
    obj_dir.mkdir(parents=True, exist_ok=True)

    def compile_one(src: Path) -> Path:
        obj = obj_dir / (src.stem + ".o")
        cmd = [nvcc, *NVCC_FLAGS, *extra_flags, "-I", str(SRC_DIR), "-c", str(src), "-o", str(obj)]
        if verbose:
            print(" ".join(cmd), flush=True)
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError(f"nvcc failed on {src.name}:\n{r.stdout}\n{r.stderr}")
        return obj

    with ThreadPoolExecutor(max_workers=min(8, len(_sources()) or 1)) as ex:
        objs = list(ex.map(compile_one, _sources()))
    # link beside the target and rename into place: a process that dlopens the library at this
    # moment sees the old file or the new one, never a half-written one; the stamp comes last
    fd, tmp = tempfile.mkstemp(prefix=out.stem + ".", suffix=".so.tmp", dir=str(out.parent))
    os.close(fd)
    try:
        link = [nvcc, "-shared", "-gencode", "arch=compute_100a,code=sm_100a", "-o", tmp] + [str(o) for o in objs]
        if verbose:
            print(" ".join(link), flush=True)
        r = subprocess.run(link, capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError(f"link failed:\n{r.stdout}\n{r.stderr}")
        os.chmod(tmp, 0o755)
        os.replace(tmp, out)
    finally:
        if os.path.exists(tmp):
            os.unlink(tmp)
    if default_target:
        _write_stamp(STAMP_PATH, source_hash(extra_flags))
    return out


def _write_stamp(path: Path, text: str) -> None:
    tmp = path.with_suffix(".stamp.tmp")
    tmp.write_text(text)
    os.replace(tmp, path)


# ---------------------------------------------------------------- host extension
def host_hash() -> str:
    """Sources and flags, and the PyTorch and Python whose object layouts are compiled in."""
    import torch

    h = hashlib.sha256()
    for f in (HOST_SOURCE, SRC_DIR / "fo_api.h"):
        h.update(f.read_bytes())
    h.update(" ".join([*HOST_FLAGS, torch.__version__, sys.version]).encode())
    return h.hexdigest()


def host_is_current() -> bool:
    return HOST_PATH.exists() and HOST_STAMP_PATH.exists() and HOST_STAMP_PATH.read_text().strip() == host_hash()


def build_host(force: bool = False, verbose: bool = False) -> Path:
    """Compile ``csrc/fo_host.cpp`` into ``_lib/_fo_host.so``; returns its path."""
    if not force and host_is_current():
        return HOST_PATH
    import sysconfig

    import torch
    from torch.utils import cpp_extension

    cxx = os.environ.get("CXX") or shutil.which("g++")
    if cxx is None:
        raise RuntimeError(f"no C++ compiler: cannot build {HOST_PATH.name} (set CXX, or ship a prebuilt _lib/)")
    cuda_home = Path(os.environ.get("CUDA_HOME", "/usr/local/cuda"))
    includes = [*cpp_extension.include_paths(), sysconfig.get_paths()["include"], str(cuda_home / "include")]
    with _build_lock(LIB_DIR):
        if not force and host_is_current():
            return HOST_PATH
        fd, tmp = tempfile.mkstemp(prefix="_fo_host.", suffix=".so.tmp", dir=str(LIB_DIR))
        os.close(fd)
        try:
            cmd = [cxx, *HOST_FLAGS, f"-D_GLIBCXX_USE_CXX11_ABI={int(torch.compiled_with_cxx11_abi())}"]
            for d in includes:
                cmd += ["-isystem", d]
            cmd += [str(HOST_SOURCE), "-o", tmp]
            for d in cpp_extension.library_paths():
                cmd += ["-L", d]
            cmd += ["-lc10", "-ltorch_cpu", "-ltorch_python", "-lc10_cuda"]
            if verbose:
                print(" ".join(cmd), flush=True)
            r = subprocess.run(cmd, capture_output=True, text=True)
            if r.returncode != 0:
                raise RuntimeError(f"{cxx} failed on {HOST_SOURCE.name}:\n{r.stdout}\n{r.stderr}")
            os.chmod(tmp, 0o755)
            os.replace(tmp, HOST_PATH)
        finally:
            if os.path.exists(tmp):
                os.unlink(tmp)
        _write_stamp(HOST_STAMP_PATH, host_hash())
    return HOST_PATH


if __name__ == "__main__":
    path = build(force="--force" in sys.argv, verbose=True)
    print(f"built {path}")
    print(f"built {build_host(force='--force' in sys.argv, verbose=True)}")
