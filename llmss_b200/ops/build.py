"""Build the sm_100a kernel library in-tree with nvcc (no GPU needed: cross-compiles).

``python -m llmss_b200.ops.build`` or ``build_library()``.  Objects are cached under
``build/obj`` keyed by a hash of the source, its local includes and the flags, and the final
``llmss_b200/_C/libllmss_b200.so`` is what ``llmss_b200.ops._lib`` dlopens (ctypes).  The
.so is git-ignored but travels with the working tree to the GPU box.
"""
from __future__ import annotations

import hashlib
import os
import shutil
import subprocess
import sys
from concurrent.futures import ThreadPoolExecutor
from pathlib import Path

ROOT = Path(__file__).resolve().parents[2]
CSRC = ROOT / "csrc"
OBJ_DIR = ROOT / "build" / "obj"
LIB_DIR = ROOT / "llmss_b200" / "_C"
LIB_PATH = LIB_DIR / "libllmss_b200.so"

BASE_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-O3", "-std=c++17", "-lineinfo",
    "-Xcompiler", "-fPIC", "-Xcompiler", "-fvisibility=hidden",
    "--expt-relaxed-constexpr",
]
# include paths are location dependent and must not enter the staleness digest: the tree (with its
# prebuilt .so) is copied to other machines under a different root.
NVCC_FLAGS = BASE_FLAGS + ["-I", str(ROOT / "include"), "-I", str(CSRC)]


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and Path(cand).exists():
            return cand
    raise RuntimeError("nvcc not found (set NVCC=/path/to/nvcc)")


def sources():
    return sorted(CSRC.glob("*.cu"))


def _digest(src: Path) -> str:
    h = hashlib.sha256()
    h.update(" ".join(BASE_FLAGS).encode())
    h.update(src.read_bytes())
    for inc in sorted(list(CSRC.glob("*.cuh")) + list((ROOT / "include").glob("*.h"))):
        h.update(inc.read_bytes())
    return h.hexdigest()[:16]


def _compile(src: Path, verbose: bool) -> Path:
    obj = OBJ_DIR / f"{src.stem}.{_digest(src)}.o"
    if obj.exists():
        return obj
    for old in OBJ_DIR.glob(f"{src.stem}.*.o"):
        old.unlink()
    cmd = [_nvcc(), *NVCC_FLAGS, "-c", str(src), "-o", str(obj)]
    if verbose:
        print("[build]", " ".join(cmd), flush=True)
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"nvcc failed for {src.name}:\n{r.stdout}\n{r.stderr}")
    return obj


def tree_digest() -> str:
    """Digest of everything that determines the library contents."""
    return hashlib.sha256("".join(_digest(s) for s in sources()).encode()).hexdigest()[:24]


def is_current() -> bool:
    stamp = LIB_DIR / "build.stamp"
    return LIB_PATH.exists() and stamp.exists() and stamp.read_text().strip() == tree_digest()


def _calls_current() -> bool:
    from . import _lib, calls

    return calls.module_path(LIB_DIR, {**_lib._SIGS, **_lib._OPTIONAL}).exists()


def _build_calls():
    """The entries as plain functions (calls.py).  Every call works without them, so that nothing here stops the library."""
    from . import _lib, calls

    try:
        OBJ_DIR.mkdir(parents=True, exist_ok=True)
        if not calls.build(LIB_DIR, OBJ_DIR, {**_lib._SIGS, **_lib._OPTIONAL}):
            print("[build] no C compiler or Python headers: library calls go through ctypes", file=sys.stderr)
    except (OSError, RuntimeError) as e:
        print(f"[build] library calls go through ctypes: {e}", file=sys.stderr)


def build_library(verbose: bool = False, force: bool = False) -> Path:
    from . import calls

    # e.g. on the GPU box: the .so files travelled with the tree.  A library that is current needs no lock where the calls' module cannot be built
    current = not force and is_current()
    if current and (_calls_current() or calls.compiler() is None):
        return LIB_PATH
    # one builder at a time (torchrun starts N ranks at once); the others wait, then see a current library
    import fcntl

    try:
        LIB_DIR.mkdir(parents=True, exist_ok=True)
        lock = open(LIB_DIR / ".build.lock", "w")
    except OSError:
        if current:          # a read-only installation: calls go through ctypes
            return LIB_PATH
        raise
    with lock:
        fcntl.flock(lock, fcntl.LOCK_EX)
        try:
            path = LIB_PATH if not force and is_current() else _build_locked(verbose, force)
            if not _calls_current():
                _build_calls()
            return path
        finally:
            fcntl.flock(lock, fcntl.LOCK_UN)


def _build_locked(verbose: bool, force: bool) -> Path:
    OBJ_DIR.mkdir(parents=True, exist_ok=True)
    if force:
        for o in OBJ_DIR.glob("*.o"):
            o.unlink()
    srcs = sources()
    with ThreadPoolExecutor(max_workers=min(8, len(srcs))) as ex:
        objs = list(ex.map(lambda s: _compile(s, verbose), srcs))
    stamp = LIB_DIR / "build.stamp"
    want = tree_digest()
    tmp = LIB_PATH.with_suffix(f".so.tmp{os.getpid()}")
    cmd = [_nvcc(), "-shared", "-o", str(tmp), *map(str, objs)]
    if verbose:
        print("[build]", " ".join(cmd), flush=True)
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"link failed:\n{r.stdout}\n{r.stderr}")
    os.replace(tmp, LIB_PATH)  # atomic: a concurrent dlopen never sees a half-written file
    stamp.write_text(want)
    return LIB_PATH


if __name__ == "__main__":
    p = build_library(verbose=True, force="--force" in sys.argv)
    print(f"built {p} ({p.stat().st_size / 1e6:.1f} MB)")
