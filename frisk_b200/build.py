"""Builds libfrisk_b200.so in-tree with nvcc for sm_100a.

    python -m frisk_b200.build [--force] [--verbose]

Each ``csrc/*.cu`` is compiled to an object (in parallel, only when it or a header
is newer than the object) and linked into ``frisk_b200/lib/libfrisk_b200.so``.
nvcc cross-compiles without a GPU.  ``csrc/recognise.cpp``, a host-only CPython module, is compiled by g++ into
``frisk_b200/lib/_recognise`` + the interpreter's extension suffix; where g++ or Python's headers are missing the package does without.
"""
import concurrent.futures
import importlib.machinery
import os
import pathlib
import shutil
import subprocess
import sys
import sysconfig

PKG = pathlib.Path(__file__).resolve().parent
CSRC = PKG / "csrc"
OBJ = PKG / "build"
LIB = PKG / "lib" / "libfrisk_b200.so"
RECOGNISE = PKG / "lib" / ("_recognise" + importlib.machinery.EXTENSION_SUFFIXES[0])  # (names the interpreter's ABI)
INCLUDE = PKG.parent / "include"

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC", "--expt-relaxed-constexpr", "-Xptxas", "-v",
]


def _nvcc():
    exe = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(exe):
        raise RuntimeError("nvcc not found: libfrisk_b200 cannot be built")
    return exe


def _stale(target, deps):
    if not target.exists():
        return True
    t = target.stat().st_mtime
    return any(d.stat().st_mtime > t for d in deps)


def build_recognise(force=False):
    """The native recogniser, or None where it cannot be built here: ``execute`` then recognises in Python, more slowly."""
    source, target = CSRC / "recognise.cpp", RECOGNISE
    if not force and not _stale(target, [source]):
        return target
    gxx, headers = shutil.which("g++"), sysconfig.get_paths()["include"]
    if gxx is None or not os.path.exists(os.path.join(headers, "Python.h")) or sys.version_info < (3, 10):
        sys.stderr.write("frisk_b200: no g++ or no headers of Python 3.10 or newer: built without the native recogniser\n")
        target.unlink(missing_ok=True)  # (one of an older source)
        return None
    target.parent.mkdir(exist_ok=True)
    res = subprocess.run([gxx, "-O2", "-std=c++17", "-shared", "-fPIC", "-I", headers, str(source), "-o", str(target)],
                         capture_output=True, text=True)
    if res.returncode:
        sys.stderr.write(res.stdout + res.stderr)
        raise RuntimeError("g++ failed on recognise.cpp")
    return target


def build(force=False, verbose=False):
    nvcc = _nvcc()
    OBJ.mkdir(exist_ok=True)
    LIB.parent.mkdir(exist_ok=True)
    headers = list(CSRC.glob("*.cuh")) + list(INCLUDE.glob("*.h"))
    sources = sorted(CSRC.glob("*.cu"))
    jobs = []
    for src in sources:
        obj = OBJ / (src.stem + ".o")
        if force or _stale(obj, [src] + headers):
            jobs.append((src, obj))

    def compile_one(job):
        src, obj = job
        cmd = [nvcc, *NVCC_FLAGS, "-I", str(INCLUDE), "-c", str(src), "-o", str(obj)]
        res = subprocess.run(cmd, capture_output=True, text=True)
        (OBJ / (src.stem + ".log")).write_text(res.stdout + res.stderr)
        return src, res

    with concurrent.futures.ThreadPoolExecutor(max_workers=min(8, max(1, len(jobs)))) as pool:
        for src, res in pool.map(compile_one, jobs):
            if verbose or res.returncode:
                sys.stderr.write(res.stdout + res.stderr)
            if res.returncode:
                raise RuntimeError(f"nvcc failed on {src.name}")
    objs = [OBJ / (s.stem + ".o") for s in sources]
    if force or jobs or _stale(LIB, objs):
        cmd = [nvcc, "-shared", "-gencode", "arch=compute_100a,code=sm_100a", "-o", str(LIB), *map(str, objs)]
        res = subprocess.run(cmd, capture_output=True, text=True)
        if res.returncode:
            sys.stderr.write(res.stdout + res.stderr)
            raise RuntimeError("link of libfrisk_b200.so failed")
    build_recognise(force)
    return LIB


if __name__ == "__main__":
    path = build(force="--force" in sys.argv, verbose="--verbose" in sys.argv)
    print(path)
