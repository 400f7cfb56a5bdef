"""Builds the native pieces in-tree:

  graphtok_b200/lib/libgtok.so      CUDA kernels + engine + C ABI, sm_100a only
  graphtok_b200/datagen/datagen     synthetic text / vocabulary generator (host only)
  graphtok_b200/cli/gpu_bpe_tokenize   command-line tool over libgtok.so
  graphtok_b200/_host.so            CPython extension: Python objects to and from libgtok.so (left out,
                                    with a line that says so, where Python's or numpy's headers are missing)

nvcc cross-compiles without a GPU.  Run as `python -m graphtok_b200.build`.
"""
import os
import shutil
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
LIB_DIR = os.path.join(HERE, "lib")
LIB = os.path.join(LIB_DIR, "libgtok.so")
DATAGEN = os.path.join(HERE, "datagen", "datagen")

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "-O3", "-lineinfo",
    "-Xcompiler", "-fPIC", "--shared", "--threads", "8",
    "-Xlinker", "--version-script=" + os.path.join(CSRC, "gtok.map"),
]
SOURCES = ["encode_kernels.cu", "tiny_kernel.cu", "engine.cu", "gtok_abi.cc", "vocab_host.cc", "tables_build.cc", "nfc_host.cc", "host_text.cc"]


def _newer(target, deps):
    if not os.path.exists(target):
        return True
    t = os.path.getmtime(target)
    return any(os.path.getmtime(d) > t for d in deps)


def source_hash():
    """Short hash of the native sources (csrc/ and the C ABI header): identifies the build a
    measurement or a profile summary was taken from."""
    import hashlib
    h = hashlib.sha256()
    for name in sorted(os.listdir(CSRC)):
        if name.endswith((".h", ".cu", ".cc", ".map")):
            with open(os.path.join(CSRC, name), "rb") as f:
                h.update(name.encode() + b"\0" + f.read())
    with open(os.path.join(HERE, "..", "include", "gtok.h"), "rb") as f:
        h.update(f.read())
    return h.hexdigest()[:16]


def _nvcc():
    return shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"


def build_lib(force=False, verbose=False):
    deps = [os.path.join(CSRC, f) for f in os.listdir(CSRC)] + [os.path.join(HERE, "..", "include", "gtok.h")]
    if not force and not _newer(LIB, deps):
        return LIB
    os.makedirs(LIB_DIR, exist_ok=True)
    cmd = [_nvcc()] + NVCC_FLAGS + (["-Xptxas", "-v"] if verbose else []) + ["-o", LIB + ".part"] + [os.path.join(CSRC, s) for s in SOURCES]
    subprocess.run(cmd, check=True)
    os.replace(LIB + ".part", LIB)               # a build that was cut short leaves no library behind
    return LIB


def build_datagen(force=False):
    src = [os.path.join(HERE, "datagen", f) for f in ("datagen.cc", "seqsplit.h")] + [os.path.join(CSRC, f) for f in ("unicode_class_table.h", "unicode_wide_table.h")]
    if not force and not _newer(DATAGEN, src):
        return DATAGEN
    subprocess.run(["g++", "-std=c++17", "-O2", "-o", DATAGEN, src[0]], check=True)
    return DATAGEN


CLI = os.path.join(HERE, "cli", "gpu_bpe_tokenize")


def build_cli(force=False):
    """The command-line tool over libgtok.so (the reference's gpu_bpe_tokenize modes and output files)."""
    src = os.path.join(HERE, "cli", "gpu_bpe_tokenize.cc")
    if not force and not _newer(CLI, [src, os.path.join(HERE, "..", "include", "gtok.h"), LIB]):
        return CLI
    subprocess.run(["g++", "-std=c++17", "-O2", "-o", CLI, src, "-L" + LIB_DIR, "-l:libgtok.so", "-Wl,-rpath," + LIB_DIR], check=True)
    return CLI


HOST = os.path.join(HERE, "_host.so")


def _host_includes():
    """Folders with the headers of this interpreter and of numpy, or the name of what is missing."""
    import sysconfig
    python = [d for d in (sysconfig.get_paths().get(k) for k in ("include", "platinclude")) if d and os.path.exists(os.path.join(d, "Python.h"))]
    if not python:
        return "Python.h"
    try:
        import numpy
    except ImportError:
        return "numpy"
    if not os.path.exists(os.path.join(numpy.get_include(), "numpy", "arrayobject.h")):
        return "numpy/arrayobject.h"
    return python[:1] + [numpy.get_include()]


def build_host(force=False):
    """The CPython extension between the Python classes and libgtok.so; None where it cannot be built, and the classes
    then go by ctypes (ctypes_host.py)."""
    src = os.path.join(HERE, "pyhost", "host_module.cc")
    if not force and not _newer(HOST, [src, os.path.join(HERE, "pyhost", "result_memory.h"), os.path.join(HERE, "..", "include", "gtok.h")]):
        return HOST
    if os.path.exists(HOST):
        os.remove(HOST)          # an outdated one must not be loaded
    why = _host_includes()
    if not isinstance(why, str):
        cmd = ["g++", "-std=c++17", "-O3", "-fPIC", "-shared", "-fvisibility=hidden"] + ["-I" + d for d in why] + [
            "-o", HOST, src]
        done = subprocess.run(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
        if done.returncode == 0:
            return HOST
        why = next((line for line in done.stdout.splitlines() if "error" in line), "g++ exit code %d" % done.returncode)
    print("graphtok_b200: extension _host left out, ctypes in its place (%s)" % why, flush=True)
    return None


def main():
    force = "--force" in sys.argv
    build_lib(force=force, verbose="-v" in sys.argv)
    build_datagen(force=force)
    build_cli(force=force)
    host = build_host(force=force)
    print(LIB)
    print(DATAGEN)
    print(CLI)
    if host:
        print(host)


if __name__ == "__main__":
    main()
