"""Build the C-ABI CUDA library in-tree with nvcc for sm_100a, and the C++ module of the eager path against it and torch.

    python -m flashnystrom_b200.build            # build if sources are newer than the .so
    python -m flashnystrom_b200.build --force

The results are flashnystrom_b200/lib/libflashnystrom_b200.so and the module beside it; nothing is installed elsewhere.  The module's
name holds a digest of its source, the header, the flags and the versions of torch and Python: another one of these
means another file, so that a module is never taken that does not fit.  FNB_LIB_NAME names a variant of the CUDA library for
measurements, which nothing here loads; the module is always linked to the library that the package loads.

Files are written under a temporary name and renamed, one process at a time: ranks of a job that meet a tree
without them build once, and none loads half a file.
"""
import contextlib
import fcntl
import glob
import hashlib
import os
import shutil
import subprocess
import sys
import sysconfig

PKG = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(PKG, "csrc")
LIB_DIR = os.path.join(PKG, "lib")
PACKAGE_LIB = os.path.join(LIB_DIR, "libflashnystrom_b200.so")
LIB_PATH = os.path.join(LIB_DIR, os.environ.get("FNB_LIB_NAME", os.path.basename(PACKAGE_LIB)))
SOURCES = ["fnb_api.cu"]
NATIVE_SOURCE = os.path.join(CSRC, "native.cpp")
NATIVE_FLAGS = ["-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden"]
HEADER = os.path.join(os.path.dirname(PKG), "include", "flashnystrom_b200.h")

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC", "-Xcompiler", "-fvisibility=hidden", "-shared",
]
if os.environ.get("FNB_PTXAS_VERBOSE"):      # registers, spills, shared memory per kernel
    NVCC_FLAGS += ["-Xptxas", "-v"]
NVCC_FLAGS += os.environ.get("FNB_EXTRA_NVCC_FLAGS", "").split()   # e.g. -DFNB_NS_TRACE for a profiling build


def _nvcc():
    exe = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(exe):
        raise RuntimeError("nvcc not found; the CUDA toolkit is required to build flashnystrom_b200")
    return exe


@contextlib.contextmanager
def _one_at_a_time():
    os.makedirs(LIB_DIR, exist_ok=True)
    fd = os.open(LIB_DIR, os.O_RDONLY)
    try:
        with contextlib.suppress(OSError):      # (a file system without locks: the work may be done twice, the files are whole)
            fcntl.flock(fd, fcntl.LOCK_EX)
        yield
    finally:
        os.close(fd)


def _compile(cmd, path, what, verbose):
    """cmd with its output brought to `path` when it is complete."""
    part = f"{path[:-3]}.part{os.getpid()}.so"
    cmd = cmd + ["-o", part]
    if verbose:
        print(" ".join(cmd))
    try:
        res = subprocess.run(cmd, capture_output=True, text=True)
        if res.returncode != 0:
            raise RuntimeError(f"{what} failed:\n" + res.stdout + res.stderr)
        os.replace(part, path)
    finally:
        with contextlib.suppress(FileNotFoundError):
            os.remove(part)
    return res.stdout + res.stderr


def _stale(path):
    if not os.path.exists(path):
        return True
    t = os.path.getmtime(path)
    deps = [os.path.join(CSRC, f) for f in os.listdir(CSRC) if not f.endswith(".cpp")]
    deps.append(HEADER)
    return any(os.path.getmtime(d) > t for d in deps if os.path.exists(d))


def native_path():
    """Where the C++ module for this source, interpreter and torch is."""
    import torch
    versions = f"{sys.implementation.cache_tag}-torch{torch.__version__}"
    digest = hashlib.sha256(repr((versions, NATIVE_FLAGS)).encode())
    for name in (NATIVE_SOURCE, HEADER):
        with open(name, "rb") as f:
            digest.update(f.read())
    return os.path.join(LIB_DIR, f"_native.{versions}.{digest.hexdigest()[:16]}.so")


def build_native(force=False, verbose=False):
    """The C++ module: host code only, linked to the CUDA library that the package loads."""
    path = native_path()
    if not force and os.path.exists(path):
        return path
    build_library(verbose=verbose, path=PACKAGE_LIB)
    import torch
    from torch.utils import cpp_extension
    cuda = os.path.dirname(os.path.dirname(_nvcc()))
    torch_lib = os.path.join(os.path.dirname(torch.__file__), "lib")
    cmd = [os.environ.get("CXX", "g++")] + NATIVE_FLAGS
    cmd += ["-I" + p for p in cpp_extension.include_paths()]
    cmd += ["-I" + sysconfig.get_paths()["include"], "-I" + os.path.join(cuda, "include"),
            f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}", NATIVE_SOURCE,
            "-L" + torch_lib, "-lc10", "-lc10_cuda", "-ltorch", "-ltorch_cpu", "-ltorch_cuda", "-ltorch_python",
            "-L" + LIB_DIR, "-l:" + os.path.basename(PACKAGE_LIB), "-Wl,-rpath,$ORIGIN"]
    with _one_at_a_time():
        if not force and os.path.exists(path):      # (another process was faster)
            return path
        _compile(cmd, path, "the C++ compiler", verbose)
        for old in glob.glob(glob.escape(path.rsplit(".", 2)[0]) + ".*.so"):      # of this interpreter and torch
            if old != path and ".part" not in old:
                os.remove(old)
    return path


def build(force=False, verbose=False):
    """Both, the CUDA library first; its path."""
    path = build_library(force, verbose)
    if path == PACKAGE_LIB:
        build_native(force, verbose)
    return path


def build_library(force=False, verbose=False, path=None):
    path = path or LIB_PATH
    if not force and not _stale(path):
        return path
    cmd = [_nvcc()] + NVCC_FLAGS + [os.path.join(CSRC, s) for s in SOURCES]
    with _one_at_a_time():
        if not force and not _stale(path):
            return path
        log = _compile(cmd, path, "nvcc", verbose)
    if verbose or os.environ.get("FNB_PTXAS_VERBOSE"):
        print(log)
    return path


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose=True))
