"""In-tree build of the native library ``fastfold_b200/lib/libffb200.so``.

Every ``csrc/*.cu`` is compiled for sm_100a only (``-gencode
arch=compute_100a,code=sm_100a``) with relocatable device code and linked into
one shared object that the Python side loads through ``ctypes``.  The kernel
sources do not include PyTorch headers and build in well under a minute; the one
file that does, ``csrc/host/dispatch.cpp`` (the native side of the operator
calls), becomes the extension module ``lib/_ffb_dispatch.so``, linked against
the kernel library and tied to the PyTorch it was built with.

Replaces the reference's ``setup.py`` CUDAExtension build (setup.py:89-125),
which targets sm_70/sm_80.
"""
import fcntl
import hashlib
import importlib.util
import os
import subprocess
import sys
from concurrent.futures import ThreadPoolExecutor

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
LIBDIR = os.path.join(HERE, "lib")
LIBNAME = "libffb200.so"
DISPATCH = "_ffb_dispatch"
NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "-rdc=true", "-Xcompiler", "-fPIC", "-Xptxas", "-v",
]


def _nvcc():
    cand = os.environ.get("NVCC") or os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "bin", "nvcc")
    return cand if os.path.exists(cand) else "nvcc"


def sources():
    return sorted(os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith(".cu"))


def _hash(paths, *texts):
    h = hashlib.sha256()
    for f in paths:
        with open(f, "rb") as fh:
            h.update(os.path.basename(f).encode())
            h.update(fh.read())
    h.update(" ".join(texts).encode())
    return h.hexdigest()


def _csrc(*suffixes):
    return sorted(os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith(suffixes))


def _digest():
    """What the kernel library is made from."""
    return _hash(_csrc(".cu", ".cuh", ".h"), *NVCC_FLAGS)


def _dispatch_digest():
    """What the extension module is made from: the PyTorch and the Python whose headers it includes belong to that."""
    import torch
    return _hash(_csrc(".h") + [os.path.join(CSRC, "host", "dispatch.cpp")], torch.__version__, sys.version)


def lib_path():
    return os.path.join(LIBDIR, LIBNAME)


def dispatch_path():
    return os.path.join(LIBDIR, DISPATCH + ".so")


def _stamp(name):
    try:
        with open(os.path.join(LIBDIR, name)) as fh:
            return fh.read().strip()
    except FileNotFoundError:
        return None


def kernels_current():
    return os.path.exists(lib_path()) and _stamp("build.stamp") == _digest()


def dispatch_current():
    return os.path.exists(dispatch_path()) and _stamp("dispatch.stamp") == _dispatch_digest()


def is_current():
    return kernels_current() and dispatch_current()


def stale():
    """Why the built files must not be loaded, or None.  Files that came without their stamps are taken as they are."""
    for path, stamp, digest, what in ((lib_path(), "build.stamp", _digest, "other sources"),
                                      (dispatch_path(), "dispatch.stamp", _dispatch_digest, "other sources or another PyTorch or Python")):
        if not os.path.exists(path):
            return "%s is missing" % path
        if _stamp(stamp) not in (None, digest()):
            return "%s was built from %s" % (path, what)
    return None


def ensure():
    """Builds what is missing or stale; RuntimeError where that is not possible."""
    why = stale()
    if why is None:
        return
    try:
        build(verbose=False)
    except Exception as e:  # no compiler, no right to write
        raise RuntimeError("fastfold_b200: native code: %s and could not be rebuilt (%s). Run `python -m fastfold_b200._build` on a "
                           "machine with nvcc and a C++ compiler." % (why, e))


def build(force=False, verbose=True):
    """Compile and link what is not current; returns the path of the kernel library.  One process at a time: the ranks of a
    job may all find the same stale file."""
    have_torch = importlib.util.find_spec("torch") is not None

    def todo():
        return force or not kernels_current(), have_torch and (force or not dispatch_current())

    if not any(todo()):
        return lib_path()
    os.makedirs(LIBDIR, exist_ok=True)
    with open(os.path.join(LIBDIR, ".lock"), "w") as lock, ThreadPoolExecutor(max_workers=1) as ex:
        fcntl.flock(lock, fcntl.LOCK_EX)
        kernels, dispatch = todo()
        host = ex.submit(_compile_dispatch) if dispatch else None
        if kernels:
            _build_kernels()
        if dispatch:
            _link_dispatch(*host.result())               # against the kernel library, whose symbols it needs
    if verbose:
        print("built", lib_path() if kernels else "", dispatch_path() if dispatch else "")
        if not have_torch:
            print("fastfold_b200: no PyTorch here; %s is built when it is first used" % dispatch_path())
    return lib_path()


def _run(cmd, what):
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError("%s failed:\n%s" % (what, r.stdout + r.stderr))
    return r.stdout + r.stderr


def _install(built, path, stamp, digest):
    """A file that a running process may have loaded is replaced, never written over."""
    os.replace(built, path)
    with open(os.path.join(LIBDIR, stamp), "w") as fh:
        fh.write(digest)


def _objdir():
    objdir = os.path.join(LIBDIR, "obj")
    os.makedirs(objdir, exist_ok=True)
    return objdir


def _build_kernels():
    objdir, nvcc, srcs, logs = _objdir(), _nvcc(), sources(), {}

    def compile_one(src):
        obj = os.path.join(objdir, os.path.basename(src)[:-3] + ".o")
        logs[src] = _run([nvcc] + NVCC_FLAGS + ["-I", CSRC, "-c", src, "-o", obj], "nvcc on %s" % src)
        return obj

    with ThreadPoolExecutor(max_workers=min(8, len(srcs))) as ex:
        objs = list(ex.map(compile_one, srcs))
    built = os.path.join(objdir, LIBNAME)
    _run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "--shared", "-Xcompiler", "-fPIC", "-o", built] + objs + ["-lcudart"], "link")
    with open(os.path.join(LIBDIR, "ptxas.log"), "w") as fh:
        for s in srcs:
            fh.write("==== %s\n%s\n" % (os.path.basename(s), logs[s]))
    _install(built, lib_path(), "build.stamp", _digest())


def _compile_dispatch():
    import sysconfig
    import torch
    tdir = os.path.dirname(torch.__file__)
    src, obj = os.path.join(CSRC, "host", "dispatch.cpp"), os.path.join(_objdir(), "dispatch.o")
    inc = [CSRC, os.path.join(tdir, "include"), os.path.join(tdir, "include", "torch", "csrc", "api", "include"),
           os.path.join(os.path.dirname(os.path.dirname(_nvcc())) or "/usr/local/cuda", "include"), sysconfig.get_paths()["include"]]
    cmd = ["g++", "-O2", "-std=c++17", "-fPIC", "-fvisibility=hidden", "-DTORCH_EXTENSION_NAME=" + DISPATCH,
           "-D_GLIBCXX_USE_CXX11_ABI=%d" % int(torch._C._GLIBCXX_USE_CXX11_ABI)]
    _run(cmd + [a for d in inc for a in ("-I", d)] + ["-c", src, "-o", obj], "g++ on %s" % src)
    return obj, os.path.join(tdir, "lib")


def _link_dispatch(obj, torch_lib):
    built = os.path.join(_objdir(), DISPATCH + ".so")
    _run(["g++", "-shared", "-o", built, obj, "-L", LIBDIR, "-lffb200", "-Wl,-rpath,$ORIGIN", "-L", torch_lib,
          "-ltorch", "-ltorch_cpu", "-ltorch_python", "-lc10", "-lc10_cuda"], "link")
    _install(built, dispatch_path(), "dispatch.stamp", _dispatch_digest())


if __name__ == "__main__":
    build(force="--force" in sys.argv)
