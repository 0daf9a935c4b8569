"""Builds ``libjitnn_b200.so`` in-tree with nvcc for sm_100a and, where a torch with CUDA is installed, the native front of Python's calls on torch tensors.

    python -m jitnn_b200.build [--force] [--verbose]

Each ``csrc/*.cu`` is compiled to an object under ``csrc/build/`` (only when it or a header is
newer than its object) and the objects are linked into ``jitnn_b200/libjitnn_b200.so``. The front (``csrc/front.cpp``) is a convenience of
the Python binding: the library does not need it, and is built whatever becomes of it.
"""
import concurrent.futures
import glob
import os
import shutil
import subprocess
import sys
import sysconfig
from importlib.util import find_spec

from jitnn_b200 import _lib

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
OBJ = os.path.join(CSRC, "build")
LIB = os.path.join(HERE, "libjitnn_b200.so")
FRONT_SRC = os.path.join(CSRC, "front.cpp")

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC", "-Xcompiler", "-fvisibility=hidden", "--expt-relaxed-constexpr",
]


def nvcc():
    path = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(path):
        raise RuntimeError("nvcc not found: the CUDA toolkit is needed to build libjitnn_b200.so")
    return path


def _newest_header():
    heads = glob.glob(os.path.join(CSRC, "*.cuh")) + glob.glob(os.path.join(HERE, "..", "include", "*.h"))
    return max(os.path.getmtime(h) for h in heads)


def _compile(src, obj, verbose, extra):
    cmd = [nvcc()] + NVCC_FLAGS + extra + ["-c", src, "-o", obj]
    res = subprocess.run(cmd, capture_output=True, text=True)
    if res.returncode != 0:
        raise RuntimeError("nvcc failed for %s:\n%s\n%s" % (src, res.stdout, res.stderr))
    if verbose:
        sys.stderr.write(res.stdout + res.stderr)


def build_front(force=False):
    """The front for this Python and the installed torch, whose versions its name carries; None where there is no torch with CUDA to build it against."""
    front, spec = _lib.front_path(), find_spec("torch")
    if front is None or spec is None or spec.origin is None:
        return None
    torch = os.path.dirname(spec.origin)
    if not os.path.exists(os.path.join(torch, "lib", "libtorch_cuda.so")):
        return None
    if not force and os.path.exists(front) and os.path.getmtime(front) >= os.path.getmtime(FRONT_SRC):
        return front
    cuda = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(nvcc()))), "include")
    cmd = [shutil.which("g++") or "c++", "-O2", "-std=c++17", "-shared", "-fPIC", "-fvisibility=hidden"]
    cmd += ["-I" + d for d in (os.path.join(torch, "include"), os.path.join(torch, "include", "torch", "csrc", "api", "include"), sysconfig.get_path("include"), cuda)]
    cmd += [FRONT_SRC, "-o", front, "-L" + os.path.join(torch, "lib"), "-ltorch_python", "-ltorch", "-ltorch_cpu", "-ltorch_cuda", "-lc10", "-lc10_cuda"]
    res = subprocess.run(cmd, capture_output=True, text=True)
    if res.returncode != 0:
        raise RuntimeError("the build of %s failed:\n%s\n%s" % (os.path.basename(front), res.stdout, res.stderr))
    for old in glob.glob(os.path.join(os.path.dirname(front), "_front*.so")):
        if old != front:
            os.remove(old)  # another torch's
    return front


def build(force=False, verbose=False, ptxas_info=False):
    os.makedirs(OBJ, exist_ok=True)
    sources = sorted(glob.glob(os.path.join(CSRC, "*.cu")))
    header_time = _newest_header()
    jobs = []
    objects = []
    extra = ["-Xptxas", "-v"] if ptxas_info else []
    for src in sources:
        obj = os.path.join(OBJ, os.path.basename(src)[:-3] + ".o")
        objects.append(obj)
        stale = force or not os.path.exists(obj) or os.path.getmtime(obj) < max(os.path.getmtime(src), header_time)
        if stale:
            jobs.append((src, obj))
    with concurrent.futures.ThreadPoolExecutor(max_workers=max(1, os.cpu_count() or 1)) as pool:
        front = pool.submit(build_front, force)
        for f in [pool.submit(_compile, s, o, verbose or ptxas_info, extra) for s, o in jobs]:
            f.result()
    if jobs or not os.path.exists(LIB):
        cmd = [nvcc(), "-shared", "-o", LIB] + objects + ["-gencode", "arch=compute_100a,code=sm_100a", "-cudart", "static"]
        res = subprocess.run(cmd, capture_output=True, text=True)
        if res.returncode != 0:
            raise RuntimeError("link failed:\n%s\n%s" % (res.stdout, res.stderr))
    try:
        front.result()
    except (RuntimeError, OSError) as e:
        sys.stderr.write("%s\nCalls on torch tensors go without the native front.\n" % e)
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="--verbose" in sys.argv, ptxas_info="--ptxas" in sys.argv))
