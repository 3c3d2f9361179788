"""Builds libexact_b200.so (the C-ABI CUDA library) in-tree with nvcc for sm_100a."""
import os
import subprocess
from concurrent.futures import ThreadPoolExecutor

PKG = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(PKG)
CSRC = os.path.join(PKG, "csrc")
INCLUDE = os.path.join(ROOT, "include")
LIBDIR = os.path.join(PKG, "lib")
OBJDIR = os.path.join(PKG, "build")
LIB = os.path.join(LIBDIR, "libexact_b200.so")
NATIVE = os.path.join(LIBDIR, "_native.so")   # the host path on torch tensors (csrc/native*.cpp)

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC", "-Xcompiler", "-fvisibility=hidden", "-I", INCLUDE, "-I", CSRC,
]


def _nvcc():
    for cand in (os.environ.get("NVCC"), "/usr/local/cuda/bin/nvcc", "nvcc"):
        if cand and (os.path.sep not in cand or os.path.exists(cand)):
            return cand
    return "nvcc"


def sources():
    return sorted(os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith(".cu"))


def _stale(target, deps):
    if not os.path.exists(target):
        return True
    t = os.path.getmtime(target)
    return any(os.path.getmtime(d) > t for d in deps)


def build_native(force=False):
    """Compile csrc/native*.cpp against this interpreter's torch and link lib/_native.so.  Returns its path."""
    import sysconfig
    import torch
    from torch.utils.cpp_extension import include_paths
    os.makedirs(LIBDIR, exist_ok=True)
    os.makedirs(OBJDIR, exist_ok=True)
    torch_lib = os.path.join(os.path.dirname(torch.__file__), "lib")
    cuda = os.path.dirname(os.path.dirname(_nvcc())) if os.path.sep in _nvcc() else "/usr/local/cuda"
    flags = ["-O2", "-std=c++17", "-fPIC", "-fvisibility=hidden", "-D_GLIBCXX_USE_CXX11_ABI=%d" % torch._C._GLIBCXX_USE_CXX11_ABI,
             "-I", INCLUDE, "-I", CSRC, "-isystem", sysconfig.get_paths()["include"], "-isystem", os.path.join(cuda, "include")]
    for inc in include_paths():
        flags += ["-isystem", inc]
    deps = [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.startswith("native") and f.endswith(".h")]
    deps += [os.path.join(INCLUDE, f) for f in os.listdir(INCLUDE)]
    jobs, objs = [], []
    for f in sorted(os.listdir(CSRC)):
        if f.endswith(".cpp"):
            src, obj = os.path.join(CSRC, f), os.path.join(OBJDIR, f[:-4] + ".host.o")
            objs.append(obj)
            if force or _stale(obj, [src] + deps):
                jobs.append(["g++"] + flags + ["-c", src, "-o", obj])
    _run_all(jobs)
    if jobs or force or _stale(NATIVE, objs):
        _run(["g++", "-shared", "-o", NATIVE] + objs + ["-L", torch_lib, "-Wl,-rpath," + torch_lib, "-ltorch_python", "-ltorch",
              "-ltorch_cuda", "-ltorch_cpu", "-lc10_cuda", "-lc10", "-L", os.path.join(cuda, "lib64"), "-lcudart", "-ldl"])
    return NATIVE


def _run(cmd):
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError("%s failed: %s\n%s\n%s" % (os.path.basename(cmd[0]), " ".join(cmd), r.stdout, r.stderr))
    return r.stderr


def _run_all(jobs):
    if not jobs:
        return []
    with ThreadPoolExecutor(max_workers=min(8, len(jobs))) as ex:
        return list(ex.map(_run, jobs))


def build(force=False, verbose=False):
    """Compile every .cu under csrc/ and link lib/libexact_b200.so, then the host path.  Returns the library path."""
    os.makedirs(LIBDIR, exist_ok=True)
    os.makedirs(OBJDIR, exist_ok=True)
    headers = [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith((".cuh", ".h"))]
    headers += [os.path.join(INCLUDE, f) for f in os.listdir(INCLUDE)]
    nvcc = _nvcc()
    jobs = []
    objs = []
    for src in sources():
        obj = os.path.join(OBJDIR, os.path.basename(src)[:-3] + ".o")
        objs.append(obj)
        if force or _stale(obj, [src] + headers):
            jobs.append([nvcc] + NVCC_FLAGS + (["-Xptxas", "-v"] if verbose else []) + ["-c", src, "-o", obj])

    logs = _run_all(jobs)
    if jobs and verbose:
        print("\n".join(logs))
    if jobs or force or _stale(LIB, objs):
        _run([nvcc, "-shared", "-o", LIB] + objs + ["-gencode", "arch=compute_100a,code=sm_100a"])
    build_native(force)
    return LIB


if __name__ == "__main__":
    import sys
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
