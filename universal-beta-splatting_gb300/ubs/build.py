"""Build the GB300 rasteriser library (libubs_gb300.so) from csrc/ with nvcc and
the host extension module on top of it (ubs_native.so, csrc/host/) with g++.

Translation units are compiled in parallel for sm_103a only and linked into
one shared library inside the package tree (_build/), which is what the
ctypes loader in ubs._lib opens; the module links to that library.
"""
import concurrent.futures as cf
import hashlib
import os
import shutil
import subprocess
import sys
import sysconfig

PKG_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(PKG_ROOT, "csrc")
INCLUDE = os.path.join(os.path.dirname(PKG_ROOT), "include")
BUILD = os.path.join(PKG_ROOT, "_build")
LIB_NAME = "libubs_gb300.so"
LIB_PATH = os.path.join(BUILD, LIB_NAME)
HOST_SRC = os.path.join(CSRC, "host", "native.cpp")
NATIVE_PATH = os.path.join(BUILD, "ubs_native.so")

ARCH = ["-gencode", "arch=compute_103a,code=sm_103a"]
NVCC_FLAGS = ["-O3", "-lineinfo", "-std=c++17", "-Xcompiler", "-fPIC",
              "--expt-relaxed-constexpr", "-diag-suppress", "128"]
# Every translation unit is built with fast math, as the reference's own CUDA
# operators are (submodules/setup.py), except those that must round like
# PyTorch's IEEE elementwise kernels (the parameter activations of the fused
# render: scene_act.cu).
FAST_MATH = ["--use_fast_math"]
IEEE_SOURCES = ("scene_act.cu",)


def _flags(src):
    return NVCC_FLAGS + ([] if os.path.basename(src) in IEEE_SOURCES else FAST_MATH)


def _nvcc():
    for c in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if c and os.path.exists(c):
            return c
    raise RuntimeError("nvcc not found: the GB300 rasteriser needs the CUDA toolkit to build")


def _sources():
    return sorted(os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith(".cu"))


def _host_compile(obj):
    """g++ command of the extension module's object (PyTorch's headers)."""
    import torch
    from torch.utils import cpp_extension
    inc = cpp_extension.include_paths("cuda") + [sysconfig.get_paths()["include"]]
    return (["g++", "-O2", "-std=c++17", "-fPIC", "-Wall", "-Wno-sign-compare",
             "-DTORCH_API_INCLUDE_EXTENSION_H",
             "-D_GLIBCXX_USE_CXX11_ABI=%d" % int(torch._C._GLIBCXX_USE_CXX11_ABI)]
            + [a for i in inc for a in ("-isystem", i)] + ["-c", HOST_SRC, "-o", obj])


def _host_link(obj, out):
    from torch.utils import cpp_extension
    return (["g++", "-shared", obj, "-o", out, "-L" + BUILD, "-l:" + LIB_NAME,
             "-Wl,-rpath,$ORIGIN"]
            + ["-L" + d for d in cpp_extension.library_paths("cuda")]
            + ["-ltorch_python", "-ltorch", "-ltorch_cuda", "-ltorch_cpu", "-lc10_cuda", "-lc10",
               "-lcudart"])


def _fingerprint():
    import torch
    h = hashlib.sha256()
    h.update(torch.__version__.encode())
    files = _sources() + sorted(os.path.join(CSRC, f) for f in os.listdir(CSRC)
                                if f.endswith((".cuh", ".h")))
    files += [os.path.join(INCLUDE, "ubs.h"), HOST_SRC]
    for f in files:
        h.update(f.encode())
        with open(f, "rb") as fh:
            h.update(fh.read())
    h.update(" ".join(ARCH + NVCC_FLAGS + FAST_MATH + list(IEEE_SOURCES)).encode())
    return h.hexdigest()


def build(force=False, verbose=False, jobs=None):
    """Compile (if sources changed) and return the path of the shared library."""
    os.makedirs(BUILD, exist_ok=True)
    stamp = os.path.join(BUILD, "stamp.txt")
    fp = _fingerprint()
    if not force and all(map(os.path.exists, (LIB_PATH, NATIVE_PATH, stamp))):
        with open(stamp) as f:
            if f.read().strip() == fp:
                return LIB_PATH
    nvcc = _nvcc()
    objs = []
    cmds = []
    for src in _sources():
        obj = os.path.join(BUILD, os.path.basename(src)[:-3] + ".o")
        objs.append(obj)
        cmds.append([nvcc] + ARCH + _flags(src) + ["-I", INCLUDE, "-c", src, "-o", obj])

    host_obj = os.path.join(BUILD, "native.o")
    cmds.append(_host_compile(host_obj))

    def run(cmd):
        if verbose:
            print(" ".join(cmd), flush=True)
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError("build failed:\n%s\n%s" % (" ".join(cmd), r.stderr[-4000:]))
        return r

    with cf.ThreadPoolExecutor(max_workers=jobs or min(len(cmds), os.cpu_count() or 4)) as ex:
        list(ex.map(run, cmds))
    tmp = LIB_PATH + ".tmp%d" % os.getpid()
    run([nvcc] + ARCH + ["-shared", "-cudart", "static", "-o", tmp] + objs)
    os.replace(tmp, LIB_PATH)
    tmp = NATIVE_PATH + ".tmp%d" % os.getpid()
    run(_host_link(host_obj, tmp))
    os.replace(tmp, NATIVE_PATH)
    with open(stamp, "w") as f:
        f.write(fp)
    return LIB_PATH


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose=True))
