"""Builds ``libscn_b200.so`` (the C-ABI library declared in ``include/scn_b200.h``) in-tree.

Every ``csrc/*.cu`` is compiled for sm_100a only
(``-gencode arch=compute_100a,code=sm_100a``) and linked into one shared library next to
this file.  nvcc cross-compiles without a GPU.  ``csrc/binding.cpp`` (the operator calls of ``SCN.py`` as a
CPython module on torch tensors) becomes ``_binding*.so`` beside it.

Usage:  python sparseconvnet_b200/build.py [--force] [--verbose]
(run as a script: importing the package needs the library this builds)
"""
import concurrent.futures as cf
import glob
import os
import subprocess
import sys
import sysconfig

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
LIB = os.path.join(HERE, "libscn_b200.so")
BINDING = os.path.join(HERE, "_binding" + (sysconfig.get_config_var("EXT_SUFFIX") or ".so"))
NVCC = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
         "-Xcompiler", "-fPIC", "-Xcompiler", "-fvisibility=hidden", "--expt-relaxed-constexpr"]


def _sources():
    return sorted(glob.glob(os.path.join(CSRC, "*.cu")))


def _deps():
    return _sources() + glob.glob(os.path.join(CSRC, "*.cuh")) + \
        glob.glob(os.path.join(HERE, "..", "include", "*.h"))


def _binding_deps():
    return [os.path.join(CSRC, "binding.cpp")] + glob.glob(os.path.join(HERE, "..", "include", "*.h"))


def _older(target, deps):
    return not os.path.exists(target) or any(os.path.getmtime(f) > os.path.getmtime(target) for f in deps)


def needs_build():
    return _older(LIB, _deps())


def build_binding():
    """g++ against torch's headers; finds libscn_b200.so beside itself."""
    import torch
    root = os.path.dirname(torch.__file__)
    cmd = [os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden",
           os.path.join(CSRC, "binding.cpp"), "-o", BINDING,
           "-D_GLIBCXX_USE_CXX11_ABI=%d" % int(torch._C._GLIBCXX_USE_CXX11_ABI),
           "-I" + os.path.join(root, "include"), "-I" + os.path.join(root, "include", "torch", "csrc", "api", "include"),
           "-I" + os.path.join(os.path.dirname(os.path.dirname(NVCC)), "include"),
           "-I" + sysconfig.get_paths()["include"],
           "-L" + os.path.join(root, "lib"), "-ltorch_python", "-ltorch", "-ltorch_cpu", "-lc10", "-lc10_cuda",
           "-L" + HERE, "-l:libscn_b200.so", "-Wl,-rpath,$ORIGIN"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError("binding failed:\n%s" % r.stderr[-6000:])


def _compile(src, verbose):
    obj = os.path.join(HERE, "build", os.path.basename(src)[:-3] + ".o")
    hdr_t = max(os.path.getmtime(f) for f in _deps() if not f.endswith(".cu"))
    if os.path.exists(obj) and os.path.getmtime(obj) > max(os.path.getmtime(src), hdr_t):
        return obj
    cmd = [NVCC, "-c", src, "-o", obj] + FLAGS + (["-Xptxas", "-v"] if verbose else [])
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError("nvcc failed on %s:\n%s" % (src, r.stderr[-6000:]))
    if verbose:
        sys.stderr.write(r.stderr)
    return obj


def build(force=False, verbose=False):
    if not force and not needs_build():
        if _older(BINDING, _binding_deps()):
            build_binding()
        return LIB
    os.makedirs(os.path.join(HERE, "build"), exist_ok=True)
    if force:
        for f in glob.glob(os.path.join(HERE, "build", "*.o")):
            os.remove(f)
    with cf.ThreadPoolExecutor(max(1, min(8, os.cpu_count() or 1))) as ex:
        objs = list(ex.map(lambda s: _compile(s, verbose), _sources()))
    cmd = [NVCC, "-shared", "-o", LIB] + objs + ["-gencode", "arch=compute_100a,code=sm_100a",
                                                   "-lcudart"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError("link failed:\n%s" % r.stderr[-4000:])
    if force or _older(BINDING, _binding_deps()):
        build_binding()
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="--verbose" in sys.argv))
