"""Compile the CUDA sources under caif_b200/csrc into caif_b200/libcaifq.so.

The torch side of the Python binding (binding/torch_binding.cpp) becomes caif_b200/_torch_binding.so.

sm_100a only (`-gencode arch=compute_100a,code=sm_100a`); nvcc cross-compiles
without a GPU.  Objects are cached under caif_b200/build/ and rebuilt when a
source or header is newer.
"""
import os
import subprocess
import sys
import sysconfig
from concurrent.futures import ThreadPoolExecutor

PKG = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(PKG)
CSRC = os.path.join(PKG, "csrc")
OBJ_DIR = os.path.join(PKG, "build")
LIB = os.path.join(PKG, "libcaifq.so")
BINDING_SRC = os.path.join(PKG, "binding", "torch_binding.cpp")
BINDING = os.path.join(PKG, "_torch_binding.so")

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC", "-Xcompiler", "-fvisibility=hidden",
    "-I", os.path.join(ROOT, "include"), "-I", CSRC,
]


def _sources():
    return sorted(f for f in os.listdir(CSRC) if f.endswith(".cu"))


def _headers():
    hs = [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith((".cuh", ".h"))]
    hs.append(os.path.join(ROOT, "include", "caifq.h"))
    return hs


def _compile_one(src, verbose):
    obj = os.path.join(OBJ_DIR, src[:-3] + ".o")
    deps = [os.path.join(CSRC, src)] + _headers()
    if os.path.exists(obj) and all(os.path.getmtime(d) <= os.path.getmtime(obj) for d in deps):
        return obj, False
    cmd = ["nvcc"] + NVCC_FLAGS + (["-Xptxas", "-v"] if verbose else []) + ["-c", os.path.join(CSRC, src), "-o", obj]
    res = subprocess.run(cmd, capture_output=True, text=True)
    if verbose and res.stderr:
        sys.stderr.write(res.stderr)
    if res.returncode != 0:
        raise RuntimeError("nvcc failed for %s:\n%s\n%s" % (src, res.stdout, res.stderr))
    return obj, True


def build_binding(force=False):
    deps = [BINDING_SRC, os.path.join(ROOT, "include", "caifq.h")]
    if not force and os.path.exists(BINDING) and all(os.path.getmtime(d) <= os.path.getmtime(BINDING) for d in deps):
        return BINDING
    import torch

    t = os.path.dirname(torch.__file__)
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    cmd = ["g++", "-std=c++20", "-O2", "-fPIC", "-shared", "-fvisibility=hidden", "-Wno-stringop-overflow",
           "-D_GLIBCXX_USE_CXX11_ABI=%d" % torch._C._GLIBCXX_USE_CXX11_ABI, "-I", os.path.join(ROOT, "include"),
           "-I", os.path.join(t, "include"), "-I", os.path.join(t, "include", "torch", "csrc", "api", "include"),
           "-I", os.path.join(cuda, "include"), "-I", sysconfig.get_paths()["include"], BINDING_SRC, "-o", BINDING,
           "-L", os.path.join(t, "lib"), "-ltorch_python", "-ltorch_cpu", "-ltorch_cuda", "-lc10", "-lc10_cuda", "-ldl"]
    res = subprocess.run(cmd, capture_output=True, text=True)
    if res.returncode != 0:
        raise RuntimeError("g++ failed for %s:\n%s" % (BINDING_SRC, res.stderr))
    return BINDING


def build(verbose=False, force=False):
    os.makedirs(OBJ_DIR, exist_ok=True)
    if force:
        for f in os.listdir(OBJ_DIR):
            if f.endswith(".o"):
                os.remove(os.path.join(OBJ_DIR, f))
    with ThreadPoolExecutor(max_workers=min(8, os.cpu_count() or 1)) as pool:
        results = list(pool.map(lambda s: _compile_one(s, verbose), _sources()))
    objs = [o for o, _ in results]
    changed = any(c for _, c in results)
    if changed or not os.path.exists(LIB):
        # hidden visibility by default; the extern "C" entry points carry default visibility
        cmd = ["nvcc", "-shared", "-gencode", "arch=compute_100a,code=sm_100a", "-o", LIB] + objs + ["-ldl"]
        subprocess.check_call(cmd)
    build_binding(force)
    return LIB


if __name__ == "__main__":
    print(build(verbose="-v" in sys.argv, force="--force" in sys.argv))
