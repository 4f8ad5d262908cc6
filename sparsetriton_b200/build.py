"""Build libsparsetriton_b200.so in-tree with nvcc for sm_100a.

    python -m sparsetriton_b200.build [--force] [--verbose]

The library is a plain C-ABI shared object (see include/sparsetriton_b200.h); it links
only against the CUDA runtime.  Beside it stands _st_host.so, the native host side (host/*.cpp: torch's C++
interface over that C ABI).  Objects are rebuilt when a source or header is newer.
"""
import os
import shutil
import subprocess
import sys

PKG = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(PKG, "csrc")
INCLUDE = os.path.join(os.path.dirname(PKG), "include")
OBJ_DIR = os.path.join(CSRC, "build")
LIB_PATH = os.path.join(PKG, "_native", "libsparsetriton_b200.so")
HOST_SRC = os.path.join(PKG, "host")
HOST_PATH = os.path.join(PKG, "_native", "_st_host.so")

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-O3", "-std=c++17", "-lineinfo", "-Wno-deprecated-gpu-targets",
    "-Xcompiler", "-fPIC",
    "--expt-relaxed-constexpr",
]


def _nvcc():
    exe = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(exe):
        raise RuntimeError("nvcc not found: cannot build libsparsetriton_b200.so")
    return exe


def sources():
    return sorted(os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith(".cu"))


def _headers():
    hs = [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith(".cuh")]
    hs += [os.path.join(INCLUDE, f) for f in os.listdir(INCLUDE) if f.endswith(".h")]
    return hs


def build(force=False, verbose=False):
    """Compile every .cu under csrc/ and link the shared library.  Returns its path."""
    nvcc = _nvcc()
    os.makedirs(OBJ_DIR, exist_ok=True)
    os.makedirs(os.path.dirname(LIB_PATH), exist_ok=True)
    newest_header = max(os.path.getmtime(h) for h in _headers())
    objs, rebuilt = [], False
    procs = []
    for src in sources():
        obj = os.path.join(OBJ_DIR, os.path.basename(src)[:-3] + ".o")
        objs.append(obj)
        stale = (force or not os.path.exists(obj)
                 or os.path.getmtime(obj) < max(os.path.getmtime(src), newest_header))
        if stale:
            cmd = [nvcc, *NVCC_FLAGS, "-I", INCLUDE, "-c", src, "-o", obj]
            if verbose:
                cmd.insert(1, "-Xptxas")
                cmd.insert(2, "-v")
                print(" ".join(cmd))
            procs.append((src, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
            rebuilt = True
    failed = False
    for src, p in procs:
        out, _ = p.communicate()
        if p.returncode != 0 or verbose:
            print(out)
        if p.returncode != 0:
            print(f"nvcc failed on {src}", file=sys.stderr)
            failed = True
    if failed:
        raise RuntimeError("nvcc failed")
    if rebuilt or not os.path.exists(LIB_PATH):
        cmd = [nvcc, "-shared", "-o", LIB_PATH, *objs, "-lcudart"]
        subprocess.check_call(cmd)
    build_host(force, verbose)
    return LIB_PATH


def build_host(force=False, verbose=False):
    """Compile host/*.cpp against torch and link _st_host.so beside the library it calls."""
    import sysconfig

    import torch
    from torch.utils import cpp_extension
    header = os.path.join(HOST_SRC, "host.h")
    abi = os.path.join(INCLUDE, "sparsetriton_b200.h")
    newest = max(os.path.getmtime(header), os.path.getmtime(abi))
    cuda = os.path.dirname(os.path.dirname(os.path.realpath(_nvcc())))
    includes = cpp_extension.include_paths() + [sysconfig.get_paths()["include"], os.path.join(cuda, "include")]
    flags = ["-O2", "-std=c++17", "-fPIC", "-fvisibility=hidden", "-w", "-DTORCH_API_INCLUDE_EXTENSION_H",
             "-DTORCH_EXTENSION_NAME=_st_host", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}"]
    objs, procs = [], []
    for name in sorted(os.listdir(HOST_SRC)):
        if not name.endswith(".cpp"):
            continue
        src, obj = os.path.join(HOST_SRC, name), os.path.join(OBJ_DIR, "host_" + name[:-4] + ".o")
        objs.append(obj)
        if force or not os.path.exists(obj) or os.path.getmtime(obj) < max(os.path.getmtime(src), newest):
            cmd = ["g++", *flags, *(f"-I{i}" for i in includes), "-c", src, "-o", obj]
            procs.append((src, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
    failed = False
    for src, p in procs:
        out, _ = p.communicate()
        if p.returncode != 0 or verbose:
            print(out)
        if p.returncode != 0:
            print(f"g++ failed on {src}", file=sys.stderr)
            failed = True
    if failed:
        raise RuntimeError("g++ failed")
    if procs or not os.path.exists(HOST_PATH):
        libs = os.path.join(os.path.dirname(torch.__file__), "lib")
        subprocess.check_call(["g++", "-shared", "-o", HOST_PATH, *objs, f"-L{libs}", "-lc10", "-lc10_cuda", "-ltorch_cpu",
                               "-ltorch_cuda", "-ltorch", "-ltorch_python", f"-L{os.path.dirname(LIB_PATH)}",
                               "-lsparsetriton_b200", f"-L{os.path.join(cuda, 'lib64')}", "-lcudart",
                               "-Wl,-rpath,$ORIGIN"])
    return HOST_PATH


if __name__ == "__main__":
    path = build(force="--force" in sys.argv, verbose="--verbose" in sys.argv)
    print(path)
