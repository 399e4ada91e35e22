"""Build libcdssm_b200.so (the C-ABI CUDA library) with nvcc for sm_100a and _cdssm_host.so (the native host path of the
operator and model API, a CPython extension over torch and that library) in-tree."""
import os
import subprocess
import sys
import sysconfig

PKG_DIR = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(PKG_DIR, "csrc")
HOST_SRC = os.path.join(CSRC, "host")
LIB_NAME = "libcdssm_b200.so"
HOST_NAME = "_cdssm_host.so"
NVCC_FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3",
              "-std=c++17", "-Xcompiler", "-fPIC", "-Xcompiler", "-fvisibility=hidden"]


def sources():
    return sorted(os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith(".cu"))


def lib_path():
    return os.path.join(PKG_DIR, LIB_NAME)


def host_path():
    return os.path.join(PKG_DIR, HOST_NAME)


def _stale(out, deps):
    if not os.path.exists(out):
        return True
    t = os.path.getmtime(out)
    return any(os.path.getmtime(d) > t for d in deps)


def _start_host(objdir, header, force, verbose):
    """Starts the compilations of the host extension: ([objects], [(command, process)])."""
    from torch.utils import cpp_extension as ext
    import torch
    headers = [os.path.join(HOST_SRC, f) for f in os.listdir(HOST_SRC) if f.endswith(".h")] + [header]
    objs, procs = [], []
    for name in sorted(f for f in os.listdir(HOST_SRC) if f.endswith(".cpp")):
        src, obj = os.path.join(HOST_SRC, name), os.path.join(objdir, "host_" + name[:-4] + ".o")
        objs.append(obj)
        if force or _stale(obj, [src] + headers):
            cmd = ["g++", "-O2", "-std=c++17", "-fPIC", "-fvisibility=hidden",
                   f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}", "-c", src, "-o", obj]
            cmd += [f"-isystem{p}" for p in ext.include_paths(device_type="cuda") + [sysconfig.get_paths()["include"]]]
            if verbose:
                print(" ".join(cmd))
            procs.append((cmd, subprocess.Popen(cmd)))
    return objs, procs


def build(force=False, verbose=False):
    """Compile every .cu under csrc/ and link the shared library, then the host extension.  Returns the library's path."""
    nvcc = os.environ.get("NVCC", "nvcc")
    headers = [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith((".cuh", ".h"))]
    headers.append(os.path.join(PKG_DIR, "..", "include", "cdssm_b200.h"))
    objdir = os.path.join(PKG_DIR, "build")
    os.makedirs(objdir, exist_ok=True)
    objs, procs = [], []
    for src in sources():
        obj = os.path.join(objdir, os.path.basename(src)[:-3] + ".o")
        objs.append(obj)
        if force or _stale(obj, [src] + headers):
            cmd = [nvcc] + NVCC_FLAGS + ["-c", src, "-o", obj]
            if verbose:
                print(" ".join(cmd))
            procs.append((cmd, subprocess.Popen(cmd)))
    host_objs, host_procs = _start_host(objdir, headers[-1], force, verbose)
    for cmd, p in procs + host_procs:
        if p.wait() != 0:
            raise RuntimeError("compilation failed: " + " ".join(cmd))
    out = lib_path()
    if force or procs or _stale(out, objs):
        cmd = [nvcc, "-shared", "-o", out] + objs + ["-lcudart"]
        if verbose:
            print(" ".join(cmd))
        subprocess.check_call(cmd)
    if force or host_procs or _stale(host_path(), host_objs):
        from torch.utils import cpp_extension as ext
        cmd = ["g++", "-shared", "-o", host_path()] + host_objs + [f"-L{p}" for p in ext.library_paths(device_type="cuda")]
        cmd += ["-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch_cuda", "-ltorch_python", "-lcublasLt", f"-L{PKG_DIR}", f"-l:{LIB_NAME}", "-Wl,-rpath,$ORIGIN"]
        if verbose:
            print(" ".join(cmd))
        subprocess.check_call(cmd)
    return out


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose=True))
