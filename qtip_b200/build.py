"""Build the in-tree binaries: libqtip_b200.so (sm_100a, nvcc) and _host.so, the native host path of a layer call
(C++ against torch's headers, linked to the library beside it).  `python -m qtip_b200.build`."""
import glob
import os
import subprocess
import sys
import sysconfig

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
SO = os.path.join(HERE, "libqtip_b200.so")
HOST_SRC = os.path.join(CSRC, "host.cpp")
HOST_SO = os.path.join(HERE, "_host.so")
NVCC_FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-lineinfo", "-std=c++17",
              "-Xcompiler", "-fPIC", "-shared", "--threads", "0"]


def sources():
    return sorted(glob.glob(os.path.join(CSRC, "*.cu")))


def needs_build():
    if not os.path.exists(SO):
        return True
    t = os.path.getmtime(SO)
    deps = sources() + glob.glob(os.path.join(CSRC, "*.cuh")) + glob.glob(os.path.join(HERE, "..", "include", "*.h"))
    return any(os.path.getmtime(d) > t for d in deps)


def build(force=False, verbose=False):
    if not force and not needs_build():
        build_host()
        return SO
    nvcc = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
    cmd = [nvcc] + NVCC_FLAGS + (["-Xptxas", "-v"] if verbose else []) + ["-o", SO] + sources()
    env = dict(os.environ)
    env.pop("CC", None)
    env.pop("CXX", None)
    subprocess.check_call(cmd + ["-ccbin", "/usr/bin/g++"], env=env)
    build_host(force=force)
    return SO


def host_needs_build():
    if not os.path.exists(HOST_SO):
        return True
    deps = [HOST_SRC, os.path.join(HERE, "..", "include", "qtip_b200.h")]
    return any(os.path.getmtime(d) > os.path.getmtime(HOST_SO) for d in deps)


def build_host(force=False):
    """_host.so: a plain CPython extension (no binding generator); needs torch's headers and libqtip_b200.so."""
    if not force and not host_needs_build():
        return HOST_SO
    import torch
    root = os.path.dirname(torch.__file__)
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    inc = [os.path.join(root, "include"), os.path.join(root, "include", "torch", "csrc", "api", "include"),
           os.path.join(cuda, "include"), sysconfig.get_paths()["include"]]
    cmd = ["/usr/bin/g++", "-O2", "-std=c++17", "-fPIC", "-shared", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}"]
    cmd += [f"-I{d}" for d in inc] + [HOST_SRC, "-o", HOST_SO, f"-L{os.path.join(root, 'lib')}", "-ltorch_python", "-ltorch",
                                      "-ltorch_cpu", "-ltorch_cuda", "-lc10", "-lc10_cuda", f"-L{HERE}", "-l:libqtip_b200.so", "-Wl,-rpath,$ORIGIN"]
    subprocess.check_call(cmd)
    return HOST_SO


if __name__ == "__main__":
    build(force=True, verbose="-v" in sys.argv)
    print(SO)
