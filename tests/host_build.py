"""Host builds of the library's own headers for CPU tests: C++ source that
includes them, compiled with g++ into a shared object."""
import ctypes
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def compile_host(source, tmp_path, name):
    src, lib = os.path.join(str(tmp_path), name + ".cpp"), os.path.join(str(tmp_path), name + ".so")
    with open(src, "w") as f:
        f.write(source)
    cuda = os.environ.get("CUDA_HOME") or "/usr/local/cuda"
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-I", os.path.join(ROOT, "qradient_gb300", "csrc"),
                    "-I", os.path.join(cuda, "include"), "-o", lib, src], check=True)
    return ctypes.CDLL(lib)
