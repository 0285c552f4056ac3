"""Small host programs that call the library's host side without a GPU.

Each tests/host/<name>.cu is compiled against the library's headers and linked
to libasph.so.  The CUDA runtime calls of tests/host/fake_cuda.cpp, where it is
linked in, take the place of the runtime's own, in the library too: the dynamic
linker binds the executable's definitions first."""
import os
import subprocess

from sph_cuda_gb300 import _build

HERE = os.path.dirname(os.path.abspath(__file__))


def build(name, tmp, fake=True):
    """Compile tests/host/<name>.cu, with or without the stand-in runtime; returns the program's path."""
    src, out = [os.path.join(HERE, "host", name + ".cu")], os.path.join(str(tmp), name)
    if fake:
        src.append(os.path.join(HERE, "host", "fake_cuda.cpp"))
    r = subprocess.run([_build.nvcc(), "-O1", "-std=c++17", "--expt-relaxed-constexpr", "-cudart", "shared",
                        *_build.ARCH, "-I", _build.CSRC, *src, "-o", out, "-L", _build.BUILD, "-lasph",
                        "-Xlinker", "-rpath", "-Xlinker", _build.BUILD], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return out


def run(program, *args):
    return subprocess.run([program, *map(str, args)], capture_output=True, text=True, timeout=120)
