"""Small host programs that call the library's host side without a GPU.

Each tests/host/<name>.cu is compiled against the library's headers and linked
to libasph.so.  CUDA runtime calls that a program defines itself take the
place of the runtime's own, in the library too (the dynamic linker binds the
executable's definitions first), so a program may hold a fake of a call."""
import os
import subprocess

from sph_cuda_gb300 import _build

HERE = os.path.dirname(os.path.abspath(__file__))


def build(name, tmp):
    """Compile tests/host/<name>.cu; returns the program's path."""
    src, out = os.path.join(HERE, "host", name + ".cu"), os.path.join(str(tmp), name)
    r = subprocess.run([_build.nvcc(), "-O1", "-std=c++17", "--expt-relaxed-constexpr", "-cudart", "shared",
                        *_build.ARCH, "-I", _build.CSRC, src, "-o", out, "-L", _build.BUILD, "-lasph",
                        "-Xlinker", "-rpath", "-Xlinker", _build.BUILD], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return out


def run(program, *args):
    return subprocess.run([program, *map(str, args)], capture_output=True, text=True, timeout=120)
