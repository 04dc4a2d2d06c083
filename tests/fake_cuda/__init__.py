"""The kernel library's launchers on a CUDA runtime that has devices, streams and limits but no GPU (``runtime.cpp``)."""
import ctypes as C
import os
import subprocess

from eagersgd_b200 import _build

HERE = os.path.dirname(os.path.abspath(__file__))


def build(to: str) -> C.CDLL:
    """Link the objects of ``libesgd_cuda.so`` with the fake runtime.  Nothing of it is visible to other libraries."""
    _build.build_cuda()
    objects = [os.path.join(_build.LIBDIR, "obj", os.path.basename(s) + ".o") for s in _build._sources("cuda", [".cu"])]
    if not all(os.path.exists(o) for o in objects):
        _build.build_cuda(force=True)
    include = os.path.join(os.path.dirname(os.path.dirname(_build.nvcc_path())), "include")
    subprocess.run(["g++", "-O1", "-std=c++17", "-fPIC", "-shared", "-pthread", "-I", include, os.path.join(HERE, "runtime.cpp")] + objects +
                   ["-o", to, "-Wl,-Bsymbolic", "-Wl,--version-script=" + os.path.join(HERE, "exports.map")], check=True)
    lib = C.CDLL(to)
    lib.fake_stream.restype = C.c_void_p
    lib.fake_launch.restype = C.c_char_p
    lib.fake_launch.argtypes = [C.c_int, C.c_void_p]
    lib.fake_attributes.restype = C.c_longlong
    return lib


def launches(lib) -> list:
    """(kernel, device, threads, dynamic shared memory, cluster, blocks) of what has been launched since the last call."""
    out = (C.c_int * 5)()
    rows = []
    for i in range(lib.fake_launches()):
        name = lib.fake_launch(i, out).decode()
        rows.append((name,) + tuple(out))
    lib.fake_clear()
    return rows
