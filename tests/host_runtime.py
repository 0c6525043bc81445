"""libsph_cuda's own objects linked with stand-ins for the CUDA runtime
(host_runtime.cpp): its host code without a GPU."""
import ctypes
import os
import re
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))


def load(out_dir):
    """The library as a ctypes handle, with the signatures of sph_gb300._lib."""
    from sph_gb300 import _lib, build
    build.build()
    objs = [os.path.join(build.OBJ, os.path.basename(s)[:-3] + ".o") for s in build.sources()]
    if not all(map(os.path.exists, objs)):
        build.build(force=True)
    src = os.path.join(HERE, "host_runtime.cpp")
    names = re.findall(r"W\((\w+)\)\(", open(src).read())
    cuda = os.path.dirname(os.path.dirname(os.path.realpath(build.nvcc())))
    lib = os.path.join(str(out_dir), "libsph_host.so")
    subprocess.run(["g++", "-shared", "-fPIC", "-std=c++17", "-O1", "-o", lib, src] + objs +
                   ["-I", os.path.join(cuda, "include"), "-L", os.path.join(cuda, "lib64"),
                    "-Wl,-Bsymbolic"] + [f"-Wl,--wrap={n}" for n in sorted(set(names))] +
                   ["-lcudart_static", "-ldl", "-lrt", "-lpthread"], check=True)
    h = ctypes.CDLL(lib)
    for name, (res, args) in _lib._SIGS.items():
        f = getattr(h, name)
        f.restype, f.argtypes = res, args
    h.host_log.restype = ctypes.c_char_p
    h.host_stream.restype = ctypes.c_void_p
    return h
