"""The operator layer linked against a backend in host memory (fake_backend.c): its host code on the CPU, and what it
queued. Kernels do nothing there, so results are not looked at."""
import ctypes as C
import os
import subprocess

from computeql_gb300 import build, native as N

_lib = None


def load(directory):
    """the library, built once per process"""
    global _lib
    if _lib is None:
        path = os.path.join(directory, "libcqlops_fake.so")
        sources = [os.path.join(build.HOST, f) for f in build.C_SOURCES] + [os.path.join(os.path.dirname(os.path.abspath(__file__)), "fake_backend.c")]
        subprocess.run(["gcc", "-std=c99", "-O1", "-fPIC", "-shared", "-Wl,-Bsymbolic", "-I", build.INCLUDE, "-I", build.HOST, "-o", path,
                        *sources, "-lm", "-lpthread"], check=True)
        _lib = C.CDLL(path)
        N._bind(_lib, N.OPS_API)
        for name, res, args in [("fake_reset", None, []), ("fake_clear_log", None, []), ("fake_fail_name", None, [C.c_char_p]), ("fake_log_count", C.c_uint32, []),
                                ("fake_log", C.c_char_p, [C.c_uint32]), ("fake_pooled_data", C.c_void_p, [C.c_char_p]),
                                ("cqlcuda_buffer_alloc", C.c_void_p, [C.c_uint64, C.c_uint32, C.c_void_p])]:
            f = getattr(_lib, name)
            f.restype, f.argtypes = res, args
    _lib.fake_reset()
    return _lib


def column(lib, ctype, array, zone=None):
    c = N.CqlColumn()
    c.type, c.rows = ctype, len(array)
    c.buffer = lib.cqlcuda_buffer_alloc(max(array.nbytes, 16), 0, array.ctypes.data)
    if zone is not None:
        c.has_range, c.zone_min, c.zone_max = 1, float(zone[0]), float(zone[1])
    return c


def log(lib, kind):
    """the names logged as `kind` ("run", "compile", "refused"), in order"""
    lines = [lib.fake_log(i).decode().split(" ", 1) for i in range(lib.fake_log_count())]
    return [name for k, name in lines if k == kind]
