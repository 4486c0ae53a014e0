"""libdesgpu's objects linked with tests/fake_cudart.c: the library's host side
without a GPU, and what it asked of the runtime."""
import contextlib
import ctypes as C
import os
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))


def load(directory):
    """(library with the entry points' signatures, fake runtime) built into `directory`."""
    from dynearthsol_gb300 import build, capi
    build.build()
    objs = [os.path.join(build.BUILD, s.replace(".cu", ".o")) for s in build.SOURCES]
    if not all(map(os.path.exists, objs)):
        build.build(force=True)
    fake, path = os.path.join(directory, "fake.o"), os.path.join(directory, "libdesgpu_fake.so")
    subprocess.check_call(["gcc", "-O1", "-fPIC", "-c", os.path.join(HERE, "fake_cudart.c"), "-o", fake])
    subprocess.check_call(["g++", "-shared", "-Wl,-Bsymbolic", "-o", path, *objs, fake])
    lib = capi.load_library(path)
    lib.fake_first_violation.restype = C.c_char_p
    lib.fake_allocated.restype = C.c_size_t
    lib.fake_block_of.argtypes = [C.c_char_p]
    lib.fake_malloc_limit.argtypes = [C.c_size_t]
    return lib


@contextlib.contextmanager
def installed(lib):
    """DeviceModel works on `lib` meanwhile."""
    from dynearthsol_gb300 import capi
    real, capi._lib = capi._lib, lib
    lib.fake_reset()
    try:
        yield
    finally:
        capi._lib = real
