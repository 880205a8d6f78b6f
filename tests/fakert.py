"""The library linked with the stand-in runtime of fake_cudart.cpp, loaded as api's library: its host
code runs on plain memory, `hook(kernel, args)` sees every launch, and allocations can be made to fail."""
import contextlib
import ctypes as C
import glob
import os
import subprocess

from storm_b200 import api, build

HOOK = C.CFUNCTYPE(None, C.c_char_p, C.POINTER(C.c_void_p))
CUDA_INC = "/usr/local/cuda/include"


def make(folder) -> str:
    build.build()
    so = os.path.join(str(folder), "libstormgpu_fake.so")
    here = os.path.dirname(os.path.abspath(__file__))
    objs = [os.path.join(build.PKG, "_build", s.replace(".cu", ".o")) for s in build.CU_SOURCES]
    subprocess.run(["g++", "-O1", "-g", "-std=c++17", "-fPIC", "-shared", "-Wl,-Bsymbolic", "-I" + CUDA_INC,
                    os.path.join(here, "fake_cudart.cpp")] + objs + ["-lpthread", "-o", so], check=True)
    return so


class Fake:
    def __init__(self, L):
        self.L = L
        for f in ("fake_live", "fake_live_bytes", "fake_fail_left", "fake_room"):
            getattr(L, f).restype = C.c_longlong
        L.fake_room.argtypes = [C.c_void_p, C.POINTER(C.c_void_p)]
        L.fake_fail_in.argtypes = [C.c_longlong]
        self.live = L.fake_live
        self.fail_in = L.fake_fail_in
        self.fail_left = L.fake_fail_left

    def room(self, p):
        """(bytes from p to the end of its allocation, the allocation)"""
        base = C.c_void_p()
        return self.L.fake_room(p, C.byref(base)), base.value

    @contextlib.contextmanager
    def hook(self, f):
        """f(kernel name, args) at every launch; what it raises comes out at the end."""
        raised = []

        def call(name, args):
            try:
                f(name.decode(), args)
            except BaseException as e:  # noqa: BLE001 (a callback cannot raise)
                raised.append(e)
        h = HOOK(call)
        self.L.fake_set_hook(h)
        try:
            yield
        finally:
            self.L.fake_set_hook(HOOK())
        if raised:
            raise raised[0]


def arg(args, i, t=C.c_int64):
    return C.cast(args[i], C.POINTER(t))[0]


def have_compiler() -> bool:
    return os.path.exists(os.path.join(CUDA_INC, "cuda_runtime_api.h")) and bool(glob.glob("/usr/bin/g++*"))


@contextlib.contextmanager
def loaded(so):
    path, lib = api.LIB_PATH, api._lib
    api.LIB_PATH, api._lib = so, None
    try:
        yield Fake(api.lib())
    finally:
        api.LIB_PATH, api._lib = path, lib
