"""The library on a CUDA runtime without a device (fake_cudart.cc): its host
code runs as it does on a GPU, kernels do nothing.  For tests of what the host
queues, waits for, allocates and does when a call fails; they need no GPU and
run on one machine as on the other."""
from __future__ import annotations

import contextlib
import ctypes as C
import os
import shutil
import subprocess
import tempfile

import numpy as np
import pytest

import kraken2_gb300 as k2g
from kraken2_gb300 import build as kb

HERE = os.path.dirname(os.path.abspath(__file__))
OUT_OF_MEMORY = 2           # cudaErrorMemoryAllocation
UNKNOWN = 999               # cudaErrorUnknown: nothing that asking again would mend
_HOOK = C.CFUNCTYPE(None, C.c_char_p, C.POINTER(C.c_void_p))
_built = None


def _build() -> str:
    """The library's objects linked to the runtime above."""
    global _built
    if _built is None:
        gxx = shutil.which("g++")
        try:
            nvcc = kb.nvcc()
        except RuntimeError:
            nvcc = None
        if not gxx or not nvcc:
            pytest.skip("g++ and nvcc are needed")
        objs = [os.path.join(kb.OUT, s + ".o") for s in kb.CU_SOURCES + kb.CC_SOURCES]
        lib = kb.build()
        if not all(os.path.exists(o) and os.path.getmtime(o) <= os.path.getmtime(lib) for o in objs):
            lib = kb.build(force=True)
        include = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(nvcc))), "include")
        out = os.path.join(tempfile.mkdtemp(prefix="fake_cuda_"), "libk2g_fake.so")
        subprocess.run([gxx, "-O1", "-std=c++17", "-fPIC", "-shared", "-Wl,-Bsymbolic", "-I", include,
                        os.path.join(HERE, "fake_cudart.cc"), *objs, "-lpthread", "-o", out], check=True)
        _built = out
    return _built


class Fake:
    def __init__(self, lib):
        self.lib = lib
        lib.fake_fault.restype = C.c_char_p
        lib.fake_pending.argtypes = [C.c_void_p]
        for f in ("fake_pending", "fake_pending_all", "fake_used", "fake_kept", "fake_launches"):
            getattr(lib, f).restype = C.c_uint64
        lib.fake_tail_of_copy.argtypes, lib.fake_tail_of_copy.restype = [C.c_size_t], C.c_long
        lib.fake_room.argtypes, lib.fake_room.restype = [C.c_void_p], C.c_long
        lib.fake_limit.argtypes = [C.c_uint64]
        lib.fake_fail.argtypes = [C.c_char_p, C.c_long, C.c_int]
        lib.fake_launches.argtypes = [C.c_char_p]
        lib.fake_hook.argtypes = [_HOOK]
        lib.fake_fault.argtypes = [C.c_long]
        lib.fake_faults.restype = C.c_long

    def pending(self, stream=None) -> int:
        return self.lib.fake_pending(stream)

    def pending_all(self) -> int:
        return self.lib.fake_pending_all()

    def launches(self, part: str) -> int:
        return self.lib.fake_launches(part.encode())

    def fail(self, fn: str, skip: int, err: int = UNKNOWN):
        self.lib.fake_fail(fn.encode(), skip, err)

    def failed(self) -> bool:
        """Whether the call that was to fail has."""
        return bool(self.lib.fake_failed())

    def limit(self, bytes_: int):
        self.lib.fake_limit(bytes_)

    def used(self) -> int:
        """Device memory held, without what the pool keeps."""
        return self.lib.fake_used()

    def kept(self) -> int:
        """What the pool keeps of the memory given back to it."""
        return self.lib.fake_kept()

    def room(self, p: int) -> int:
        """Bytes from p to the end of its allocation (-1: none)."""
        return self.lib.fake_room(p)

    def tail_of_copy(self, n: int) -> int:
        """Bytes of the allocation behind the last host-to-device copy of n bytes (-1: none)."""
        return self.lib.fake_tail_of_copy(n)

    def faults(self) -> list:
        return [self.lib.fake_fault(i).decode() for i in range(self.lib.fake_faults())]

    def hook(self, fn):
        """fn(kernel name, argument pointers) at each launch."""
        self._hook = _HOOK(lambda name, args: fn(name.decode(), args))
        self.lib.fake_hook(self._hook)

    def stream(self) -> int:
        s = C.c_void_p()
        self.lib.cudaStreamCreateWithFlags(C.byref(s), 1)
        return s.value

    def device(self, a: np.ndarray) -> int:
        """The array in an allocation of the fake device."""
        p = C.c_void_p()
        self.lib.cudaMalloc(C.byref(p), C.c_size_t(max(a.nbytes, 1) + 16))
        assert p.value
        if a.nbytes:
            C.memmove(p.value, a.ctypes.data, a.nbytes)
        return p.value


@contextlib.contextmanager
def fake_cuda():
    """kraken2_gb300 on the fake runtime, within the block."""
    path = _build()
    real, real_path = k2g._lib, k2g.LIB_PATH
    k2g._lib, k2g.LIB_PATH = _fake_lib.get("lib"), path
    try:
        _fake_lib["lib"] = k2g.lib()
        f = Fake(_fake_lib["lib"])
        f.lib.fake_reset()
        yield f
        f.lib.fake_reset()
    finally:
        k2g._lib, k2g.LIB_PATH = real, real_path


_fake_lib: dict = {}
