"""The library's host code on a CUDA runtime of host memory (fake_runtime.cpp): contexts of two devices, memory
limits and failing calls without a GPU."""

import ctypes as C
import hashlib
import os
import subprocess

from pyalbsim_gb300 import _native
from pyalbsim_gb300.build import ARCH, CSRC, INCLUDE, LIB_DIR, nvcc_path

HERE = os.path.dirname(os.path.abspath(__file__))


def build() -> str:
    files = [os.path.join(HERE, f) for f in ("fake_runtime.cpp", "fake_units.cu")]
    files += [os.path.join(CSRC, f) for f in ("albgpu.cu", "noalloc.cu")]
    flags = [*ARCH, "-O1", "-std=c++17", "-Xcompiler", "-fPIC", "--expt-relaxed-constexpr", "-I", INCLUDE, "-I", CSRC]
    h = hashlib.sha256(" ".join(flags).encode())
    for f in files + [os.path.join(HERE, "fake_cuda.h")] + [os.path.join(CSRC, x) for x in sorted(os.listdir(CSRC)) if x.endswith((".cuh", ".h"))]:
        with open(f, "rb") as fh:
            h.update(fh.read())
    out = os.path.join(LIB_DIR, "host_" + h.hexdigest()[:16])
    lib = os.path.join(out, "libalbhost.so")
    if not os.path.exists(lib):
        os.makedirs(out, exist_ok=True)
        # symbols of the library resolve to the stand-in, whatever runtime the process has loaded
        cmd = [nvcc_path(), *flags, "-shared", "-cudart", "none", "-Xlinker", "-Bsymbolic", "-o", lib + ".tmp", *files]
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError(r.stderr)
        os.replace(lib + ".tmp", lib)
    return lib


def load():
    """The stand-in library with the argument types of the real one."""
    before, _native._lib = _native._lib, None
    try:
        lib = _native.load_library(build())
    finally:
        _native._lib = before
    for name in ("fake_used", "fake_peak", "fake_traced"):
        getattr(lib, name).restype = C.c_uint64
    lib.fake_limit.argtypes = [C.c_int, C.c_uint64]
    lib.fake_rates.argtypes = [C.c_void_p, C.c_void_p]
    return lib


def violations(lib) -> str:
    buf = C.create_string_buffer(4096)
    n = lib.fake_violations(buf, 4096)
    return f"{n}: {buf.value.decode()}" if n else ""
