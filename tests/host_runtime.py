"""The library's host code linked against a CUDA runtime without a GPU (fake_cudart.cc): built once per test run."""
import concurrent.futures
import ctypes as C
import glob
import os
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)


def build(out):
    """The shared library in directory `out`; kernels are compiled to unoptimised PTX only, they never run."""
    from cupythia_b200 import build as b
    srcs = b.sources()
    objs = [os.path.join(out, os.path.basename(s) + ".o") for s in srcs]
    nvcc = [b.NVCC, "-gencode", "arch=compute_100a,code=compute_100a", "-Xcicc", "-O0", "-std=c++17", "-Xcompiler",
            "-fPIC", "--expt-relaxed-constexpr", "-c"]

    def run(cmd):
        r = subprocess.run(cmd, capture_output=True, text=True)
        assert r.returncode == 0, r.stderr

    with concurrent.futures.ThreadPoolExecutor(os.cpu_count() or 4) as ex:
        list(ex.map(run, [nvcc + [s, "-o", o] for s, o in zip(srcs, objs)]))
    so = os.path.join(out, "libhost.so")
    run(["g++", "-O1", "-std=c++17", "-fPIC", "-shared", "-I" + os.path.join(b.CUDA_HOME, "include"),
         os.path.join(HERE, "fake_cudart.cc")] + objs + ["-o", so, "-Wl,-Bsymbolic"])
    return so


def load(so):
    from cupythia_b200 import _lib
    lib = C.CDLL(so)
    for name, args in _lib.SIGNATURES.items():
        f = getattr(lib, name)
        f.argtypes, f.restype = args, C.c_int
    lib.cp_last_error.argtypes, lib.cp_last_error.restype = [C.c_void_p], C.c_char_p
    lib.fake_fail_above.argtypes = [C.c_size_t]
    lib.fake_fail_nth.argtypes = [C.c_long]
    lib.fake_count.argtypes = lib.fake_first.argtypes = [C.c_char_p]
    lib.fake_watch.argtypes = [C.c_char_p, C.c_int]
    lib.fake_watched.restype = C.c_void_p
    lib.fake_is_device.argtypes = [C.c_void_p, C.c_size_t]
    for f in (lib.fake_device_bytes, lib.fake_device_allocations, lib.fake_pinned_allocations):
        f.restype = C.c_size_t
    return lib
