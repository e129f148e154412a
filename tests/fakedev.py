"""The library over the stand-in CUDA runtime of fake_cudart.cpp: what its calls launch, on a
machine without a GPU. `run` executes a script in a process of its own, where the stand-in
is preloaded; the script has this module's names and prints what it found as JSON."""
import ctypes as C
import json
import os
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
PKG = os.path.join(ROOT, "nemo-fmi-devel_gb300")


def build():
    """Compile the library and the stand-in; the stand-in's path."""
    from nemo_gpu import build as b
    b.build()
    out = os.path.join(HERE, "_build", "libfake_cudart.so")
    src = os.path.join(HERE, "fake_cudart.cpp")
    if not os.path.exists(out) or os.path.getmtime(out) < os.path.getmtime(src):
        os.makedirs(os.path.dirname(out), exist_ok=True)
        include = os.path.join(os.path.dirname(os.path.dirname(b._nvcc())), "include")
        subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-I" + include, "-o", out, src], check=True)
    return out


def run(script):
    env = dict(os.environ, LD_PRELOAD=build(), FAKE_CUDART=build(), PYTHONPATH=os.pathsep.join((HERE, PKG, ROOT)))
    r = subprocess.run([sys.executable, "-c", "from fakedev import *\n" + script], env=env, capture_output=True,
                       text=True, timeout=600)
    assert r.returncode == 0, r.stdout + r.stderr
    return json.loads(r.stdout.splitlines()[-1])


if "FAKE_CUDART" in os.environ:
    from nemo_gpu import _ffi, gyre, shelf  # noqa: F401
    from nemo_gpu import build as _b

    fake = C.CDLL(os.environ["FAKE_CUDART"])
    fake.fake_launches.restype = C.c_char_p
    fake.fake_held.restype = C.c_size_t
    lib = _ffi.load(_b.library_path())

    HOTPATH = ("AVT", "AH_WSLP2", "AKZ", "TSB", "TSN", "TSA", "UN", "VN", "WN", "USLP", "VSLP", "WSLPI", "WSLPJ", "UA", "VA",
               "UB", "VB", "SSHN", "SSHB", "UN_B", "VN_B", "UB_B", "VB_B", "UTAU", "VTAU", "EMP", "RCDU_BOT", "SSHA",
               "UA_B", "VA_B", "UN_ADV", "VN_ADV", "UB2_B", "VB2_B", "UN_BF", "VN_BF")  # fields of stp_hotpath

    def launches():
        """[(kernel, grid x y z, block x y, shared memory)] since the last call"""
        out = [line.split() for line in fake.fake_launches().decode().splitlines()]
        fake.fake_clear()
        return [(k, *map(int, rest)) for k, *rest in out]

    class Ctx:
        def __init__(self, dom, nam, prec="mixed", nmem=1):
            self.h, self.nmem, self.dom = C.c_void_p(), nmem, dom
            st = lib.nemo_gpu_create(C.byref(_ffi.make_desc(dom)), C.byref(_ffi.make_namelist(nam)), nmem,
                                     _ffi.PREC_FP64 if prec == "fp64" else _ffi.PREC_MIXED, None, C.byref(self.h))
            assert st == 0, st
            self.n3 = dom["jpi"] * dom["jpj"] * dom["jpk"]

        def array(self, n):
            """device memory of n doubles a member"""
            p = C.c_void_p()
            assert fake.cudaMalloc(C.byref(p), C.c_size_t(8 * n * self.nmem)) == 0
            return p

        def bind(self, *names):
            for n in names:
                p = self.array(lib.nemo_gpu_field_numel(self.h, _ffi.F[n]))
                assert lib.nemo_gpu_bind(self.h, _ffi.F[n], p) == 0, n

        def __call__(self, routine, *args):
            st = getattr(lib, "nemo_gpu_" + routine)(self.h, *args)
            assert st == 0, routine + ": " + lib.nemo_gpu_last_error(self.h).decode()

        def close(self):
            lib.nemo_gpu_destroy(self.h)
