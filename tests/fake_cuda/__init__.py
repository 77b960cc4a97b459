"""libewt's host code over a stand-in for the CUDA runtime (fake_cuda.cpp), for
tests of what it does around the kernels: no GPU, no kernel runs."""
import ctypes as C
import glob
import os
import subprocess

_HERE = os.path.dirname(os.path.abspath(__file__))
_OUT = os.path.join(os.path.dirname(_HERE), "cpp", "bin")


def load():
    import ecl_wavelet_gb300 as E
    from ecl_wavelet_gb300 import buildlib as B

    E.build()
    os.makedirs(_OUT, exist_ok=True)
    so = os.path.join(_OUT, "libewt_fake_cuda.so")
    src = os.path.join(_HERE, "fake_cuda.cpp")
    objs = [os.path.join(B.OBJ_DIR, os.path.basename(s) + ".o") for s in B.sources()]
    deps = objs + [src]
    if not os.path.exists(so) or any(os.path.getmtime(d) > os.path.getmtime(so) for d in deps):
        inc = os.path.join(os.path.dirname(os.path.dirname(B.nvcc())), "include")
        tmp = so + ".%d" % os.getpid()
        r = subprocess.run(["g++", "-O1", "-std=c++17", "-fPIC", "-shared", "-Wl,-Bsymbolic",
                            "-I", inc, src] + objs + ["-o", tmp, "-lpthread", "-ldl"],
                           capture_output=True, text=True)
        assert r.returncode == 0, r.stderr
        os.replace(tmp, so)
    L = C.CDLL(so)
    for name, (res, args) in E.SIGNATURES.items():
        f = getattr(L, name)
        f.restype, f.argtypes = res, args
    for name, (res, args) in {
            "fake_reset": (None, []), "fake_set": (None, [C.c_char_p, C.c_long]),
            "fake_fail": (None, [C.c_char_p, C.c_long]),
            "fake_calls": (C.c_long, [C.c_char_p]),
            "fake_patch": (None, [C.c_uint64] * 3), "fake_live": (C.c_uint64, []),
            "fake_peak": (C.c_uint64, []), "fake_pending": (C.c_long, []),
            "fake_journal": (C.c_char_p, [])}.items():
        f = getattr(L, name)
        f.restype, f.argtypes = res, args
    return L


def build(L, text, alphabet, patch=None):
    """A tree of the stand-in; patch: (entries, from, value) of the count table
    that the passes would have written."""
    out = C.c_void_p()
    L.fake_reset()
    if patch:
        L.fake_patch(patch[0] * 8, patch[1], patch[2])
    sigma = 0 if alphabet is None else alphabet.size
    st = L.ewt_build(text.ctypes.data, text.size, text.itemsize,
                     None if alphabet is None else alphabet.ctypes.data, sigma, 0, C.byref(out))
    assert st == 0, L.ewt_last_error()
    return out
