"""The reference mode's FP64 lines in pairs of floats (csrc/lb_ff.cuh), compiled
for the host and compared with the FP64 lines themselves."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def host(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("ff") / "libff_host.so")
    cuda = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-shared", "-fPIC",
                    "-I" + cuda, os.path.join(HERE, "ff_host.cpp"), "-o", out], check=True)
    lib = ctypes.CDLL(out)
    lib.ratio_wrong.restype = ctypes.c_long
    lib.psi_error.restype = ctypes.c_double
    return lib


def ptr(a):
    return a.ctypes.data_as(ctypes.c_void_p)


@pytest.mark.parametrize("add", [0.0, -1.0], ids=["density", "velocity"])
@pytest.mark.parametrize("v", [1.0, 0.7, 3e-30, 1e-38, 1e28, 1e30, 1.3e31, 1e33, 1e34, 7e34, 1e35,
                               1e36, 3e38, -1e34])
def test_face_quotients(host, v, add):
    """populations of the divisor's own size, so that the quotient is of order one:
    every value that the form decides is the FP64 line's"""
    rng = np.random.default_rng(5)
    n = 20000
    a, b = (np.float32(v) * rng.uniform(0.1, 0.9, (2, n))).astype(np.float32)
    assert host.ratio_wrong(ptr(a), ptr(b), ctypes.c_long(n), ctypes.c_double(v),
                            ctypes.c_float(add)) == 0


# a sweep over the whole range, and every float where the reduced argument is at
# its largest for several k (rho = 200 / ((k + 1/2) ln 2))
@pytest.mark.parametrize("lo,hi,step", [(8.0, 2.0 ** 20, 61)] + [
    (200 / ((k + 0.5) * np.log(2)) * (1 - 2e-3), 200 / ((k + 0.5) * np.log(2)) * (1 + 2e-3), 1)
    for k in (0, 1, 2, 5, 12, 20, 35)])
def test_psi(host, lo, hi, step):
    """the form's error is at most half of what its rounding check allows (2^-35), and
    no value that the check decides differs from the FP64 line"""
    wrong = ctypes.c_long()
    err = host.psi_error(ctypes.c_float(lo), ctypes.c_float(hi), ctypes.c_int(step),
                         ctypes.byref(wrong))
    assert wrong.value == 0
    assert err <= 2.0 ** -36, np.log2(err)
