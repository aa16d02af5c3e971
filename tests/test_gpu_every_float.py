"""GPU: the reciprocal and the pseudo-potentials of the paired and float-pair forms give
the bits of the operations they stand for, on all 2^32 floats."""
import ctypes
import importlib.util
import os
import subprocess

import pytest

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def probe(pkg, tmp_path_factory):
    pkg_dir = os.path.dirname(os.path.abspath(pkg.__file__))
    spec = importlib.util.spec_from_file_location("lbgb300_build",
                                                  os.path.join(pkg_dir, "build.py"))
    b = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(b)
    lib = str(tmp_path_factory.mktemp("probe") / "libpairs_probe.so")
    subprocess.run([b._nvcc()] + b.NVCC_FLAGS + ["-shared", os.path.join(HERE, "pairs_probe.cu"),
                   "-o", lib], check=True)
    fn = ctypes.CDLL(lib).probe_every_float
    fn.restype = ctypes.c_long
    return fn


@pytest.mark.parametrize("form", [0, 1, 2, 3],
                         ids=["reciprocal", "two-reciprocals", "psi-exp", "psi-reference"])
def test_same_bits(probe, form):
    assert probe(form) == 0
