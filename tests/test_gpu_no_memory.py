"""GPU: device memory that runs out while a lattice is set up.  The failure is made
on the host: the context's translation unit is compiled once more with a cudaMalloc
that can be told to fail, and linked with the library's other objects."""
import glob
import importlib.util
import os
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def failing(pkg, tmp_path_factory):
    pkg_dir = os.path.dirname(os.path.abspath(pkg.__file__))
    spec = importlib.util.spec_from_file_location("lbgb300_build",
                                                  os.path.join(pkg_dir, "build.py"))
    b = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(b)
    tmp = str(tmp_path_factory.mktemp("failing"))
    obj, lib = os.path.join(tmp, "lb_context.o"), os.path.join(tmp, "liblbgb300_failing.so")
    subprocess.run([b._nvcc()] + b.NVCC_FLAGS + ["-include", os.path.join(HERE, "failing_malloc.h"),
                   "-c", os.path.join(b.CSRC, "lb_context.cu"), "-o", obj], check=True)
    others = [o for o in glob.glob(os.path.join(b.OBJ_DIR, "*.o"))
              if os.path.basename(o) != "lb_context.o"]
    subprocess.run([b._nvcc()] + b.ARCH + ["-shared", "-o", lib, obj] + others, check=True)
    return pkg.abi.load(lib)


@pytest.mark.parametrize("steps", [(1,), (3, 7), (200,)])
def test_walls_without_memory_for_their_masks(pkg, failing, monkeypatch, steps):
    """a lattice of the marching strips whose wall masks cannot be allocated keeps its
    walls: the bits of one step per launch, before and after memory is back"""
    W, H = 1028, 700
    N = W * H
    rng = np.random.default_rng(1)
    walls = [np.zeros(N, np.uint8) for _ in range(2)]
    for w in walls:
        w[rng.random(N) < 0.05] = 1
        w[rng.random(N) < 0.02] = 3
    rho = (1 + 0.02 * rng.standard_normal(N)).astype(np.float32)

    def run(tuning, fail):
        lat = pkg.Lattice(9, W, H, tau_inv=np.float32(1 / 0.7), wall_u=(0.03, 0, 0), tuning=tuning)
        out = []
        for i, w in enumerate(walls):
            if fail:
                failing.lb_test_no_memory(i == 0)
            lat.set_flags(w)
            lat.init_equilibrium(rho)
            for n in steps:
                lat.step(n)
            out.append(lat.populations()[:, (w & 1) == 0])
        lat.close()
        return out

    want = run(0x108, False)
    monkeypatch.setattr(pkg.lattice, "_lib", lambda: failing)
    try:
        got = run(0, True)
    finally:
        failing.lb_test_no_memory(0)
    for a, b in zip(got, want):
        assert np.array_equal(a.view(np.uint32), b.view(np.uint32))
