"""GPU: the staged D3Q19 Shan-Chen step in its two tiles (64 and 32 columns)
and with chunks of planes that do not divide the depth gives the bits of the
two-pass step: one tile and one chunk per plane, widths of an odd number of
tiles, and lattices large enough for chunks of several planes."""
import ctypes

import numpy as np
import pytest

from conftest import load_package
from golden_io import bits

pytestmark = pytest.mark.gpu

STAGED, TWO_PASS = 0x100 | 0x040, 0x100


@pytest.fixture(scope="module")
def pkg():
    p = load_package()
    n = ctypes.c_int(0)
    assert p.lib().lb_device_count(ctypes.byref(n)) == 0 and n.value >= 1, "no CUDA device"
    return p


@pytest.mark.parametrize("shape", [(32, 8, 4), (64, 8, 4), (192, 24, 12), (256, 256, 200)],
                         ids=lambda s: "x".join(map(str, s)))
@pytest.mark.parametrize("storage", [0, 1, 2], ids=["f32", "f16", "bf16"])
def test_matches_two_pass(pkg, shape, storage):
    W, H, D = shape
    rng = np.random.default_rng(5)
    # densities around and beyond the coexistence densities
    rho = (0.693 * (1 + rng.uniform(-0.5, 0.5, W * H * D))).astype(np.float32)
    u = [rng.uniform(-0.05, 0.05, W * H * D).astype(np.float32) for _ in range(3)]
    out = []
    for tuning in (STAGED, TWO_PASS):
        lat = pkg.Lattice(19, W, H, D, tau_inv=1.0, G=-5.0, psi_form=pkg.abi.LB_PSI_EXP1,
                          force=(0.0, np.float32(3e-6), 0.0), storage=storage, rho_ref=0.693,
                          tuning=tuning, graph_steps=2)
        lat.set_flags(np.zeros(W * H * D, np.uint8))
        lat.init_equilibrium(rho, *u)
        lat.step(5)
        out.append((lat.populations(), *lat.moments()))
        lat.close()
    assert np.isfinite(out[0][0]).all()
    for a, b in zip(*out):
        assert np.array_equal(bits(a), bits(b))
