"""GPU: the D2Q9 marching strips (LB_TUNE_MARCH: one launch advances several
steps, the time levels in between in registers) give the bits of the per-step
path: strips and marches that do not divide the lattice, lattices narrower than
a strip or lower than a march, odd widths, walls (also moving ones) anywhere,
step counts that leave a remainder, and the cursor probe."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

PLAIN, MARCH = 0x100 | 0x008, 0x100 | 0x002


def beq(a, b):
    a, b = np.ascontiguousarray(a), np.ascontiguousarray(b)
    return a.shape == b.shape and np.array_equal(a.view(np.uint8), b.view(np.uint8))


def run(pkg, W, H, tuning, walls, steps=(1, 2, 7, 23)):
    N = W * H
    rng = np.random.default_rng(N + W)
    flags = np.zeros(N, np.uint8)
    if walls:
        flags[rng.random(N) < 0.08] = 1
        flags[rng.random(N) < 0.03] = 3
    u = [(0.03 * rng.standard_normal(N)).astype(np.float32) for _ in range(2)]
    rho = (1 + 0.02 * rng.standard_normal(N)).astype(np.float32)
    lat = pkg.Lattice(9, W, H, tau_inv=np.float32(1 / 0.7), force=(2e-5, -1e-5, 0),
                      wall_u=(0.03, -0.01, 0), tuning=tuning, graph_steps=8)
    lat.set_flags(flags)
    lat.init_equilibrium(rho, *u)
    out = []
    for s in steps:
        lat.step(s)
        out += list(lat.moments()[:3])
    v = np.full(4, np.nan, np.float32)
    for s, x, y in ((7, 0, 0), (4, W // 2, H // 2), (2, W - 1, H - 1)):
        rc = pkg.lib().lb_run_probe(lat.h, s, x, y, 0, v.ctypes.data_as(ctypes.c_void_p))
        assert rc == 0
        out.append(v.copy())
    out.append(lat.populations()[:, (flags & 1) == 0])
    out.append(np.array([lat.steps_done()]))
    lat.close()
    return out


@pytest.mark.parametrize("walls", [False, True], ids=["periodic", "walls"])
@pytest.mark.parametrize("W,H", [(1, 1), (2, 3), (7, 5), (56, 16), (60, 41), (64, 33), (130, 71),
                                 (253, 90), (1000, 7)])
def test_matches_per_step_path(pkg, W, H, walls):
    for a, b in zip(run(pkg, W, H, MARCH, walls), run(pkg, W, H, PLAIN, walls)):
        assert beq(a, b)


@pytest.mark.parametrize("W,H", [(1028, 1024), (729, 721)])
def test_default_on_a_large_lattice(pkg, W, H):
    """100 steps of more than 2^19 nodes are 33 launches of three and one single step"""
    out = []
    for tuning, launches in ((0, 34), (PLAIN, 100)):
        lat = pkg.Lattice(9, W, H, tau_inv=np.float32(1 / 0.6), tuning=tuning)
        lat.set_flags(np.zeros(W * H, np.uint8))
        rng = np.random.default_rng(4)
        lat.init_equilibrium((1 + 0.02 * rng.standard_normal(W * H)).astype(np.float32))
        before = lat.launches()
        lat.step(100)
        assert lat.launches() - before == launches
        out.append(lat.populations())
        lat.close()
    assert beq(*out)
