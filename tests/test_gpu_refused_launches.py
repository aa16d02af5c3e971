"""GPU: a launch that the runtime refuses (more rows than a grid takes) is reported
by the call that made it, and by no later call."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROWS = 65536  # one more than a grid's y extent


def later_calls_work(pkg):
    """calls whose launches report cudaGetLastError"""
    lat = pkg.Lattice(9, 64, 40, tau_inv=1.0)
    lat.set_flags(np.zeros(64 * 40, np.uint8))
    lat.init_equilibrium(np.ones(64 * 40, np.float32))
    lat.step(3)
    assert lat.steps_done() == 3
    lat.close()


@pytest.mark.parametrize("Q", [9, 19])
def test_entry_points(pkg, Q):
    L, F = pkg.lib(), ctypes.c_float
    dd = pkg.DeviceData(Q, 1, ROWS, 1)
    g, b = pkg.abi.dim3(1, 1, 1), pkg.abi.dim3(32, 4, 1)
    w = pkg.W2 if Q == 9 else pkg.W3

    def stream():
        (L.streaming_d2q9 if Q == 9 else L.streaming_d3q19)(dd.ptr(), g, b)

    def collide():
        plot, z = ctypes.c_void_p(dd.plot), F(0)
        if Q == 9:
            L.collision_d2q9(plot, dd.ptr(), F(w[0]), F(w[1]), F(w[2]), F(1), z, z, F(1), z, z, z,
                             z, g, b, z, z, z, z)
        else:
            L.collision_d3q19(plot, dd.ptr(), F(w[0]), F(w[1]), F(w[2]), F(1), z, z, z, F(1), z,
                              z, z, z, g, b)

    for call in (stream, collide):
        L.lb_abi_clear_error()
        call()
        assert L.lb_abi_last_error()
        L.lb_abi_clear_error()
        later_calls_work(pkg)
        assert not L.lb_abi_last_error()
    dd.close()


@pytest.mark.parametrize("Q,G", [(9, 0.0), (9, -5.0), (19, 0.0), (19, -5.0)])
def test_contexts(pkg, Q, G):
    lat = pkg.Lattice(Q, 1, ROWS, 1, tau_inv=1.0, G=G, tuning=0x108)
    lat.set_flags(np.zeros(ROWS, np.uint8))
    lat.init_equilibrium(np.ones(ROWS, np.float32))
    with pytest.raises(pkg.LBError):
        lat.step(1)
    later_calls_work(pkg)
    lat.close()
