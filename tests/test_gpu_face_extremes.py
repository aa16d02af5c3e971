"""GPU: the reference mode's Zou-He faces give the oracle's bits for inlet
velocities and outlet densities so large that their reciprocal's low part would be
a subnormal float, with populations of the same size."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def same(a, b):
    a, b = np.asarray(a), np.asarray(b)
    eq = (a.view(np.uint32) == b.view(np.uint32)) | (np.isnan(a) & np.isnan(b))
    return a.shape == b.shape and bool(eq.all())


@pytest.mark.parametrize("size", [1e30, 1e32, 1e34, 7e34, 1e35, 1e36, 1e37])
@pytest.mark.parametrize("Q", [9, 19])
def test_outlet_density_and_inlet_velocity(pkg, oracle, Q, size):
    W, H, D = (12, 4000, 1) if Q == 9 else (9, 60, 60)
    N = W * H * D
    rng = np.random.default_rng(7)
    w = oracle.D2_W if Q == 9 else oracle.D3_W
    f = (w[:, None] * size * (1 + 0.3 * rng.standard_normal((Q, N)))).astype(np.float32)
    ux_in, rho_out, tau_inv = np.float32(-size), np.float32(size), np.float32(1.25)
    zero = np.zeros(N, np.uint8)
    lat = pkg.Lattice(Q, W, H, D, mode=pkg.abi.LB_MODE_REFERENCE, tau_inv=tau_inv,
                      u_in=(ux_in, 0, 0), rho_out=rho_out)
    lat.set_flags(zero)
    lat.set_populations(f)
    lat.step(1)
    mom = [np.zeros(N, np.float32) for _ in range(4)]
    with np.errstate(all="ignore"):
        if Q == 9:
            sc = [np.zeros(N, np.float32) for _ in range(3)]
            oracle.d2q9_stream(f, zero, W, H)
            oracle.d2q9_collide(f, zero, mom[:3], sc, W, H, *pkg.W2, tau_inv, ux_in, 0, rho_out,
                                0, 0, 0.0, 0.0)
        else:
            oracle.d3q19_stream(f, zero, W, H, D)
            oracle.d3q19_collide(f, zero, mom, W, H, D, *pkg.W3, tau_inv, ux_in, 0, 0, rho_out)
    got = lat.moments()[:3] if Q == 9 else lat.moments()
    ux, rho = (got[1], got[0])
    assert same(rho, mom[2] if Q == 9 else mom[3]) and same(ux, mom[0])
    assert same(lat.populations(), f)
    lat.close()
