"""GPU: psi = 4 exp(-200/rho) of a million densities per range, in the reference
mode's collision, gives the oracle's bits."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lo,hi", [(8.0, 700.0), (576.0, 578.5), (52.3, 52.6), (700.0, 1.1e6)])
def test_psi(pkg, oracle, lo, hi):
    W = H = 1024
    N = W * H
    rho = np.exp(np.linspace(np.log(lo), np.log(hi), N)).astype(np.float32)
    f = (oracle.D2_W[:, None] * rho[None, :]).astype(np.float32)
    zero = np.zeros(N, np.uint8)
    lat = pkg.Lattice(9, W, H, mode=pkg.abi.LB_MODE_REFERENCE, tau_inv=1.0, G=-120.0,
                      rho_out=float(rho[N // 2]), psi_form=pkg.abi.LB_PSI_REF)
    lat.set_flags(zero)
    lat.set_populations(f)
    lat.step(1)
    mom = [np.zeros(N, np.float32) for _ in range(3)]
    sc = [np.zeros(N, np.float32) for _ in range(3)]
    oracle.d2q9_stream(f, zero, W, H)
    oracle.d2q9_collide(f, zero, mom, sc, W, H, *pkg.W2, np.float32(1.0), 0.0, 0,
                        np.float32(rho[N // 2]), 0, 0, -120.0, 0.0)
    got = lat.populations()
    assert np.array_equal(got.view(np.uint32), f.view(np.uint32))
    lat.close()
