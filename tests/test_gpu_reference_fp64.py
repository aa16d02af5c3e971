"""GPU: the reference mode's FP64 lines (Zou-He faces, psi = 4 exp(-200/rho))
give the oracle's bits where the library forms them in pairs of floats, at the
edges of that form's range and outside it: densities from tiny to huge, flows
at rest, inlet velocities and outlet densities whose reciprocal is not finite."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

STEPS = 2


def same(a, b):
    a, b = np.asarray(a), np.asarray(b)
    eq = (a.view(np.uint32) == b.view(np.uint32)) | (np.isnan(a) & np.isnan(b))
    return a.shape == b.shape and bool(eq.all())


def state(w, N, scale, noise):
    rng = np.random.default_rng(N)
    return (w[:, None] * scale * (1 + noise * rng.standard_normal((len(w), N)))).astype(np.float32)


FACES = [(0.05, 1.0), (0.0, 1.0), (-0.3, 0.7), (0.999999, 1e-3), (1.0, 1.0), (0.02, 0.0)]
STATES = [(1.0, 0.0), (1.0, 0.05), (200.0, 0.01), (1e-30, 0.05)]


@pytest.mark.parametrize("scale,noise", STATES)
@pytest.mark.parametrize("ux_in,rho_out", FACES)
def test_faces_d2q9(pkg, oracle, ux_in, rho_out, scale, noise):
    W, H = 33, 40
    N = W * H
    f = state(oracle.D2_W, N, scale, noise)
    tau_inv = np.float32(1 / 0.8)
    zero = np.zeros(N, np.uint8)
    lat = pkg.Lattice(9, W, H, mode=pkg.abi.LB_MODE_REFERENCE, tau_inv=tau_inv,
                      u_in=(ux_in, 0, 0), rho_out=rho_out)
    lat.set_flags(zero)
    lat.set_populations(f)
    lat.step(STEPS)
    mom = [np.zeros(N, np.float32) for _ in range(3)]
    sc = [np.zeros(N, np.float32) for _ in range(3)]
    with np.errstate(all="ignore"):
        for _ in range(STEPS):
            oracle.d2q9_stream(f, zero, W, H)
            oracle.d2q9_collide(f, zero, mom, sc, W, H, *pkg.W2, tau_inv, np.float32(ux_in), 0,
                                np.float32(rho_out), 0, 0, 0.0, 0.0)
    assert same(lat.populations(), f)
    lat.close()


@pytest.mark.parametrize("scale,noise", STATES)
@pytest.mark.parametrize("ux_in,rho_out", FACES)
def test_faces_d3q19(pkg, oracle, ux_in, rho_out, scale, noise):
    W, H, D = 9, 20, 11
    N = W * H * D
    f = state(oracle.D3_W, N, scale, noise)
    tau_inv = np.float32(1 / 0.8)
    zero = np.zeros(N, np.uint8)
    lat = pkg.Lattice(19, W, H, D, mode=pkg.abi.LB_MODE_REFERENCE, tau_inv=tau_inv,
                      u_in=(ux_in, 0, 0), rho_out=rho_out)
    lat.set_flags(zero)
    lat.set_populations(f)
    lat.step(STEPS)
    mom = [np.zeros(N, np.float32) for _ in range(4)]
    for _ in range(STEPS):
        oracle.d3q19_stream(f, zero, W, H, D)
        oracle.d3q19_collide(f, zero, mom, W, H, D, *pkg.W3, tau_inv, np.float32(ux_in), 0, 0,
                             np.float32(rho_out))
    assert same(lat.populations(), f)
    lat.close()


@pytest.mark.parametrize("lo,hi", [(0.5, 8.0), (7.99, 8.01), (8.0, 700.0), (700.0, 3e6),
                                   (1048575.0, 1048577.0)])
def test_reference_psi(pkg, oracle, lo, hi):
    W, H = 64, 64
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
    assert same(lat.populations(), f)
    lat.close()
