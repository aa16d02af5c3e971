"""GPU: every launch form of the ensemble, with both forms of psi, gives the bits of
the domains run alone."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DIMS = [(33, 20), (5, 7), (64, 32), (1, 9), (70, 41)]
FORMS = [(0, n, 3) for n in range(1, 13)] + [(64, 2, 4)]


@pytest.mark.parametrize("psi,G,rho0", [(1, -5.0, 0.693), (0, -120.0, 200.0)],
                         ids=["exp1", "reference"])
def test_every_form(pkg, psi, G, rho0):
    nx = np.array([d[0] for d in DIMS], np.int32)
    ny = np.array([d[1] for d in DIMS], np.int32)
    rng = np.random.default_rng(8)
    rho = (rho0 * (1 + rng.uniform(-0.01, 0.01, int((nx * ny).sum())))).astype(np.float32)
    Gs = np.full(len(DIMS), G, np.float32)
    want = []
    for form in FORMS:
        ens = pkg.Ensemble(nx, ny, Gs, psi_form=psi)
        ens.set_launch(*form)
        ens.init_equilibrium(rho)
        ens.step(41)
        f = ens.populations()
        for d, (W, H) in enumerate(DIMS):
            if len(want) <= d:
                lat = pkg.Lattice(9, W, H, tau_inv=1.0, G=G, psi_form=psi)
                lat.set_flags(np.zeros(W * H, np.uint8))
                lat.init_equilibrium(ens.domain(rho, d))
                lat.step(41)
                want.append(lat.populations().view(np.uint32))
                lat.close()
            got = np.ascontiguousarray(ens.domain(f, d)).view(np.uint32)
            assert np.array_equal(got, want[d]), (form, W, H)
        ens.close()
