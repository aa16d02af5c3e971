"""GPU: the ensemble's strips of column pairs (forms 10 to 12) evolve every
domain bit for bit like the same domain alone, with one and with two steps per
launch (form 10 on 2^20 nodes and more): domains of one node to several strips,
rows that start on 16 bytes and rows that do not, odd step counts, both psi
forms, graphs and direct launches."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DIMS = [(64, 64), (56, 8), (5, 7), (60, 33), (57, 19), (1, 1), (128, 70), (113, 24), (64, 2),
        (2, 90), (300, 9)]


def beq(a, b):
    a, b = np.ascontiguousarray(a), np.ascontiguousarray(b)
    return a.shape == b.shape and np.array_equal(a.view(np.uint8), b.view(np.uint8))


@pytest.mark.parametrize("psi,G0,rho0", [(1, -5.0, 0.693), (0, -120.0, 200.0)],
                         ids=["exp1", "reference"])
@pytest.mark.parametrize("form,large", [(10, False), (11, False), (12, False), (10, True)],
                         ids=["one-step", "64-rows", "16-rows", "two-steps"])
def test_matches_single_domain_runs(pkg, form, large, psi, G0, rho0):
    dims = DIMS + [(1024, 1024)] if large else DIMS
    nx = np.array([d[0] for d in dims], np.int32)
    ny = np.array([d[1] for d in dims], np.int32)
    rng = np.random.default_rng(3)
    G = (G0 * (1 + 0.05 * rng.uniform(-1, 1, len(dims)))).astype(np.float32)
    tau_inv = rng.uniform(0.8, 1.2, len(dims)).astype(np.float32)
    rho = (rho0 * (1 + rng.uniform(-0.01, 0.01, int((nx * ny).sum())))).astype(np.float32)
    ens = pkg.Ensemble(nx, ny, G, tau_inv=tau_inv, psi_form=psi)
    ens.set_launch(0, form, 12)
    ens.init_equilibrium(rho)
    steps = (1, 2, 35, 70)
    for n in steps:
        ens.step(n)
    f, mom = ens.populations(), ens.moments()
    for d, (W, H) in enumerate(dims):
        lat = pkg.Lattice(9, W, H, tau_inv=float(tau_inv[d]), G=float(G[d]), psi_form=psi)
        lat.set_flags(np.zeros(W * H, np.uint8))
        lat.init_equilibrium(ens.domain(rho, d))
        lat.step(sum(steps))
        assert beq(ens.domain(f, d), lat.populations()), (W, H)
        for a, b in zip(mom, lat.moments()[:3]):
            assert beq(ens.domain(a, d), b), (W, H)
        lat.close()
    ens.close()


def test_default_takes_two_steps_on_large_ensembles(pkg):
    n = np.full(5, 512, np.int32)  # 1.3 M nodes
    ens = pkg.Ensemble(n, n, np.full(5, -5.0, np.float32))
    ens.init_equilibrium(np.full(5 * 512 * 512, 0.7, np.float32))
    before = ens.launches()
    ens.step(101)  # one step, then pairs
    assert ens.launches() - before == 51
    ens.close()
