"""GPU: which lattices the D2Q9 marching strips are left out for."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tuning", [0, 0x102], ids=["default", "march"])
@pytest.mark.parametrize("walls", [False, True], ids=["periodic", "walls"])
def test_more_rows_than_a_grid_takes(pkg, walls, tuning):
    """65 536 rows: the flags are taken, and every step is refused before anything
    has moved, whatever the number of steps"""
    W, H = 9, 65536
    N = W * H
    lat = pkg.Lattice(9, W, H, tau_inv=1.0, tuning=tuning)
    flags = np.zeros(N, np.uint8)
    flags[::1001] = walls
    lat.set_flags(flags)
    rng = np.random.default_rng(1)
    lat.init_equilibrium((1 + 0.01 * rng.standard_normal(N)).astype(np.float32))
    f = lat.populations()
    for n in (1, 3, 7):
        with pytest.raises(pkg.LBError):
            lat.step(n)
        assert lat.steps_done() == 0
    assert np.array_equal(f.view(np.uint32), lat.populations().view(np.uint32))
    lat.close()


@pytest.mark.parametrize("W,H,launches", [(700001, 1, 6), (263000, 2, 6), (140000, 5, 6),
                                          (53125, 16, 6), (50001, 20, 2), (525000, 4, 2),
                                          (17000, 32, 2), (729, 721, 2)])
def test_lattices_of_few_rows(pkg, W, H, launches):
    """six steps by default: two launches of three where the strips are the faster form,
    six where the rows an item reads beyond its own outweigh them; the same bits"""
    N = W * H
    rng = np.random.default_rng(2)
    rho = (1 + 0.01 * rng.standard_normal(N)).astype(np.float32)
    out = []
    for tuning in (0, 0x108):
        lat = pkg.Lattice(9, W, H, tau_inv=np.float32(1 / 0.6), tuning=tuning)
        lat.set_flags(np.zeros(N, np.uint8))
        lat.init_equilibrium(rho)
        before = lat.launches()
        lat.step(6)
        if tuning == 0:
            assert lat.launches() - before == launches
        out.append(lat.populations())
        lat.close()
    assert np.array_equal(out[0].view(np.uint32), out[1].view(np.uint32))
