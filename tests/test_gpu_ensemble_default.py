"""GPU: the ensemble's default launch form follows the shapes of its domains, and gives
the bits of the form it replaces."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def ensemble(pkg, dims):
    nx, ny = (np.array([d[i] for d in dims], np.int32) for i in (0, 1))
    ens = pkg.Ensemble(nx, ny, np.full(len(dims), -5.0, np.float32))
    rng = np.random.default_rng(4)
    ens.init_equilibrium((0.693 * (1 + rng.uniform(-0.01, 0.01, ens.NT))).astype(np.float32))
    return ens


@pytest.mark.parametrize("dims,form", [
    ([(8, 8)] * 8192, 6),               # 64-column strips would store 8 columns each
    ([(10, 10)] * 6000, 6),             # and copy node by node
    ([(8, 8)] * 16384, 6),              # 2^20 nodes: two steps per launch otherwise
    ([(16, 16)] * 64, 10),              # too few for one round of strips
    ([(64, 64)] * 1024, 10),
    ([(10, 10)] * 50 + [(512, 512)] * 8, 10),
], ids=["8", "10", "8-two-steps", "few-16", "64", "mixed"])
def test_default_form(pkg, dims, form):
    got = []
    for other in (0, 10, 6):
        ens = ensemble(pkg, dims)
        if other:
            ens.set_launch(0, other, 6)
        else:
            shape = np.zeros(3, np.int32)
            assert pkg.lib().lb_ensemble_get_launch(ens.h, shape.ctypes.data) == 0
            assert tuple(shape[:2]) == (0, form)
        ens.step(37)
        got.append([np.ascontiguousarray(v).view(np.uint32)
                    for v in (ens.populations(), *ens.moments())])
        ens.close()
    for g in got[1:]:
        assert all(np.array_equal(a, b) for a, b in zip(got[0], g))
