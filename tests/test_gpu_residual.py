"""lbm_residual_fp64 on states out of the ordinary: an infinite population makes it non-finite (reported as a
divergence) whichever its direction, and ordinary states give what plain NumPy gives."""
import numpy as np
import pytest

from helpers import lb

pytestmark = pytest.mark.gpu

DIVERGED = -4
EQ = lb.EQUILIBRIUM | lb.SET_RHO | lb.SET_UX | lb.SET_UY | lb.SET_UZ


def fixed_velocity(lattice, storage, shape):
    """Every cell is an equilibrium cell of class 0: whatever it receives, the state after a step is finite."""
    d = lb.make_desc(lattice, lb.BGK, storage, shape, omega=1.3)
    lb.set_classes(d, [(EQ, 1.0, 0.05, 0.0, 0.0)])
    return d


@pytest.mark.parametrize("storage", [lb.F32, lb.F64, lb.BF16S])
@pytest.mark.parametrize("lattice,shape", [(lb.D2Q9, (40, 30)), (lb.D3Q27, (20, 12, 10))])
def test_an_infinite_population_is_a_divergence(lattice, shape, storage):
    n = int(np.prod(shape))
    w = lb.velocities(lattice)[3]
    for direction in (0, 1, len(w) - 1):
        F = np.repeat(w, n).astype(np.float32)
        F[direction * n + n // 2] = np.inf
        with lb.Lattice(fixed_velocity(lattice, storage, shape)) as lat:
            lat.set_populations(F)
            lat.step(1)
            with pytest.raises(lb.LbmError) as e:
                lat.residual()
            assert e.value.code == DIVERGED


@pytest.mark.parametrize("storage", [lb.F32, lb.F64])
@pytest.mark.parametrize("lattice,shape", [(lb.D2Q9, (61, 47)), (lb.D3Q27, (20, 12, 11))])
def test_residual_of_ordinary_states(lattice, shape, storage):
    n = int(np.prod(shape))
    cx, cy, cz, w, _ = lb.velocities(lattice)
    rng = np.random.default_rng(n)
    F = (np.repeat(w, n) * (1 + 0.02 * rng.standard_normal(len(w) * n))).astype(np.float32)
    states = []
    with lb.Lattice(lb.make_desc(lattice, lb.BGK, storage, shape, omega=1.3)) as lat:
        lat.set_populations(F)
        for _ in range(2):
            lat.step(1)
            states.append(lat.get_populations(np.float64).reshape(len(w), n).astype(np.longdouble))
        got = lat.residual()
    u = [np.stack([(np.asarray(c)[:, None] * f).sum(0) for c in (cx, cy, cz)]) / f.sum(0) for f in states]
    want = np.sqrt(((u[1] - u[0]) ** 2).sum() / (u[1] ** 2).sum())
    # |u| and |du| are some 1e-2; a velocity carries at most 30 roundings of 2^-53 of terms below 0.5
    assert abs(got - want) <= want * 1e-12
