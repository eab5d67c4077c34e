"""Tiles that stay in their CTAs exchange the cells at their edges in rounds (csrc/tiles.cuh): what happens where they
cannot."""
import numpy as np
import pytest

from helpers import lb

pytestmark = pytest.mark.gpu


def lattice(nx, ny, storage, kernel=lb.KERNEL_AUTO):
    d = lb.make_desc(lb.D2Q9, lb.BGK, storage, (nx, ny), omega=1.25)
    lat = lb.Lattice(d, lb.setup_channel2d(d, 0.04, nx // 5, ny // 2, ny // 10, 1))
    lat.set_kernel(kernel)
    _, _, _, w, _ = lb.velocities(lb.D2Q9)
    rng = np.random.default_rng(nx * ny)
    lat.set_populations((np.repeat(w, nx * ny) * (1 + 0.02 * rng.standard_normal(9 * nx * ny))).astype(np.float32))
    return lat


@pytest.mark.parametrize("storage", [lb.F32, lb.F16S, lb.F64])
@pytest.mark.parametrize("nx,ny", [(128, 128), (180, 164), (301, 199)])
def test_without_memory_for_the_exchange(nx, ny, storage):
    """One launch per few steps, with the same results; lbm_step does not allocate."""
    with lattice(nx, ny, storage) as lat, lattice(nx, ny, storage, lb.KERNEL_PLAIN) as ref:
        lat.step(31)
        assert lat.test_last_tiles()[3] == 1
        lat.test_without_exchange()
        for n in (3, 9, 10, 31):
            lat.step(n)
            shape, _, _, rounds = lat.test_last_tiles()
            assert shape in (1, 2) and rounds == 0
        ref.step(31 + 3 + 9 + 10 + 31)
        assert np.array_equal(lat.get_populations(np.float64), ref.get_populations(np.float64))
