"""The tiles' packed FP32 arithmetic against the scalar one at its limits."""
import ctypes as C

import numpy as np
import pytest

from helpers import lb

pytestmark = pytest.mark.gpu


def bits(x):
    return int(np.float32(x).view(np.uint32))


def test_reciprocal_equals_the_division():
    """Every float of the range that densities take, of both signs (2.5 thousand million)."""
    differ = C.c_int64(-1)
    first, last = bits(2.0 ** -24), bits(2.0 ** 126)
    assert lb.lib().lbm_test_reciprocal(first, last - first, C.byref(differ)) == 0
    assert differ.value == 0
    # the count does count: the reciprocal of zero is NaN here and infinite as a division
    assert lb.lib().lbm_test_reciprocal(0, 1, C.byref(differ)) == 0
    assert differ.value == 2


@pytest.mark.parametrize("storage", [lb.F32, lb.F16S, lb.BF16S, lb.F64])
@pytest.mark.parametrize("collision,kind,nx,ny", [(lb.BGK, 1, 260, 190), (lb.BGK, 2, 128, 120), (lb.BGK, None, 1200, 1000),
                                                  (lb.SHANCHEN, None, 200, 136)])
def test_a_diverging_lattice_diverges_alike(collision, kind, nx, ny, storage):
    """From populations of order one to infinities and NaN: as single steps do, value by value."""
    out = []
    for kernel in (lb.KERNEL_AUTO, lb.KERNEL_PLAIN):
        d = lb.make_desc(lb.D2Q9, collision, storage, (nx, ny), omega=1.99, sc_G=-5.0)
        m = None if kind is None else lb.setup_channel2d(d, 0.04, nx // 5, ny // 2, ny // 10, kind)
        _, _, _, w, _ = lb.velocities(lb.D2Q9)
        noise = 0.6 * np.random.default_rng(1).standard_normal(9 * nx * ny)
        with lb.Lattice(d, m) as lat:
            lat.set_kernel(kernel)
            lat.set_populations((np.repeat(w, nx * ny) * (1 + noise)).astype(np.float32))
            states = []
            for _ in range(7):
                lat.step(8)
                states.append(lat.get_populations(np.float64))
            out.append(states)
    for a, b in zip(*out):
        assert np.array_equal(a, b, equal_nan=True)
    assert not np.abs(out[1][-1]).max() < 1e20 or storage == lb.F16S  # it did
