"""Tiles at the sizes that are run in earnest: tall tiles, which have inner cells that no neighbour needs and long lists of
outlet cells, and runs beyond the steps of one launch.  Each case states the tiles it has to take, so that a plan that
stopped taking tiles does not pass unseen."""
import numpy as np
import pytest

from helpers import lb

pytestmark = pytest.mark.gpu

SMALL, MID, PIECES, STREAM, SHANCHEN = 1, 2, 3, 4, 5


def lattice(kind, nx, ny, storage, kernel=lb.KERNEL_AUTO, arithmetic=lb.ARITH_DEVIATION):
    if kind == "shanchen":
        d, m = lb.make_desc(lb.D2Q9, lb.SHANCHEN, storage, (nx, ny), omega=1.1, sc_G=-5.0), None
        amp = 0.02
    else:
        d = lb.make_desc(lb.D2Q9, lb.BGK, storage, (nx, ny), omega=1.25, arithmetic=arithmetic)
        m = lb.setup_cavity2d(d, 0.1) if kind == "lid" else lb.setup_channel2d(d, 0.04, nx // 5, ny // 2, ny // 10, kind)
        amp = 0.01
    lat = lb.Lattice(d, m)
    lat.set_kernel(kernel)
    _, _, _, w, _ = lb.velocities(lb.D2Q9)
    rng = np.random.default_rng(nx * 31 + ny)
    lat.set_populations((np.repeat(w, nx * ny) * (0.7 + amp * rng.standard_normal(9 * nx * ny))).astype(np.float32))
    return lat


def same_as_plain(kind, nx, ny, storage, runs, shape, rows, steps, rounds, arithmetic=lb.ARITH_DEVIATION):
    with lattice(kind, nx, ny, storage, arithmetic=arithmetic) as a, \
            lattice(kind, nx, ny, storage, lb.KERNEL_PLAIN, arithmetic) as b:
        for n in runs:
            a.step(n)
            b.step(n)
            assert a.test_last_tiles() == (shape, rows, steps, rounds) and b.test_last_tiles()[0] == 0
            assert np.array_equal(a.get_populations(np.float64), b.get_populations(np.float64), equal_nan=True)
            assert a.residual() == b.residual()


@pytest.mark.parametrize("storage", [lb.F32, lb.F16S, lb.BF16S])
@pytest.mark.parametrize("kind,nx,ny,rows", [(0, 1024, 256, 30), (1, 1024, 256, 30), (2, 1024, 256, 30), ("lid", 512, 512, 30),
                                             (0, 1000, 300, 34), (1, 1000, 300, 34), ("lid", 500, 512, 30)])
def test_tall_tiles_that_stay_for_a_run(kind, nx, ny, rows, storage):
    same_as_plain(kind, nx, ny, storage, (13, 34), MID, rows, 4, 1)


@pytest.mark.parametrize("nx,ny,kind,rows", [(640, 400, 1, 30), (641, 401, "lid", 32), (576, 500, 1, 32)])
def test_tall_double_precision_tiles(nx, ny, kind, rows):
    same_as_plain(kind, nx, ny, lb.F64, (13, 34), MID, rows, 4, 1)


def test_tall_tiles_in_absolute_arithmetic():
    same_as_plain(1, 1000, 300, lb.F32, (13, 34), MID, 34, 4, 1, lb.ARITH_ABSOLUTE)


@pytest.mark.parametrize("storage", [lb.F32, lb.F16S])
@pytest.mark.parametrize("kind,nx,ny,shape,rows,steps", [("lid", 128, 128, SMALL, 8, 8), ("lid", 192, 176, SMALL, 16, 4),
                                                         (1, 260, 190, MID, 8, 4)])
def test_runs_beyond_one_launch(kind, nx, ny, shape, rows, steps, storage):
    """4096 steps a launch: the rounds of the second launch go on from those of the first."""
    same_as_plain(kind, nx, ny, storage, (4099, 8200), shape, rows, steps, 1)


@pytest.mark.parametrize("kind,nx,ny,storage,shape,rows,steps", [
    ("lid", 1024, 512, lb.F32, PIECES, 30, 4),
    ("lid", 1501, 1201, lb.F32, PIECES, 34, 4),
    (1, 1200, 1000, lb.F32, STREAM, 34, 4),
    (1, 1030, 1000, lb.F64, STREAM, 12, 4),
    ("shanchen", 1024, 1024, lb.BF16S, SHANCHEN, 28, 2),
    ("shanchen", 1025, 769, lb.F32, SHANCHEN, 30, 2),
])
def test_many_tiles_a_cta(kind, nx, ny, storage, shape, rows, steps):
    same_as_plain(kind, nx, ny, storage, (7, 18), shape, rows, steps, 0)


@pytest.mark.parametrize("kind,nx,ny,storage,few,enough", [
    ("lid", 64, 64, lb.F32, (3, 10, 23), 24),        # one cluster
    ("lid", 48, 40, lb.F64, (4, 63), 64),
    ("lid", 80, 80, lb.F16S, (4, 13), 14),
    ("lid", 100, 100, lb.F32, (4,), 10),
    (1, 1200, 1000, lb.F32, (3, 4), 5),              # single steps
    (1, 641, 401, lb.F64, (3, 4), 5),
    (0, 1001, 300, lb.F16S, (3, 4), 5),
    ("lid", 1501, 1201, lb.F32, (3, 4), 5),
])
def test_runs_too_short_for_tiles(kind, nx, ny, storage, few, enough):
    with lattice(kind, nx, ny, storage) as a, lattice(kind, nx, ny, storage, lb.KERNEL_PLAIN) as b:
        for n in (*few, enough):
            a.step(n)
            a.sync()  # (small lattices with runs beside one another take single steps or clusters anyway)
            b.step(n)
            b.sync()
            if a.kernel() == lb.KERNEL_CLUSTER or a.desc.cells > 16384:
                assert (a.test_last_tiles()[0] != 0) == (n == enough)
            assert np.array_equal(a.get_populations(np.float64), b.get_populations(np.float64), equal_nan=True)
