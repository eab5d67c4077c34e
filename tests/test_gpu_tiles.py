"""Several steps per launch on overlapped tiles (csrc/tiles.cuh): a D2Q9 BGK lattice whose kernel family is
left to the engine gives the same populations, macros and residual as one stepped by the plain kernel, bit
for bit: every storage and arithmetic, each tile shape, remainders of tiles and of steps, all boundary
classes."""
import numpy as np
import pytest

from helpers import lb

pytestmark = pytest.mark.gpu

DEV, ABS = lb.ARITH_DEVIATION, lb.ARITH_ABSOLUTE


def problem(kind, nx, ny, storage, arithmetic):
    d = lb.make_desc(lb.D2Q9, lb.BGK, storage, (nx, ny), omega=1.25, arithmetic=arithmetic)
    if kind == "lid":
        m = lb.setup_cavity2d(d, 0.1)
    elif kind == "periodic":
        m = None
    elif kind == "outlets":  # zero-gradient cells in neighbouring columns, without a mask's help
        lb.set_classes(d, [(lb.ZEROGRAD_XP, 1.0, 0.0, 0.0, 0.0)])
        m = None
    else:  # channel with the given boundaries
        m = lb.setup_channel2d(d, 0.04, nx // 5, ny // 2, ny // 10, kind)
    return d, m


def start(nx, ny):
    _, _, _, w, _ = lb.velocities(lb.D2Q9)
    rng = np.random.default_rng(nx * 10007 + ny)
    return (np.repeat(w, nx * ny) * (1 + 0.02 * rng.standard_normal(9 * nx * ny))).astype(np.float32)


def run(d, m, F, kernel, runs):
    out = []
    with lb.Lattice(d, m) as lat:
        lat.set_kernel(kernel)
        lat.set_populations(F)
        for n in runs:
            lat.step(n)
            rho, u = lat.macros(np.float32)
            out += [lat.get_populations(np.float64), rho, u, np.float64(lat.residual())]
        lat.sync()
        assert lat.steps_done == sum(runs)
    return out


def same(kind, nx, ny, storage, arithmetic, runs):
    d, m = problem(kind, nx, ny, storage, arithmetic)
    F = start(nx, ny)
    a = run(d, m, F, lb.KERNEL_AUTO, runs)
    b = run(d, m, F, lb.KERNEL_PLAIN, runs)
    for x, y in zip(a, b):
        assert np.array_equal(x, y, equal_nan=True)


@pytest.mark.parametrize("storage", [lb.F32, lb.F16S, lb.BF16S, lb.F64])
@pytest.mark.parametrize("kind,nx,ny", [
    ("lid", 32, 18),        # the smallest lattice and the smallest tile
    ("lid", 128, 128),      # whole tiles of the small shape
    ("periodic", 133, 97),  # remainders in x and y, odd rows
    (1, 130, 101),          # equilibrium inlet, zero-gradient outlet
    (2, 134, 90),           # Zou-He boundaries
    ("lid", 180, 164),      # small shape, four steps
    (0, 260, 190),          # mid shape, the reference's channel
    (1, 301, 199),          # mid shape, rows that start anywhere
    ("outlets", 96, 80),
])
def test_tiles_equal_plain_steps(kind, nx, ny, storage):
    same(kind, nx, ny, storage, DEV, (1, 2, 3, 4, 9, 10, 31))


@pytest.mark.parametrize("storage", [lb.F32, lb.F64])
@pytest.mark.parametrize("kind,nx,ny", [("lid", 100, 100), (1, 131, 80), (0, 300, 100)])
def test_tiles_equal_plain_steps_in_absolute_arithmetic(kind, nx, ny, storage):
    same(kind, nx, ny, storage, ABS, (3, 20))


@pytest.mark.parametrize("kind,nx,ny", [
    (1, 1200, 1000),          # streamed tiles
    ("periodic", 1068, 1067), # a short last tile in x and y
    ("lid", 1501, 1201),      # one region at a time: rows that start anywhere
])
def test_large_fp32_lattices(kind, nx, ny):
    same(kind, nx, ny, lb.F32, DEV, (7, 12))


def test_nearest_rounding_and_cell_offset():
    """Tiles hash the same cell indices and step numbers as single steps; round-to-nearest too."""
    for rounding in (lb.ROUND_STOCHASTIC, lb.ROUND_NEAREST):
        d = lb.make_desc(lb.D2Q9, lb.BGK, lb.F16S, (144, 120), omega=1.3, rounding=rounding)
        m = lb.setup_cavity2d(d, 0.1)
        out = []
        for kernel in (lb.KERNEL_AUTO, lb.KERNEL_PLAIN):
            with lb.Lattice(d, m) as lat:
                lat.set_kernel(kernel)
                lat.set_cell_offset(12345)
                lat.set_populations(start(144, 120))
                lat.step(29)
                out.append(lat.get_populations(np.float64))
        assert np.array_equal(out[0], out[1])


def test_two_lattices_on_two_streams():
    """Interleaved runs of two lattices (each on its own stream) do not disturb one another."""
    sizes = ((128, 128), (260, 190))
    alone = []
    for nx, ny in sizes:
        d, m = problem("lid", nx, ny, lb.F32, DEV)
        with lb.Lattice(d, m) as lat:
            lat.set_populations(start(nx, ny))
            lat.step(60)
            alone.append(lat.get_populations(np.float64))
    ds = [problem("lid", nx, ny, lb.F32, DEV) for nx, ny in sizes]
    with lb.Lattice(*ds[0]) as a, lb.Lattice(*ds[1]) as b:
        for lat, (nx, ny) in zip((a, b), sizes):
            lat.set_populations(start(nx, ny))
        for _ in range(3):
            a.step(20)
            b.step(20)
        assert np.array_equal(a.get_populations(np.float64), alone[0])
        assert np.array_equal(b.get_populations(np.float64), alone[1])
