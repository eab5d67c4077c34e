"""Several steps per launch on overlapped tiles (csrc/tiles.cuh): a D2Q9 lattice whose kernel family is
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
    ("outlets", 300, 200),  # more zero-gradient cells than threads
    ("lid", 129, 105),      # last tiles of one column and one row
    (1, 257, 199),
])
def test_tiles_equal_plain_steps(kind, nx, ny, storage):
    same(kind, nx, ny, storage, DEV, (1, 2, 3, 4, 9, 10, 31))


@pytest.mark.parametrize("storage", [lb.F32, lb.F64])
@pytest.mark.parametrize("kind,nx,ny", [("lid", 100, 100), (1, 131, 80), (0, 300, 100)])
def test_tiles_equal_plain_steps_in_absolute_arithmetic(kind, nx, ny, storage):
    same(kind, nx, ny, storage, ABS, (3, 20))


@pytest.mark.parametrize("storage,kind,nx,ny", [
    (lb.F32, "lid", 1024, 512),        # in L2, two waves: moved in pieces
    (lb.F32, 1, 1200, 1000),           # streamed by bulk copies
    (lb.F32, "periodic", 1068, 1067),  # a short last tile in x and y
    (lb.F32, 1, 1501, 1201),           # rows that start anywhere: moved in pieces
    (lb.F64, 1, 1030, 1000),           # streamed by bulk copies
    (lb.F32, "outlets", 1200, 1000),
])
def test_many_tiles_per_cta(storage, kind, nx, ny):
    same(kind, nx, ny, storage, DEV, (7, 12))


@pytest.mark.parametrize("storage", [lb.F32, lb.F16S, lb.BF16S])
@pytest.mark.parametrize("walls", [False, True])
@pytest.mark.parametrize("nx,ny", [
    (80, 10),     # the smallest
    (133, 97),    # remainders; rows that start anywhere (FP32; 16-bit words step singly)
    (136, 61),
    (520, 500),   # one wave of full tiles
    (1000, 900),  # several tiles a CTA
])
def test_shan_chen_tiles_equal_the_two_passes(nx, ny, walls, storage):
    d = lb.make_desc(lb.D2Q9, lb.SHANCHEN, storage, (nx, ny), omega=1.1, sc_G=-5.0)
    m = None
    if walls:  # solid rows, a forced-density equilibrium block, a row of forced velocity
        m = np.zeros((nx, ny), np.uint8)
        m[:, 0] = m[:, -1] = 1
        m[nx // 3:nx // 3 + 5, ny // 2:ny // 2 + 4] = 2
        m[:, ny // 4] = 3
        solid = lb.BOUNCE | lb.SET_RHO | lb.SET_UX | lb.SET_UY
        lb.set_classes(d, [(0, 1.0, 0.0, 0.0, 0.0), (solid, 0.3, 0.0, 0.0, 0.0),
                           (lb.EQUILIBRIUM | lb.SET_RHO, 0.8, 0.0, 0.0, 0.0), (lb.SET_UX, 1.0, 0.01, 0.0, 0.0)])
    _, _, _, w, _ = lb.velocities(lb.D2Q9)
    rho = 0.693 + np.random.default_rng(nx + ny).uniform(-0.05, 0.05, nx * ny)
    F = (w[:, None] * rho[None, :]).astype(np.float32).ravel()
    a = run(d, m, F, lb.KERNEL_AUTO, (1, 2, 3, 6, 9))
    b = run(d, m, F, lb.KERNEL_PLAIN, (1, 2, 3, 6, 9))
    for x, y in zip(a, b):
        assert np.array_equal(x, y, equal_nan=True)


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
