"""lbm_step inside a stream capture: a captured even run is replayed from the buffer that it was captured from, any
number of times and between live runs, and advances the lattice each time, whatever family the engine chose."""
import numpy as np
import pytest

from helpers import lb

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def lattice(collision, nx, ny, storage):
    d = lb.make_desc(lb.D2Q9, collision, storage, (nx, ny), omega=1.3, sc_G=-5.0)
    m = lb.setup_cavity2d(d, 0.1) if collision == lb.BGK else None
    _, _, _, w, _ = lb.velocities(lb.D2Q9)
    rng = np.random.default_rng(nx + ny)
    F = (np.repeat(w, nx * ny) * (0.7 + 0.02 * rng.standard_normal(9 * nx * ny))).astype(np.float32)
    lat = lb.Lattice(d, m)
    lat.set_populations(F)
    return lat


@pytest.mark.parametrize("n", [2, 4, 10, 26])
@pytest.mark.parametrize("collision,nx,ny,storage", [
    (lb.BGK, 128, 128, lb.F32),     # captured: one cluster
    (lb.BGK, 128, 128, lb.F16S),
    (lb.BGK, 260, 190, lb.F32),     # live: tiles that stay for a run
    (lb.BGK, 300, 200, lb.BF16S),
    (lb.BGK, 1200, 1000, lb.F32),   # live: four steps a launch
    (lb.BGK, 1030, 1000, lb.F64),
    (lb.SHANCHEN, 200, 136, lb.F32),  # live: two steps a launch
])
def test_replays_between_live_runs(collision, nx, ny, storage, n):
    stream = torch.cuda.Stream()
    with lattice(collision, nx, ny, storage) as lat, lattice(collision, nx, ny, storage) as ref:
        ref.set_kernel(lb.KERNEL_PLAIN)
        lat.set_stream(stream)

        def same():
            torch.cuda.synchronize()
            return np.array_equal(lat.get_populations(np.float64), ref.get_populations(np.float64), equal_nan=True)

        lat.step(7)
        lat.sync()
        ref.step(7)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            lat.step(n)
        for _ in range(2):
            with torch.cuda.stream(stream):
                graph.replay()
            ref.step(n)
        assert same()
        for live in (2, 4, 6, 10, 12, 36):
            lat.step(live)
            ref.step(live)
            assert same()
            with torch.cuda.stream(stream):
                graph.replay()
            ref.step(n)
            assert same()
        torch.cuda.synchronize()
        del graph


def test_long_captured_and_live_runs_in_one_cluster():
    """More than the 4096 steps of one launch, captured and live."""
    stream = torch.cuda.Stream()
    with lattice(lb.BGK, 64, 48, lb.F32) as lat, lattice(lb.BGK, 64, 48, lb.F32) as ref:
        ref.set_kernel(lb.KERNEL_PLAIN)
        lat.set_kernel(lb.KERNEL_CLUSTER)
        lat.set_stream(stream)
        lat.step(2)
        lat.sync()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            lat.step(4100)
        for _ in range(2):
            with torch.cuda.stream(stream):
                graph.replay()
        lat.step(10000)
        with torch.cuda.stream(stream):
            graph.replay()
        torch.cuda.synchronize()
        ref.step(2 + 3 * 4100 + 10000)
        assert np.array_equal(lat.get_populations(np.float64), ref.get_populations(np.float64))
        del graph


@pytest.mark.parametrize("built", [False, True])
@pytest.mark.parametrize("lattice_id,shape,storage", [(lb.D2Q9, (150, 97), lb.F16S), (lb.D3Q27, (48, 20, 16), lb.F32)])
def test_captures_before_and_after_the_engines_own_graphs(lattice_id, shape, storage, built):
    """Long live runs of single steps replay graphs of the engine's own; a capture may come before or after the first one."""
    stream = torch.cuda.Stream()
    d = lb.make_desc(lattice_id, lb.BGK, storage, shape, omega=1.3)
    n = int(np.prod(shape))
    w = lb.velocities(lattice_id)[3]
    F = (np.repeat(w, n) * (1 + 0.02 * np.random.default_rng(n).standard_normal(len(w) * n))).astype(np.float32)
    with lb.Lattice(d) as lat, lb.Lattice(d) as ref:
        for a in (lat, ref):
            a.set_kernel(lb.KERNEL_PLAIN)
            a.set_populations(F)
        lat.set_stream(stream)
        lat.step(700 if built else 2)
        ref.step(700 if built else 2)
        lat.sync()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            lat.step(600)
        for _ in range(2):
            with torch.cuda.stream(stream):
                graph.replay()
        ref.step(1200)
        torch.cuda.synchronize()
        assert np.array_equal(lat.get_populations(np.float64), ref.get_populations(np.float64))
        lat.step(700)
        ref.step(700)
        with torch.cuda.stream(stream):
            graph.replay()
        ref.step(600)
        torch.cuda.synchronize()
        assert np.array_equal(lat.get_populations(np.float64), ref.get_populations(np.float64))
        del graph
