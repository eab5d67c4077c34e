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
        for n in (5, 9, 10, 31):
            lat.step(n)
            shape, _, _, rounds = lat.test_last_tiles()
            assert shape in (1, 2) and rounds == 0
        ref.step(31 + 5 + 9 + 10 + 31)
        assert np.array_equal(lat.get_populations(np.float64), ref.get_populations(np.float64))


@pytest.mark.parametrize("captured", [False, True])
@pytest.mark.parametrize("nx,ny,storage", [(128, 128, lb.F32), (180, 164, lb.F16S), (301, 199, lb.F64)])
def test_where_the_ctas_cannot_all_be_resident(nx, ny, storage, captured):
    """A refused launch in rounds is made again as one launch per few steps, in the same run and with the same results, also
    where a captured run has fixed the parity of the buffers; rounds come back once they are launched."""
    with lattice(nx, ny, storage) as lat, lattice(nx, ny, storage, lb.KERNEL_PLAIN) as ref:
        lat.step(31)
        done = 31
        if captured:
            torch = pytest.importorskip("torch")
            stream = torch.cuda.Stream()
            lat.set_stream(stream)
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph, stream=stream):
                lat.step(2)
        for refused in (True, False):
            lat.test_refuse_rounds(refused)
            for n in (30, 31, 46):
                at = lat.device_populations()[0]
                lat.step(n)
                done += n
                shape, _, _, rounds = lat.test_last_tiles()
                assert shape in (1, 2) and rounds == (0 if refused else 1)
                if captured and n % 2 == 0:
                    assert lat.device_populations()[0] == at
                lat.sync()
        if captured:
            with torch.cuda.stream(stream):
                graph.replay()
            torch.cuda.synchronize()
            done += 2
            del graph
        ref.step(done)
        assert np.array_equal(lat.get_populations(np.float64), ref.get_populations(np.float64))


TIMEOUT = -8


@pytest.mark.parametrize("nx,ny,storage,tile", [(128, 128, lb.F32, 77), (180, 164, lb.F16S, 0), (301, 199, lb.F64, 3)])
def test_tiles_that_wait_in_vain_report_a_timeout(nx, ny, storage, tile):
    """A tile's neighbours and it give up after two seconds, then theirs; the next run is a clean one."""
    with lattice(nx, ny, storage) as lat, lattice(nx, ny, storage, lb.KERNEL_PLAIN) as ref:
        F = lat.get_populations(np.float64)
        lat.step(30)  # (chooses the family of the single steps)
        assert lb.lib().lbm_sync(lat._h) == 0
        lat.test_stall_tiles(tile)
        lat.step(30)
        assert lat.test_last_tiles()[3] == 1
        assert lb.lib().lbm_sync(lat._h) == TIMEOUT
        assert b"neighbours' records" in lb.lib().lbm_last_error()
        assert lb.lib().lbm_sync(lat._h) == 0  # reported once
        ref.step(60)  # (the random words go by the step's number)
        for other in (lat, ref):
            other.set_populations(F)
        for n in (30, 31, 5):
            lat.step(n)
            assert lb.lib().lbm_sync(lat._h) == 0
            ref.step(n)
            assert np.array_equal(lat.get_populations(np.float64), ref.get_populations(np.float64))


def test_the_stall_needs_tiles_that_exchange():
    with lb.Lattice(lb.make_desc(lb.D3Q27, lb.BGK, lb.F32, (32, 32, 32))) as lat:
        with pytest.raises(lb.LbmError):
            lat.test_stall_tiles(0)
    with lattice(128, 128, lb.F32) as lat:
        for tile in (-1, 100000):
            with pytest.raises(lb.LbmError):
                lat.test_stall_tiles(tile)
