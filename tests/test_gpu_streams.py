"""Lattices on several streams: small ones with runs under way beside one another take forms that share the GPU (single
steps or one cluster each, as the tiles of one lattice take every SM), with the same results; alone they take tiles."""
import threading

import numpy as np
import pytest

from helpers import lb

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def start(k, nx, ny):
    _, _, _, w, _ = lb.velocities(lb.D2Q9)
    rng = np.random.default_rng(1000 * k + nx)
    return (np.repeat(w, nx * ny) * (1 + 0.02 * rng.standard_normal(9 * nx * ny))).astype(np.float32)


def lattice(k, nx, ny, storage=lb.F32, collision=lb.BGK):
    d = lb.make_desc(lb.D2Q9, collision, storage, (nx, ny), omega=1.25, sc_G=-5.0)
    lat = lb.Lattice(d, lb.setup_cavity2d(d, 0.1) if collision == lb.BGK else None)
    lat.set_populations(start(k, nx, ny))
    return lat


def plain(k, nx, ny, steps, storage=lb.F32, collision=lb.BGK):
    with lattice(k, nx, ny, storage, collision) as lat:
        lat.set_kernel(lb.KERNEL_PLAIN)
        lat.step(steps)
        return lat.get_populations(np.float64)


def shape(lat):
    return lat.test_last_tiles()[0]


@pytest.mark.parametrize("wait", [False, True])
@pytest.mark.parametrize("nx,ny,storage,collision,count,n", [
    (64, 64, lb.F32, lb.BGK, 2, 37),          # in a cluster each
    (128, 128, lb.F16S, lb.BGK, 3, 37),
    (130, 101, lb.F64, lb.BGK, 2, 37),
    (192, 180, lb.F32, lb.BGK, 4, 37),
    (192, 192, lb.F16S, lb.BGK, 4, 37),
    (260, 190, lb.F32, lb.BGK, 3, 800),       # single steps
    (128, 96, lb.BF16S, lb.SHANCHEN, 6, 800),
])
def test_small_lattices_share_the_gpu(nx, ny, storage, collision, count, n, wait):
    lats = [lattice(k, nx, ny, storage, collision) for k in range(count)]
    try:
        for turn in range(3):
            for lat in lats:
                lat.step(n)
            shapes = [shape(lat) for lat in lats]
            if wait:
                for lat in lats:
                    lat.sync()
            if turn:
                assert shapes == [0] * count
        for k, lat in enumerate(lats):
            assert np.array_equal(lat.get_populations(np.float64), plain(k, nx, ny, 3 * n, storage, collision))
        # alone again, from the second run on (each has been waited for)
        for _ in range(2):
            lats[0].step(n)
            lats[0].sync()
        assert shape(lats[0]) != 0
        assert np.array_equal(lats[0].get_populations(np.float64), plain(0, nx, ny, 5 * n, storage, collision))
    finally:
        for lat in lats:
            lat.close()


def test_short_runs_keep_their_tiles():
    """Single steps of a short run are launched one by one, which costs more than tiles that wait for one another."""
    lats = [lattice(k, 260, 190) for k in range(4)]
    for _ in range(3):
        for lat in lats:
            lat.step(10)
    assert all(shape(lat) != 0 for lat in lats)
    assert np.array_equal(lats[1].get_populations(np.float64), plain(1, 260, 190, 30))
    for lat in lats:
        lat.close()


def test_large_lattices_keep_their_tiles():
    lats = [lattice(k, 1200, 1000) for k in range(4)]
    for _ in range(2):
        for lat in lats:
            lat.step(9)
    assert all(shape(lat) != 0 for lat in lats)
    assert np.array_equal(lats[3].get_populations(np.float64), plain(3, 1200, 1000, 18))
    for lat in lats:
        lat.close()


def test_lattices_of_one_stream_keep_their_tiles():
    stream = torch.cuda.Stream()
    lats = [lattice(k, 128, 128) for k in range(4)]
    for lat in lats:
        lat.set_stream(stream)
    for _ in range(2):
        for lat in lats:
            lat.step(20)
    assert all(shape(lat) != 0 for lat in lats)
    assert np.array_equal(lats[2].get_populations(np.float64), plain(2, 128, 128, 40))
    for lat in lats:
        lat.close()


def test_a_lattice_waited_for_by_other_means_holds_no_other_back():
    with lattice(0, 64, 64) as a, lattice(1, 64, 64) as b:
        a.step(30)
        torch.cuda.synchronize()  # (the engine does not learn of it)
        for _ in range(3):
            b.step(30)
            b.sync()
        assert shape(b) != 0


def test_lattices_on_threads_of_their_own():
    out, errors = {}, []

    def work(k, nx, ny):
        try:
            with lattice(k, nx, ny) as lat:
                for _ in range(30):
                    lat.step(11)
                    lat.macros(np.float32)
                out[k] = lat.get_populations(np.float64)
        except Exception as e:  # noqa: BLE001
            errors.append(e)

    sizes = [(128, 128), (64, 64), (260, 190), (128, 128), (96, 70), (300, 200)]
    threads = [threading.Thread(target=work, args=(k, *s)) for k, s in enumerate(sizes)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors
    for k, s in enumerate(sizes):
        assert np.array_equal(out[k], plain(k, *s, 330))


def test_hundreds_of_lattices_under_way():
    """The last 32 runs are looked at: a step call costs the host the same beside hundreds of lattices as beside a few."""
    lats = [lattice(k, 64, 48) for k in range(200)]
    for _ in range(2):
        for lat in lats:
            lat.step(7)
    assert shape(lats[0]) == shape(lats[-1]) == 0
    for k in (0, 99, 199):
        assert np.array_equal(lats[k].get_populations(np.float64), plain(k, 64, 48, 14))
    for lat in lats:
        lat.close()
