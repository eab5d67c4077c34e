"""bench.py's bytes and launch counts of runs on tiles (host code): populations cross HBM once per launch of several steps,
and the figure stays a rate that the hardware can have."""
import sys

import pytest

from helpers import ROOT, lb

sys.path.insert(0, str(ROOT))
import bench  # noqa: E402

TILES = "void lbm::k_step_tiles<float, false, ...>(...)"
PLAIN = "void lbm::k_step_bgk<lbm::D2Q9, float, ...>(...)"
PSI = "void lbm::k_sc_psi<float>(...)"
SC = "void lbm::k_step_sc<float>(...)"


def test_tiled_run():
    d = lb.make_desc(lb.D2Q9, lb.BGK, lb.F32, (4096, 4096))
    counted = bench.launch_counts([TILES] * 12 + [PLAIN] * 2 + ["Memcpy DtoH"], 50)
    assert counted == {"launches": 14, "crossings": 14, "kernels": ["k_step_bgk", "k_step_tiles"]}
    assert bench.crossed_bytes(d, 50, counted) == 14 * 72 * 4096 ** 2
    r = bench.roofline_of(d, 50, 50 * 121e-6, counted, 6542.0)
    assert r["frac"] < 1 and r["bound"] != "hbm"


def test_single_steps():
    d = lb.make_desc(lb.D2Q9, lb.BGK, lb.F16S, (1000, 300))
    counted = bench.launch_counts([PLAIN] * 20, 20)
    assert bench.crossed_bytes(d, 20, counted) == 36 * 300000 * 20
    assert bench.roofline_of(d, 20, 1e-3, counted, 6542.0)["bound"] == "hbm"
    s = lb.make_desc(lb.D2Q9, lb.SHANCHEN, lb.F32, (256, 256))
    counted = bench.launch_counts([PSI, SC] * 20, 20)
    assert counted["launches"] == 40 and bench.crossed_bytes(s, 20, counted) == 80 * 65536 * 20
    t = lb.make_desc(lb.D3Q27, lb.MRT, lb.F16S, (256, 256, 256))
    assert bench.crossed_bytes(t, 20, None) == 108 * 256 ** 3 * 20


@pytest.mark.parametrize("steps", [1, 20])
def test_nothing_profiled(steps):
    counted = bench.launch_counts([], steps)
    assert counted["launches"] == counted["crossings"] == steps
