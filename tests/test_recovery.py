"""After a wait gave up: lbm_sync and lbm_batch_sync report it once and clear what it left in the order of the stream
that steps run on, so that a run issued right behind them finds everything cleared and keeps its own error.  No test
here makes the GPU fault: the waits have short limits and the launches return."""
import re

import numpy as np
import pytest

from helpers import ROOT, cavity3d, lb

TIMEOUT = -8


def test_clears_are_ordered_with_the_steps():
    """cudaMemset takes the legacy default stream, which a lattice's (non-blocking) stream does not wait for, and returns
    before it is done: it may not clear what a step of an existing lattice or ensemble reads or writes."""
    text = (ROOT / "lbm-arrayfire_b200" / "csrc" / "runtime.cu").read_text()
    assert not re.findall(r"\bcudaMemset\(", text)
    text = (ROOT / "lbm-arrayfire_b200" / "csrc" / "batch.cu").read_text()
    body = text[text.index("int lbm_batch_sync("):]
    body = body[:body.index("\n}")]
    assert "cudaMemsetAsync(b->err" in body and not re.findall(r"\bcudaMemset\(", body)


def test_movers_that_give_up_wait_for_their_copies():
    """Bulk copies under way land in shared memory: the warps that issued them may not leave the CTA before, also when a
    wait gave up."""
    text = (ROOT / "lbm-arrayfire_b200" / "csrc" / "tiles.cuh").read_text()
    gives_up = text[text.index("if (vote(2, MT, !ok)) {"):]
    gives_up = gives_up[:gives_up.index("break;")]
    assert gives_up.count("mbar_wait_bounded(&full[") == 2  # the tile at hand and the next one


@pytest.mark.gpu
def test_every_stalled_run_reports_its_own_timeout():
    d, m, F0 = cavity3d(n=(64, 48, 40), u_lid=0.1, omega=1.3)
    with lb.Lattice(d, m) as lat:
        lat.set_kernel(lb.KERNEL_ROWS)
        lat.set_populations(F0)
        lat.step(1)
        assert lb.lib().lbm_sync(lat._h) == 0
        for _ in range(20):  # the next run is issued right behind the clear
            lat.test_stall_next_step(item=0, wait_clocks=1 << 14)
            lat.step(1)
            assert lb.lib().lbm_sync(lat._h) == TIMEOUT
        lat.set_populations(F0)
        lat.step(5)
        assert lb.lib().lbm_sync(lat._h) == 0
        a = lat.get_populations(np.float64)
    with lb.Lattice(d, m) as lat:
        lat.set_kernel(lb.KERNEL_PLAIN)
        lat.set_populations(F0)
        lat.step(5)
        assert np.array_equal(a, lat.get_populations(np.float64))
