"""The guard on the number of tile activations ends a launch whose queue is full: its
workers leave it, instead of only marking it as failed.  The launches here are
ordinary ones that a low limit cuts short."""
import pytest

import mrcuda
from mrcuda import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("schedule,fields", [(1, False), (1, True), (2, False), (3, False)])
def test_activation_limit_ends_the_launch(schedule, fields):
    eng = mrcuda.Engine(0)
    wl = W.congestion_board(seed=5, n_nets=256)
    b = eng.board(wl.grid, wl.x, wl.y, wl.vias, wl.directed)
    bt = mrcuda.Batch(b, list(wl.nets) * 6, list(wl.windows) * 6, retry_full=False, keep_fields=fields)
    bt.set_schedule(schedule)
    bt.launch()
    want = bt.finish()
    whole = bt.stats()["activations"]
    bt.set_activation_limit(1)
    bt.launch()
    with pytest.raises(mrcuda.IterationLimit):
        bt.finish()
    # a worker leaves after 64 activations at most (the device holds 1184 CTAs of 128
    # threads, or as many warps of the warp schedule as CTAs x 4, each 32 activations)
    assert bt.stats()["activations"] < whole // 2, (bt.stats(), whole)
    bt.set_activation_limit(0)
    bt.launch()
    got = bt.finish()
    assert (got.costs == want.costs).all() and (got.cells == want.cells).all()
    bt.close()
    b.close()
    eng.close()
