"""A tile height asked for leaves the default schedule as fast as it is: its kernel has
tiles of its own."""
import pytest

import mrcuda
from mrcuda import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fields", [False, True])
def test_default_schedule_keeps_its_tiles(fields):
    eng = mrcuda.Engine(0)
    wl = W.plain_board(seed=1)
    b = eng.board(wl.grid, wl.x, wl.y, wl.vias)
    bt = mrcuda.Batch(b, wl.nets, wl.windows, time_kernels=True, keep_fields=fields)

    def solve():
        ms = []
        for _ in range(8):
            bt.launch()
            got = bt.finish()
            ms.append(bt.relax_ms())
        return min(ms[2:]), got

    least, want = solve()
    for tile_h in (8, 16, 32, 64):
        for threads in (128, 256):
            bt.set_config(tile_h, threads)
            assert bt.config() == {"tile_h": tile_h, "threads": threads, "schedule": 1}
            ms, got = solve()
            assert got.paths == want.paths and got.search_costs == want.search_costs
            assert ms < 1.3 * least, (tile_h, threads, ms, least)
    bt.close()
    b.close()
    eng.close()
