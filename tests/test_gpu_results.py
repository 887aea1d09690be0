"""Result memory: fields and distance fields live in blocks that are lent to
their arrays and reused after them, never before."""
import gc

import numpy as np
import pytest

import mrcuda
from mrcuda import api
from mrcuda import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("limit", [256 << 20, 0], ids=["page-locked", "ordinary"])
def test_held_results_are_not_overwritten_and_outlive_the_engine(oracle, monkeypatch, limit):
    monkeypatch.setattr(api._ResultBlock, "LIMIT", limit)
    boards = [W.plain_board(seed=s, w=70 + s, h=33, n_nets=5) for s in (1, 2, 3)]
    engine = mrcuda.Engine(0)
    held = []
    for turn in range(2):
        for wl in boards:
            r = engine.route_isolated_batch(wl.request(), keep_fields=True)
            d = engine.distance_fields(wl.grid, [n.src for n in wl.nets] + [len(wl.grid.dims)])
            held.append((wl, r, d))
            tmp = engine.route_isolated_batch(wl.request(), keep_fields=True)  # freed at once
            del tmp
    engine.close()
    gc.collect()
    for wl, r, d in held:
        for i, n in enumerate(wl.nets):
            dist, _ = oracle.isolated_field(wl.grid, wl.x, wl.y, wl.vias, n, wl.windows[i])
            np.testing.assert_array_equal(r.fields[i], dist)
            np.testing.assert_array_equal(d[i], oracle.bfs_distance_field(wl.grid, n.src))
        assert (d[-1] == mrcuda.COST_MAX).all()


def test_paths_longer_than_the_first_download(oracle):
    """More path cells than a batch's first download holds (256 a net)."""
    w, h = 64, 41
    cost = np.ones((h, w), np.uint32)
    cost[1::2, :] = mrcuda.OBSTACLE
    for k, y in enumerate(range(1, h, 2)):
        cost[y, w - 1 if k % 2 == 0 else 0] = 1
    grid = mrcuda.Grid(mrcuda.Dims(w, h), cost.reshape(-1))
    engine = mrcuda.Engine(0)
    try:
        got = engine.route_lee(grid, [mrcuda.NetEndpoints("a", 0, w * h - 1), mrcuda.NetEndpoints("b", w * h - 1, 3)])
        exp = [oracle.lee_route_one(grid, n) for n in (mrcuda.NetEndpoints("a", 0, w * h - 1),
                                                       mrcuda.NetEndpoints("b", w * h - 1, 3))]
        assert [(r.path, r.cost) for r in got.results] == exp and len(exp[0][0]) > 512
    finally:
        engine.close()
