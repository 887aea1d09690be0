"""Large prices: any price the interface takes gives the oracle's paths and fields, and the
time of a search does not hang on how large its prices are."""
import numpy as np
import pytest

import mrcuda
from mrcuda import workloads as W
from mrcuda.types import COST_MAX, Dims, Grid, IsolatedRouteRequest, IsolatedRouteWindow, NetEndpoints

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def eng():
    e = mrcuda.Engine(0)
    yield e
    e.close()


def _check(eng, oracle, grid, x, y, vias, nets, wins, directed=None):
    req = IsolatedRouteRequest(grid, nets, wins, np.asarray(x, np.uint32), np.asarray(y, np.uint32), vias, directed)
    want, costs = oracle.isolated_batch(req, retry_full=False, mode="field")
    for keep in (False, True):
        got = eng.route_isolated_batch(req, keep_fields=keep, retry_full=False)
        assert got.search_costs == costs
        assert got.paths == want
    for i, net in enumerate(nets):
        dist, _ = oracle.isolated_field(grid, req.x_edge_costs, req.y_edge_costs, vias, net, wins[i], directed)
        assert np.array_equal(got.fields[i], dist), i


# both sides of what packed price words hold, of what plain ones hold, and of the largest
@pytest.mark.parametrize("price", [2**19 - 1, 2**19, 2**24 + 1, 2**29 - 1, 2**29, 2**31 - 2, 2**31 - 1, 2**31, 2**32 - 2])
@pytest.mark.parametrize("layers", [1, 3, 6])
def test_price_limits(eng, oracle, price, layers):
    """Uniform gaps (ties everywhere), one dear line, and dear cells on a cheap board."""
    rng = np.random.default_rng(price % 1000 + layers)
    dims = Dims(43, 37, layers)
    n = len(dims)
    full = IsolatedRouteWindow(0, 0, 42, 36)
    for form in ("all", "line", "cells"):
        cost = np.ones(n, np.uint32)
        cost[rng.random(n) < 0.15] = COST_MAX
        x, y, vias = [2] * 42, [2] * 36, [3] * (layers - 1)
        if form == "all":
            x, y, vias = [price] * 42, [price] * 36, [price] * (layers - 1)
        elif form == "line":
            x[20], y[18] = price, price
        else:
            cost[(rng.random(n) < 0.3) & (cost == 1)] = price
        free = np.flatnonzero(cost != COST_MAX)
        nets = []
        for k in range(6):
            s, t = (int(v) for v in rng.choice(free, 2))
            if form == "all" and k < 4:  # within what such prices can pay for
                sx, sy = dims.xy(s)
                near = [c for c in free if abs(dims.xy(int(c))[0] - sx) + abs(dims.xy(int(c))[1] - sy) <= 1 + 2 * k]
                t = int(rng.choice(near))
            nets.append(NetEndpoints(f"n{k}", s, t))
        _check(eng, oracle, Grid(dims, cost), x, y, vias, nets, [full] * len(nets))


@pytest.mark.parametrize("price", [2**19, 2**25, 2**31 - 1])
def test_directed_price_limits(eng, oracle, price):
    rng = np.random.default_rng(price % 1000)
    dims = Dims(70, 41, 2)
    n = len(dims)
    cost = np.ones(n, np.uint32)
    cost[rng.random(n) < 0.1] = COST_MAX
    d = np.where(rng.random((n, 4)) < 0.2, price, rng.integers(1, 50, (n, 4))).astype(np.uint32)
    d[rng.random((n, 4)) < 0.05] = COST_MAX
    free = np.flatnonzero(cost != COST_MAX)
    nets = [NetEndpoints(f"n{k}", *(int(v) for v in rng.choice(free, 2))) for k in range(8)]
    _check(eng, oracle, Grid(dims, cost), [1] * 69, [1] * 40, [40], nets, [IsolatedRouteWindow(0, 0, 69, 40)] * 8,
           d.reshape(-1))


def _times(eng, factor):
    """Least device times (relax, walk) in ms of a board with its prices times `factor`."""
    import torch

    wl = W.congestion_board(seed=5, n_nets=128)
    up = lambda a: (np.asarray(a, np.uint64) * factor).astype(np.uint32)
    directed = np.where(wl.directed == COST_MAX, COST_MAX, wl.directed.astype(np.uint64) * factor).astype(np.uint32)
    b = eng.board(wl.grid, up(wl.x), up(wl.y), [v * factor for v in wl.vias], directed)
    bt = mrcuda.Batch(b, wl.nets, wl.windows, retry_full=False, time_kernels=True)
    st = torch.cuda.Stream()
    relax, walk = [], []
    for _ in range(8):
        e0, e1 = (torch.cuda.Event(enable_timing=True) for _ in range(2))
        e0.record(st)
        bt.launch(st.cuda_stream)
        e1.record(st)
        bt.finish()
        relax.append(bt.relax_ms())
        walk.append(e0.elapsed_time(e1) - relax[-1])
    bt.close()
    b.close()
    return min(relax[2:]), min(walk[2:])


@pytest.mark.parametrize("factor", [1000, 2500, 20000])
def test_walk_time_does_not_depend_on_the_prices(eng, factor):
    """The same search in larger units: labels of a window spread over more than 2^19, then
    single prices above it."""
    _, small = _times(eng, 1)
    _, large = _times(eng, factor)
    assert large < 2 * small, (small, large)
