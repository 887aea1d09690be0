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
@pytest.mark.parametrize("layers", [1, 3, 6, 12])
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


def test_boards_of_small_and_large_prices_in_one_batch(eng, oracle):
    """A launch over both, replayed as a graph, with and without fields."""
    boards = [W.plain_board(seed=3, w=70, h=50, n_nets=6), W.plain_board(seed=4, w=90, h=40, n_nets=6)]
    reqs = []
    for wl, gap in zip(boards, (3, 70_000)):
        d = wl.grid.dims
        reqs.append(IsolatedRouteRequest(wl.grid, wl.nets, wl.windows, np.full(d.w - 1, gap, np.uint32),
                                         np.full(d.h - 1, gap + 1, np.uint32), [2 * gap]))
    held = [eng.board(r.grid, r.x_edge_costs, r.y_edge_costs, r.via_edge_costs) for r in reqs]
    want = [oracle.isolated_batch(r, retry_full=False, mode="field") for r in reqs]
    for keep in (False, True):
        bt = mrcuda.Batch(held, [n for r in reqs for n in r.nets], [w for r in reqs for w in r.windows], retry_full=False,
                          keep_fields=keep, net_board=[k for k, r in enumerate(reqs) for _ in r.nets])
        bt.capture_graph()
        for _ in range(3):
            bt.launch()
            got = bt.finish()
            assert got.paths == want[0][0] + want[1][0] and got.search_costs == want[0][1] + want[1][1]
        bt.close()
    for b in held:
        b.close()


@pytest.mark.parametrize("factor,weight", [(4000, 16), (1, 1 << 18)])
def test_negotiation_with_large_prices(eng, oracle, factor, weight):
    """Price overrides (a clearance) on a board of large prices, and large penalties on a
    board of small ones."""
    from test_gpu_negotiation import _run_both

    wl = W.snapshot_board(w=96, h=80, layers=3, n_nets=24, median=40)
    directed = np.where(wl.directed == COST_MAX, COST_MAX, wl.directed.astype(np.uint64) * factor).astype(np.uint32)
    req = IsolatedRouteRequest(wl.grid, wl.nets, wl.windows, wl.x, wl.y, [v * factor for v in wl.vias], directed)
    _run_both(eng, oracle, req, rounds=3, weight=weight, clearance=1)
    _run_both(eng, oracle, req, rounds=3, weight=weight)


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


@pytest.mark.parametrize("factor", [1000, 2500, 20000])
def test_relax_time_hardly_depends_on_the_prices(eng, factor):
    """Tiles whose labels don't fit 32-bit words take more work, on 64-bit ones, but no
    attempt on 32 bits each time."""
    small, _ = _times(eng, 1)
    large, _ = _times(eng, factor)
    assert large < 3.2 * small, (small, large)  # what a relax on 64-bit labels throughout took


def test_a_dear_corner_costs_the_rest_of_the_board_nothing(eng):
    """A few cells of a large price: the tiles without them stay on 32-bit words."""
    wl = W.plain_board(seed=1)
    cost = wl.grid.cost.copy()
    cost[:3] = 10**6
    times = []
    for c in (wl.grid.cost, cost):
        b = eng.board(Grid(wl.grid.dims, c, wl.grid.board_constraint, wl.grid.via_forbidden), wl.x, wl.y, wl.vias)
        bt = mrcuda.Batch(b, wl.nets, wl.windows, time_kernels=True)
        ms = []
        for _ in range(8):
            bt.launch()
            bt.finish()
            ms.append(bt.relax_ms())
        times.append(min(ms[2:]))
        bt.close()
        b.close()
    assert times[1] < 1.5 * times[0], times
