"""The layer kernel (32-bit tile labels, a warp per layer) against the oracle at
the sizes where it can go wrong: window widths and heights around its 32 x 8
tiles, window columns off its 4-column grid, every layer count class, and
prices and path costs on both sides of what a packed word holds."""
import numpy as np
import pytest

import mrcuda
from mrcuda.types import COST_MAX, Dims, Grid, IsolatedRouteRequest, IsolatedRouteWindow, NetEndpoints
from test_gpu_parity import _assert_fields

pytestmark = pytest.mark.gpu


def _board(rng, layers, price):
    dims = Dims(72, 21, layers)
    n = len(dims)
    cost = np.ones(n, np.uint32)
    cost[rng.random(n) < 0.15] = COST_MAX
    d = rng.integers(max(price // 2, 1), price + 1, (n, 4)).astype(np.uint32)
    d[rng.random((n, 4)) < 0.05] = COST_MAX
    grid = Grid(dims, cost)
    free = np.flatnonzero(cost != COST_MAX)
    nets, wins = [], []
    for x0 in range(5):  # every offset off the 4-column grid, and the next
        for ww, wh in ((31, 7), (32, 8), (33, 9), (64, 16), (65, 17), (1, 20), (67 - x0, 1)):
            x1, y0 = x0 + ww - 1, int(rng.integers(0, 21 - wh + 1))
            inside = [int(c) for c in free if x0 <= c % 72 <= x1 and y0 <= (c // 72) % 21 < y0 + wh]
            if not inside:
                continue
            src, dst = (int(v) for v in rng.choice(inside, 2))
            nets.append(NetEndpoints(f"n{len(nets)}", src, dst))
            wins.append(IsolatedRouteWindow(x0, y0, x1, y0 + wh - 1))
    return IsolatedRouteRequest(grid, nets, wins, np.ones(71, np.uint32), np.ones(20, np.uint32),
                                [int(v) for v in rng.integers(1, 2 * price + 1, layers - 1)], d)


@pytest.mark.parametrize("layers", [1, 2, 4, 5, 8, 9, 16])
@pytest.mark.parametrize("price", [1, 30, (1 << 16) - 1, 1 << 16, (1 << 17) - 1, 1 << 17, 1 << 25])
def test_tile_edges_and_word_limits(oracle, layers, price):
    req = _board(np.random.default_rng(1000 * layers + price % 997), layers, price)
    engine = mrcuda.Engine(0)
    try:
        exp = oracle.isolated_batch(req, retry_full=False, mode="field")
        got = engine.route_isolated_batch(req, retry_full=False, keep_fields=True)
        assert (got.paths, got.search_costs) == exp
        _assert_fields(oracle, req, got)
        paths_only = engine.route_isolated_batch(req, retry_full=False)
        assert (paths_only.paths, paths_only.search_costs) == exp
    finally:
        engine.close()


@pytest.mark.parametrize("layers", [1, 2, 3, 4])
@pytest.mark.parametrize("price", [1, 40, (1 << 14) - 1, (1 << 16) + 1, 1 << 25])
def test_axis_gaps_tie(oracle, layers, price):
    """Boards priced by axis gaps, where many paths cost the same and the canonical
    one hangs on every tie, up to prices of which a word holds only a few steps:
    windows around 32 x 16 tiles, with and without own pads."""
    rng = np.random.default_rng(77 * layers + price % 991)
    w, h = 72, 37
    dims = Dims(w, h, layers)
    cost = np.ones(len(dims), np.uint32)
    cost[rng.random(len(dims)) < 0.12] = COST_MAX
    cost[rng.random(len(dims)) < 0.2] = 3
    gx = rng.integers(max(price // 2, 1), price + 1, w - 1).astype(np.uint32)
    gy = rng.integers(max(price // 2, 1), price + 1, h - 1).astype(np.uint32)
    free = np.flatnonzero(cost != COST_MAX)
    cells = np.arange(len(dims))
    nets, wins = [], []
    for x0 in range(4):
        for ww, wh in ((31, 15), (32, 16), (33, 17), (64, 32), (65, 33), (1, 36), (68, 1), (40, 23), (34, 24)):
            y0 = int(rng.integers(0, h - wh + 1))
            box = (cells % w >= x0) & (cells % w < x0 + ww) & (cells // w % h >= y0) & (cells // w % h < y0 + wh)
            inside = free[box[free]]
            if len(inside) < 2:
                continue
            src, dst = (int(v) for v in rng.choice(inside, 2))
            walls = np.flatnonzero(box & (cost == COST_MAX))
            pads = sorted({src, dst, *(int(c) for c in walls[rng.random(len(walls)) < 0.3])})
            nets.append(NetEndpoints(f"n{len(nets)}", src, dst, pads if len(nets) % 2 else []))
            wins.append(IsolatedRouteWindow(x0, y0, x0 + ww - 1, y0 + wh - 1))
    vias = [int(v) for v in rng.integers(1, 2 * price + 1, layers - 1)]
    req = IsolatedRouteRequest(Grid(dims, cost), nets, wins, gx, gy, vias)
    engine = mrcuda.Engine(0)
    try:
        exp = oracle.isolated_batch(req, retry_full=False, mode="field")
        got = engine.route_isolated_batch(req, retry_full=False, keep_fields=True)
        assert (got.paths, got.search_costs) == exp
        _assert_fields(oracle, req, got)
        paths_only = engine.route_isolated_batch(req, retry_full=False)
        assert (paths_only.paths, paths_only.search_costs) == exp
    finally:
        engine.close()


@pytest.mark.parametrize("layers,w,h", [(1, 200, 40), (2, 40, 32), (4, 64, 32), (8, 64, 16)])
@pytest.mark.parametrize("price", [1, 3, (1 << 19) - 1, 1 << 19])
def test_long_ways_inside_a_tile(oracle, layers, w, h, price):
    """More hops inside a tile and its border than a word holds: a serpentine on
    every layer, joined by single vias into one way, and equal costs beside it."""
    cost = np.ones((layers, h, w), np.uint32)
    cost[:, 1::2, :] = COST_MAX
    for k, y in enumerate(range(1, h, 2)):
        cost[:, y, w - 1 if k % 2 == 0 else 0] = 1
    rng = np.random.default_rng(layers + w)
    holes = rng.random(cost.shape) < 0.01
    cost[holes & (cost == COST_MAX)] = 2
    dims = Dims(w, h, layers)
    last = (h - 2) * w if (h // 2) % 2 == 0 else (h - 2) * w + w - 1
    forbidden = np.ones((layers, h * w), np.uint8)
    for l in range(layers - 1):
        forbidden[l:l + 2, 0 if l % 2 else last] = 0
    full = IsolatedRouteWindow.full(dims)
    far = (layers - 1) * w * h
    nets = [NetEndpoints("a", 0, far + last), NetEndpoints("b", far, 4), NetEndpoints("c", 2 * w + 1, far + 2 * w + 1)]
    req = IsolatedRouteRequest(Grid(dims, cost.reshape(-1), None, forbidden.reshape(-1)), nets, [full] * 3,
                               np.full(w - 1, price, np.uint32), np.full(h - 1, price, np.uint32), [price] * (layers - 1))
    engine = mrcuda.Engine(0)
    try:
        exp = oracle.isolated_batch(req, retry_full=False, mode="field")
        got = engine.route_isolated_batch(req, retry_full=False, keep_fields=True)
        assert (got.paths, got.search_costs) == exp
        _assert_fields(oracle, req, got)
        paths_only = engine.route_isolated_batch(req, retry_full=False)
        assert (paths_only.paths, paths_only.search_costs) == exp
    finally:
        engine.close()


def test_a_field_that_leaves_the_packed_range(oracle):
    """Long hop counts and costs: a serpentine whose labels spread past one word
    inside a tile (walls every other row, a gap at alternating ends)."""
    w, h, layers = 64, 40, 2
    cost = np.ones((layers, h, w), np.uint32)
    cost[:, 1::2, :] = COST_MAX
    for k, y in enumerate(range(1, h, 2)):
        cost[:, y, w - 1 if k % 2 == 0 else 0] = 1
    grid = Grid(Dims(w, h, layers), cost.reshape(-1))
    full = IsolatedRouteWindow.full(grid.dims)
    nets = [NetEndpoints("a", 0, w * h - w), NetEndpoints("b", w * h - w, 5)]
    engine = mrcuda.Engine(0)
    try:
        for step in (1, 900, 60000):
            req = IsolatedRouteRequest(grid, nets, [full, full], np.full(w - 1, step, np.uint32),
                                       np.full(h - 1, step, np.uint32), [7])
            exp = oracle.isolated_batch(req, retry_full=False, mode="field")
            got = engine.route_isolated_batch(req, retry_full=False, keep_fields=True)
            assert (got.paths, got.search_costs) == exp, step
            _assert_fields(oracle, req, got)
    finally:
        engine.close()


@pytest.mark.parametrize("nets,copies", [(1, 1), (9, 3), (9, 16)])
@pytest.mark.parametrize("layers", [1, 4, 5])
def test_tile_height_rule(oracle, layers, nets, copies):
    """Both tile heights on the same nets: the batch alone, and so often repeated
    that it has more tiles than the taller ones are taken for; five layers and
    prices per cell always run on the lower ones."""
    rng = np.random.default_rng(31 * layers)
    dims = Dims(640, 400, layers)
    cost = np.ones(len(dims), np.uint32)
    cost[rng.random(len(dims)) < 0.1] = COST_MAX
    free = np.flatnonzero(cost != COST_MAX)
    ends = [(int(a), int(b)) for a, b in rng.choice(free, (nets, 2))]
    full = IsolatedRouteWindow.full(dims)
    base = [NetEndpoints(f"n{k}", a, b) for k, (a, b) in enumerate(ends)]
    grid, gx, gy = Grid(dims, cost), np.full(639, 2, np.uint32), rng.integers(1, 9, 399).astype(np.uint32)
    vias = [5] * (layers - 1)
    engine = mrcuda.Engine(0)
    try:
        paths, costs = oracle.isolated_batch(IsolatedRouteRequest(grid, base, [full] * nets, gx, gy, vias),
                                             retry_full=False, mode="field")
        req = IsolatedRouteRequest(grid, base * copies, [full] * (nets * copies), gx, gy, vias)
        got = engine.route_isolated_batch(req, retry_full=False)
        assert (got.paths, got.search_costs) == (list(paths) * copies, list(costs) * copies)
    finally:
        engine.close()
