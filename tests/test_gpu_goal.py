"""The goal-directed relax kernel (path-only batches of many tiles) against the
oracle: the searches it cuts short give the same canonical paths and costs."""
import numpy as np
import pytest

import mrcuda
from mrcuda import workloads as W
from mrcuda.types import IsolatedRouteRequest
from test_gpu_parity import _random_case

pytestmark = pytest.mark.gpu


def _tiles(req):
    return sum(((w.x1 - w.x0 + 32) // 32) * ((w.y1 - w.y0 + 8) // 8) for w in req.windows)


@pytest.mark.parametrize("directed", [False, True], ids=["axis", "directed"])
@pytest.mark.parametrize("zero", [False, True], ids=["positive", "zeros"])
def test_goal_directed_batches_equal_the_oracle(oracle, directed, zero):
    """Adversarial boards (saturating and MAX - 1 prices, own pads entered below
    the cheapest cell, masks, unreachable targets, ragged windows), with prices
    that bound the rest of a path and with zeros that do not; the nets are
    repeated until the launch has enough tiles to run goal-directed."""
    rng = np.random.default_rng(71 + 2 * directed + zero)
    reqs = []
    for trial in range(40):
        req = _random_case(rng, trial, directed, max_side=90, max_layers=9 if trial % 8 == 0 else 4)
        if req is None:
            continue
        if not zero:  # every step has a price: 3 x the cheapest cell, gaps of at least 5
            g = req.grid
            cheap = g.cost < 100
            g.cost[cheap] = 3 * (g.cost[cheap] + 1)
            req.x_edge_costs = np.maximum(req.x_edge_costs, 5).astype(np.uint32)
            req.y_edge_costs = np.maximum(req.y_edge_costs, 5).astype(np.uint32)
            if directed:
                req.directed_in_costs = np.maximum(req.directed_in_costs, 5).astype(np.uint32)
        reqs.append(req)
    per = sum(_tiles(r) for r in reqs)
    times = -(-12000 // per)
    many = [IsolatedRouteRequest(r.grid, list(r.nets) * times, list(r.windows) * times, r.x_edge_costs,
                                 r.y_edge_costs, r.via_edge_costs, r.directed_in_costs) for r in reqs]
    engine = mrcuda.Engine(0)
    try:
        for retry in (False, True):
            got = engine.route_instances(many, retry_full=retry)
            for k, (r, out) in enumerate(zip(reqs, got)):
                paths, costs = oracle.isolated_batch(r, retry_full=retry, mode="field")
                assert out.paths == paths * times, (k, retry)
                assert out.search_costs == costs * times, (k, retry)
    finally:
        engine.close()


@pytest.mark.parametrize("seed", [2, 7])
def test_congestion_board_paths_only(oracle, seed):
    """Prices whose bound is loose (a path costs 1.4 x it), so that improvements
    wait for the target and are released in several steps."""
    req = W.congestion_board(seed=seed).request()
    exp = oracle.isolated_batch(req, mode="astar")
    engine = mrcuda.Engine(0)
    try:
        for _ in range(3):
            got = engine.route_isolated_batch(req)
            assert (got.paths, got.search_costs) == exp
    finally:
        engine.close()
