"""Boards of more than 16 layers on the default schedule: the oracle's paths and fields, and
no cliff in time behind 16 layers."""
import numpy as np
import pytest

import mrcuda
from mrcuda import workloads as W
from mrcuda.types import COST_MAX, Dims, Grid, IsolatedRouteRequest, NetEndpoints
from test_gpu_parity import _assert_fields

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def eng():
    e = mrcuda.Engine(0)
    yield e
    e.close()


@pytest.mark.parametrize("layers", [17, 20, 23, 24])
@pytest.mark.parametrize("price", [3, 60_000])
def test_many_layers_match_the_oracle(eng, oracle, layers, price):
    rng = np.random.default_rng(layers + price)
    dims = Dims(37, 19, layers)
    n = len(dims)
    cost = np.ones(n, np.uint32)
    cost[rng.random(n) < 0.2] = COST_MAX
    free = np.flatnonzero(cost != COST_MAX)
    flags = (rng.random(n) < 0.05).astype(np.uint8)
    for directed in (None, rng.integers(1, price + 1, 4 * n).astype(np.uint32)):
        nets = []
        for k in range(8):
            s, t = (int(v) for v in rng.choice(free, 2))
            pads = sorted({int(c) for c in rng.choice(n, 5)} | {s}) if k % 2 else []
            nets.append(NetEndpoints(f"n{k}", s, t, pads, pads[:2]))
        req = IsolatedRouteRequest(Grid(dims, cost, None, flags), nets, mrcuda.net_windows(dims, nets),
                                   rng.integers(1, price + 1, 36).astype(np.uint32),
                                   rng.integers(1, price + 1, 18).astype(np.uint32),
                                   [int(v) for v in rng.integers(1, 2 * price, layers - 1)], directed)
        want = oracle.isolated_batch(req, mode="field")
        for keep in (False, True):
            got = eng.route_isolated_batch(req, keep_fields=keep)
            assert (got.paths, got.search_costs) == want
        _assert_fields(oracle, req, got)


def test_time_behind_16_layers(eng):
    times = []
    for layers in (16, 20):
        wl = W.congestion_board(seed=5, w=160, h=160, layers=layers, n_nets=64)
        b = eng.board(wl.grid, wl.x, wl.y, wl.vias, wl.directed)
        bt = mrcuda.Batch(b, wl.nets, wl.windows, retry_full=False, time_kernels=True)
        ms = []
        for _ in range(6):
            bt.launch()
            bt.finish()
            ms.append(bt.relax_ms())
        times.append(min(ms[2:]))
        bt.close()
        b.close()
    assert times[1] < 3 * times[0], times
