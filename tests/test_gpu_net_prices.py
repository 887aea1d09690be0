"""Cells priced for the net itself (own pads, via pads), more of them in one tile and one
window of the path walk than their lists hold, and goal-directed batches of each layer
class alone (a launch takes the kernel of its largest board)."""
import numpy as np
import pytest

import mrcuda
from mrcuda.types import COST_MAX, Dims, Grid, IsolatedRouteRequest, NetEndpoints
from test_gpu_parity import _assert_fields, _random_case

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def eng():
    e = mrcuda.Engine(0)
    yield e
    e.close()


def _check(eng, oracle, req):
    want = oracle.isolated_batch(req, retry_full=False, mode="field")
    for keep in (False, True):
        got = eng.route_isolated_batch(req, retry_full=False, keep_fields=keep)
        assert (got.paths, got.search_costs) == want
    _assert_fields(oracle, req, got)
    assert all(p is not None for p in want[0])


# own pads in a block of w x h x layers: past 512 a tile, past 256 a walk window (each via pad counts thrice there)
@pytest.mark.parametrize("layers,block", [(1, (32, 16)), (2, (32, 8)), (2, (20, 16)), (4, (32, 8)), (4, (40, 20)), (7, (16, 8)),
                                          (16, (12, 8)), (20, (9, 9))])
@pytest.mark.parametrize("directed", [False, True])
@pytest.mark.parametrize("gap", [9, 40_000])
def test_large_pads(eng, oracle, layers, block, directed, gap):
    """Large pads of obstacle cells on every layer, which only their own net may enter and
    leave by their vias; the paths run through them, the other nets around."""
    rng = np.random.default_rng(layers * 100 + block[0] + directed)
    dims = Dims(90, 45, layers)
    n = len(dims)
    cost = rng.integers(1, 4, n).astype(np.uint32)
    flags = np.zeros(n, np.uint8)
    nets, bw, bh = [], *block
    for k, (x0, y0) in enumerate(((3, 2), (45, 21))):
        pad = [dims.idx3(x, y, l) for l in range(layers) for y in range(y0, y0 + bh) for x in range(x0, x0 + bw)]
        cost[pad] = COST_MAX
        flags[pad] = 1  # static via mask: open to the pad's own net alone
        src = dims.idx3(x0 + bw // 2, y0 + bh // 2, layers // 2)
        dst = dims.idx3(85 if k == 0 else 1, 22, 0)
        nets.append(NetEndpoints(f"pad{k}", src, dst, sorted(pad), sorted(pad[::2])))
        nets.append(NetEndpoints(f"through{k}", dims.idx3(0, y0, 0), dims.idx3(89, y0 + bh - 1, 0), sorted(pad), sorted(pad[1::3])))
    free = [int(c) for c in rng.choice(np.flatnonzero(cost != COST_MAX), 4)]
    nets += [NetEndpoints("around0", free[0], free[1]), NetEndpoints("around1", free[2], free[3])]
    cost[[nt.dst for nt in nets if cost[nt.dst] == COST_MAX and nt.dst not in nt.passable_pads]] = 1
    for nt in nets:
        for c in (nt.src, nt.dst):
            if cost[c] == COST_MAX and c not in nt.passable_pads:
                cost[c] = 1
    d = rng.integers(1, gap + 1, 4 * n).astype(np.uint32) if directed else None
    _check(eng, oracle, IsolatedRouteRequest(Grid(dims, cost, None, flags), nets, mrcuda.net_windows(dims, nets),
                                             rng.integers(1, gap + 1, 89).astype(np.uint32),
                                             rng.integers(1, gap + 1, 44).astype(np.uint32), [2 * gap] * (layers - 1), d))


@pytest.mark.parametrize("directed", [False, True])
@pytest.mark.parametrize("classes", [(1, 4), (5, 8), (9, 12), (17, 18)])
def test_layer_classes_alone(eng, oracle, classes, directed):
    """Adversarial boards of one layer class to a launch, without and with fields."""
    rng = np.random.default_rng(classes[0] + directed)
    reqs = [r for r in (_random_case(rng, t, directed, max_side=80 if classes[1] <= 8 else 50, max_layers=classes[1],
                                     min_layers=classes[0]) for t in range(12)) if r is not None]
    want = [oracle.isolated_batch(r, retry_full=False, mode="field") for r in reqs]
    for keep in (False, True):
        for r, out, w in zip(reqs, eng.route_instances(reqs, retry_full=False, keep_fields=keep), want):
            assert (out.paths, out.search_costs) == w
            if keep:
                _assert_fields(oracle, r, out)
