"""Performance cases of the routing engine, through its public Python entry points.

Every case is a plain dict; ``prepare`` builds what a program holds before the
call (the boards and nets of one seed, an engine, resident boards, a staged
batch, a running request loop), ``run`` makes one pass and returns all of its
outputs.  Outputs are whole numbers (path offsets and cells, search costs,
distance fields, occupancy), so ``exact`` has nothing to add to them.

The kinds:

* ``call``      — Engine.route_isolated_batch: one board and its nets from host
                  arrays, the provider seam of the negotiated router.
* ``resident``  — Board + Batch.launch/finish: the board stays in HBM and a staged
                  net set is solved again, with paths only or with fields.
* ``instances`` — Engine.route_instances: many small boards of uneven size in one
                  launch, from page-locked or ordinary host arrays.
* ``multi``     — the same instances resident, replayed as a CUDA graph.
* ``lee``       — Engine.route_lee: unit steps on single layers, whole-board windows.
* ``fields``    — Engine.distance_fields: complete distance fields of many sources.
* ``negotiate`` — a snapshot negotiation from its creation through several rounds.
* ``serve``     — a burst of requests through the continuous-batching request loop.
"""
from __future__ import annotations

import math
import os
import random
import sys

import numpy as np

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "metal-route_b200"))

import mrcuda  # noqa: E402
from mrcuda import workloads as W  # noqa: E402
from mrcuda.types import IsolatedRouteWindow  # noqa: E402

_ENGINE = None


def _engine():
    """One engine per process, as a program keeps it."""
    global _ENGINE
    if _ENGINE is None:
        _ENGINE = mrcuda.Engine(0)
    return _ENGINE


def listed():
    return [
        # the smallest call: one short net on a small two-layer board (a retried or hand-edited net)
        dict(name="call one net", kind="call", board="axis", w=48, h=40, layers=2, nets=1, pinned=False),
        # the provider seam of the reference's router: axis gap prices, own pads, via and board masks, odd sizes
        dict(name="call pads", kind="call", board="pads", w=233, h=187, layers=4, nets=48, pinned=False),
        # an ordinary congested board from page-locked host arrays; some windows too tight, retried on the whole board
        dict(name="call directed", kind="call", board="directed", w=389, h=301, layers=3, nets=96, pinned=True),
        # the plain workload: 128x128x2, whole-board windows, complete fields and paths
        dict(name="resident fields", kind="resident", board="plain", w=128, h=128, layers=2, nets=60, fields=True),
        # the congestion workload: 512x512x4, directed prices, polygon outline, 256 nets, paths
        dict(name="resident congestion", kind="resident", board="directed", w=512, h=512, layers=4, nets=256,
             fields=False),
        # a large board with long nets (median 300 cells): the deepest wavefronts
        dict(name="resident large", kind="resident", board="snapshot", w=1280, h=1153, layers=6, nets=160,
             fields=False),
        # uneven instances from page-locked host arrays, one call
        dict(name="instances call", kind="instances", count=256, pinned=True),
        # uneven instances resident, one launch replayed as a graph
        dict(name="instances resident", kind="multi", count=640),
        # Lee routing of a single-layer board
        dict(name="lee", kind="lee", w=201, h=160, layers=1, nets=40),
        # complete distance fields of many sources
        dict(name="fields", kind="fields", w=192, h=176, layers=2, sources=32),
        # negotiation from its creation through six rounds, connection groups
        dict(name="negotiate", kind="negotiate", w=512, h=480, layers=4, nets=300, rounds=6, groups=True,
             clearance=0),
        # a burst of requests of different sizes on resident boards
        dict(name="serve burst", kind="serve", boards=6, lo=64, hi=512, requests=18, max_nets=128),
    ]


def _log(rng: random.Random, lo: int, hi: int) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["call", "call", "resident", "resident", "instances", "multi", "lee", "fields", "negotiate",
                       "serve"])
    if kind == "call":
        board = rng.choice(["axis", "pads", "directed"])
        return dict(kind=kind, board=board, w=_log(rng, 40, 420), h=_log(rng, 40, 420), layers=rng.randint(2, 6),
                    nets=_log(rng, 1, 128), pinned=rng.random() < 0.5)
    if kind == "resident":
        board = rng.choice(["plain", "directed", "snapshot", "pads"])
        big = 1000 if board == "snapshot" else 128 if board == "plain" else 512
        return dict(kind=kind, board=board, w=_log(rng, 48, big), h=_log(rng, 48, big), layers=rng.randint(1, 6),
                    nets=_log(rng, 4, 60 if board == "plain" else 256),
                    fields=board == "plain" and rng.random() < 0.5)
    if kind == "instances":
        return dict(kind=kind, count=_log(rng, 16, 384), pinned=rng.random() < 0.5)
    if kind == "multi":
        return dict(kind=kind, count=_log(rng, 16, 768))
    if kind == "lee":
        return dict(kind=kind, w=_log(rng, 40, 320), h=_log(rng, 40, 320), layers=1, nets=_log(rng, 1, 64))
    if kind == "fields":
        return dict(kind=kind, w=_log(rng, 48, 256), h=_log(rng, 48, 256), layers=rng.randint(1, 3),
                    sources=_log(rng, 1, 40))
    if kind == "negotiate":
        clear = rng.choice([0, 0, 1])
        return dict(kind=kind, w=_log(rng, 96, 480), h=_log(rng, 96, 480), layers=rng.randint(2, 5),
                    nets=_log(rng, 24, 256), rounds=rng.randint(2, 6), groups=not clear and rng.random() < 0.5,
                    clearance=clear)
    return dict(kind="serve", boards=rng.randint(2, 6), lo=64, hi=_log(rng, 96, 512), requests=rng.randint(4, 18),
                max_nets=_log(rng, 24, 128))


# -- inputs -------------------------------------------------------------------

def _axis_board(seed, w, h, layers, n_nets, pads):
    """A board on non-uniform lines: per-axis gap prices (length x 16), unit
    enter weights, ~10% obstacles; with `pads` also a courtyard mask along the
    rim, a static via mask, own pads around both endpoints, and no vias into the
    last layer of a board of more than three (a plane layer without pins)."""
    rng = np.random.default_rng(seed)
    dims = mrcuda.Dims(w, h, layers)
    cost = np.ones((layers, h, w), dtype=np.uint32)
    while (cost == mrcuda.OBSTACLE).mean() < 0.10:
        rw, rh = int(rng.integers(2, 9)), int(rng.integers(2, 9))
        x0, y0 = int(rng.integers(0, w - rw)), int(rng.integers(0, h - rh))
        cost[int(rng.integers(0, layers)), y0:y0 + rh, x0:x0 + rw] = mrcuda.OBSTACLE
    board = via = None
    if pads:
        rim = np.zeros((layers, h, w), dtype=np.uint8)
        for s in (np.s_[:, :2, :], np.s_[:, -2:, :], np.s_[:, :, :2], np.s_[:, :, -2:]):
            rim[s] |= mrcuda.BOARD_TRACE_NODE | mrcuda.BOARD_VIA_NODE
        board = rim.reshape(-1)
        via = (rng.random(w * h * layers) < 0.02).astype(np.uint8)
    closed = pads and layers > 3
    nets = []
    for i in range(n_nets):
        ends, own = [], []
        for _ in range(2):
            x, y, l = int(rng.integers(4, w - 4)), int(rng.integers(4, h - 4)), int(rng.integers(0, layers - closed))
            ends.append(dims.idx3(x, y, l))
            if pads:  # a 3 x 3 pad; its cells are obstacles to every other net
                cost[l, y - 1:y + 2, x - 1:x + 2] = mrcuda.OBSTACLE
                own += [dims.idx3(x + dx, y + dy, l) for dy in (-1, 0, 1) for dx in (-1, 0, 1)]
            else:
                cost[l, y, x] = 1
        own = sorted(set(own))
        nets.append(mrcuda.NetEndpoints(f"a{i}", ends[0], ends[1], own, own[:1] if pads else []))
    grid = mrcuda.Grid(dims, cost.reshape(-1), board, via)
    vias = [80] * (layers - 1)
    if closed:
        vias[-1] = None
    x = (16 * rng.integers(1, 9, w - 1)).astype(np.uint32)
    y = (16 * rng.integers(1, 9, h - 1)).astype(np.uint32)
    return W.Workload("axis", grid, nets, mrcuda.net_windows(dims, nets), x, y, vias)


def _board(c, seed):
    w, h, layers, n = c["w"], c["h"], c["layers"], c["nets"]
    if c["board"] in ("axis", "pads"):
        return _axis_board(seed, w, h, layers, n, c["board"] == "pads")
    if c["board"] == "plain":
        return W.plain_board(seed=seed, w=w, h=h, layers=layers, n_nets=n)
    if c["board"] == "snapshot":
        return W.snapshot_board(seed=seed, w=w, h=h, layers=layers, n_nets=n)
    wl = W.congestion_board(seed=seed, w=w, h=h, layers=layers, n_nets=n)
    if c["kind"] == "call":  # every 16th window without a margin: some cannot hold a path and are retried
        for i in range(0, n, 16):
            (ax, ay), (bx, by) = wl.grid.dims.xy(wl.nets[i].src), wl.grid.dims.xy(wl.nets[i].dst)
            wl.windows[i] = IsolatedRouteWindow(min(ax, bx), min(ay, by), max(ax, bx), max(ay, by))
    return wl


class _Out:
    """The outputs in buffers of one size per case, as the paths' total length
    differs from seed to seed: arrays placed one after another, zeros behind."""

    def __init__(self, capacity):
        self.buf = np.zeros(capacity, np.int64)

    def put(self, arrays):
        at = 0
        for a in arrays:
            self.buf[at:at + a.size] = a
            at += a.size
        return self.buf


def _cell_capacity(c):
    """More cells than the case's paths have together."""
    if c["kind"] in ("instances", "multi"):
        return 600 * c["count"] + 4096
    if c["kind"] == "serve":
        return c["requests"] * c["max_nets"] * c["hi"] + 4096
    return 2 * c.get("nets", 0) * (c["w"] + c["h"]) + 4096


def prepare(case, seed):
    c, e = dict(case), _engine()
    kind = c["kind"]
    out = _Out(_cell_capacity(c))
    if kind == "call":
        wl = _board(c, seed)
        if c["pinned"]:
            W.pin_boards(e, [wl])
        return kind, out, e, wl.request()
    if kind == "resident":
        wl = _board(c, seed)
        board = e.board(wl.grid, wl.x, wl.y, wl.vias, wl.directed)
        return kind, out, mrcuda.Batch(board, wl.nets, wl.windows, keep_fields=c["fields"])
    if kind in ("instances", "multi"):
        s = W.uneven_instances(seed=seed, n_instances=c["count"])
        if kind == "instances":
            if c["pinned"]:
                W.pin_boards(e, s.instances)
            return kind, out, e, s.requests()
        boards = [e.board(wl.grid, wl.x, wl.y, wl.vias) for wl in s.instances]
        nets = [wl.nets[0] for wl in s.instances]
        wins = [wl.windows[0] for wl in s.instances]
        batch = mrcuda.Batch(boards, nets, wins, net_board=list(range(len(boards))))
        batch.capture_graph()
        return kind, out, batch
    if kind == "lee":
        wl = W.plain_board(seed=seed, w=c["w"], h=c["h"], layers=c["layers"], n_nets=c["nets"])
        return kind, out, e, wl.grid, wl.nets
    if kind == "fields":
        wl = W.plain_board(seed=seed, w=c["w"], h=c["h"], layers=c["layers"], n_nets=c["sources"])
        return kind, out, e, wl.grid, [nt.src for nt in wl.nets]
    if kind == "negotiate":
        side = (c["w"] + c["h"]) / 4
        wl = W.snapshot_board(seed=seed, w=c["w"], h=c["h"], layers=c["layers"], n_nets=c["nets"], median=side)
        for i, nt in enumerate(wl.nets):
            nt.net = f"s{i // 4}#{i % 4}"
        return kind, out, e, wl.request(), c
    # serve: boards generated as the congestion board, nets drawn per request
    rng = np.random.default_rng(seed)
    pool = W.serving_pool(seed=seed % 100003, n_boards=c["boards"], lo=c["lo"], hi=c["hi"])
    trace = W.serving_trace(pool, 1.0, c["requests"], seed=int(rng.integers(1 << 30)), max_nets=c["max_nets"])
    boards = [e.board(wl.grid, wl.x, wl.y, wl.vias, wl.directed) for wl in pool]
    reqs = [(boards[wl.meta["board_index"]], wl.nets, wl.windows) for _, wl in trace]
    return kind, out, e.server(), reqs, _Out(2 * c["requests"] * (c["max_nets"] + 1))


def _paths(r, out):
    return [r.offsets, out.put([r.cells]), r.costs]


def run(state):
    kind, out = state[0], state[1]
    if kind == "call":
        return _paths(state[2].route_isolated_batch(state[3]), out)
    if kind in ("resident", "multi"):
        state[2].launch()
        r = state[2].finish()
        return _paths(r, out) + (r.fields or [])
    if kind == "instances":
        return _paths(state[2].route_instances(state[3], split=False), out)
    if kind == "lee":
        r = state[2].route_lee(state[3], state[4])
        return [r.congestion, out.put([np.array([v for x in r.results for v in (x.cost, len(x.path), *x.path)])])]
    if kind == "fields":
        return state[2].distance_fields(state[3], state[4])
    if kind == "negotiate":
        _, _, e, req, c = state
        neg = e.negotiation(req, groups="connections" if c["groups"] else None, clearance=c["clearance"],
                            via_keepout=2 * c["clearance"])
        try:
            stats = [neg.round() for _ in range(c["rounds"])]
            paths = neg.paths()
        finally:
            neg.close()
        return [np.array([[s["dirty"], s["routed"], s["retried"], s["overused_edges"], s["path_cells"]] for s in stats],
                         np.int64),
                np.array([len(p) if p else 0 for p in paths], np.int64),
                out.put([np.array([x for p in paths if p for x in p], np.int64)])]
    _, _, server, reqs, ends = state
    tickets = [server.submit_resident(b, nets, wins) for b, nets, wins in reqs]
    got = [server.wait(t)[0] for t in tickets]
    return [out.put([r.cells for r in got]), ends.put([a for r in got for a in (r.offsets, r.costs)])]


def exact(case, seed):
    """Every output is a whole number: there is no rounding to measure."""
    return None


def work(case):
    """Board words read once (enter weights 4 B, masks 1 B, directed prices 16 B a
    cell), paths written once at the nets' mean length, fields written once.
    A label-correcting search does no floating-point work."""
    c = case
    kind = c["kind"]
    if kind in ("instances", "multi"):
        # mean instance: LogNormal(ln 96, 0.5) per side, 5 layers, 5 B a cell; paths about a side long
        cells = c["count"] * (96 * math.exp(0.125)) ** 2 * 5
        return {"bytes": cells * 5 + c["count"] * 110 * 4, "flops": 0}
    if kind == "serve":
        lo, hi = c["lo"], c["hi"]
        side2 = (hi ** 2 - lo ** 2) / (2 * math.log(hi / lo))
        nets = c["requests"] * (c["max_nets"] - 16) / math.log(c["max_nets"] / 16)
        return {"bytes": c["boards"] * side2 * 4 * 21 + nets * math.sqrt(side2) * 0.7 * 4, "flops": 0}
    cells = c["w"] * c["h"] * c["layers"]
    if kind == "fields":
        return {"bytes": cells * 4 * (1 + c["sources"]), "flops": 0}
    board = c.get("board", "snapshot" if kind == "negotiate" else "plain")
    per = {"axis": 4, "plain": 4, "pads": 6, "directed": 21, "snapshot": 20}[board]
    length = (c["w"] + c["h"]) / 3
    passes = c.get("rounds", 1)
    total = cells * per * passes + c["nets"] * length * 4 * passes
    if c.get("fields"):
        total += c["nets"] * cells * 4
    return {"bytes": total, "flops": 0}
