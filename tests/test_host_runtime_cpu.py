"""The host runtime (csrc/engine.cu) on a CUDA runtime made of host memory
(fake_cuda.cpp): what it does with streams, page-locked memory and failing calls.
Each test is a child process, so that this one keeps the real library."""
import os
import shutil
import subprocess
import sys

import pytest

from conftest import ROOT

CUDA = next((d for d in (os.environ.get("CUDA_HOME"), "/usr/local/cuda") if d and os.path.exists(d + "/include/cuda.h")), None)
pytestmark = pytest.mark.skipif(CUDA is None or shutil.which("g++") is None, reason="needs g++ and the CUDA headers")

PROLOGUE = """
import ctypes as C, sys
import numpy as np
import mrcuda
from mrcuda.types import *
L = mrcuda.load_library(sys.argv[1])
L.fake_fail.argtypes = [C.c_char_p, C.c_int]
L.fake_pinned_bytes.restype = C.c_uint64
eng = mrcuda.Engine(0)
fail = lambda call, nth=1: L.fake_fail(call.encode(), nth)
def grid(w, h, layers=1):
    return Grid(Dims(w, h, layers), np.ones(w * h * layers, np.uint32))
def board(w, h, layers=1, gap=1):
    return eng.board(grid(w, h, layers), [gap] * (w - 1), [gap] * (h - 1), [1] * (layers - 1))
def nets(w, h, n=1):
    return [NetEndpoints(f"n{i}", 0, w * h - 1) for i in range(n)]
"""


@pytest.fixture(scope="session")
def fake_library(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("fake") / "libfake.so")
    csrc = os.path.join(ROOT, "metal-route_b200", "csrc")
    subprocess.check_call(["g++", "-x", "c++", "-std=c++17", "-O1", "-w", "-fPIC", "-shared", "-D__ldg(p)=(*(p))",
                           "-I", CUDA + "/include", "-I", os.path.join(ROOT, "include"), "-I", csrc,
                           os.path.join(csrc, "engine.cu"), os.path.join(ROOT, "tests", "fake_cuda.cpp"),
                           "-Wl,--wrap=malloc", "-Wl,--no-undefined", "-lpthread", "-o", so])
    return so


@pytest.fixture
def run(fake_library):
    def go(body):
        env = dict(os.environ, PYTHONPATH=os.path.join(ROOT, "metal-route_b200"))
        p = subprocess.run([sys.executable, "-c", PROLOGUE + body, fake_library], env=env, capture_output=True,
                           text=True, timeout=120)
        assert p.returncode == 0, p.stdout + p.stderr
    return go


def test_no_copy_is_in_flight_after_a_failed_finish(run):
    """Host memory for the fields runs out: the call returns with nothing on its way
    into the context's download block, which the next call of any stream uses."""
    run("""
bt = mrcuda.Batch(board(40, 30), nets(40, 30), keep_fields=True)
bt.launch()
fail("cudaHostAlloc", 2); fail("malloc")  # (the first page-locked block is the download block)
try: bt.finish(); assert False
except mrcuda.OutOfMemory: pass
assert L.fake_pending_host_writes() == 0
bt.finish()
""")


def test_no_copy_is_in_flight_after_failed_distance_fields(run):
    """A copy fails after others were put on the stream: none of those still writes into
    the caller's rows, which the caller may free."""
    run("""
g = grid(40, 30); g.cost[1] = COST_MAX
fail("copy to host", 3)  # status, rows before the refused source, rows after it
try: eng.distance_fields(g, [0, 1, 2]); assert False
except mrcuda.BackendUnavailable: pass
assert L.fake_pending_host_writes() == 0
""")


def test_page_locked_boards_leave_results_page_locked(run):
    """Only results count toward what results may hold page-locked: a program with many
    page-locked boards still gets its fields page-locked."""
    run("""
held = [eng.pinned_empty((16 << 20,), np.uint32) for _ in range(9)]  # 576 MB of boards
bt = mrcuda.Batch(board(400, 300), nets(400, 300, 8), keep_fields=True)
bt.launch(); first = bt.finish()  # (also takes the download block)
before = L.fake_pinned_bytes()
bt.launch(); second = bt.finish()
assert L.fake_pinned_bytes() - before >= second.fields[0].nbytes * 8
""")


def test_a_failed_page_locked_allocation_is_tried_again_without_the_kept_blocks(run):
    run("""
kept = eng.pinned_empty((4 << 20,), np.uint32); del kept
before = L.fake_pinned_bytes()
fail("cudaHostAlloc")
big = eng.pinned_empty((16 << 20,), np.uint32)  # larger than any kept block
assert L.fake_pinned_bytes() == before - (16 << 20) + (64 << 20)
""")


def test_downloads_lock_no_more_pages_than_they_need(run):
    """A small call locks about what it brings back; a call of very many nets no more
    than a bound."""
    run("""
bt = mrcuda.Batch(board(20, 20), nets(20, 20))
bt.launch(); bt.finish()
assert L.fake_pinned_bytes() <= 2 << 20
many = mrcuda.Batch(board(20, 20), nets(20, 20, 70000))
many.launch(); many.finish()
assert L.fake_pinned_bytes() <= 24 << 20
""")


def test_autotuned_fields_leave_path_batches_alone(run):
    """Complete fields and paths alone are different searches: what an autotuner finds for
    one says nothing about the other.  (The timings here make it take its last candidate.)"""
    run("""
b = board(128, 128, 2)
mk = lambda keep: mrcuda.Batch(b, nets(128, 128), keep_fields=keep)
default = mk(False).config()
tuned = mk(True).autotune()
assert tuned["schedule"] != default["schedule"]
assert mk(False).config() == default
assert mk(True).config() == {k: tuned[k] for k in default}
""")
