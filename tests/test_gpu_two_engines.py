"""Engines of different launch shapes side by side: what one sets for a kernel
must not take the other's shared memory away.

Tolerance: the exact (straight, diagonal) optimum and the move count must be
identical from both engines, before and after the other's solves."""
from __future__ import annotations

import time

import pytest

from uastar_gb300 import Engine, GridInstance, PuzzleInstance
from uastar_gb300 import _lib as L
from uastar_gb300 import engine as E

pytestmark = pytest.mark.gpu
SMALL = {"heap_top_levels": -1}  # least shared memory: no heap levels but the root


@pytest.mark.parametrize("dedup", [0, 1])
def test_grids_in_turn(dedup):
    H, W, s, g = 200, 220, (0, 0), (199, 219)
    words = E.gen_grid(9, H, W, 0.25, s, g)
    with Engine(0, dedup=dedup) as a, Engine(0, dedup=dedup, **SMALL) as b:
        got = [e.grid_solve(words, H, W, s, g) for e in (a, b, a, b, a)]
        assert all(r.ok for r in got) and len({(r.straight, r.diagonal) for r in got}) == 1


def test_puzzles_in_turn():
    tiles = E.gen_puzzle(3, 3, 80)
    with Engine(0) as a, Engine(0, **SMALL) as b:
        for e in (a, b):
            e.pdb_build(3)
        assert len({e.puzzle_solve(3, tiles).steps for e in (a, b, a, b, a)}) == 1


def test_serving_beside_a_batch_of_small_teams():
    insts = [GridInstance(E.gen_grid(9, 200, 200, 0.25, (0, 0), (199, 199)), 200, 200, (0, 0), (199, 199)),
             PuzzleInstance(3, E.gen_puzzle(3, 3, 80))]
    with Engine(0) as a, Engine(0) as b:
        for e in (a, b):
            e.pdb_build(3)
        a.serve_start(hbm_budget_gb=8.0)
        want, _ = b.batch_solve(insts, threads_per_instance=32, threads_per_heap=32)
        ids = [a.serve_submit(i) for i in insts]
        got, end = {}, time.time() + 20
        while len(got) < len(ids) and time.time() < end:
            got.update(a.serve_poll())
            time.sleep(0.001)
        a.serve_stop()
        for i, w in zip(ids, want):
            r = got[i]
            assert r["status"] == w["status"] == L.OK
            assert (r["steps"], r["straight"], r["diagonal"]) == (w["steps"], w["straight"], w["diagonal"])
