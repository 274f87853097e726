"""The last instances of a batch's waves, which move on to larger teams.

Tolerance: the exact (straight, diagonal) optimum must be identical to the
oracle's."""
from __future__ import annotations

import numpy as np
import pytest

from uastar_gb300 import Engine, GridInstance, PuzzleInstance
from uastar_gb300 import _lib as L
from uastar_gb300 import engine as E

pytestmark = pytest.mark.gpu


def open_grid(H, W, est_nodes=0):
    """All cells open, corner to corner: min(H, W) - 1 diagonal steps, the rest straight."""
    words = np.full(E.grid_words(H, W), np.uint64(0xFFFFFFFFFFFFFFFF), dtype=np.uint64)
    return GridInstance(words, H, W, (0, 0), (H - 1, W - 1), est_nodes)


# what a program may give its engine for plain solves, and too little of it for these instances
LIMITS = [{"hash_log2_slots": 12}, {"heap_capacity": 3, "heaps": 32, "block_threads": 32, "threads_per_heap": 1,
                                    "heap_top_levels": -1},
          {"heaps": 1 << 20}]


@pytest.mark.parametrize("limit", range(len(LIMITS)))
def test_limits_of_plain_solves_refuse_no_instance(limit):
    grids = [open_grid(2100, 2300), open_grid(1200, 1300)]
    with Engine(0, **LIMITS[limit]) as eng:
        eng.pdb_build(4)
        for insts in (grids[:1], grids[1:], grids + [PuzzleInstance(4, E.gen_puzzle(1001, 4, 200))]):
            res, _ = eng.batch_solve(insts)
            for i, r in zip(insts, res):
                assert r["status"] == L.OK, r
                if isinstance(i, GridInstance):
                    assert (r["straight"], r["diagonal"]) == (abs(i.H - i.W), min(i.H, i.W) - 1)
                else:
                    assert r["steps"] == 50


@pytest.mark.parametrize("ctas", [1, 8])
def test_no_early_end_while_instances_wait(ctas):
    # grids of ~600 steps on few teams: only those running when the queue has
    # run empty may be handed on, so all but one team's worth finish where they
    # began (est_nodes: with room for every cell, none overflows)
    grids = [open_grid(600, 400 + 7 * i, 600 * (400 + 7 * i)) for i in range(4 * ctas)]
    with Engine(0) as eng:
        res, _ = eng.batch_solve(grids, ctas=ctas)
    assert all(r["status"] == L.OK for r in res)
    assert sum(r["attempts"] == 1 for r in res) >= len(grids) - ctas


def test_short_grids_finish_where_they_began():
    grids = [open_grid(200 + 3 * i, 320, 320 * 320) for i in range(36)]
    with Engine(0) as eng:
        res, stats = eng.batch_solve(grids)
    assert stats["waves"] == 1 and stats["escalated"] == 0
    assert all(r["status"] == L.OK and r["attempts"] == 1 for r in res)


@pytest.mark.parametrize("W,escalated", [(513, 0), (514, 0), (2049, 0), (2050, 1)])
def test_a_grid_alone_is_started_once(W, escalated):
    # 2 x 256 and 2 x 1024 steps are where one team or a cluster is sure not to keep it
    with Engine(0) as eng:
        (r,), stats = eng.batch_solve([open_grid(300, W, 300 * W)])
    assert r["status"] == L.OK and (r["straight"], r["diagonal"]) == (W - 300, 299)
    assert r["attempts"] == 1 and stats["escalated"] == escalated


@pytest.mark.parametrize("tier1", [1, 1 << 20])
def test_small_budgets_lose_no_instance(tier1):
    # (200 moves from the goal: more than the 256 steps after which a lone puzzle
    # moves on, and than the 64 of the second tier)
    tiles = E.gen_puzzle(1008, 4, 200)
    with Engine(0, hash_log2_slots=8) as eng:
        eng.pdb_build(4)
        (r,), _ = eng.batch_solve([PuzzleInstance(4, tiles)], tier1_rounds=tier1, tier2_puzzle_rounds=64)
    assert r["status"] == L.OK and r["steps"] == 46
