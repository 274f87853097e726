"""What a batch leaves as it was: instances that it hands to the plain engine
must not replace the caller's loaded grid or last solution.

Tolerance: the exact (straight, diagonal) optimum and the path's cells must be
identical before and after."""
from __future__ import annotations

import numpy as np
import pytest

import oracle as O
from uastar_gb300 import Engine, GridInstance, PuzzleInstance
from uastar_gb300 import _lib as L
from uastar_gb300 import engine as E
from uastar_gb300 import workloads as WL

pytestmark = pytest.mark.gpu


def handed_on():
    """Instances that overflow both team tiers (est_nodes) and end on the plain engine."""
    sp = WL.screened_grid(400, 400, 0.2, 3, exact=True)
    return [GridInstance(sp.words(), sp.H, sp.W, sp.start, sp.goal, est_nodes=1),
            PuzzleInstance(4, E.gen_puzzle(1008, 4, 200), est_nodes=1)]


def test_loaded_grid_survives_a_batch():
    H, W, s, g = 90, 70, (0, 0), (89, 69)
    words = E.gen_grid(5, H, W, 0.2, s, g)
    ref, _ = O.grid_astar(words, H, W, s, g, want_path=False)
    with Engine(0) as eng:
        eng.pdb_build(4)
        eng.grid_load(words, H, W)
        assert ref.solved
        for insts in (handed_on()[:1], handed_on()):
            res, stats = eng.batch_solve(insts)
            assert stats["escalated"] == len(insts) and all(r["status"] == L.OK for r in res)
            r = eng.grid_solve_loaded(s, g)
            assert r.ok and (r.straight, r.diagonal) == (ref.straight, ref.diagonal)
            a, b, _ = E.validate_grid_path(words, H, W, s, g, eng.grid_path())
            assert (a, b) == (ref.straight, ref.diagonal)


def test_last_solution_survives_a_batch():
    H, W, s, g = 90, 70, (0, 0), (89, 69)
    words = E.gen_grid(5, H, W, 0.2, s, g)
    with Engine(0) as eng:
        eng.pdb_build(4)
        assert eng.grid_solve(words, H, W, s, g).ok
        path = eng.grid_path()
        _, stats = eng.batch_solve(handed_on())
        assert stats["escalated"] == 2
        assert np.array_equal(eng.grid_path(), path)
        tiles = E.gen_puzzle(40, 4, 40)
        assert eng.puzzle_solve(4, tiles).ok
        moves = eng.puzzle_moves()
        eng.batch_solve(handed_on())
        assert eng.puzzle_moves() == moves
