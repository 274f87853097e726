"""Rounds that expand improved successors at once (ga_search's continuation
passes under its bound on f) against the oracle, where the passes meet an edge:
maps one word wide or narrower, ends on the border, a start next to the goal,
no relaxer warps, candidate regions of a few heaps, a limit on expansion steps.

Tolerance: the exact (straight, diagonal) optimum must be identical; no
path of n cells can have been found in fewer than n - 1 expansion steps."""
from __future__ import annotations

import numpy as np
import pytest

import oracle as O
from uastar_gb300 import Engine
from uastar_gb300 import _lib as L
from uastar_gb300 import engine as E

pytestmark = pytest.mark.gpu

SHAPES = [{}, {"heaps": 32, "block_threads": 32, "threads_per_heap": 1},
          {"heaps": 64, "block_threads": 64, "threads_per_heap": 32}, {"heaps": 1000, "block_threads": 96}]
MAPS = [(1, 700, 0.0), (3, 400, 0.1), (31, 33, 0.2), (64, 32, 0.3), (65, 129, 0.35), (300, 200, 0.3), (500, 777, 0.25)]


@pytest.mark.parametrize("shape", range(len(SHAPES)))
@pytest.mark.parametrize("H,W,rate", MAPS)
def test_grids_at_the_edges(shape, H, W, rate):
    rng = np.random.default_rng(H * 1000 + W)
    ends = [((0, 0), (H - 1, W - 1)), ((H - 1, 0), (0, W - 1)), ((H // 2, W // 2), (H // 2, W // 2 + 1)),
            (tuple(int(rng.integers(0, n)) for n in (H, W)), tuple(int(rng.integers(0, n)) for n in (H, W)))]
    with Engine(0, **SHAPES[shape]) as eng:
        for i, (s, g) in enumerate(ends):
            words = E.gen_grid(77 + i, H, W, rate, s, g)
            ref, _ = O.grid_astar(words, H, W, s, g, want_path=False)
            r = eng.grid_solve(words, H, W, s, g)
            if not ref.solved:
                assert r.status == L.NO_SOLUTION
                continue
            assert r.ok and (r.straight, r.diagonal) == (ref.straight, ref.diagonal), (H, W, s, g)
            assert r.rounds >= r.path_len - 1
            assert r.expanded <= r.generated or r.generated == 0


@pytest.mark.parametrize("limit", [1, 2, 3, 7, 50])
def test_step_limit_is_exact(limit):
    H, W = 200, 300
    words = E.gen_grid(3, H, W, 0.2, (0, 0), (H - 1, W - 1))
    with Engine(0, max_rounds=limit) as eng:
        r = eng.grid_solve(words, H, W, (0, 0), (H - 1, W - 1))
        assert r.status == L.ITER_LIMIT and r.rounds == limit
