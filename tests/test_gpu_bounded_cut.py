"""The memory-bounded mode where its parts meet an edge: the smallest table
caps (fewer heaps than usual; a pause after few rounds), boards next to the goal
(the exact phase's cut meets it), boards whose whole tree below the threshold
ends inside the cut, and the three board sizes.

Tolerance: the exact phase proves its answer, so steps and lower bound must
both be the plain engine's optimum, and the moves must replay to the goal."""
from __future__ import annotations

import pytest

from uastar_gb300 import Engine
from uastar_gb300 import _lib as L
from uastar_gb300 import engine as E

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def beng():
    with Engine(0, exact_ms=30000) as eng:
        for n in (3, 4, 5):
            eng.pdb_build(n)
        yield eng


@pytest.mark.parametrize("n,walks", [(3, (0, 1, 2, 40, 100)), (4, (0, 1, 3, 25, 60, 120)), (5, (0, 1, 3, 25, 50))])
@pytest.mark.parametrize("log2", [16, 17, 18, 20])
def test_bounded_equals_plain(beng, n, walks, log2):
    for w in walks:
        tiles = E.gen_puzzle(900 + w, n, w)
        ref = beng.puzzle_solve(n, tiles)
        r = beng.puzzle_solve_bounded(n, tiles, log2)
        assert ref.ok and r["status"] == L.OK
        assert r["steps"] == r["lower_bound"] == ref.steps, (n, w, log2, r)
        mv = beng.puzzle_moves()
        assert len(mv) == ref.steps and E.validate_puzzle_moves(n, tiles, mv)
