"""Plain solves with the smallest tables (2 to 8 slots): every state past the
load limit is counted, on a fresh table as on one used before.

Corridors of open cells, one cell wide: a search from cell s of n stores one
state more per step, so the status is a whole number known beforehand."""
from __future__ import annotations

import numpy as np
import pytest

from uastar_gb300 import Engine
from uastar_gb300 import _lib as L
from uastar_gb300 import engine as E

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("log2", [1, 2, 3])
def test_corridors_fill_the_table(log2):
    n = 64  # cells: more than the table's bytes hold at 8 a cell
    words = E.pack_words(np.ones((1, n), dtype=np.uint8))
    with Engine(0, hash_log2_slots=log2) as eng:
        for _ in range(2):
            for s in range(0, n - 1):
                r = eng.grid_solve(words, 1, n, (0, s), (0, n - 1 if s < n // 2 else 0))
                assert r.status == L.HASH_FULL and r.table_used > 0.8 * 2**log2, s
                r = eng.grid_solve(words, 1, n, (0, s), (0, s))
                assert r.ok and r.path_len == 1


def test_near_goals_fit_a_tiny_table():
    # 8 slots hold 6 states; a goal two cells away takes at most five, if nothing
    # away from it is expanded
    n = 64
    words = E.pack_words(np.ones((1, n), dtype=np.uint8))
    with Engine(0, hash_log2_slots=3) as eng:
        for s in range(2, n - 2):
            for g in (s - 2, s - 1, s + 1, s + 2):
                r = eng.grid_solve(words, 1, n, (0, s), (0, g))
                assert r.ok and r.path_len == abs(g - s) + 1, (s, g)
