"""The memory-bounded mode keeps within its table cap, also where the growth by
4x would step over it: a board with more states than the cap's load limit needs
several segments, one with fewer needs one.

Tolerance: the plain engine's optimum must be identical, and at least as large
as the lower bound where the exact phase is off."""
from __future__ import annotations

import pytest

from uastar_gb300 import Engine
from uastar_gb300 import _lib as L
from uastar_gb300 import engine as E

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def beng():
    with Engine(0, exact_ms=-1) as eng:
        eng.pdb_build(4)
        yield eng


# (11 M states each, as the plain engine counts them: 6.7 M fit 2^23 slots, 13.4 M 2^24)
@pytest.mark.parametrize("seed", [1021, 1047])
def test_odd_cap_is_not_stepped_over(beng, seed):
    tiles = E.gen_puzzle(seed, 4, 200)
    ref = beng.puzzle_solve(4, tiles)
    assert ref.ok and ref.table_used > 0.9 * 2**23
    r = beng.puzzle_solve_bounded(4, tiles, 23)
    assert r["status"] == L.OK and r["segments"] > 1
    assert r["lower_bound"] <= ref.steps <= r["steps"]


@pytest.mark.parametrize("log2", [23, 25])
def test_odd_cap_is_used(beng, log2):
    tiles = E.gen_puzzle(1039, 4, 200)  # 3.2 M states: past the first table's growth point
    r = beng.puzzle_solve_bounded(4, tiles, log2)
    assert r["status"] == L.OK and r["segments"] == 1
    assert r["steps"] == r["lower_bound"] == beng.puzzle_solve(4, tiles).steps
