"""The bench's model of a grid search's bytes counts no access that the search
cannot make: nodes expanded without a heap have no heap entry, and a push's node
is the word that its relax wrote.  CPU only; whole numbers."""
from __future__ import annotations

import sys

import pytest

from conftest import ROOT

sys.path.insert(0, str(ROOT))
import bench  # noqa: E402


@pytest.mark.parametrize("popped,continued,generated,left", [(0, 0, 0, 0), (1, 0, 8, 0), (53, 39, 268, 0),
                                                             (10, 500, 900, 25), (40, 3, 100, 60)])
def test_no_more_than_the_accesses(popped, continued, generated, left):
    pushed = popped + left  # (`left` stay in the heaps)
    sectors = 3 * (popped + continued) + generated + pushed + 2 * popped
    model = bench.grid_bytes(popped + continued, generated, pushed)
    assert model >= 32 * sectors
    if left == 0:
        assert model == 32 * sectors
    assert model <= 32 * (sectors + 2 * left)
    expanded = popped + continued  # the model as it reads
    assert model == eval(bench.GRID_BYTES_MODEL)
