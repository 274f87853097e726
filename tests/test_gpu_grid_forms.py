"""Maps at the sizes where a default solve changes between the word per cell and
the hashed table (838 860 | 838 861 and 2^20 | 2^20 + 1 cells).

Tolerance: the exact (straight, diagonal) optimum must be identical to that of
the sorted mode, which is hashed at every size, and the path must re-validate."""
from __future__ import annotations

import pytest

from uastar_gb300 import Engine
from uastar_gb300 import engine as E

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H,W,hashed", [(916, 915, False), (916, 916, True), (1024, 1024, True), (1024, 1025, False)])
def test_default_form_at_its_edges(H, W, hashed):
    s, g = (0, 0), (H - 1, W - 1)
    words = E.gen_grid(11, H, W, 0.25, s, g)
    with Engine(0) as eng, Engine(0, dedup=1) as sorted_eng:
        r, ref = eng.grid_solve(words, H, W, s, g), sorted_eng.grid_solve(words, H, W, s, g)
        assert ref.ok and r.ok and (r.straight, r.diagonal) == (ref.straight, ref.diagonal)
        a, b, _ = E.validate_grid_path(words, H, W, s, g, eng.grid_path())
        assert (a, b) == (r.straight, r.diagonal)
        # a word per cell has nothing to grow
        assert hashed or r.table_grows == 0
