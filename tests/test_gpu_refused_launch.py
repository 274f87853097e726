"""A call that the CUDA runtime refuses is reported once, by that call: the next
solve of this or another engine goes on.

Tolerance: the exact (straight, diagonal) optimum must be identical before and
after."""
from __future__ import annotations

import pytest

from uastar_gb300 import Engine, GridInstance, PuzzleInstance
from uastar_gb300 import engine as E
from uastar_gb300.engine import EngineError

pytestmark = pytest.mark.gpu
H, W, S, G = 60, 70, (0, 0), (59, 69)
# more shared memory than a CTA can have
TOO_LARGE = {"block_threads": 512, "threads_per_heap": 1}


def test_after_a_refused_shape():
    words = E.gen_grid(5, H, W, 0.2, S, G)
    with Engine(0) as a:
        want = a.grid_solve(words, H, W, S, G)
        for _ in range(2):
            with Engine(0, **TOO_LARGE) as b, pytest.raises(EngineError):
                b.grid_solve(words, H, W, S, G)
            r = a.grid_solve(words, H, W, S, G)
            assert r.ok and (r.straight, r.diagonal) == (want.straight, want.diagonal)
            with Engine(0) as c:
                assert c.grid_solve(words, H, W, S, G).ok


@pytest.mark.parametrize("kw", [{"threads_per_instance": 512, "threads_per_heap": 1, "cluster_size": 16},
                                {"threads_per_instance": 512, "cluster_size": 16}, {"cluster_size": 16}])
def test_after_a_batch_without_clusters(kw):
    words = E.gen_grid(5, H, W, 0.2, S, G)
    with Engine(0) as a:
        a.pdb_build(3)
        want = a.grid_solve(words, H, W, S, G)
        insts = [GridInstance(words, H, W, S, G), PuzzleInstance(3, E.gen_puzzle(1, 3, 30))]
        try:
            a.batch_solve(insts, **kw)
        except EngineError:
            pass
        r = a.grid_solve(words, H, W, S, G)
        assert r.ok and (r.straight, r.diagonal) == (want.straight, want.diagonal)
