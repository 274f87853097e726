"""The path read-out in windows of cells (walk_grid) where a window can go
wrong: maps narrower than one, wider by a cell, paths that leave a window on
every side or turn back in it, one cell, one step, more cells than the solve's
own room for its path, a caller's buffer that is exactly long enough or not.

Tolerance: none.  A path is right when the host's validation finds it to run
from start to goal over free cells with the oracle's straight and diagonal steps."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

import oracle as O
from uastar_gb300 import Engine
from uastar_gb300 import _lib as L
from uastar_gb300 import engine as E

pytestmark = pytest.mark.gpu


def serpentine(H, W, lanes_of):
    """Walls across the map with a gap at alternating ends, lanes_of rows apart."""
    free = np.ones((H, W), bool)
    for j, x in enumerate(range(lanes_of, H - 1, lanes_of + 1)):
        free[x] = False
        free[x, -1 if j % 2 == 0 else 0] = True
    return free


def noalloc(words, H, W, s, g, cap):
    torch = pytest.importorskip("torch")
    dev = torch.device("cuda", 0)
    d_words = torch.from_numpy(words.view(np.int64).copy()).to(dev)
    d_path = torch.full((cap + 1,), -1, dtype=torch.int32, device=dev)
    d_res = torch.zeros(C.sizeof(L.NoallocGridResult), dtype=torch.uint8, device=dev)
    rc = L.load().uastar_grid_solve_noalloc(C.c_void_p(d_words.data_ptr()), H, W, *s, *g,
                                            C.c_void_p(d_path.data_ptr()), cap, C.c_void_p(d_res.data_ptr()),
                                            C.c_void_p(torch.cuda.current_stream(dev).cuda_stream))
    assert rc == L.OK
    torch.cuda.synchronize(dev)
    path = d_path.cpu().numpy()
    assert path[cap] == -1  # nothing behind the caller's buffer
    return L.NoallocGridResult.from_buffer_copy(d_res.cpu().numpy().tobytes()), path


@pytest.mark.parametrize("H,W,lanes", [(1, 1, 0), (1, 2, 0), (1, 4097, 0), (130, 1, 0), (64, 64, 0), (65, 63, 0),
                                       (127, 129, 1), (200, 90, 5), (61, 1500, 2), (700, 333, 40)])
def test_paths(H, W, lanes):
    free = serpentine(H, W, lanes) if lanes else np.ones((H, W), bool)
    words = E.pack_words(free)
    corners = [(0, 0), (H - 1, W - 1), (H - 1, 0), (0, W - 1), (H // 2, W // 2)]
    with Engine(0) as eng:
        for s, g in [(corners[0], corners[1]), (corners[1], corners[0]), (corners[2], corners[3]),
                     (corners[4], corners[0]), (corners[1], corners[4])]:
            if not (free[s] and free[g]):
                continue
            ref, _ = O.grid_astar(words, H, W, s, g, want_path=False)
            r = eng.grid_solve(words, H, W, s, g)
            assert r.ok == ref.solved
            if not r.ok:
                continue
            n = ref.straight + ref.diagonal + 1
            assert r.path_len == n
            assert E.validate_grid_path(words, H, W, s, g, eng.grid_path())[:2] == (ref.straight, ref.diagonal)
            for cap in (n, n + 7, max(1, n - 1)):
                res, path = noalloc(words, H, W, s, g, cap)
                if cap < n:
                    assert res.status == L.ARENA_FULL and res.path_len == 0
                    continue
                assert res.status == L.OK and res.path_len == n
                assert E.validate_grid_path(words, H, W, s, g, path[:n])[:2] == (ref.straight, ref.diagonal)
