"""Grids searched with a word per cell (GridDirect) and the rule that chooses
it: single-number costs in the right order, every setting of the table's size
that moves a map between the word and the hashed form, costs that leave the
word's range.

Tolerance: none.  Costs are exact pairs of step counts; both forms must return
the oracle's optimum and a path that the host validates."""
from __future__ import annotations

import ctypes as C
import re
from fractions import Fraction
from pathlib import Path

import numpy as np
import pytest

import oracle as O
from uastar_gb300 import Engine
from uastar_gb300 import _lib as L
from uastar_gb300 import engine as E

SRC = (Path(__file__).resolve().parents[1] / "uastar_gb300" / "csrc" / "ga_problems.cuh").read_text()
FRAC = int(re.search(r"kFrac = (\d+);", SRC).group(1))
DIAG = int(re.search(r"kDiag = (\d+)ull;", SRC).group(1))
LIMIT = int(re.search(r"kLimit = (\d+)ull << kFrac;", SRC).group(1))


def test_numbers_compare_as_costs():
    """sign((a1 + b1 sqrt2) - (a2 + b2 sqrt2)) for costs below the limit, where
    it is hardest: differences that are convergents of sqrt2, and near them."""
    top = int(LIMIT / 2**0.5)
    assert DIAG % 2 == 1 and abs(Fraction(DIAG, 2**FRAC) ** 2 - 2) < Fraction(3, 2**FRAC)
    p, q, checked = 1, 1, 0
    while q <= top:
        for dp in range(-2, 3):
            for dq in range(-2, 3):
                s, d = p + dp, q + dq  # s straight steps against d diagonal ones
                if s < 0 or not 0 <= d <= top:
                    continue
                exact = (s * s > 2 * d * d) - (s * s < 2 * d * d)
                number = (s << FRAC) - d * DIAG
                assert (number > 0) - (number < 0) == exact, (s, d)
                checked += 1
        p, q = p + 2 * q, p + q
    assert checked > 300
    inv = pow(DIAG, -1, 1 << FRAC)
    for a, b in ((0, 0), (1, 0), (0, 1), (LIMIT - 1, 0), (0, top), (12345, 67890), (400000, 282000)):
        c = (a << FRAC) + b * DIAG
        assert c < LIMIT << FRAC or (a, b) == (0, top)
        assert ((c * inv) & ((1 << FRAC) - 1), (c - b * DIAG) >> FRAC) == (b, a)
        assert (2 * c) << 3 < 1 << 64  # g and f = g + h, with the move's three bits


def _same(eng, words, H, W, s, g):
    ref, _ = O.grid_astar(words, H, W, s, g, want_path=False)
    r = eng.grid_solve(words, H, W, s, g)
    assert r.ok == ref.solved
    if r.ok:
        assert (r.straight, r.diagonal) == (ref.straight, ref.diagonal)
        assert E.validate_grid_path(words, H, W, s, g, eng.grid_path())[:2] == (ref.straight, ref.diagonal)
    return r


@pytest.mark.gpu
@pytest.mark.parametrize("H,W", [(1, 3), (3, 1), (64, 64), (61, 67), (129, 500), (512, 1024), (727, 719)])
@pytest.mark.parametrize("log2", [0, 10, 12, 17, 20])
def test_word_and_hashed_tables_agree(H, W, log2):
    words = E.gen_grid(H + W, H, W, 0.2, (0, 0), (H - 1, W - 1))
    room = int(0.8 * (1 << log2)) if log2 else 1 << 40
    with Engine(0, hash_log2_slots=log2, max_load=0.8) as eng:
        if H * W <= room:  # else the search may report a full table, in either form
            _same(eng, words, H, W, (0, 0), (H - 1, W - 1))
            _same(eng, words, H, W, (H - 1, W // 2), (0, 0))
        else:
            r = eng.grid_solve(words, H, W, (0, 0), (H - 1, W - 1))
            assert r.status in (L.OK, L.HASH_FULL)
            assert r.status != L.OK or r.table_used <= room


@pytest.mark.gpu
def test_costs_beyond_the_word():
    # the goal is out of reach and 1500 cells behind the start drive f over the limit
    W, start = LIMIT - 100, 1500
    free = np.ones((1, W), np.uint8)
    free[0, start + 1] = 0
    words, s, g = E.pack_words(free), (0, start), (0, W - 1)
    with Engine(0) as eng:
        r = eng.grid_solve(words, 1, W, s, g)
        assert r.status == L.NO_SOLUTION and r.table_used == start + 1
        # a straight way across that is longer than the limit, and a short query there
        free = np.ones((1, LIMIT + 64), np.uint8)
        _same(eng, E.pack_words(free), 1, LIMIT + 64, (0, 5), (0, 700))
    torch = pytest.importorskip("torch")
    dev = torch.device("cuda", 0)
    for w, width, s, g, want in ((words, W, start, W - 1, L.NO_SOLUTION),
                                 (E.pack_words(free), LIMIT + 64, 5, 700, L.OK)):
        d_words = torch.from_numpy(w.view(np.int64).copy()).to(dev)
        d_path = torch.full((2000,), -1, dtype=torch.int32, device=dev)
        d_res = torch.zeros(C.sizeof(L.NoallocGridResult), dtype=torch.uint8, device=dev)
        rc = L.load().uastar_grid_solve_noalloc(C.c_void_p(d_words.data_ptr()), 1, width, 0, s, 0, g,
                                                C.c_void_p(d_path.data_ptr()), 2000, C.c_void_p(d_res.data_ptr()),
                                                C.c_void_p(torch.cuda.current_stream(dev).cuda_stream))
        assert rc == L.OK
        torch.cuda.synchronize(dev)
        res = L.NoallocGridResult.from_buffer_copy(d_res.cpu().numpy().tobytes())
        assert res.status == want
        if want == L.OK:
            assert (res.straight, res.diagonal) == (695, 0)
            assert (d_path.cpu().numpy()[:696] == np.arange(5, 701)).all()
