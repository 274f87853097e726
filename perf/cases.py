"""Workloads of the engine: what a program that uses it has it solve.

Grids are seeded Bernoulli maps (10..35 % blocked) solved corner to corner
unless a case says otherwise; puzzle boards are random walks from the goal.
Every input is made from the seed alone.  A state holds host bitmaps and
boards (the engine's calls take host buffers) or, for the allocation-free
call, the caller's device buffers; engines and their resident pattern tables
are kept over all states, as a program keeps them over all its requests.

Outputs are what every correct solve has in common: status, exact cost,
steps, path length.  Which of several equally short paths comes back depends
on the order in which the GPU's threads meet, so paths are fetched as a user
would, and their length is returned, not their cells (nor the float32 cost
accumulated along them, nor node counts), with the cells at its two ends.
"""
from __future__ import annotations

import ctypes
import heapq
import math
import random
import time

import numpy as np
import torch

from uastar_gb300 import Engine, GridInstance, PuzzleInstance, gen_grid, grid_reachable
from uastar_gb300 import _lib as L
from uastar_gb300.engine import grid_screen

SQRT2 = math.sqrt(2.0)


def listed():
    return [
        # one query on a small map: the fixed cost of a call
        {"name": "grid_61x67", "kind": "grid", "H": 61, "W": 67, "rate": 0.2, "near": 9},
        # the repository's ordinary map: 1000 x 1000, 30 % blocked
        {"name": "grid_1000", "kind": "grid", "H": 1000, "W": 1000, "rate": 0.3},
        # the headline map: 20000 x 20000, 30 % blocked
        {"name": "grid_20000", "kind": "grid", "H": 20000, "W": 20000, "rate": 0.3},
        # navigation: one ragged map loaded once, several start/goal queries on it
        {"name": "queries_1537x2049", "kind": "queries", "H": 1537, "W": 2049, "rate": 0.25, "queries": 6},
        # a caller that may not allocate: device buffers in, device buffers out
        {"name": "noalloc_700x1021", "kind": "noalloc", "H": 700, "W": 1021, "rate": 0.25, "near": 80},
        # 8-puzzles, one after another: a few hundred states each
        {"name": "puzzle8_x4", "kind": "puzzles", "n": 3, "walk": 100, "count": 4},
        # 15-puzzles of 200 random moves, one after another (the puzzle benchmark's boards)
        {"name": "puzzle15_x8", "kind": "puzzles", "n": 4, "walk": 200, "count": 8},
        # 24-puzzles near the goal: 16-byte keys
        {"name": "puzzle24_x3", "kind": "puzzles", "n": 5, "walk": 60, "count": 3},
        # 15-puzzles with the table capped at 2^20 slots (memory-bounded mode)
        {"name": "bounded15_x2", "kind": "bounded", "n": 4, "walk": 160, "count": 2, "log2_slots": 20},
        # a process's first puzzles: build the pattern tables, then solve
        {"name": "tables15_x2", "kind": "tables", "n": 4, "walk": 120, "count": 2},
        # many instances in one call, three puzzles to a grid as in the mixed benchmark
        {"name": "batch_96", "kind": "batch", "puzzles": 72, "grids": 24, "max_side": 1500, "walk": 200},
        # a burst of requests at the running serving loop, half puzzles and half grids
        {"name": "serve_48", "kind": "serve", "puzzles": 24, "grids": 24, "max_side": 1500, "walk": 160},
    ]


def _log(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["grid", "grid", "grid", "queries", "noalloc", "puzzles", "puzzles", "bounded", "tables",
                       "batch", "serve"])
    rate = round(rng.uniform(0.10, 0.35), 4)
    if kind in ("grid", "queries"):
        hi = 9000 if kind == "grid" else 2500
        h = _log(rng, 48, hi)
        w = max(48, min(hi, int(h * rng.uniform(0.5, 2.0))))
        c = {"kind": kind, "H": h, "W": w, "rate": rate, "near": h // 8}
        if kind == "queries":
            c["queries"] = rng.randint(2, 10)
        return c
    if kind == "noalloc":
        return {"kind": kind, "H": _log(rng, 48, 1400), "W": _log(rng, 48, 1400), "rate": rate, "near": 12}
    if kind == "puzzles":
        n = rng.choice([3, 4, 4, 5])
        return {"kind": kind, "n": n, "walk": rng.randint(20, 60 if n == 5 else 220),
                "count": rng.randint(2, 4 if n == 5 else 8)}
    if kind == "bounded":
        return {"kind": kind, "n": 4, "walk": rng.randint(60, 180), "count": rng.randint(1, 3),
                "log2_slots": rng.randint(18, 22)}
    if kind == "tables":
        n = rng.choice([3, 4, 5])
        return {"kind": kind, "n": n, "walk": rng.randint(20, 50 if n == 5 else 120), "count": rng.randint(2, 4)}
    many = _log(rng, 4, 40)
    return {"kind": kind, "puzzles": many * (3 if kind == "batch" else 1), "grids": many,
            "max_side": _log(rng, 300, 2000), "walk": rng.randint(80, 220)}


# ------------------------------------------------------------------ inputs
def _engine(key, n=()):
    """The program's engine for one kind of work, its pattern tables resident."""
    if key not in _ENGINES:
        _ENGINES[key] = Engine(0)
    eng = _ENGINES[key]
    for side in n:
        if (key, side) not in _TABLES:
            eng.pdb_build(side)
            _TABLES.add((key, side))
    return eng


_ENGINES: dict = {}
_TABLES: set = set()


def _grid(H, W, rate, seed, i, near=0):
    """A map and a query from one corner to the opposite one (each end moved
    by up to `near` cells), connected as far as a bounded search tells."""
    rng = random.Random(seed * 1000003 + i)
    while True:
        start = rng.randint(0, min(near, H - 1)), rng.randint(0, min(near, W - 1))
        goal = H - 1 - rng.randint(0, min(near, H - 1)), W - 1 - rng.randint(0, min(near, W - 1))
        words = gen_grid(rng.getrandbits(32), H, W, rate, start, goal)
        if start != goal and grid_screen(words, H, W, start, goal) != 0:
            return GridInstance(words, H, W, start, goal)


def _board(n, walk, rng):
    """`walk` random blank moves from the goal, none undoing the one before."""
    b = list(range(1, n * n)) + [0]
    at, back = n * n - 1, -1
    for _ in range(walk):
        x, y = divmod(at, n)
        to = [p * n + q for p, q in ((x + 1, y), (x - 1, y), (x, y + 1), (x, y - 1))
              if 0 <= p < n and 0 <= q < n and p * n + q != back]
        q = rng.choice(to)
        b[at], b[q] = b[q], b[at]
        at, back = q, at
    return np.array(b, dtype=np.uint8)


def _boards(case, seed):
    rng = random.Random(seed)
    return [_board(case["n"], case["walk"], rng) for _ in range(case["count"])]


def _mixture(case, seed):
    """Puzzles of 60..walk moves and square grids of 256..max_side cells a side."""
    rng = random.Random(seed)
    out = [PuzzleInstance(4, _board(4, rng.randint(60, case["walk"]), rng)) for _ in range(case["puzzles"])]
    for j in range(case["grids"]):
        side = rng.randint(256, case["max_side"])
        out.append(_grid(side, side, round(rng.uniform(0.10, 0.35), 4), seed, j))
    return out


def _ends(inst, count, seed):
    """`count` start/goal pairs on the map, in open cells that the engine's host search connects."""
    rng = random.Random(seed)
    out = []
    while len(out) < count:
        s, g = ((rng.randrange(inst.H), rng.randrange(inst.W)) for _ in range(2))
        if grid_reachable(inst.words, inst.H, inst.W, s, g):
            out.append((s, g))
    return out


def prepare(case, seed):
    k = case["kind"]
    if k == "grid":
        return {"kind": k, "eng": _engine("grid"), "inst": _grid(case["H"], case["W"], case["rate"], seed, 0, case.get("near", 0))}
    if k == "queries":
        inst = _grid(case["H"], case["W"], case["rate"], seed, 0, case.get("near", 0))
        return {"kind": k, "eng": _engine("grid"), "inst": inst, "ends": _ends(inst, case["queries"], seed)}
    if k == "noalloc":
        inst = _grid(case["H"], case["W"], case["rate"], seed, 0, case.get("near", 0))
        words = torch.from_numpy(inst.words.view(np.int64)).cuda()
        return {"kind": k, "inst": inst, "words": words,
                "path": torch.empty(inst.H * inst.W + 1, dtype=torch.int32, device="cuda"),
                "result": torch.zeros(ctypes.sizeof(L.NoallocGridResult) // 8, dtype=torch.int64, device="cuda")}
    if k in ("puzzles", "bounded"):
        return {"kind": k, "eng": _engine("puzzle", (case["n"],)), "n": case["n"], "boards": _boards(case, seed),
                "log2_slots": case.get("log2_slots", 0)}
    if k == "tables":
        return {"kind": k, "eng": _engine("tables"), "n": case["n"], "boards": _boards(case, seed)}
    if k == "batch":
        return {"kind": k, "eng": _engine("batch", (4,)), "insts": _mixture(case, seed)}
    if k == "serve":
        fresh = "serve" not in _ENGINES
        eng = _engine("serve", (4,))
        if fresh:
            eng.serve_start(hbm_budget_gb=32.0)
        return {"kind": k, "eng": eng, "insts": _mixture(case, seed)}
    raise ValueError(f"unknown kind {k}")


# -------------------------------------------------------------------- runs
def _grid_out(sol, path):
    found = [sol.status, sol.straight, sol.diagonal, len(path), path[0], path[-1]]
    return {"cost": float(sol.cost_exact), "found": np.array(found)}


def _solve_boards(eng, n, boards):
    out = []
    for b in boards:
        s = eng.puzzle_solve(n, b)
        out.append([s.status, s.steps, len(eng.puzzle_moves())])
    return np.array(out)


def _result_rows(rows):
    return np.array([[r["status"], r["steps"], r["straight"], r["diagonal"]] for r in rows])


def run(state):
    k = state["kind"]
    if k == "grid":
        g = state["inst"]
        sol = state["eng"].grid_solve(g.words, g.H, g.W, g.start, g.goal)
        return _grid_out(sol, state["eng"].grid_path())
    if k == "queries":
        g, eng, out = state["inst"], state["eng"], []
        eng.grid_load(g.words, g.H, g.W)
        for s, t in state["ends"]:
            out.append(_grid_out(eng.grid_solve_loaded(s, t), eng.grid_path()))
        return out
    if k == "noalloc":
        g = state["inst"]
        rc = L.load().uastar_grid_solve_noalloc(
            ctypes.c_void_p(state["words"].data_ptr()), g.H, g.W, g.start[0], g.start[1], g.goal[0], g.goal[1],
            ctypes.c_void_p(state["path"].data_ptr()), state["path"].numel(),
            ctypes.c_void_p(state["result"].data_ptr()), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
        if rc != L.OK:
            raise RuntimeError(f"uastar_grid_solve_noalloc: {rc}")
        # the record's status, straight, diagonal and path length words, and the path's first cell
        return [state["result"][0:3], state["result"][6:7], state["path"][0:1]]
    if k == "puzzles":
        return _solve_boards(state["eng"], state["n"], state["boards"])
    if k == "tables":
        state["eng"].pdb_build(state["n"])
        return _solve_boards(state["eng"], state["n"], state["boards"])
    if k == "bounded":
        out = []
        for b in state["boards"]:
            r = state["eng"].puzzle_solve_bounded(state["n"], b, state["log2_slots"])
            out.append([r["status"], r["steps"], r["lower_bound"], len(state["eng"].puzzle_moves())])
        return np.array(out)
    if k == "batch":
        rows, _ = state["eng"].batch_solve(state["insts"])
        return _result_rows(rows)
    if k == "serve":
        eng = state["eng"]
        ids = [eng.serve_submit(i) for i in state["insts"]]
        got = {}
        while len(got) < len(ids):
            done = eng.serve_poll()
            got.update(done)
            if not done:
                time.sleep(0.0002)
        return _result_rows([got[i] for i in ids])
    raise ValueError(f"unknown kind {k}")


# ------------------------------------------------------------ work and truth
def work(case):
    """Bytes a solve cannot do without: its map or board in, its path out (and the tables it builds)."""
    k = case["kind"]

    def grid(h, w):
        return h * w / 8 + 4 * (h + w)

    def board(n):
        return n * n + 4 * {3: 24, 4: 50, 5: 60}[n]

    if k in ("grid", "noalloc"):
        b = grid(case["H"], case["W"])
    elif k == "queries":
        b = case["H"] * case["W"] / 8 + case["queries"] * 2 * (case["H"] + case["W"])
    elif k in ("puzzles", "bounded"):
        b = case["count"] * board(case["n"])
    elif k == "tables":
        b = case["count"] * board(case["n"]) + {3: 362880, 4: 576576000, 5: 510048000}[case["n"]]
    else:
        side = (256 + case["max_side"]) / 2
        b = case["puzzles"] * board(4) + case["grids"] * grid(side, side)
    return {"bytes": float(b), "flops": 0.0}


def _astar(cells, H, W, start, goal):
    """Exact optimal cost by sequential A* in float64 on a list of 0/1 cells."""
    gx, gy = goal

    def h(x, y):
        dx, dy = abs(x - gx), abs(y - gy)
        return max(dx, dy) + (SQRT2 - 1.0) * min(dx, dy)

    s, t = start[0] * W + start[1], gx * W + gy
    best = {s: (0, 0)}
    closed = set()
    heap = [(h(*start), s)]
    while heap:
        _, u = heapq.heappop(heap)
        if u == t:
            a, d = best[u]
            return a + d * SQRT2
        if u in closed:
            continue
        closed.add(u)
        x, y = divmod(u, W)
        if not cells[u]:
            continue
        a, d = best[u]
        for dx in (-1, 0, 1):
            for dy in (-1, 0, 1):
                p, q = x + dx, y + dy
                if (not dx and not dy) or not (0 <= p < H and 0 <= q < W):
                    continue
                v = p * W + q
                if v in closed or not (cells[v] or v == t):
                    continue
                c = (a, d + 1) if dx and dy else (a + 1, d)
                old = best.get(v)
                if old is None or c[0] + c[1] * SQRT2 < old[0] + old[1] * SQRT2 - 1e-9:
                    best[v] = c
                    heapq.heappush(heap, (c[0] + c[1] * SQRT2 + h(p, q), v))
    return math.inf


def exact(case, seed):
    """Optimal grid costs in 64 bits.  The other outputs are whole numbers."""
    k = case["kind"]
    if k not in ("grid", "queries") or case["H"] * case["W"] * case.get("queries", 1) > 1_200_000:
        return None
    g = _grid(case["H"], case["W"], case["rate"], seed, 0, case.get("near", 0))
    bits = np.unpackbits(np.asarray(g.words).view(np.uint8), bitorder="little")[: g.H * g.W].tolist()
    ends = _ends(g, case["queries"], seed) if k == "queries" else [(g.start, g.goal)]
    out = [{"cost": _astar(bits, g.H, g.W, a, b), "found": None} for a, b in ends]
    return out if k == "queries" else out[0]
