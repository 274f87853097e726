"""The memory that the memory-bounded mode's exact phase takes beside the table:
less than a table of 2^24 slots, and none that it could not do without.

Boards that need several segments at 2^16 slots.  Without memory for the exact
phase the segments' solution must come back, as with the phase switched off;
with memory for few roots the answer is the optimum all the same."""
from __future__ import annotations

import subprocess
import sys
from pathlib import Path

import pytest

from uastar_gb300 import Engine
from uastar_gb300 import _lib as L
from uastar_gb300 import build as B
from uastar_gb300 import engine as E

pytestmark = pytest.mark.gpu
ROOT = Path(__file__).resolve().parents[1]
CAP = 16


def board():
    return E.gen_puzzle(1008, 4, 200)  # 46 moves, 0.3 M states


def test_footprint():
    torch = pytest.importorskip("torch")
    # (the stacks of the passes' threads belong to the process: there before the measurement)
    with Engine(0, exact_ms=30000) as first:
        first.pdb_build(4)
        assert first.puzzle_solve_bounded(4, board(), CAP)["exact_optimal"] == 1
    with Engine(0, exact_ms=30000) as eng, Engine(0, exact_ms=-1) as without:
        used = []
        for e in (without, eng):
            e.pdb_build(4)
            e.puzzle_solve_bounded(4, E.gen_puzzle(900, 4, 10), CAP)
            before = torch.cuda.mem_get_info(0)[0]
            r = e.puzzle_solve_bounded(4, board(), CAP)
            assert r["status"] == L.OK and r["segments"] > 1
            used.append(before - torch.cuda.mem_get_info(0)[0])
        assert used[1] - used[0] <= 16 * 2**24 * 0.6, used


CHILD = """
import ctypes, sys
sys.path[:0] = [sys.argv[2], sys.argv[2] + "/tests"]
from pathlib import Path
from uastar_gb300 import _lib as L
L.LIB_PATH = Path(sys.argv[1])
from uastar_gb300 import Engine
import test_gpu_bounded_memory as T
limit = L.load().fake_malloc_limit
limit.argtypes = [ctypes.c_size_t]
for bytes_, passes in ((100 << 10, False), (8 << 20, True)):
    with Engine(0, exact_ms=30000) as eng:
        eng.pdb_build(4)
        want = eng.puzzle_solve(4, T.board()).steps
        # (an easy board: the table and the heaps are there, the exact phase's memory not yet)
        assert eng.puzzle_solve_bounded(4, T.E.gen_puzzle(900, 4, 10), T.CAP)["segments"] == 1
        limit(bytes_)
        r = eng.puzzle_solve_bounded(4, T.board(), T.CAP)
        limit(2**64 - 1)
        assert r["status"] == L.OK and r["segments"] > 1, r
        assert r["lower_bound"] <= want <= r["steps"] == len(eng.puzzle_moves()), r
        assert (r["exact_passes"] > 0) == passes and r["exact_optimal"] == int(passes), r
        assert not passes or r["steps"] == want, r
        r = eng.puzzle_solve_bounded(4, T.board(), T.CAP)
        assert r["exact_optimal"] == 1 and r["steps"] == want, r
"""


def test_without_the_memory(tmp_path):
    lib = tmp_path / "libuastar_fake.so"
    objs = [B.OUT_DIR / (s + ".o") for s in B.CUDA_SOURCES + B.HOST_SOURCES]
    subprocess.run(["g++", "-O1", "-fPIC", "-c", str(ROOT / "tests" / "cpp" / "fake_malloc.cpp"), "-o",
                    str(tmp_path / "fake.o")], check=True)
    subprocess.run([B._nvcc(), *B.ARCH, "-shared", "-o", str(lib), *map(str, objs), str(tmp_path / "fake.o"),
                    "-Xlinker", "--wrap=cudaMalloc", "-lpthread"], check=True)
    r = subprocess.run([sys.executable, "-c", CHILD, str(lib), str(ROOT)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stderr[-2000:]
