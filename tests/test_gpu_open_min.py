"""The minimum over a paused search's open list (ga_open.cuh k_best_open): it
must be the least current entry also where all of a heap's least entries are
stale, since the memory-bounded mode takes it for a lower bound.

The result is a whole number: it must be identical to the host's."""
from __future__ import annotations

import subprocess
from pathlib import Path

import pytest

from uastar_gb300 import build as B

pytestmark = pytest.mark.gpu
ROOT = Path(__file__).resolve().parents[1]


def test_least_current_entry_of_parked_heaps(tmp_path):
    exe = tmp_path / "open_min"
    subprocess.run([B._nvcc(), *B.ARCH, "-O1", "-std=c++17", "--expt-relaxed-constexpr", "-o", str(exe),
                    str(ROOT / "tests" / "cuda" / "open_min.cu")], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout
