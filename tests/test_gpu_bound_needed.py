"""A puzzle's slots and entries hold g in 8 bits, which only a bound on f keeps
it in: ga_search refuses a puzzle search that is set up without one.

Status and move count are whole numbers: they must be identical."""
from __future__ import annotations

import subprocess
from pathlib import Path

import pytest

from uastar_gb300 import build as B

pytestmark = pytest.mark.gpu
ROOT = Path(__file__).resolve().parents[1]


def test_puzzle_without_a_bound_is_refused(tmp_path):
    exe = tmp_path / "bound_needed"
    subprocess.run([B._nvcc(), *B.ARCH, "-O1", "-std=c++17", "--expt-relaxed-constexpr", "-o", str(exe),
                    str(ROOT / "tests" / "cuda" / "bound_needed.cu")], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout
