"""The float32 shortcut of the exact cost comparison (ga_problems.cuh
sqrt2_sign) restated in numpy, with and without a fused multiply-add: wherever
its error bound lets it decide, it must agree with integers.  CPU only."""
from __future__ import annotations

import re
from pathlib import Path

import numpy as np

SRC = (Path(__file__).resolve().parents[1] / "uastar_gb300" / "csrc" / "ga_problems.cuh").read_text()
BOUND = np.float32(re.search(r"fabsf\(v\) > ([0-9.e-]+)f \* \(fabsf\(fd\) \+ 2\.f \* fabsf\(fe\)\)", SRC).group(1))
ROOT = np.float32(re.search(r"v = fd - ([0-9.]+)f \* fe;", SRC).group(1))


def exact(d: int, e: int) -> int:
    """sign(d - e * sqrt(2)) by squares."""
    if d >= 0 and e <= 0:
        return 0 if d == e == 0 else 1
    if d <= 0 and e >= 0:
        return -1
    s = (d * d > 2 * e * e) - (d * d < 2 * e * e)
    return s if d > 0 else -s


def pairs():
    rng = np.random.default_rng(3)
    for bits in (1, 3, 8, 16, 24, 31):
        for d, e in rng.integers(-(2**bits) + 1, 2**bits, (3000, 2)):
            yield int(d), int(e)
    p, q = 1, 1
    while p < 2**31:  # convergents of sqrt(2) and their neighbours
        for dp in range(-3, 4):
            for dq in range(-3, 4):
                for s in (1, -1):
                    if max(abs(p + dp), abs(q + dq)) < 2**31:
                        yield s * (p + dp), s * (q + dq)
        p, q = p + 2 * q, p + q


def test_shortcut_agrees_with_integers():
    decided = total = 0
    for d, e in pairs():
        fd, fe = np.float32(d), np.float32(e)
        for v in (np.float32(fd - np.float32(ROOT * fe)),  # two roundings
                  np.float32(np.float64(fd) - np.float64(ROOT) * np.float64(fe))):  # one
            total += 1
            if abs(v) > BOUND * np.float32(abs(fd) + np.float32(2) * abs(fe)):
                decided += 1
                assert (1 if v > 0 else -1) == exact(d, e), (d, e)
    assert decided > 0.8 * total  # it is a shortcut
