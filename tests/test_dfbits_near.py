"""Scaled rounding to integers by bit patterns (csrc/dfbits.cuh, the digit slicing of the
FP64-accurate products) against exact rational arithmetic on the CPU: halves away from zero."""
import os
import shutil
import subprocess
from fractions import Fraction

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


def nearest(x, sh):
    v = abs(Fraction(x)) * Fraction(2) ** sh
    q = int(v + Fraction(1, 2))
    return -q if x < 0 else q


def test_near_int(tmp_path):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("g++ not available")
    exe = str(tmp_path / "near")
    subprocess.run([gxx, "-O2", "-std=c++17", "-o", exe, os.path.join(HERE, "native", "dfbits_near_driver.cpp")], check=True)
    rng = np.random.default_rng(5)
    x, sh = [], []
    for s in range(2, 9):  # a row of exponent e: |x| < 2^e, sh = 6 - e + 7 (s - 1)
        for e in (-1000, -300, 0, 1, 300, 900):
            v = rng.uniform(-1, 1, 60) * 2.0 ** e * np.exp2(-rng.integers(0, 70, 60).astype(float))
            v[0], v[1], v[2] = np.nextafter(2.0 ** e, 0), -np.nextafter(2.0 ** e, 0), 0.0
            t = 6 - e + 7 * (s - 1)
            with np.errstate(under="ignore", over="ignore"):
                v[3:13] = np.ldexp(rng.integers(-40, 40, 10) + 0.5, -t)  # halves
            x.append(v)
            sh.append(np.full(60, t))
    x.append(np.array([np.inf, -np.inf, np.nan, 5e-324, -0.0, 2.0 ** 60, 5e-324]))
    sh.append(np.array([48, 48, 48, 48, 48, 0, 1074]))
    x, sh = np.concatenate(x), np.concatenate(sh).astype(np.int64)
    buf = np.empty(len(x), dtype=[("x", "<f8"), ("s", "<i8")])
    buf["x"], buf["s"] = x, sh
    out = np.frombuffer(subprocess.run([exe], input=buf.tobytes(), capture_output=True, check=True).stdout, dtype="<i8").reshape(-1, 2)
    fin = np.isfinite(x)
    assert not out[~fin, 0].any()
    assert out[-2, 0] == 0 and out[-1, 0] == 0  # beyond 2^55; a denormal that does not vanish
    normal = fin & ((np.abs(x) >= 2.0 ** -1022) | (x == 0)) & (sh < 1000)
    big = np.zeros(len(x), bool)
    big[-2] = True
    assert out[normal & ~big, 0].all()
    for i in np.flatnonzero(out[:, 0]):
        assert out[i, 1] == nearest(x[i], int(sh[i])), (x[i], sh[i])
