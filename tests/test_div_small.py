"""Quotients by integers from a rounded reciprocal (csrc/divsmall.cuh, the Legendre recurrences) against
the division, on the CPU: every divisor that a table or a rule reaches (l <= 8,532, n <= 12,800), at random
numerators and at those whose quotients lie next to midpoints of two numbers."""
import os
import shutil
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


def test_div_small(tmp_path):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("g++ not available")
    exe = str(tmp_path / "div")
    subprocess.run([gxx, "-O2", "-std=c++17", "-ffp-contract=off", "-o", exe,
                    os.path.join(HERE, "native", "divsmall_driver.cpp")], check=True)
    rng = np.random.default_rng(11)
    c = np.arange(1, 12801)
    n = [rng.uniform(-1, 1, c.size) * np.exp2(rng.integers(-300, 300, c.size).astype(float)) for _ in range(8)]
    for _ in range(24):
        # the 53-bit n next to (m + 1/2) c for a random 53-bit m
        m = rng.integers(2**52, 2**53, c.size)
        for k in (-1, 0, 1):
            num = [(2 * int(a) + 1) * int(b) for a, b in zip(m, c)]  # 2 n
            sh = [max(0, x.bit_length() - 54) for x in num]
            n.append(np.array([float(((x >> (s + 1)) + k) << s) for x, s in zip(num, sh)]))
    n.append(np.zeros(c.size))
    num, den = np.concatenate(n), np.tile(c.astype(float), len(n))
    buf = np.stack([num, den], 1)
    out = np.frombuffer(subprocess.run([exe], input=buf.tobytes(), capture_output=True, check=True).stdout).reshape(-1, 2)
    assert out.shape == buf.shape and np.array_equal(out[:, 0], out[:, 1])
