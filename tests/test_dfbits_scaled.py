"""A float times a power of two as FP64 bits (csrc/dfbits.cuh, the final step of the
FP64-accurate tensor-core products), bit for bit against ldexp on the CPU."""
import os
import shutil
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


def test_scaled_matches_ldexp(tmp_path):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("g++ not available")
    exe = str(tmp_path / "scaled")
    subprocess.run([gxx, "-O2", "-std=c++17", "-o", exe, os.path.join(HERE, "native", "dfbits_scaled_driver.cpp")], check=True)
    rng = np.random.default_rng(3)
    u = rng.integers(0, 1 << 32, 40000, dtype=np.uint64).astype(np.uint32)
    e = rng.integers(-1000, 1001, 40000).astype(np.int32)
    edge = np.array([0, 1 << 31, 1, 0x007fffff, 0x00800000, 0x7f7fffff, 0x7f800000, 0xff800000, 0x7fc00000, 0x3f800000,
                     0xbf800001], dtype=np.uint32)
    ee = np.array([-2147483648, -891, -890, -149, 0, 149, 890, 891, 2147483647], dtype=np.int32)
    u = np.concatenate([u, np.repeat(edge, len(ee))])
    e = np.concatenate([e, np.tile(ee, len(edge))])
    out = subprocess.run([exe], input=np.stack([u, e.view(np.uint32)], 1).astype(np.uint32).tobytes(), capture_output=True,
                         check=True).stdout
    out = np.frombuffer(out, dtype=[("ok", "<i8"), ("x", "<f8")])
    f = u.view(np.float32)
    zero = (u << np.uint32(1)) == 0
    ex = (u >> 23) & 255
    covered = zero | ((ex > 0) & (ex < 255) & (np.abs(e.astype(np.int64)) <= 890))
    assert np.array_equal(out["ok"] == 1, covered)
    c = covered & ~zero
    assert np.array_equal(out["x"][c], np.ldexp(f[c].astype(np.float64), e[c]))
    assert np.array_equal(out["x"][zero].view(np.uint64), f[zero].astype(np.float64).view(np.uint64))
