"""The one-correction reciprocal and reciprocal square root of csrc/df64.cuh, built for the
host with g++ and checked against FP64."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.mark.parametrize("op", [0, 1])
def test_one_correction_reaches_double_float(tmp_path, op):
    out = str(tmp_path / "df64_fast.so")
    r = subprocess.run(["g++", "-O2", "-ffp-contract=off", "-std=c++17", "-shared", "-fPIC", "-o", out,
                        os.path.join(HERE, "df64_fast_host.cpp")], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    L = C.CDLL(out)
    P = C.POINTER(C.c_double)
    L.bd_df64_fast.argtypes = [C.c_int, P, C.c_int, P]
    rng = np.random.default_rng(op)
    a = np.concatenate([10.0 ** rng.uniform(-12, 12, 20000), 1.0 + rng.uniform(0, 11, 20000), 2.0 ** np.arange(-30, 31.0)])
    if op == 1:
        a = a * rng.choice([-1.0, 1.0], len(a))
    got = np.zeros(len(a))
    L.bd_df64_fast(op, a.ctypes.data_as(P), len(a), got.ctypes.data_as(P))
    ref = 1.0 / np.sqrt(a) if op == 0 else 1.0 / a
    # the input's own double-float rounding (2^-48) and a few units of 2^-47 of the result
    assert np.max(np.abs(got / ref - 1.0)) < 2.0 ** -45
