"""The stage update's division by three equals the division, bit for bit: signed
zeros, subnormals, infinities, NaN, the largest values and random bit patterns
of every exponent."""
import ctypes
import os
import subprocess

import numpy as np

from cases import ROOT


def test_third_is_the_division(tmp_path):
    src, so = str(tmp_path / "third.cpp"), str(tmp_path / "third.so")
    with open(src, "w") as f:
        f.write('#include "dgp_round.h"\n'
                'extern "C" void thirds(const double* x, double* y, long n) {\n'
                '  for (long i = 0; i < n; ++i) y[i] = dgp::third(x[i]);\n}\n')
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-shared", "-fPIC",
                    "-I" + os.path.join(ROOT, "dg-parallel_b200", "csrc"), src, "-o", so], check=True)
    rng = np.random.default_rng(3)
    tiny = np.arange(2000, dtype=np.uint64)  # the smallest subnormals, around the smallest normal and the largest value
    edges = [tiny, np.uint64(0x0010000000000000) - tiny, np.uint64(0x0010000000000000) + tiny,
             np.uint64(0x0030000000000000) + tiny, np.uint64(0x7FF0000000000000) - tiny,
             np.array([0x7FF8000000000000], dtype=np.uint64)]
    bits = np.concatenate(edges + [rng.integers(0, 1 << 63, 1_000_000, dtype=np.uint64)])
    x = np.concatenate([bits, bits | np.uint64(1 << 63)]).view(np.float64)
    y = np.empty_like(x)
    p = ctypes.POINTER(ctypes.c_double)
    lib = ctypes.CDLL(so)
    lib.thirds(x.ctypes.data_as(p), y.ctypes.data_as(p), ctypes.c_long(len(x)))
    with np.errstate(all="ignore"):
        want = x / 3.0
    nan = np.isnan(want)
    assert np.isnan(y[nan]).all()
    assert np.array_equal(y[~nan].view(np.uint64), want[~nan].view(np.uint64))
