"""Conversions that the tensor-core kernels make by integer operations, in
place of the FP64 pipe's or the conversion unit's, against CUDA's own: bit for
bit, over every f32, every digit and accumulator that the bounds allow, and
integers of up to 62 bits at the edges of rounding."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    from block_gb300 import build

    out = str(tmp_path_factory.mktemp("conversions") / "conversions.so")
    csrc = os.path.join(ROOT, "block_gb300", "csrc", "cuda")
    subprocess.run([build._nvcc(), *build.ARCH, "-std=c++17", "-O3", "-Xcompiler", "-fPIC", "-shared", "-I", csrc, "-o", out,
                    os.path.join(ROOT, "tests", "conversions.cu")], check=True)
    so = ctypes.CDLL(out)
    for f in (so.check_f32_to_f64, so.check_integers, so.check_scaled):
        f.restype = ctypes.c_longlong
    return so


def test_every_f32(lib):
    assert lib.check_f32_to_f64() == 0


def test_digits_and_accumulators(lib):
    assert lib.check_integers() == 0


def test_scaled_integers(lib):
    rng = np.random.default_rng(3)
    a = [0, 1, -1, 2**53 - 1, 2**53, 2**53 + 1, 2**53 + 2, 2**53 + 3, 2**62 - 1, 2**61, -(2**62) + 1]
    for bits in range(1, 63):  # all ones, a half, just below and above a half of the last place
        a += [2**bits - 1, 2 ** (bits - 1)]
        if bits > 54:
            last = 2 ** (bits - 53)
            for odd in (0, 1):
                m = 2 ** (bits - 1) + odd * last
                a += [m + last // 2 + d for d in (-1, 0, 1)]
    a += [int(x) >> int(s) for x, s in zip(rng.integers(0, 2**62, 20000), rng.integers(0, 62, 20000))]
    a = np.array([v for v in a if v < 2**62], np.int64)
    a = np.concatenate([a, -a])
    p = a.ctypes.data_as(ctypes.POINTER(ctypes.c_longlong))
    assert lib.check_scaled(p, a.size) == 0
