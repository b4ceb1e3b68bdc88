"""RECYCLE and LONG kernels on the CPU (csrc/recycle.cuh, csrc/longline.cuh), and
the literal factors of the long primes.

The GPU kernels are variants of their extents and are run with all others by
test_gpu_parity.py."""
import ctypes

import numpy as np
import pytest

import oracle
from conftest import field
from test_hostcheck import C64_TOL, C128_TOL, run

# (shape, precision, ring planes, rows of a chunk, batch): batches below, at and above the emulated grid of 3
RECYCLE = [((16, 16, 32), 0, 27, 8, 8), ((23, 23, 23), 0, 23, 12, 2), ((23, 23, 23), 0, 27, 12, 7),
           ((24, 24, 24), 0, 24, 8, 3), ((30, 30, 30), 1, 30, 10, 4), ((16, 16, 16), 0, 16, 8, 10)]
# (shape, precision, outputs a task, volumes a CTA, batch): whole and partial groups
LONG = [((97, 2, 1), 0, 6, 16, 33), ((83, 2, 1), 0, 6, 16, 16), ((47, 3, 2), 0, 8, 8, 11),
        ((97, 2, 1), 1, 4, 16, 1), ((83, 2, 1), 1, 7, 16, 20), ((47, 3, 2), 1, 8, 8, 17)]


def check(hostcheck, shape, prec, sign, alg, vpc, nvol):
    rng = np.random.default_rng(12000 + sum(shape) + alg + nvol)
    x = field(rng, (nvol,) + shape, dist="normal", dtype=np.complex128 if prec == 0 else np.complex64)
    got = run(hostcheck, x, shape, prec, sign, alg, vpc)
    x64 = x.astype(np.complex128)
    want = oracle.fft3d(x64) if sign < 0 else oracle.ifft3d(x64)
    # the tolerances of the other passes: the same line sums, or direct sums of at most 97 terms in double
    assert oracle.rel_error_per_volume(got, want).max() < (C128_TOL if prec == 0 else C64_TOL)


@pytest.mark.parametrize("shape,prec,planes,rows,nvol", RECYCLE)
@pytest.mark.parametrize("sign", [-1, +1])
def test_recycled_rows(hostcheck, shape, prec, planes, rows, nvol, sign):
    check(hostcheck, shape, prec, sign, 900 + planes, rows, nvol)


@pytest.mark.parametrize("shape,prec,outputs,vpc,nvol", LONG)
@pytest.mark.parametrize("sign", [-1, +1])
def test_long_prime_lines(hostcheck, shape, prec, outputs, vpc, nvol, sign):
    check(hostcheck, shape, prec, sign, 2000 + outputs, vpc, nvol)


@pytest.mark.parametrize("n", [19, 23])
def test_literal_factors_are_the_tables(hostcheck, n):
    lit, tab = np.zeros((n, 2)), np.zeros((n, 2))
    hostcheck.hostcheck_literal_factors.argtypes = [ctypes.c_int, ctypes.c_void_p, ctypes.c_void_p]
    assert hostcheck.hostcheck_literal_factors(n, lit.ctypes.data, tab.ctypes.data) == 0
    assert np.array_equal(lit, tab)
