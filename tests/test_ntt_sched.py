"""CPU check of the transforms' centring schedules (csrc/ntt_sched.hpp): the
double-precision forward and inverse with the compiled-in schedule, formed row
twiddles included, give the exact residues and stay inside every stated
bound, for every ring dimension, on primes just below 2^50 (where the bounds are
tight) and 40-bit ones, random, zero and extreme residues, the inverse also from
centred ones."""
import ctypes
import os
import subprocess

import pytest

from test_exact_arith import _ntt_primes, _psi

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def emu(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("emu") / "libsched.so")
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-frounding-math", "-shared", "-fPIC",
                    os.path.join(HERE, "ntt_sched_emu.cpp"), "-o", out], check=True)
    lib = ctypes.CDLL(out)
    lib.emu_sched_check.argtypes = [ctypes.c_int, ctypes.c_uint64, ctypes.c_uint64, ctypes.c_uint64, ctypes.c_int]
    return lib


@pytest.mark.parametrize("logn", range(8, 17))
def test_schedule_exact_and_bounded(emu, logn):
    two_n = 2 << logn
    for top in (1 << 50, 1 << 40):
        for p in _ntt_primes(top, 2, two_n):
            for pattern in range(4):
                assert emu.emu_sched_check(logn, p, _psi(p, two_n), 17 * logn + pattern, pattern) == 0, (p, pattern)
