"""CPU checks of the exactness arguments behind the FP64 and tensor-core paths.

The CUDA kernels compute the same residues as the integer arithmetic only
because of value bounds (fp64.cuh, ks.cu, conv_tc.cu; the transforms' in
test_ntt_sched.py).  These tests restate the device arithmetic on the host and
run it against exact integer arithmetic on the cases the bounds are tight for
(tests/exact_arith_emu.c, C99 fma):

* the FP64 key-switch sums of rotations, and of products with their tensor
  product: up to 8 digits, the signed own-digit product, digit values as the
  row pass leaves them, maximal operands;
* the FP64 plaintext dot products in runs of seven, and element-wise products;
* the int8-split conversion: byte layout of A and B in the canonical K-major
  shared-memory form, the matrix product of the tensor-core MMAs, the
  reassembly of V' and its reduction by a 32-bit quotient for every prime size
  and digit size, the lift of a dropped top limb (numpy / Python ints).
The GPU parity tests then check the kernels themselves against the oracle.
"""
import ctypes
import math
import os
import random
import subprocess
from fractions import Fraction

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


def _is_prime(n):
    if n < 2:
        return False
    for a in (2, 3, 5, 7, 11, 13, 17, 19, 23, 29, 31, 37):
        if n % a == 0:
            return n == a
    d, s = n - 1, 0
    while d % 2 == 0:
        d //= 2
        s += 1
    for a in (2, 3, 5, 7, 11, 13, 17, 19, 23, 29, 31, 37):
        x = pow(a, d, n)
        if x in (1, n - 1):
            continue
        for _ in range(s - 1):
            x = x * x % n
            if x == n - 1:
                break
        else:
            return False
    return True


def _ntt_primes(top, count, two_n=1 << 17):
    out, p = [], (top - 1) // two_n * two_n + 1
    while len(out) < count:
        if p < top and _is_prime(p):
            out.append(p)
        p -= two_n
    return out


def _psi(p, two_n=1 << 17):
    rng = random.Random(p)
    while True:
        w = pow(rng.randrange(2, p - 1), (p - 1) // two_n, p)
        if pow(w, two_n // 2, p) == p - 1:
            return w


@pytest.fixture(scope="module")
def emu(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("emu") / "libemu.so")
    subprocess.run(["gcc", "-O2", "-ffp-contract=off", "-frounding-math", "-shared", "-fPIC",
                    os.path.join(HERE, "exact_arith_emu.c"), "-o", out, "-lm"], check=True)
    lib = ctypes.CDLL(out)
    u64, i32 = ctypes.c_uint64, ctypes.c_int
    lib.emu_ks_check.argtypes = [u64, i32, i32, u64, i32, i32]
    lib.emu_hmult_check.argtypes = [u64, i32, i32, i32, u64, i32, i32]
    lib.emu_dot_check.argtypes = [u64, i32, i32, u64, i32, i32]
    return lib


PRIMES_50 = _ntt_primes(1 << 50, 3) + _ntt_primes((1 << 49) + (1 << 47), 1)


@pytest.mark.parametrize("p", PRIMES_50[:2])
def test_fp64_keyswitch_sums_exact(emu, p):
    for nd in range(1, 7):
        for c0 in (0, 1):
            assert emu.emu_ks_check(p, nd, c0, nd, 20000, 0) == 0, nd
            assert emu.emu_ks_check(p, nd, c0, nd, 4, 1) == 0, nd


@pytest.mark.parametrize("p", PRIMES_50)
def test_fp64_product_sums_exact(emu, p):
    """Up to 8 digits in the kernel of its own, up to 6 fused into the row pass
    (lazy digit values); own: the digit of the limb, -1 for a special limb."""
    for lazy in (0, 1):
        for nd in range(1, 7 if lazy else 9):
            for own in range(-1, nd):
                assert emu.emu_hmult_check(p, nd, own, lazy, 10 * nd + own, 2000, 0) == 0, (lazy, nd, own)
                assert emu.emu_hmult_check(p, nd, own, lazy, 1, 16, 1) == 0, (lazy, nd, own)


@pytest.mark.parametrize("p", PRIMES_50)
def test_fp64_dot_products_exact(emu, p):
    for n in (1, 6, 7, 8, 15, 64):
        for accumulate in (0, 1):
            assert emu.emu_dot_check(p, n, accumulate, n, 2000, 0) == 0, n
            assert emu.emu_dot_check(p, n, accumulate, n, 2, 1) == 0, n


M32, M64 = (1 << 32) - 1, (1 << 64) - 1


def _tc_mod(p, cnt):
    """conv_tc.cu tc_mod: (s, k, M), from the context's double 1/p (rounded up below 2^50)."""
    inv = 1.0 / float(p)
    if p < 1 << 50 and Fraction(inv) * p < 1:
        inv = math.nextafter(inv, 1.0)
    bits = p.bit_length()
    s = max(16, bits + (2040 * cnt).bit_length() - 32)
    k = max(0, bits - 1 - s)
    m = int(math.ldexp(inv, 32 + k + s))
    assert 0 < m - 1 <= M32  # the device's 32 bits hold it
    return s, k, m - 1


def _reduce_cols(c, p, mod):
    """conv_tc.cu reduce_cols in 32- and 64-bit words."""
    s, k, M = mod
    w = [c[2 * i] + (c[2 * i + 1] << 8) for i in range(4)]
    assert max(w) <= M32
    e, o = (w[2] << 32) | w[0], (w[3] << 32) | w[1]
    h = (e >> 16) + o
    T = h >> (s - 16)
    assert h <= M64 and s - 16 < 32 and T <= M32
    q = (T * M >> 32) >> k
    np_ = -p & M64
    a = (q * (np_ & M32) + e) & M64
    r = (a + (((q * (np_ >> 32)) & M32) << 32) + (o << 16)) & M64
    assert r < 2 * p, (p, q)
    return r if r < p else r - p


def _conv_tc_emulate(ck, cnt, ntar, bits, seed):
    """Byte layouts, MMA and epilogue of the pre-shifted int8 conversion;
    returns the number of outputs that differ from sum_i x_i M_i mod p."""
    rnd = random.Random(seed)
    rows, lbo_a = 128, 2048
    ntar2 = (ntar + 1) & ~1
    lbo_b = ntar2 * 128
    A = np.zeros(2 * ck * lbo_a, np.uint8)
    B = np.zeros(2 * ck * lbo_b, np.uint8)
    ps = [rnd.randrange(2 ** (bits - 1), 2 ** bits) | 1 for _ in range(ntar)]
    x = [[(2 ** 62 - 1) if rnd.random() < 0.5 else rnd.randrange(2 ** 62) for _ in range(rows)] for _ in range(cnt)]
    M = [[ps[m] - 1 if rnd.random() < 0.5 else rnd.randrange(ps[m]) for m in range(ntar)] for _ in range(cnt)]
    for i in range(cnt):
        for r in range(rows):
            off = (i >> 1) * lbo_a + (r >> 3) * 128 + (r & 7) * 16 + (i & 1) * 8
            A[off:off + 8] = np.frombuffer(x[i][r].to_bytes(8, "little"), np.uint8)
    for u in range(2 * ck * ntar2):
        c, m = divmod(u, ntar2)
        mp = [0] * 16
        for h in range(2):
            i = 2 * c + h
            live = i < cnt and m < ntar
            v = M[i][m] if live else 0
            for a in range(8):
                mp[8 * h + a] = v
                if live and a < 7:
                    v = (v << 8) % ps[m]
        for sb in range(8):
            nn = m * 8 + sb
            off = c * lbo_b + (nn >> 3) * 128 + (nn & 7) * 16
            B[off:off + 16] = np.frombuffer(bytes((mp[pos] >> (8 * sb)) & 255 for pos in range(16)), np.uint8)

    def operand(buf, start, lbo, nrows):  # canonical K-major, no swizzle, K = 32 bytes
        idx = np.array([[start + (k // 16) * lbo + (r // 8) * 128 + (r % 8) * 16 + k % 16 for k in range(32)]
                        for r in range(nrows)])
        return buf[idx].astype(np.int64)

    bad = 0
    for m0 in range(0, ntar2, 32):
        nt = min(32, ntar2 - m0)
        D = np.zeros((rows, nt * 8), np.int64)
        for k in range(ck):
            D += operand(A, 2 * k * lbo_a, lbo_a, rows) @ operand(B, 2 * k * lbo_b + m0 * 128, lbo_b, nt * 8).T
        assert D.max() < 2 ** 23
        for mm in range(nt):
            m = m0 + mm
            if m >= ntar:
                continue
            p = ps[m]
            mod = _tc_mod(p, cnt)
            for r in range(0, rows, 3):
                res = _reduce_cols([int(v) for v in D[r, mm * 8:mm * 8 + 8]], p, mod)
                bad += res != sum(x[i][r] * M[i][m] for i in range(cnt)) % p
    return bad


@pytest.mark.parametrize("ck,cnt,ntar,bits", [(3, 10, 30, 50), (3, 10, 39, 60), (4, 15, 25, 62), (1, 3, 9, 50)])
def test_tensor_conversion_layout_exact(ck, cnt, ntar, bits):
    assert _conv_tc_emulate(ck, cnt, ntar, bits, ck * 100 + ntar) == 0


def _reduction_moduli():
    """18- to 62-bit odd numbers: the least and the greatest of each width, and others."""
    rnd = random.Random(11)
    for bits in range(18, 63):
        yield (1 << (bits - 1)) + 1
        yield (1 << bits) - 1
        yield rnd.randrange(1 << (bits - 1), 1 << bits) | 1


def test_tensor_conversion_reduction_bound():
    """The reassembly, the 32-bit quotient and its one correction for 18- to 62-bit
    moduli and digits of 1 to 16 limbs: V' at its greatest (bytes of 255 against
    constants p - 1), at multiples of p and beside them, and random."""
    rnd = random.Random(7)
    for p in _reduction_moduli():
        for cnt in (1, 2, 3, 4, 7, 10, 15, 16):
            mod = _tc_mod(p, cnt)
            cases = [([255] * 8 * cnt, [p - 1] * 8 * cnt), ([0] * 8 * cnt, [p - 1] * 8 * cnt),
                     ([1] + [0] * (8 * cnt - 1), [p - 1] * 8 * cnt), ([255, 1] + [255] * (8 * cnt - 2), [p - 1, 255] * 4 * cnt),
                     ([rnd.randrange(256) for _ in range(8 * cnt)], [rnd.randrange(p) for _ in range(8 * cnt)])]
            for xs, ms in cases:
                c = [sum(x * (m >> (8 * s) & 255) for x, m in zip(xs, ms)) for s in range(8)]
                v = sum(x * m for x, m in zip(xs, ms))
                assert v == sum(c[s] << (8 * s) for s in range(8)) and max(c) < 2 ** 23
                assert _reduce_cols(c, p, mod) == v % p, (p, cnt)


def test_tensor_conversion_top_limb_lift():
    """The fused ModDown adds the centred top limb: one conditional addition where
    the top modulus is below twice the target, else a reduction; v and tl at their
    ends and at the centring's edge."""
    rnd = random.Random(13)

    def signed(x):
        return x - (1 << 64) if x >> 63 else x

    for p in _reduction_moduli():
        for ql in {p + 2, 2 * p - 1, p - 2, p // 2 | 1, p // 5 | 1, 2 * p + 1, min(9 * p + 2, 2 ** 62 - 1), 2 ** 61 + 1} - {p}:
            for tl in (0, 1, ql // 2 - 1, ql // 2, ql // 2 + 1, ql - 1, rnd.randrange(ql)):
                for v in (0, 1, p // 2, p - 1, rnd.randrange(p)):
                    up = tl > ql >> 1
                    want = (v + tl - (ql if up else 0)) % p
                    if ql < 2 * p:  # kTcNear
                        x = (v + ((tl - ql) & M64 if up else tl) + (0 if up else -p & M64)) & M64
                        assert ((x + p) & M64 if signed(x) < 0 else x) == want, (p, ql, tl, v)
                    # also such a target's form beside one that is not near
                    sw = tl + (p - ql % p if up else 0)
                    assert sw <= M64
                    sw = sw % p if p < ql else sw
                    assert v + sw - (p if v + sw >= p else 0) == want, (p, ql, tl, v)
