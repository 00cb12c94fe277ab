"""Every arithmetic a limb can take, by the size of its prime, in one context:
primes of 56 bits and more (Harvey butterflies), smaller ones (three-product
quotients, or the FP64 pipes below 50 bits), and the tensor-core conversions'
reduction from 18- to 61-bit targets.  NTT and HMult + rescale bit-exact against
the oracle, random and extreme residues, integer and FP64 variants."""
import numpy as np
import pytest

from gpu_helpers import device_status, from_dev, rand_ct, rand_key, to_dev
from test_exact_arith import _is_prime

pytestmark = pytest.mark.gpu


def _pair(logN, qbits, pbits, dnum):
    import pyfideslib_b200 as F
    from oracle import oracle as O

    used = []
    for b in list(qbits) + list(pbits):  # the largest unused b-bit prime = 1 mod 2N
        step = 2 << logN
        used.append(next(x for x in range((1 << b) - step + 1, 1 << (b - 1), -step) if x not in used and _is_prime(x)))
    q, p = used[:len(qbits)], used[len(qbits):]
    cc = F.CryptoContext(log_n=logN, num_q=len(q), dnum=dnum, q=np.array(q, dtype=np.uint64),
                         p=np.array(p, dtype=np.uint64), scale=2.0 ** 30)
    return cc, O.Ctx(logN, cc.q, cc.p, dnum)


@pytest.mark.parametrize("logN", [10, 13])
@pytest.mark.parametrize("variant", [3, 9])
@pytest.mark.parametrize("conv", [0, 3, 4])
def test_mixed_prime_sizes_bitexact(logN, variant, conv):
    from pyfideslib_b200._capi import lib

    cc, oc = _pair(logN, [60, 50, 59, 41, 40, 33, 26, 61, 45, 20 if logN == 10 else 24, 49, 18 if logN == 10 else 22], [61, 60, 59, 61], 3)
    cc.set_ntt_variant(variant)
    assert lib.fides_set_conv_accumulator(cc._h, conv) == 0
    pid = list(range(len(cc.q) + len(cc.p)))
    x = oc.random(pid, 5)
    for i in pid[::2]:
        x[i] = oc.primes[i] - 1
        x[i, 1::3] = 0
    d = to_dev(x)
    cc.ntt(d.data_ptr(), 0, len(pid))
    assert np.array_equal(from_dev(d), oc.ntt(x, pid))
    cc.ntt(d.data_ptr(), 0, len(pid), inverse=True)
    assert np.array_equal(from_dev(d), x)
    kb, ka = rand_key(oc, 7)
    cc.upload_relin_key(kb, ka)
    for lv in (11, 7, 3):
        a, b = rand_ct(oc, lv, 40 + lv), rand_ct(oc, lv, 50 + lv)
        pm1 = np.array([oc.primes[i] - 1 for i in range(lv + 1)], dtype=np.uint64)[:, None]
        a = (a[0], np.ascontiguousarray(np.broadcast_to(pm1, a[1].shape)))
        got = cc.EvalMult(cc.upload(*a), cc.upload(*b), rescale=True).download()
        want = oc.hmult(lv, *a, *b, kb, ka, rescale=True)
        assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1]), lv
    assert device_status(cc) == 0


@pytest.mark.parametrize("small", ["q", "p"])
def test_moduli_below_17_bits_leave_the_tensor_cores(small):
    """The tensor-core reduction needs moduli above 2^17: with a smaller one among
    the ciphertext or the special moduli its variants are refused and every other
    one is exact."""
    from pyfideslib_b200._capi import lib

    cc, oc = _pair(9, [50, 40, 16 if small == "q" else 30, 18, 45], [60, 59, 14 if small == "p" else 58], 3)
    for conv in (3, 4):
        assert lib.fides_set_conv_accumulator(cc._h, conv) != 0
    kb, ka = rand_key(oc, 7)
    cc.upload_relin_key(kb, ka)
    for conv in (-1, 0, 2):
        assert lib.fides_set_conv_accumulator(cc._h, conv) == 0
        for lv in (4, 3, 2, 1):
            a, b = rand_ct(oc, lv, 40 + lv), rand_ct(oc, lv, 50 + lv)
            got = cc.EvalMult(cc.upload(*a), cc.upload(*b), rescale=True).download()
            want = oc.hmult(lv, *a, *b, kb, ka, rescale=True)
            assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1]), (conv, lv)
