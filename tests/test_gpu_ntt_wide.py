"""The transforms' wide instances (launches of at most 640 or 768 threads per SM, one
thread per 16 coefficients) and narrow ones: bit-exact against the oracle on each side
of both lines, with the prologues and epilogues the library uses (products, rescale,
ModUp / ModDown scales through a rotation)."""
import numpy as np
import pytest

from gpu_helpers import device_status, from_dev, make_pair, rand_ct, rand_key, to_dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("logN", [9, 12, 13, 15, 16])
@pytest.mark.parametrize("variant", [3, 9])
def test_wide_and_narrow_bitexact(logN, variant):
    cc, oc = make_pair(logN, 3, 1, 2)
    cc.set_ntt_variant(variant)
    pid = list(range(4))
    lines = [t * 148 * 16 // (4 * cc.N) for t in (640, 768)]  # polynomials of 4 limbs up to each line
    for npoly in (1, lines[0], lines[0] + 1, lines[1], lines[1] + 1):
        x = np.stack([oc.random(pid, 10 * logN + k) for k in range(npoly)])
        for i in pid:
            x[-1, i] = oc.primes[i] - 1
            x[-1, i, ::3] = 0
        want = np.stack([oc.ntt(v, pid) for v in x])
        d = to_dev(x)
        cc.ntt_batch(d.data_ptr(), 4 * cc.N, npoly, 0, 4)
        assert np.array_equal(from_dev(d), want), npoly
        cc.ntt_batch(d.data_ptr(), 4 * cc.N, npoly, 0, 4, inverse=True)
        assert np.array_equal(from_dev(d), x), npoly


@pytest.mark.parametrize("logN", [9, 11, 13, 14, 15])
@pytest.mark.parametrize("variant", [3, 9])
def test_fused_modes_bitexact(logN, variant):
    cc, oc = make_pair(logN, 5, 2, 3)
    cc.set_ntt_variant(variant)
    a, b = oc.random(list(range(5)), 3), oc.random(list(range(5)), 4)
    da, db, dc, s0, s1 = (to_dev(v) for v in (a, b, np.zeros_like(a), np.zeros_like(a), np.zeros_like(a)))
    cc.polymul(da.data_ptr(), db.data_ptr(), dc.data_ptr(), s0.data_ptr(), s1.data_ptr(), 0, 5)
    pid = list(range(5))
    p = np.array(oc.primes[:5], dtype=object)[:, None]
    prod = (oc.ntt(a, pid).astype(object) * oc.ntt(b, pid).astype(object) % p).astype(np.uint64)
    d = to_dev(from_dev(dc))
    cc.ntt(d.data_ptr(), 0, 5)
    assert np.array_equal(from_dev(d), prod)
    kb, ka = rand_key(oc, 7)
    g = cc.rotation_galois(3)
    cc.upload_relin_key(kb, ka)
    cc.upload_galois_key(g, kb, ka)
    for lv in (4, 1):
        x, y = rand_ct(oc, lv, 40 + lv), rand_ct(oc, lv, 50 + lv)
        X, Y = cc.upload(*x), cc.upload(*y)
        got = cc.EvalMult(X, Y, rescale=True).download()
        want = oc.hmult(lv, *x, *y, kb, ka, rescale=True)
        assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1]), lv
        got = cc.EvalRotate(X, 3).download()
        want = oc.rotate(lv, *x, pow(g, -1, 2 * oc.N), kb, ka)
        assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1]), lv
        got = cc.Rescale(X).download()
        assert np.array_equal(got[0], oc.rescale(lv, x[0])) and np.array_equal(got[1], oc.rescale(lv, x[1])), lv
    assert device_status(cc) == 0
