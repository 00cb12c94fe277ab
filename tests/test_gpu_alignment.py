"""Limbs that start at an odd word: the inverse transform takes them (a shifted
buffer, an odd stride between polynomials) with the same residues, the forward
one and the polynomial product's scratch need 16-byte boundaries and refuse."""
import numpy as np
import pytest

from gpu_helpers import from_dev, make_pair, to_dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("logN", [8, 9, 12, 16])
@pytest.mark.parametrize("variant", [3, 9])
def test_inverse_at_odd_words(logN, variant):
    cc, oc = make_pair(logN, 3, 1, 2)
    cc.set_ntt_variant(variant)
    pid, nl, N = [0, 1, 2, 3], 4, cc.N
    x = np.stack([oc.random(pid, 3 + logN + k) for k in range(3)])
    ev = np.stack([oc.ntt(v, pid) for v in x])
    buf = np.zeros(1 + nl * N, dtype=np.uint64)  # one polynomial, one word off
    buf[1:] = ev[0].ravel()
    d = to_dev(buf)
    cc.ntt(d.data_ptr() + 8, 0, nl, inverse=True)
    got = from_dev(d)
    assert got[0] == 0 and np.array_equal(got[1:].reshape(nl, N), x[0])
    stride = nl * N + 1  # every second polynomial one word off
    buf = np.zeros(3 * stride, dtype=np.uint64)
    for k in range(3):
        buf[k * stride:k * stride + nl * N] = ev[k].ravel()
    d = to_dev(buf)
    cc.ntt_batch(d.data_ptr(), stride, 3, 0, nl, inverse=True)
    got = from_dev(d)
    for k in range(3):
        assert np.array_equal(got[k * stride:k * stride + nl * N].reshape(nl, N), x[k]), k
        assert got[k * stride + nl * N] == 0


def test_forward_at_odd_words_is_refused():
    from pyfideslib_b200 import FidesError

    cc, oc = make_pair(9, 3, 1, 2)
    pid, nl, N = [0, 1, 2], 3, cc.N
    x = np.zeros(3 * (nl * N + 1) + 1, dtype=np.uint64)
    x[1:1 + nl * N] = oc.random(pid, 5).ravel()
    d, s = to_dev(x), to_dev(x)
    p, q = d.data_ptr(), s.data_ptr()
    for call in (lambda: cc.ntt(p + 8, 0, nl), lambda: cc.ntt_batch(p, nl * N + 1, 2, 0, nl),
                 lambda: cc.polymul(p, p, p, q + 8, q + 8 * (nl * N + 2), 0, nl)):
        with pytest.raises(FidesError):
            call()
    assert np.array_equal(from_dev(d), x)
    # operands of a product at odd words, the scratch on its boundary
    t = to_dev(np.zeros(2 * nl * N, dtype=np.uint64))
    cc.polymul(p + 8, p + 8, p + 8, t.data_ptr(), t.data_ptr() + 8 * nl * N, 0, nl)
    e = oc.ntt(x[1:1 + nl * N].reshape(nl, N), pid).astype(object)
    sq = (e * e % np.array(oc.primes[:nl], dtype=object)[:, None]).astype(np.uint64)
    got = from_dev(d)[1:1 + nl * N].reshape(nl, N)
    assert np.array_equal(oc.ntt(got, pid), sq)
