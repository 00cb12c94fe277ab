"""HMult with the tensor product inside the key switch (no tensor kernel): against
the oracle at every level, with and without rescale, for the integer and FP64
arithmetics and sums, one to eight digits, the inner product on its own or fused into the digits' row
pass (in one launch or two), squares, extreme residues, and inputs at mixed levels
in one batch."""
import numpy as np
import pytest

from gpu_helpers import device_status, make_pair, rand_ct, rand_key

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("logN,L,K,dnum", [(9, 5, 2, 3), (12, 7, 3, 3), (13, 6, 1, 6), (11, 3, 3, 1),
                                           (10, 7, 1, 7), (12, 8, 1, 8), (9, 15, 2, 8)])
@pytest.mark.parametrize("variant,ks", [(9, 1), (9, 0), (9, 11), (9, 3), (9, 10), (3, 1), (3, 0), (3, 11), (3, 2)])
def test_tensor_in_key_switch_bitexact(logN, L, K, dnum, variant, ks):
    from pyfideslib_b200._capi import lib

    cc, oc = make_pair(logN, L, K, dnum)
    kb, ka = rand_key(oc, 7)
    cc.upload_relin_key(kb, ka)
    cc.set_ntt_variant(variant)
    assert lib.fides_set_keyswitch_variant(cc._h, ks) == 0
    raw, A, B = [], [], []
    for lv in range(L):
        a, b = rand_ct(oc, lv, 40 + lv), rand_ct(oc, lv, 50 + lv)
        if lv % 2:
            pm1 = np.array([oc.primes[i] - 1 for i in range(lv + 1)], dtype=np.uint64)[:, None]
            a = tuple(np.ascontiguousarray(np.broadcast_to(pm1, v.shape)) for v in a)
            b = (a[0], b[1])
        raw.append((a, b))
        A.append(cc.upload(*a))
        B.append(cc.upload(*b))
    for rescale in (True, False):
        outs = cc.EvalMultBatch(A, B, rescale=rescale)
        for lv in range(L):
            want = oc.hmult(lv, *raw[lv][0], *raw[lv][1], kb, ka, rescale=rescale and lv > 0)
            got = outs[lv].download()
            assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1]), (lv, rescale)
    got = cc.EvalSquare(A[-1], rescale=True, out=A[-1]).download()  # the output may be the input
    want = oc.hmult(L - 1, *raw[-1][0], *raw[-1][0], kb, ka, rescale=True)
    assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1])
    assert device_status(cc) == 0
