"""The warp-local row passes and 16-column tiles at every shape of the warp
tile: N = 256 (16 lanes, one warp per limb), 512 and 1024 (one and two warps
per limb), 2048 and up (four warps per CTA); one to three row stages in the
second register group.  Bit-exact against the oracle, integer and
double-precision arithmetic, single and batched, on random and extreme
residues; the fused key-switch row pass with and without the split launch."""
import numpy as np
import pytest

from gpu_helpers import from_dev, make_pair, rand_ct, rand_key, to_dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("logN", [8, 9, 10, 11, 13, 15])
@pytest.mark.parametrize("variant", [3, 9])
def test_warp_tiles_bitexact(logN, variant):
    cc, oc = make_pair(logN, 5, 2, 2)
    nl = 7
    pid = list(range(nl))
    cc.set_ntt_variant(variant)
    x = np.stack([oc.random(pid, 31 + logN), oc.random(pid, 32 + logN), oc.random(pid, 33 + logN)])
    for i in pid:  # extremes in the second polynomial
        x[1, i] = oc.primes[i] - 1
        x[1, i, ::2] = 0
    want = np.stack([oc.ntt(v, pid) for v in x])
    d = to_dev(x)
    cc.ntt_batch(d.data_ptr(), nl * cc.N, 3, 0, nl)
    assert np.array_equal(from_dev(d), want)
    cc.ntt_batch(d.data_ptr(), nl * cc.N, 3, 0, nl, inverse=True)
    assert np.array_equal(from_dev(d), x)


@pytest.mark.parametrize("logN,dnum", [(9, 2), (11, 5), (13, 6)])
@pytest.mark.parametrize("ks", [1, 3, 11])
def test_fused_keyswitch_rows_bitexact(logN, dnum, ks):
    from pyfideslib_b200._capi import lib

    cc, oc = make_pair(logN, 6, 1, dnum) if dnum == 6 else make_pair(logN, 6, 3, dnum)
    kb, ka = rand_key(oc, 7)
    cc.upload_relin_key(kb, ka)
    assert lib.fides_set_keyswitch_variant(cc._h, ks) == 0
    for lv in (5, 2):
        a, b = rand_ct(oc, lv, 40 + lv), rand_ct(oc, lv, 50 + lv)
        got = cc.EvalMult(cc.upload(*a), cc.upload(*b), rescale=True).download()
        want = oc.hmult(lv, *a, *b, kb, ka, rescale=True)
        assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1]), lv
