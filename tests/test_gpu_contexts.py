"""Contexts side by side at one ring dimension: one with more digits runs its
fused key switch (a tile of shared memory per digit) after others with fewer
digits were made, bit-exact against the oracle."""
import numpy as np
import pytest

from gpu_helpers import make_pair, rand_ct, rand_key

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("logN", [9, 13, 16])
@pytest.mark.parametrize("ks", [3, 11])
def test_fused_key_switch_after_a_smaller_context(logN, ks):
    from pyfideslib_b200._capi import lib

    cc, oc = make_pair(logN, 6, 1, 6)
    kb, ka = rand_key(oc, 7)
    cc.upload_relin_key(kb, ka)
    assert lib.fides_set_keyswitch_variant(cc._h, ks) == 0
    others = [make_pair(logN, 4, 2, d)[0] for d in (2, 1)]
    a, b = rand_ct(oc, 5, 40), rand_ct(oc, 5, 50)
    got = cc.EvalMult(cc.upload(*a), cc.upload(*b), rescale=True).download()
    want = oc.hmult(5, *a, *b, kb, ka, rescale=True)
    assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1])
    del others
