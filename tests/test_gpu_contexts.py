"""Contexts side by side: one with more digits runs its fused key switch (a tile of
shared memory per digit) after others with fewer digits were made at its ring
dimension, bit-exact against the oracle; tensor-core conversions of two widths at once."""
import numpy as np
import pytest

from gpu_helpers import device_status, make_pair, rand_ct, rand_key

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


def test_contexts_with_both_tensor_core_widths_side_by_side():
    """Products queued in turn on two contexts (two streams), one with 32 targets
    per matrix product and one with 16, which also change in between: the residues of
    each context alone, and no wait given up."""
    from pyfideslib_b200._capi import lib

    sides = []
    for k, conv in enumerate((3, 4)):
        cc, oc = make_pair(13, 8, 3, 3)
        cc.upload_relin_key(*rand_key(oc, 7))
        a, b = cc.upload(*rand_ct(oc, 7, 40 + k)), cc.upload(*rand_ct(oc, 7, 50 + k))
        assert lib.fides_set_conv_accumulator(cc._h, 0) == 0
        want = cc.EvalMult(a, b, rescale=True).download()
        sides.append((cc, conv, a, b, want))
    outs = []
    for rep in range(20):
        for cc, conv, a, b, want in sides:
            assert lib.fides_set_conv_accumulator(cc._h, conv if rep % 4 else 7 - conv) == 0
            outs.append((cc.EvalMult(a, b, rescale=True), want))
    for ct, want in outs:
        got = ct.download()
        assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1])
    assert all(device_status(s[0]) == 0 for s in sides)
