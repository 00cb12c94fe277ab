"""N = 256, the smallest ring: products (inner product alone and fused), squares,
single, hoisted and batched rotations, rescale and a linear transform, bit-exact
against the oracle; also N = 512, one block per limb of the inner products."""
import numpy as np
import pytest

from gpu_helpers import device_status, make_pair, rand_ct, rand_key

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("logN", [8, 9])
@pytest.mark.parametrize("conv", [0, 2, 3, 4])
@pytest.mark.parametrize("ks", [0, 1, 11])
def test_products_and_rotations(logN, conv, ks):
    from pyfideslib_b200._capi import lib

    cc, oc = make_pair(logN, 6, 2, 3)
    assert lib.fides_set_conv_accumulator(cc._h, conv) == 0
    assert lib.fides_set_keyswitch_variant(cc._h, ks) == 0
    kb, ka = rand_key(oc, 7)
    cc.upload_relin_key(kb, ka)
    keys = {}
    for r in (1, 3, 5):
        g = cc.rotation_galois(r)
        keys[r] = (pow(g, -1, 2 * oc.N), rand_key(oc, 60 + 2 * r))
        cc.upload_galois_key(g, *keys[r][1])

    def same(ct, want):
        got = ct.download()
        assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1])

    raw = {lv: (rand_ct(oc, lv, 40 + lv), rand_ct(oc, lv, 50 + lv)) for lv in (5, 2, 0)}
    up = {lv: (cc.upload(*a), cc.upload(*b)) for lv, (a, b) in raw.items()}
    for lv, (a, b) in raw.items():
        for rescale in (True, False):
            same(cc.EvalMult(*up[lv], rescale=rescale), oc.hmult(lv, *a, *b, kb, ka, rescale=rescale and lv > 0))
        for r, (ginv, key) in keys.items():
            same(cc.EvalRotate(up[lv][0], r), oc.rotate(lv, *a, ginv, *key))
        for r, ct in zip(keys, cc.EvalFastRotation(up[lv][0], list(keys))):
            same(ct, oc.rotate(lv, *a, keys[r][0], *keys[r][1]))
    for ct, lv in zip(cc.EvalMultBatch([up[5][0], up[2][0]], [up[5][1], up[2][1]], rescale=True), (5, 2)):
        same(ct, oc.hmult(lv, *raw[lv][0], *raw[lv][1], kb, ka, rescale=True))
    for ct, r in zip(cc.EvalRotateBatch([up[5][0]] * 3, list(keys)), keys):
        same(ct, oc.rotate(5, *raw[5][0], keys[r][0], *keys[r][1]))
    assert device_status(cc) == 0
