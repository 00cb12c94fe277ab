"""The launches that cover a whole ciphertext operation: scalar and
element-wise operations on both components (limb counts around one launch's
64 constants), and the plaintext dot products of all giant steps in one
launch (more outputs and more terms than a launch's tables hold, sums longer
than a launch)."""
import numpy as np
import pytest

from gpu_helpers import make_pair, rand_ct, rand_key

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L,level", [(3, 0), (70, 63), (70, 64), (70, 69)])
def test_scalar_and_elementwise_bitexact(L, level):
    import pyfideslib_b200 as F

    cc = F.CryptoContext(log_n=9, num_q=L, dnum=min(8, L))
    rng = np.random.default_rng(level)
    mod = np.array(cc.q[:level + 1], dtype=object)[:, None]

    def rand():
        return np.stack([rng.integers(0, q, cc.N, dtype=np.uint64) for q in cc.q[:level + 1]])

    a, b, m = (rand(), rand()), (rand(), rand()), rand()
    A, B = cc.upload(*a), cc.upload(*b)
    o = [x.astype(object) for x in a + b] + [m.astype(object)]

    def same(ct, w0, w1):
        g = ct.download()
        assert np.array_equal(g[0].astype(object), w0 % mod) and np.array_equal(g[1].astype(object), w1 % mod)

    for v in (0.75, -3.0):
        k = int(round(v * cc.scale))
        same(cc.EvalMult(A, v), o[0] * k, o[1] * k)
        same(cc.EvalAdd(A, v), o[0] + k, o[1])
    same(cc.EvalAdd(A, B), o[0] + o[2], o[1] + o[3])
    same(cc.EvalSub(A, B), o[0] - o[2], o[1] - o[3])
    same(cc.EvalNegate(A), -o[0], -o[1])
    h = F._capi.vp()
    F._capi.check(F.lib.fides_pt_upload(cc._h, m.ctypes.data_as(F._capi.u64p), level, cc.scale, 1, cc.N // 2, h), cc._h)
    P = F.Plaintext(cc, h.value)
    same(cc.EvalMult(A, P), o[0] * o[4], o[1] * o[4])
    same(cc.EvalAdd(A, P), o[0] + o[4], o[1])
    same(cc.EvalAdd(A, A, out=A), o[0] * 2, o[1] * 2)  # an output may alias its inputs


# (offsets, baby step): 20 outputs of 3 terms (two launches of outputs), one
# output of 70 terms (two launches of terms), outputs that do not fill a launch
@pytest.mark.parametrize("offsets,bstep", [(list(range(60)), 3), (list(range(70)), 70), (list(range(-5, 45)), 20)])
def test_giant_steps_one_launch_bitexact(offsets, bstep):
    import pyfideslib_b200 as F
    from test_gpu_linear import _oracle_bsgs, _upload_pt

    cc, oc = make_pair(11, 4, 2, 2)
    keys = {}
    for i, r in enumerate(F.CryptoContext.linear_transform_rotations(offsets, bstep)):
        keys[r] = rand_key(oc, 300 + 2 * i)
        cc.upload_galois_key(cc.rotation_galois(r), *keys[r])
    level = 3
    c0, c1 = rand_ct(oc, level, 400)
    pts_r = [oc.random(list(range(level + 1)), 500 + k) for k in range(len(offsets))]
    for i in range(level + 1):  # extremes
        pts_r[1][i] = oc.primes[i] - 1
        c1[i] = oc.primes[i] - 1
    pts = [_upload_pt(cc, m, level) for m in pts_r]
    got = cc.EvalLinearTransform(cc.upload(c0, c1), offsets, pts, bstep, rescale=False).download()
    want = _oracle_bsgs(oc, level, c0, c1, offsets, pts_r, bstep, keys, cc.rotation_galois)
    assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1])
