"""What a captured plan points at: its workspace stays alive when a larger batch
on the same context takes a new one (residues against the oracle before and
after, two plans of different sizes), and a launch is refused once a buffer or a
key that the graph reads or writes has been replaced."""
import numpy as np
import pytest

from gpu_helpers import make_pair, rand_ct, rand_key

pytestmark = pytest.mark.gpu


def test_plan_survives_a_larger_batch():
    cc, oc = make_pair(12, 5, 2, 3)
    kb, ka = rand_key(oc, 31)
    cc.upload_relin_key(kb, ka)
    g = cc.rotation_galois(3)
    gk = rand_key(oc, 33)
    cc.upload_galois_key(g, *gk)

    def inputs(n, seed):
        raw = [(rand_ct(oc, 4 - i % 2, seed + 4 * i), rand_ct(oc, 4 - i % 2, seed + 4 * i + 2)) for i in range(n)]
        return raw, [cc.upload(*a) for a, _ in raw], [cc.upload(*b) for _, b in raw]

    def want(raw, rotate):
        out = []
        for a, b in raw:
            lv = len(a[0]) - 1
            r = oc.hmult(lv, *a, *b, kb, ka, rescale=True)
            out.append(oc.rotate(lv - 1, *r, pow(g, -1, 2 * oc.N), *gk) if rotate else r)
        return out

    def same(outs, ref):
        for o, w in zip(outs, ref):
            got = o.download()
            assert np.array_equal(got[0], w[0]) and np.array_equal(got[1], w[1])

    raw, A, B = inputs(3, 100)
    ref = want(raw, True)
    plan, outs = cc.plan_hmult_rotate(A, B, [3] * 3, rescale=True)
    plan.launch()
    same(outs, ref)
    raw2, A2, B2 = inputs(9, 200)
    ref2 = want(raw2, False)
    same(cc.EvalMultBatch(A2, B2, rescale=True), ref2)  # takes a workspace of nine elements
    scratch = [cc.random_ct(4, 7 + i) for i in range(40)]  # whatever was freed is in use again
    for o in outs:  # stale results would show
        cc.write(o, *rand_ct(oc, o.level, 5))
    plan.launch()
    same(outs, ref)
    plan2, outs2 = cc.plan_hmult_rotate(A2, B2, None, rescale=True)
    plan2.launch()
    plan.launch()
    same(outs2, ref2)
    same(outs, ref)
    del plan  # its workspace goes with it, the larger one stays
    plan2.launch()
    same(outs2, ref2)
    same(cc.EvalMultBatch(A2, B2, rescale=True), ref2)
    del scratch


def test_plan_refuses_replaced_buffers_and_keys():
    from pyfideslib_b200 import FidesError

    cc, oc = make_pair(11, 4, 2, 2)
    sk = cc.KeyGen(seed=5)
    cc.EvalMultKeyGen(sk)
    cc.EvalRotateKeyGen(sk, [1], seed=9)
    A, B = [cc.random_ct(3, 1), cc.random_ct(3, 2)], [cc.random_ct(3, 3), cc.random_ct(3, 4)]

    def fresh():
        plan, outs = cc.plan_hmult_rotate(A, B, [1, 1], rescale=True)
        plan.launch()
        return plan, outs

    def refused(plan):
        with pytest.raises(FidesError):
            plan.launch()

    plan, outs = fresh()
    cc.EvalAdd(A[0], A[1], out=A[0])  # an input's result buffer is a new one
    refused(plan)
    plan, outs = fresh()
    cc.EvalAdd(outs[0], outs[1], out=outs[1])
    refused(plan)
    plan, outs = fresh()
    cc.EvalRotateKeyGen(sk, [1], seed=9)  # the same compressed key again
    plan.launch()
    cc.EvalRotateKeyGen(sk, [1], seed=10)
    refused(plan)
    plan, outs = fresh()
    cc.upload_galois_key(cc.rotation_galois(1), *rand_key(oc, 3))  # both halves stored: a new allocation
    refused(plan)
    plan, outs = fresh()
    cc.upload_relin_key(*rand_key(oc, 4))
    cc.upload_galois_key(cc.rotation_galois(1), *rand_key(oc, 5))  # full keys in place: the plan reads them
    plan.launch()
    want = cc.EvalRotateBatch(cc.EvalMultBatch(A, B, rescale=True), [1, 1])
    for o, w in zip(outs, want):
        got, ref = o.download(), w.download()
        assert np.array_equal(got[0], ref[0]) and np.array_equal(got[1], ref[1])
