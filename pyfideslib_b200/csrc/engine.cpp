// engine.cpp -- the key-switching pipeline over a batch of nb <= kMaxBatch
// elements at one level, queued on the workspace's stream.  A single operation is a batch of one; batches
// share every launch (blockIdx.z or an interleaved grid dimension), so wave
// tails, launch overheads and, for HMult, switching-key reads are amortised.
//
// Reference flow (src/CKKS/LimbPartitionMGPU.cu:573-1748 modup_ksk_moddown_mgpu,
// :458-571 fusedHoistRotate; Ciphertext.cpp:409-622, :756-926, :1053-1226):
//   tensor -> INTT -> ModUp conversion -> NTT -> inner product with the key
//   -> INTT of the special limbs -> ModDown conversion -> NTT -> combine
//   (-> rescale).  Here the tensor product is formed inside the first INTT's load
//   and the inner product, ModDown and Rescale share their NTT (see
//   moddown_finish) and every step runs once for the whole batch.
#include "context.hpp"

namespace fides {

namespace {

// Digit words of a batch from which HMult's inner product runs fused into the
// digits' row pass: 768 MiB, about six times the L2.  The fused kernel's few long
// warps per SM are slower in themselves; what it saves is the digits' return
// trip to HBM, and under the power cap that trip costs clock too.  Back to back
// for a second each, us unfused / fused, N = 2^16: L = 30 (87 digit limbs) 8 pairs
// 1586 / 1649, 16 pairs 3110 / 3102, 24 pairs 4626 / 4607, 32 pairs 6161 / 6094;
// L = 20 (61) 12 pairs 1659 / 1713, 24 pairs 3261 / 3223, 32 pairs 4298 / 4283;
// N = 2^15, L = 16 (50) 32 pairs 1758 / 1786.
constexpr size_t kFuseMinWords = (size_t)96 << 20;

LimbSeg seg_ws(const uint64_t* in, uint64_t* out, int count, int nq, int q0, int level, size_t bstride) {
    LimbSeg g{};
    g.in = in;
    g.out = out;
    g.count = count;
    g.skip_lo = count;
    g.nq = nq;
    g.q0 = q0;
    g.level = level;
    g.bstride = bstride;
    return g;
}

// Special limbs of XB / XA -> INTT scaled by (P/p_k)^-1 (in place), and, for
// the fused rescale, the INTT of both halves' top limbs into T.
void special_intt(fides_ctx* c, Workspace& w, int level, int nb, bool with_top) {
    const int n = level + 1, N = c->N;
    LimbMap m{};
    m.nb = nb;
    uint64_t* xs[2] = {w.XB, w.XA};
    for (int s = 0; s < 2; ++s) {
        LimbSeg g = seg_ws(xs[s] + (size_t)n * N, xs[s] + (size_t)n * N, c->K, 0, 0, level, w.stride);
        g.lmode = IL_PLAIN;
        g.smode = IS_MODDOWN;
        m.seg[m.nseg++] = g;
        m.total += c->K;
    }
    if (with_top) {
        for (int s = 0; s < 2; ++s) {
            LimbSeg g = seg_ws(xs[s] + (size_t)level * N, w.T + (size_t)s * N, 1, 1, level, level, w.stride);
            g.lmode = IL_PLAIN;
            g.smode = IS_PLAIN;
            m.seg[m.nseg++] = g;
            m.total += 1;
        }
    }
    ntt_inverse(c->dev, m, -1, -1, w.st);
}

// ModDown of XB -> out0, XA -> out1 for every element.  product: the ciphertext
// limbs hold e + P^-1 x already (launch_ks_hmult); with `rescale` (products
// only) the result is also rescaled: out = Rescale(e + ModDown(x)), computed as
// one NTT per output limb.
void moddown_finish(fides_ctx* c, Workspace& w, int level, int nb, uint64_t* const* out0, uint64_t* const* out1,
                    bool product, bool rescale) {
    const int n = level + 1, N = c->N, L = c->L;
    special_intt(c, w, level, nb, rescale);
    MdArgs md{};
    md.y[0] = w.XB + (size_t)n * N;
    md.y[1] = w.XA + (size_t)n * N;
    md.w[0] = w.W;
    md.w[1] = w.W + (size_t)L * N;
    md.ttop[0] = rescale ? w.T : nullptr;
    md.ttop[1] = rescale ? w.T + N : nullptr;
    md.bstride = w.stride;
    launch_moddown_conv(c->dev, level, nb, md, w.st);
    LimbMap m{};
    m.nb = nb;
    m.nseg = 2;
    const uint64_t* xs[2] = {w.XB, w.XA};
    const int nout = rescale ? level : n;
    for (int s = 0; s < 2; ++s) {
        LimbSeg g = seg_ws(w.W + (size_t)s * L * N, nullptr, nout, nout, 0, level, w.stride);
        g.in2 = xs[s];
        g.out_tab = (int8_t)(s + 1);
        m.seg[s] = g;
        m.total += nout;
    }
    for (int b = 0; b < nb; ++b) {
        m.bout[0][b] = out0[b];
        m.bout[1][b] = out1[b];
    }
    ntt_forward(c->dev, m, FL_PLAIN, rescale ? FS_RESCALE : product ? FS_SUBP : FS_MODDOWN, w.st);
}

}  // namespace

// Limbs of the ModUp digits in DIG (transformed in place): digit d holds the
// Q primes outside it up to `level`, then the K special primes.
static LimbMap digit_map(fides_ctx* c, Workspace& w, int level, int nb) {
    const int n = level + 1, N = c->N;
    LimbMap dm{};
    dm.nb = nb;
    const int nd = level / c->alpha + 1;
    for (int d = 0; d < nd; ++d) {
        const int lo = d * c->alpha, hi = std::min(lo + c->alpha - 1, level), cnt = hi - lo + 1;
        uint64_t* p = w.DIG + (size_t)d * w.dig_stride * N;
        LimbSeg g = seg_ws(p, p, n - cnt + c->K, n, 0, level, w.stride);
        g.skip_lo = lo;
        g.skip_cnt = cnt;
        dm.seg[dm.nseg++] = g;
        dm.total += g.count;
    }
    return dm;
}

// ModUp conversion + NTT of the digits, from the scaled coefficients in XT.
static void modup_from_xt(fides_ctx* c, Workspace& w, int level, int nb) {
    launch_modup_conv(c->dev, level, nb, w.XT, w.DIG, w.dig_stride, w.stride, w.st);
    ntt_forward(c->dev, digit_map(c, w, level, nb), FL_PLAIN, FS_PLAIN, w.st);
}

void eng_modup(fides_ctx* c, Workspace& w, int level, int nb, const uint64_t* const* x) {
    const int n = level + 1;
    // scaled INTT of each element's input (separate buffers: one segment per
    // element) into its XT
    int done = 0;
    while (done < nb) {
        LimbMap im{};
        im.nb = 1;
        for (; done < nb && im.nseg < kMaxSeg; ++done) {
            im.seg[im.nseg++] = seg_ws(x[done], w.XT + (size_t)done * w.stride, n, n, 0, level, 0);
            im.total += n;
        }
        ntt_inverse(c->dev, im, IL_PLAIN, IS_MODUP, w.st);
    }
    modup_from_xt(c, w, level, nb);
}

void eng_hmult(fides_ctx* c, Workspace& w, int level, int nb, const uint64_t* const* a0, const uint64_t* const* a1,
               const uint64_t* const* b0, const uint64_t* const* b1, uint64_t* const* out0, uint64_t* const* out1,
               bool rescale, const SwitchKey& key) {
    const int n = level + 1;
    // fused inner product: forced (bit 1), or for batches of at least
    // kFuseMinWords words of digits (bit 2)
    const int nd = level / c->alpha + 1;
    const size_t words = (size_t)nb * (size_t)(nd * (n + c->K) - n) * (size_t)c->N;
    const bool fuse = ((c->dev.ks_variant & 2) || ((c->dev.ks_variant & 4) && words >= kFuseMinWords)) &&
                      ntt_rows_keyswitch_supported(c->dev) && key.a != nullptr;
    // scaled INTT of a1 b1 (the product in its load) and ModUp conversion
    LimbMap im{};
    im.nb = nb;
    LimbSeg g = seg_ws(nullptr, w.XT, n, n, 0, level, w.stride);
    g.in_tab = 1;
    im.seg[im.nseg++] = g;
    im.total = n;
    KsHmultArgs ka{};
    for (int b = 0; b < nb; ++b) {
        im.bin[0][b] = ka.a1[b] = a1[b];
        im.bin[1][b] = ka.b1[b] = b1[b];
        ka.a0[b] = a0[b];
        ka.b0[b] = b0[b];
    }
    ka.dig = w.DIG;
    ka.kb = key.b;
    ka.ka = key.a;
    ka.a_seed = key.a ? 0 : uniform_stream(key.a_seed, 0);
    ka.xb = w.XB;
    ka.xa = w.XA;
    ka.dig_stride = w.dig_stride;
    ka.bstride = w.stride;
    ka.level = level;
    ka.fp_sums = c->dev.ks_variant & 1;
    ntt_inverse(c->dev, im, IL_MUL, IS_MODUP, w.st);
    launch_modup_conv(c->dev, level, nb, w.XT, w.DIG, w.dig_stride, w.stride, w.st);
    // the digits' NTT and the inner product with the rest of the tensor product;
    // fused, the digits' evaluation limbs do not reach HBM
    if (fuse) {
        ntt_forward_cols(c->dev, digit_map(c, w, level, nb), FL_PLAIN, w.st);
        ntt_rows_keyswitch(c->dev, ka, nb, w.st);
    } else {
        ntt_forward(c->dev, digit_map(c, w, level, nb), FL_PLAIN, FS_PLAIN, w.st);
        launch_ks_hmult(c->dev, nb, ka, w.st);
    }
    moddown_finish(c, w, level, nb, out0, out1, true, rescale && level > 0);
}

void eng_rotate(fides_ctx* c, Workspace& w, int level, int nb, const uint64_t* const* c0, const uint64_t* const* c1,
                const SwitchKey* const* keys, const uint32_t* galois, uint64_t* const* out0, uint64_t* const* out1,
                bool hoisted) {
    if (hoisted) {
        eng_modup(c, w, level, 1, c1);
    } else {
        eng_modup(c, w, level, nb, c1);
    }
    KsArgs ka{};
    for (int b = 0; b < nb; ++b) {
        ka.own[b] = hoisted ? c1[0] : c1[b];
        ka.c0[b] = hoisted ? c0[0] : c0[b];
        ka.kb[b] = keys[b]->b;
        ka.ka[b] = keys[b]->a;
        ka.a_seed[b] = keys[b]->a ? 0 : uniform_stream(keys[b]->a_seed, 0);
        ka.galois[b] = galois[b];
    }
    ka.dig = w.DIG;
    ka.xb = w.XB;
    ka.xa = w.XA;
    ka.dig_stride = w.dig_stride;
    ka.bstride = w.stride;
    ka.dig_bstride = hoisted ? 0 : w.stride;
    launch_ks_inner(c->dev, level, nb, ka, w.st);
    moddown_finish(c, w, level, nb, out0, out1, false, false);
}

void eng_rotate_sum(fides_ctx* c, Workspace& w, int level, int nb, const uint64_t* const* c0,
                    const uint64_t* const* c1, const SwitchKey* const* keys, const uint32_t* galois, int nout,
                    const int* start, uint64_t* const* out0, uint64_t* const* out1) {
    eng_modup(c, w, level, nb, c1);
    KsArgs ka{};
    for (int b = 0; b < nb; ++b) {
        ka.own[b] = c1[b];
        ka.c0[b] = c0[b];
        ka.kb[b] = keys[b]->b;
        ka.ka[b] = keys[b]->a;
        ka.a_seed[b] = keys[b]->a ? 0 : uniform_stream(keys[b]->a_seed, 0);
        ka.galois[b] = galois[b];
    }
    ka.dig = w.DIG;
    ka.xb = w.XB;
    ka.xa = w.XA;
    ka.dig_stride = w.dig_stride;
    ka.bstride = w.stride;
    ka.dig_bstride = w.stride;
    launch_ks_inner(c->dev, level, nb, ka, w.st);
    ExtSumArgs sa{};
    sa.nout = nout;
    sa.n = level + 1;
    for (int u = 0; u <= nout; ++u) sa.start[u] = start[u];
    sa.x[0] = w.XB;
    sa.x[1] = w.XA;
    sa.bstride = w.stride;
    launch_ext_sum(c->dev, sa, w.st);
    // one ModDown per output, on a view of the workspace whose element 0 is
    // the output's first element (every per-element buffer moves together)
    for (int u = 0; u < nout; ++u) {
        Workspace v = w;
        const size_t off = (size_t)start[u] * w.stride;
        for (uint64_t** p : {&v.XT, &v.DIG, &v.XB, &v.XA, &v.W, &v.T}) *p += off;
        moddown_finish(c, v, level, 1, out0 + u, out1 + u, false, false);
    }
}

void eng_rotate_groups(fides_ctx* c, Workspace& w, int level, int ngroups, int nper, const uint64_t* const* c0,
                       const uint64_t* const* c1, const SwitchKey* const* keys, const uint32_t* galois,
                       uint64_t* const* out0, uint64_t* const* out1) {
    eng_modup(c, w, level, ngroups, c1);
    const int nb = ngroups * nper;
    KsArgs ka{};
    for (int b = 0; b < nb; ++b) {
        ka.own[b] = c1[b / nper];
        ka.c0[b] = c0[b / nper];
        ka.kb[b] = keys[b]->b;
        ka.ka[b] = keys[b]->a;
        ka.a_seed[b] = keys[b]->a ? 0 : uniform_stream(keys[b]->a_seed, 0);
        ka.galois[b] = galois[b];
        ka.dig_elem[b] = (uint8_t)(b / nper);
    }
    ka.dig = w.DIG;
    ka.xb = w.XB;
    ka.xa = w.XA;
    ka.dig_stride = w.dig_stride;
    ka.bstride = w.stride;
    ka.dig_bstride = w.stride;
    ka.dig_group = nper;
    launch_ks_inner(c->dev, level, nb, ka, w.st);
    moddown_finish(c, w, level, nb, out0, out1, false, false);
}

}  // namespace fides
