// ntt_kernels.cuh -- negacyclic NTT / INTT kernels over RNS limbs for sm_100a,
// templates on the ring dimension (ntt_n.cu instantiates one per file).
//
// Role in the reference: src/NTT.cu NTT_/INTT_ (two-pass 2-D decomposition with
// fused prologues/epilogues, NTTfusions.cuh).  The transform computed is the
// same one: natural-order coefficients -> evaluations in bit-reversed order,
//   out[i] = sum_j a_j psi^{(2 bitrev(i) + 1) j}  (mod p),
// i.e. the in-place Cooley-Tukey loop over the bit-reversed psi table, and its
// Gentleman-Sande inverse with N^-1 folded into the last stage.
//
// Layout and schedule (this file's own design):
//   * N = R x C with R = 2^LR rows of C = 2^LC contiguous coefficients.  The
//     first LR stages only pair elements of one column, the last LC stages
//     only elements of one row.  Pass 1 runs the column stages, pass 2 the
//     row stages.
//   * Each thread owns 16 elements of one column/row in registers and runs up
//     to 4 butterfly stages on them (radix-16 register blocking); the next
//     group of stages follows one shared-memory exchange.  Column passes move
//     16 consecutive columns per CTA (128-byte coalesced rows).
//   * A row pass needs no CTA-wide barrier: the 2^LC / 16 threads of a row lie
//     in one warp, which owns 512 contiguous words (RowGeo), exchanges, runs
//     the epilogue and stores on its own.  Warps drift apart, so the loads of
//     some run under the butterflies of others.  (N=2^16, 32 x 30 limbs: the
//     CTA-synchronous form waited 1.1 issue slots per instruction at
//     barriers; forward pair 505 -> 457 us, inverse 509 -> 494 us; one 2^13
//     transform of 7 limbs 14.4 -> 12.5 us.)
//   * Harvey lazy butterflies on the integer pipes, or, for primes below
//     2^50, exact butterflies on the FP64 pipes with residues held as
//     integer-valued doubles (fp64.cuh).
//   * Prologues/epilogues fuse the surrounding element-wise work (products of
//     two inputs, ModDown/Rescale combinations, per-limb CRT scalings).  The
//     mode is a per-segment field, so one launch can mix limbs with different
//     fusions.
#pragma once
#include "fp64.cuh"
#include "kernels.hpp"
#include "ntt_sched.hpp"

namespace fides {

// ---- integer butterflies ----
// MODE 0 is Harvey's form: X kept in [0, 4p) with one conditional subtraction
// per butterfly.  MODE 3 (primes below 2^56) drops the subtraction and forms
// the Shoup quotient from three of the four 32x32 partial products: it is low
// by at most 2, the product lands in [0, 4p), each stage adds at most 4p, and
// the bound after the 16 stages of a 2^16 transform is 65p < 2^63 (the Shoup
// product accepts any 64-bit input); one Barrett step in the epilogue reduces.
constexpr uint64_t kApproxPrimeBound = 1ull << 56;

// floor(a * b / 2^64) - d with d in {0, 1, 2}
__device__ __forceinline__ uint64_t mulhi64_approx(uint64_t a, uint64_t b) {
    const uint32_t a0 = (uint32_t)a, a1 = (uint32_t)(a >> 32), b0 = (uint32_t)b, b1 = (uint32_t)(b >> 32);
    uint64_t h = (uint64_t)a1 * b1;
    h += __umulhi(a1, b0);
    h += __umulhi(a0, b1);
    return h;
}

template <int MODE>
__device__ __forceinline__ void ct_bfly(uint64_t& X, uint64_t& Y, const ulonglong2 w, const uint64_t p,
                                        const uint64_t two_p) {
    if constexpr (MODE == 3) {
        const uint64_t t = Y * w.x - mulhi64_approx(Y, w.y) * p;  // [0, 4p)
        const uint64_t x = X;
        X = x + t;
        Y = x - t + 2 * two_p;
    } else {
        const uint64_t x = csub(X, two_p);
        const uint64_t t = mul_shoup_lazy(Y, w.x, w.y, p);
        X = x + t;
        Y = x - t + two_p;
    }
}

__device__ __forceinline__ void gs_bfly(uint64_t& X, uint64_t& Y, const ulonglong2 w, const uint64_t p,
                                        const uint64_t two_p) {
    const uint64_t s = csub(X + Y, two_p);
    const uint64_t d = X - Y + two_p;
    X = s;
    Y = mul_shoup_lazy(d, w.x, w.y, p);
}

// canonical residue of any forward-NTT output of the integer butterflies
__device__ __forceinline__ uint64_t reduce_fwd(uint64_t v, const PrimeConst& c) {
    return csub(reduce64_lazy(v, c), c.p);
}

// ---- double-precision butterflies (primes below 2^50) ----
// Residues are held exactly as signed integer-valued doubles (bit patterns in
// the uint64_t registers); fp64.cuh states the product, ntt_sched.hpp the
// bounds and where the stages centre.  The column pass hands its doubles to
// the row pass (and the inverse's row pass to its column pass) unconverted.

// forward; RED centres x first, to within p/2 of rsub p where rsub carries
// kRint (centre around 0) or kRint + s (around s p)
template <bool RED>
__device__ __forceinline__ void ct_bfly_fp(uint64_t& X, uint64_t& Y, const ulonglong2 w, const double p,
                                           const double pinv, const double rsub) {
    double x = as_f64(X);
    if constexpr (RED) x = __fma_rn(-__dsub_rn(__fma_rn(x, pinv, kRint), rsub), p, x);
    const double t = fp_mulw(as_f64(Y), as_f64(w.x), as_f64(w.y), p);
    X = as_u64(__dadd_rn(x, t));
    Y = as_u64(__dsub_rn(x, t));
}

// inverse: the sum is centred when CEN, the difference goes through the product
template <bool CEN>
__device__ __forceinline__ void gs_bfly_fp(uint64_t& X, uint64_t& Y, const ulonglong2 w, const double p,
                                           const double pinv) {
    const double x = as_f64(X), y = as_f64(Y);
    double s = __dadd_rn(x, y);
    if constexpr (CEN) s = fp_center(s, p, pinv);
    X = as_u64(s);
    Y = as_u64(fp_mulw(__dsub_rn(x, y), as_f64(w.x), as_f64(w.y), p));
}


__device__ __forceinline__ ulonglong2 ldg2(const uint64_t* base, size_t idx) {
    return __ldg(reinterpret_cast<const ulonglong2*>(base) + idx);
}

// 16-byte asynchronous copy into shared memory (twiddle staging: no registers
// held while the data loads go out behind it)
__device__ __forceinline__ void stage16(void* dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
}
__device__ __forceinline__ void stage_wait() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }

// A stage whose register partner bit is kb pairs k and k | (1 << kb) and uses
// twiddle group g = k >> (kb + 1), g < 8 >> kb; get(kb, g) supplies it.
//
// Integer stages KB_FIRST .. KB_END in steps of STEP.  MODE: 0 and 3 forward
// (see ct_bfly), 2 inverse.
template <int KB, int KB_END, int STEP, int MODE, class Get>
__device__ __forceinline__ void int_stages(uint64_t (&x)[16], Get get, uint64_t p, uint64_t two_p) {
    ulonglong2 w[8 >> KB];
#pragma unroll
    for (int g = 0; g < (8 >> KB); ++g) w[g] = get(KB, g);
#pragma unroll
    for (int k = 0; k < 16; ++k) {
        if (k & (1 << KB)) continue;
        if constexpr (MODE == 2)
            gs_bfly(x[k], x[k | (1 << KB)], w[k >> (KB + 1)], p, two_p);
        else
            ct_bfly<MODE>(x[k], x[k | (1 << KB)], w[k >> (KB + 1)], p, two_p);
    }
    if constexpr (KB != KB_END) int_stages<KB + STEP, KB_END, STEP, MODE>(x, get, p, two_p);
}

// forward integer group in the form of this limb's prime (uniform per CTA)
template <int KB_FIRST, class Get>
__device__ __forceinline__ void int_fwd(bool approx, uint64_t (&x)[16], Get get, uint64_t p, uint64_t two_p) {
    if (approx)
        int_stages<KB_FIRST, 0, -1, 3>(x, get, p, two_p);
    else
        int_stages<KB_FIRST, 0, -1, 0>(x, get, p, two_p);
}

// forward double-precision stages: partner bits KB .. 0, global stages S ..
template <int LOGN, int LR, int S, int KB, class Get>
__device__ __forceinline__ void fp_fwd(uint64_t (&x)[16], Get get, double p, double pinv, double rlast) {
    constexpr FwdSched sc = fwd_sched(LOGN, LR);
    ulonglong2 w[8 >> KB];
#pragma unroll
    for (int g = 0; g < (8 >> KB); ++g) w[g] = get(KB, g);
#pragma unroll
    for (int k = 0; k < 16; ++k) {
        if (k & (1 << KB)) continue;
        ct_bfly_fp<sc.red[S]>(x[k], x[k | (1 << KB)], w[k >> (KB + 1)], p, pinv, S == LOGN - 1 ? rlast : kRint);
    }
    if constexpr (KB > 0) fp_fwd<LOGN, LR, S + 1, KB - 1>(x, get, p, pinv, rlast);
}

// inverse double-precision stages: partner bits KB .. NST-1 of a group G of
// inv_sched (0 row A, 1 row B, 2 column A, 3 column B)
template <int LR, int LC, int G>
__device__ __forceinline__ constexpr unsigned inv_mask(int kb) {
    constexpr InvSched s = inv_sched(LR, LC);
    return G == 0 ? s.ra.mask[kb] : G == 1 ? s.rb.mask[kb] : G == 2 ? s.ca.mask[kb] : s.cb.mask[kb];
}
template <int LR, int LC, int G, int KB, int NST, int K = 0>
__device__ __forceinline__ void fp_inv_stage(uint64_t (&x)[16], const ulonglong2* w, double p, double pinv) {
    if constexpr (!(K & (1 << KB)))
        gs_bfly_fp<((inv_mask<LR, LC, G>(KB) >> K) & 1) != 0>(x[K], x[K | (1 << KB)], w[K >> (KB + 1)], p, pinv);
    if constexpr (K < 15) fp_inv_stage<LR, LC, G, KB, NST, K + 1>(x, w, p, pinv);
}
template <int LR, int LC, int G, int KB, int NST, class Get>
__device__ __forceinline__ void fp_inv(uint64_t (&x)[16], Get get, double p, double pinv) {
    ulonglong2 w[8 >> KB];
#pragma unroll
    for (int g = 0; g < (8 >> KB); ++g) w[g] = get(KB, g);
    fp_inv_stage<LR, LC, G, KB, NST>(x, w, p, pinv);
    if constexpr (KB + 1 < NST) fp_inv<LR, LC, G, KB + 1, NST>(x, get, p, pinv);
}

// ---- geometry ----
// Every kernel has two instances: one held to 80 registers, 24 warps per SM, and
// a wide one of up to 128 registers for launches that do not fill the SMs anyway
// (wide_threads): with all the loads of a thread in flight and no spills its
// warps are shorter, which is all that counts there.
constexpr int min_ctas(int nt, bool wide) {
    const int c = (wide ? 512 : 768) / nt;
    return c < 32 ? c : 32;
}
// Column pass: 16 consecutive columns per CTA, TPC threads per column.  (Tiles
// of 256 threads whatever the column length left a 2^13 transform of 6 limbs
// on 24 CTAs; 16 columns are the narrowest tile with 128-byte rows.)
template <int LR, int LC>
struct ColGeo {
    static constexpr int R = 1 << LR, C = 1 << LC;
    static constexpr int TPC = 1 << (LR - 4), TC = 16, NT = TPC * TC;
    static constexpr int MINB = min_ctas(NT, false), MINB_WIDE = min_ctas(NT, true);
};
// Row pass: a warp (WL lanes, 16 for N = 256) owns RW whole rows = GW
// contiguous words; W warps per CTA, independent of one another.
template <int LR, int LC>
struct RowGeo {
    static constexpr int R = 1 << LR, C = 1 << LC;
    static constexpr int TPR = 1 << (LC - 4);                    // threads per row
    static constexpr int WL = R * TPR < 32 ? R * TPR : 32;       // lanes
    static constexpr int RW = WL / TPR;                          // rows per warp
    static constexpr int GW = WL * 16, SW = GW + GW / 16;        // words, padded words
    static constexpr int GROUPS = R * C / GW;
    static constexpr int W = GROUPS < 4 ? GROUPS : 4;
    static constexpr int NT = W * WL;
    static constexpr int MINB = min_ctas(NT, false), MINB_WIDE = min_ctas(NT, true);
    static constexpr unsigned MASK = WL == 32 ? 0xffffffffu : (1u << WL) - 1;
    // staged twiddles of a warp: entry r * 15 + 2^t - 1 + g of row r's first
    // four stages, then psi_br[g], g < 8
    static constexpr int TW = RW * 15 + 8;
};

// padded position of word i of a warp's tile: both the strided and the
// contiguous register mappings hit 16 distinct bank pairs
__device__ __forceinline__ int padi(int i) { return i + (i >> 4); }

// Row-pass twiddles.  Row r's stage s' (0 <= s' < LC) uses
// psi_br[((R + r) << s') + h], h < 2^s'.  The first four stages' 15 twiddles
// are the same for all threads of the row and are staged in shared memory.
// From stage 4 on, thread th needs h = (th << m) + g, g < 2^m (m = 3 - kb), and
// since the bit reversals of disjoint bit groups add,
//   psi_br[((R + r) << s') + (th << m) + g] = D_s' psi_br[g]  (mod p),
// D_s' = the g = 0 entry: one table load per stage and thread, issued before
// the data is needed, and 2^m - 1 products on the FP64 pipes instead of up to
// 15 dependent L2 loads per group.  (Integer limbs load every entry: their
// Shoup companions cannot be formed by a product.)
template <int LR, int LC>
__device__ __forceinline__ void stage_row_tw(ulonglong2* s_tw, const uint64_t* twg, int row0, int lane) {
    using G = RowGeo<LR, LC>;
    const ulonglong2* tw2 = reinterpret_cast<const ulonglong2*>(twg);
#pragma unroll
    for (int e = lane; e < G::TW; e += G::WL) {
        if (e < G::RW * 15) {
            const int r = e / 15, j = e % 15, t = 31 - __clz(j + 1);
            stage16(s_tw + e, tw2 + ((size_t)(G::R + row0 + r) << t) + (j + 1 - (1 << t)));
        } else {
            stage16(s_tw + e, tw2 + (e - G::RW * 15));
        }
    }
}

// twiddle g of partner bit kb formed from D (exact table entry), |w| <= 0.594p;
// the quotient companion is fl(w fl(1/p))
__device__ __forceinline__ ulonglong2 form_tw(const ulonglong2 D, double gw, int g, double p, double pinv) {
    if (g == 0) return D;
    const double w = fp_mulmod(as_f64(D.x), gw, p, pinv);
    ulonglong2 r;
    r.x = as_u64(w);
    r.y = as_u64(__dmul_rn(w, pinv));
    return r;
}

// ---------------------------------------------------------------------------
// forward, pass 1: column stages 0..LR-1
// ---------------------------------------------------------------------------
template <int LR, int LC, bool FP, bool WIDE>
__global__ void __launch_bounds__(ColGeo<LR, LC>::NT, WIDE ? ColGeo<LR, LC>::MINB_WIDE : ColGeo<LR, LC>::MINB)
    k_ntt_fwd_cols(const __grid_constant__ DevCtx ctx, const __grid_constant__ LimbMap map) {
    using G = ColGeo<LR, LC>;
    constexpr int C = G::C, TC = G::TC, LOGN = LR + LC;
    __shared__ __align__(16) uint64_t sm[LR > 4 ? G::R * TC : 1];
    __shared__ ulonglong2 tws[G::R];

    pdl_trigger();
    const LimbRef lr = resolve_limb(map, blockIdx.z, blockIdx.y, ctx.N, ctx.L);
    const PrimeConst pc = ctx.pc[lr.prime];
    const bool fp = FP && pc.p < kFpPrimeBound;
    const ulonglong2* twg = reinterpret_cast<const ulonglong2*>(fp ? ctx.fwd_twf : ctx.fwd_tw) + (size_t)lr.prime * ctx.N;
    for (int i = threadIdx.x; i < G::R; i += G::NT) stage16(&tws[i], &twg[i]);

    const int c = threadIdx.x % TC, th = threadIdx.x / TC;
    const int col = blockIdx.x * TC + c;
    pdl_wait();
    uint64_t x[16];
#pragma unroll
    for (int k = 0; k < 16; ++k) x[k] = lr.in[(size_t)(th + (k << (LR - 4))) * C + col];
    const double p = __ull2double_rn(pc.p), pinv = as_f64(pc.pinv_f64);
    if (lr.lmode == FL_SWITCHMOD) {
        const uint64_t om = ctx.pc[lr.level].p;
        if (fp && om < kFpPrimeBound) {
            // the centred lift of a residue mod om is already an operand the
            // butterflies take while om <= 2p
            const double omd = __ull2double_rn(om);
            const bool wide = om > pc.two_p;
#pragma unroll
            for (int k = 0; k < 16; ++k) {
                double v = as_f64(fp_from_u(x[k]));
                if (x[k] > (om >> 1)) v = __dsub_rn(v, omd);
                if (wide) v = fp_center(v, p, pinv);
                x[k] = as_u64(v);
            }
        } else {
#pragma unroll
            for (int k = 0; k < 16; ++k) {
                x[k] = switch_modulus(x[k], om, pc);
                if (fp) x[k] = fp_from_u(x[k]);
            }
        }
    } else if (fp) {
#pragma unroll
        for (int k = 0; k < 16; ++k) x[k] = fp_from_u(x[k]);
    }
    stage_wait();
    __syncthreads();
    // stages 0..3: r = th + (k << (LR - 4)), twiddle (1 << t) + (k >> (4 - t))
    auto g1 = [&](int kb, int g) { return tws[(8 >> kb) + g]; };
    // stages 4..LR-1: r = 16 th + k
    auto g2 = [&](int kb, int g) { return tws[(1 << (LR - 1 - kb)) + (th << (3 - kb)) + g]; };
    const bool approx = pc.p < kApproxPrimeBound;
    if (fp) {
        fp_fwd<LOGN, LR, 0, 3>(x, g1, p, pinv, kRint);
    } else {
        int_fwd<3>(approx, x, g1, pc.p, pc.two_p);
    }
    if constexpr (LR > 4) {
#pragma unroll
        for (int k = 0; k < 16; ++k) sm[(th + (k << (LR - 4))) * TC + c] = x[k];
        __syncthreads();
#pragma unroll
        for (int k = 0; k < 16; ++k) x[k] = sm[((th << 4) + k) * TC + c];
        if (fp)
            fp_fwd<LOGN, LR, 4, LR - 5>(x, g2, p, pinv, kRint);
        else
            int_fwd<LR - 5>(approx, x, g2, pc.p, pc.two_p);
    }
    // double-precision limbs leave as doubles
    if constexpr (LR > 4) {
#pragma unroll
        for (int k = 0; k < 16; ++k) lr.out[(size_t)((th << 4) + k) * C + col] = x[k];
    } else {
#pragma unroll
        for (int k = 0; k < 16; ++k) lr.out[(size_t)(th + k) * C + col] = x[k];
    }
}

// ---------------------------------------------------------------------------
// forward, pass 2: row stages LR..logN-1, with fused epilogue
// ---------------------------------------------------------------------------
// The 16 words of a thread through the row stages: x[k] holds word
// th + (k << (LC - 4)) of its row, and afterwards word 16 th + k.
// srow: the warp's padded tile; s_tw: the staged twiddles.
template <int LR, int LC, bool FP>
struct RowFwd {
    using G = RowGeo<LR, LC>;
    static constexpr int NST2 = LC - 4;  // stages of the second group
    static constexpr int LOGN = LR + LC;
    ulonglong2 D[NST2 > 0 ? NST2 : 1];

    __device__ __forceinline__ void load_d(const uint64_t* twg, int row, int th) {
#pragma unroll
        for (int i = 0; i < NST2; ++i) {  // partner bit kb = NST2 - 1 - i, stage 4 + i
            const int kb = NST2 - 1 - i;
            D[i] = ldg2(twg, ((size_t)(G::R + row) << (4 + i)) + ((size_t)th << (3 - kb)));
        }
    }
    // double-precision limbs; rlast: kRint (last stage centred around 0) or
    // kRint + s (around s p)
    __device__ __forceinline__ void run_fp(uint64_t (&x)[16], uint64_t* sw, const ulonglong2* s_tw, int lane, int th,
                                           int rl, double p, double pinv, double rlast) const {
        const ulonglong2* g1 = s_tw + rl * 15;
        fp_fwd<LOGN, LR, LR, 3>(x, [&](int kb, int g) { return g1[(8 >> kb) - 1 + g]; }, p, pinv, rlast);
        if constexpr (NST2 > 0) {
            exchange(x, sw, lane, th, rl);
            const ulonglong2* gw = s_tw + G::RW * 15;
            fp_fwd<LOGN, LR, LR + 4, NST2 - 1>(
                x, [&](int kb, int g) { return form_tw(D[NST2 - 1 - kb], as_f64(gw[g].x), g, p, pinv); }, p, pinv,
                rlast);
        }
    }
    __device__ __forceinline__ void run_int(uint64_t (&x)[16], uint64_t* sw, const ulonglong2* s_tw,
                                            const uint64_t* twg, int row, int lane, int th, int rl,
                                            const PrimeConst& pc) const {
        const ulonglong2* g1 = s_tw + rl * 15;
        const bool approx = pc.p < kApproxPrimeBound;
        int_fwd<3>(approx, x, [&](int kb, int g) { return g1[(8 >> kb) - 1 + g]; }, pc.p, pc.two_p);
        if constexpr (NST2 > 0) {
            exchange(x, sw, lane, th, rl);
            int_fwd<NST2 - 1>(
                approx, x,
                [&](int kb, int g) {
                    return ldg2(twg, ((size_t)(G::R + row) << (LC - 1 - kb)) + ((size_t)th << (3 - kb)) + g);
                },
                pc.p, pc.two_p);
        }
    }
    // strided to contiguous words
    __device__ __forceinline__ void exchange(uint64_t (&x)[16], uint64_t* sw, int lane, int th, int rl) const {
        __syncwarp(G::MASK);
#pragma unroll
        for (int k = 0; k < 16; ++k) sw[padi(rl * G::C + th + (k << (LC - 4)))] = x[k];
        __syncwarp(G::MASK);
#pragma unroll
        for (int k = 0; k < 16; ++k) x[k] = sw[17 * lane + k];
    }
};

// The epilogue of one warp's tile: out[i] = f(value, in2[i]) over the
// words of the tile, two adjacent words per lane and step (16-byte accesses).
// IN2: whether in2 is read (else 0).
template <class G, bool IN2, class F>
__device__ __forceinline__ void row_epilogue(const LimbRef& lr, size_t base, const uint64_t* sw, int lane, F f) {
#pragma unroll 4
    for (int j = 0; j < 8; ++j) {
        const int i = 2 * lane + 2 * G::WL * j;
        const int wi = padi(i);
        ulonglong2 a = make_ulonglong2(0, 0), o;
        if (IN2) a = *reinterpret_cast<const ulonglong2*>(lr.in2 + base + i);
        o.x = f(sw[wi], a.x);
        o.y = f(sw[wi + 1], a.y);
        *reinterpret_cast<ulonglong2*>(lr.out + base + i) = o;
    }
}

template <int LR, int LC, bool FP, bool WIDE>
__global__ void __launch_bounds__(RowGeo<LR, LC>::NT, WIDE ? RowGeo<LR, LC>::MINB_WIDE : RowGeo<LR, LC>::MINB)
    k_ntt_fwd_rows(const __grid_constant__ DevCtx ctx, const __grid_constant__ LimbMap map) {
    using G = RowGeo<LR, LC>;
    __shared__ __align__(16) uint64_t sm[G::W * G::SW];
    __shared__ ulonglong2 s_twa[G::W * G::TW];

    pdl_trigger();
    const LimbRef lr = resolve_limb(map, blockIdx.z, blockIdx.y, ctx.N, ctx.L);
    const PrimeConst pc = ctx.pc[lr.prime];
    const bool fp = FP && pc.p < kFpPrimeBound;
    const uint64_t* twg = (fp ? ctx.fwd_twf : ctx.fwd_tw) + (size_t)lr.prime * 2 * ctx.N;

    const int w = threadIdx.x / G::WL, lane = threadIdx.x % G::WL;
    const int th = lane % G::TPR, rl = lane / G::TPR;
    const int row0 = (blockIdx.x * G::W + w) * G::RW;
    const size_t base = (size_t)row0 * G::C;
    uint64_t* sw = sm + w * G::SW;
    ulonglong2* s_tw = s_twa + w * G::TW;
    stage_row_tw<LR, LC>(s_tw, twg, row0, lane);
    RowFwd<LR, LC, FP> rf;
    if (fp) rf.load_d(twg, row0 + rl, th);
    pdl_wait();
    const uint64_t* src = lr.out + base + rl * G::C;
    uint64_t x[16];
#pragma unroll
    for (int k = 0; k < 16; ++k) x[k] = src[th + (k << (LC - 4))];
    if (lr.smode != FS_PLAIN && lr.in2 && gridDim.y > 1) {
        // the epilogue's operand for this tile (one 128-byte line per lane):
        // start its HBM reads now, under the butterflies.
        // Batched launches only: a single element's grid is about two waves,
        // where the early reads only compete with the row loads (measured
        // 1.5% slower per operation, 0.5% faster batched)
        prefetch_l2(lr.in2 + base + lane * 16);
    }
    stage_wait();
    __syncwarp(G::MASK);
    const double p = __ull2double_rn(pc.p), pinv = as_f64(pc.pinv_f64);
    // double-precision limbs end within 1.63p of 0, or of 2p when the value
    // is reduced as it is
    if (fp)
        rf.run_fp(x, sw, s_tw, lane, th, rl, p, pinv, lr.smode == FS_PLAIN ? kRint + 2.0 : kRint);
    else
        rf.run_int(x, sw, s_tw, twg, row0 + rl, lane, th, rl, pc);
    __syncwarp(G::MASK);
#pragma unroll
    for (int k = 0; k < 16; ++k) sw[17 * lane + k] = x[k];
    __syncwarp(G::MASK);
    if (fp) {
        // the combinations stay on the FP64 pipes: operands are residues (or
        // sums below 3.2p), the constants are centred with exact companions, so
        // every product is below 0.62p and the last one, shifted by p, is
        // positive.  (64-bit Shoup products here cost as many issue slots as the
        // butterflies: the final row pass of 32 products took 925 us, 58 x 32 limbs.)
        const double2 c = lr.smode == FS_PLAIN ? make_double2(0, 0)
                          : lr.smode == FS_RESCALE
                              ? *reinterpret_cast<const double2*>(ctx.rs_qinvf + 2 * ((size_t)lr.level * ctx.L + lr.prime))
                              : *reinterpret_cast<const double2*>(ctx.md_pinvf + 2 * lr.prime);
        auto conv = [](uint64_t u) { return as_f64(fp_from_u(u)); };
        if (lr.smode == FS_PLAIN)
            row_epilogue<G, false>(lr, base, sw, lane,
                                   [&](uint64_t v, uint64_t) { return fp_pos_to_u(as_f64(v), p, pinv); });
        else if (lr.smode == FS_SUBP)
            row_epilogue<G, true>(lr, base, sw, lane, [&](uint64_t v, uint64_t a) {
                return fp_pos_to_u(__dadd_rn(conv(a), fp_mulw_sh(-as_f64(v), c.x, c.y, p, kRint + 1.0)), p, pinv);
            });
        else
            row_epilogue<G, true>(lr, base, sw, lane, [&](uint64_t v, uint64_t a) {
                return fp_pos_to_u(fp_mulw_sh(__dsub_rn(conv(a), as_f64(v)), c.x, c.y, p, kRint + 1.0), p, pinv);
            });
        return;
    }
    const ulonglong2 c = lr.smode == FS_PLAIN ? make_ulonglong2(0, 0)
                         : lr.smode == FS_RESCALE ? ldg2(ctx.rs_qinv, (size_t)lr.level * ctx.L + lr.prime)
                                                  : ldg2(ctx.md_pinv, lr.prime);
    if (lr.smode == FS_PLAIN)
        row_epilogue<G, false>(lr, base, sw, lane, [&](uint64_t v, uint64_t) { return reduce_fwd(v, pc); });
    else if (lr.smode == FS_SUBP)
        row_epilogue<G, true>(lr, base, sw, lane, [&](uint64_t v, uint64_t a) {
            return sub_mod(a, mul_shoup(reduce_fwd(v, pc), c.x, c.y, pc.p), pc.p);
        });
    else
        row_epilogue<G, true>(lr, base, sw, lane, [&](uint64_t v, uint64_t a) {
            return mul_shoup(sub_mod(a, reduce_fwd(v, pc), pc.p), c.x, c.y, pc.p);
        });
}

// ---------------------------------------------------------------------------
// forward, pass 2 of the ModUp digits fused with the key-switch inner product
// ---------------------------------------------------------------------------
// One warp owns a tile of RW rows of output limb m (prime t) of batch element
// b.  First it runs the row stages of every digit limb of prime t that needs
// them (the column pass has already run in place), each into its own
// shared-memory tile; when t lies inside digit d, that digit's value is the
// original evaluation limb instead and is read in the epilogue.  Then one
// epilogue forms  XB[m] = sum_d D_d kb[d][t],  XA[m] = sum_d D_d ka[d][t]
// with the key and own-limb loads of all digits in flight together.  The
// digit limbs never return to HBM in evaluation form and are not read back
// by a separate inner-product kernel.  The prime, and so the twiddles, are
// the same for every digit of the warp.  Reference: the key-switch dot
// products fused into the NTT epilogue, ksk_dot_fusion / ksk_dot_acc_fusion
// (src/NTTfusions.cuh:295-345) in the KSK_DOT modes of NTT_ (src/NTT.cu:680-700).
//
// The own limb is the product a1 b1 of the element's inputs, formed here, and
// the ciphertext limbs' epilogue adds the rest of the tensor product, as in
// k_ks_hmult.
//
// Sums: for primes below 2^50 with fp_sums, each product is an exact FP64
// fp_mulmod of a transformed value (below 1.7p: the last row stage centres) or
// the own limb (< p) with a key residue (< p): |r| <= (1/2 + 1.7 * 3/8) p, and
// up to 6 digits sum below 6.9p < 2^53; otherwise products are accumulated in 128 bits.
// Results are canonical residues, identical to k_ks_inner's.
//
// MB: CTAs of four warps per SM the register budget is cut for (6, or 4 where
// every digit needs a tile)
template <int LR, int LC>
constexpr size_t ks_warp_words(int tiles) {
    using G = RowGeo<LR, LC>;
    return (size_t)G::SW * tiles + 2 * G::TW;
}

template <int LR, int LC, bool FP, int MB>
__global__ void __launch_bounds__(RowGeo<LR, LC>::NT, MB)
    k_ntt_fwd_rows_ks(const __grid_constant__ DevCtx ctx, const __grid_constant__ KsHmultArgs a, int tiles) {
    using G = RowGeo<LR, LC>;
    extern __shared__ __align__(16) uint64_t ks_sm[];  // per warp: twiddles, then one tile per digit needing rows

    pdl_trigger();
    const int level = a.level, n = level + 1;
    const int m = a.m0 + (int)blockIdx.z;
    const size_t boff = (size_t)blockIdx.y * a.bstride;
    const int t = m < n ? m : ctx.L + (m - n);
    const PrimeConst pc = ctx.pc[t];
    const bool fp = FP && pc.p < kFpPrimeBound;
    const uint64_t* twg = (fp ? ctx.fwd_twf : ctx.fwd_tw) + (size_t)t * 2 * ctx.N;

    const int w = threadIdx.x / G::WL, lane = threadIdx.x % G::WL;
    const int th = lane % G::TPR, rl = lane / G::TPR;
    const int row0 = (blockIdx.x * G::W + w) * G::RW;
    const size_t base = (size_t)row0 * G::C;
    const size_t kstride = (size_t)(ctx.L + ctx.K) * ctx.N;
    const size_t limb_off = (size_t)t * ctx.N + base;
    const int nd = a.nd;
    int d_own = -1;  // digit holding t (its value is the own limb)
    for (int d = 0; d < nd; ++d)
        if (m < n && (unsigned)(t - d * ctx.alpha) < (unsigned)ctx.alpha) d_own = d;
    uint64_t* wsm = ks_sm + (size_t)w * ks_warp_words<LR, LC>(tiles);
    ulonglong2* s_tw = reinterpret_cast<ulonglong2*>(wsm);
    uint64_t* s_tile = wsm + 2 * G::TW;
    stage_row_tw<LR, LC>(s_tw, twg, row0, lane);
    RowFwd<LR, LC, FP> rf;
    if (fp) rf.load_d(twg, row0 + rl, th);

    // the epilogue's key tiles (and own tile) are read once per batch from
    // HBM; start those reads now, under the transforms
    for (int d = 0; d < nd; ++d) {
        prefetch_l2(a.kb + d * kstride + limb_off + lane * 16);
        prefetch_l2(a.ka + d * kstride + limb_off + lane * 16);
    }
    pdl_wait();
    const bool tensor = m < n;
    const int bi = blockIdx.y;
    if (tensor) {
        prefetch_l2(a.a0[bi] + limb_off + lane * 16);
        prefetch_l2(a.a1[bi] + limb_off + lane * 16);
        prefetch_l2(a.b0[bi] + limb_off + lane * 16);
        prefetch_l2(a.b1[bi] + limb_off + lane * 16);
    }
    stage_wait();
    __syncwarp(G::MASK);

    const double p = __ull2double_rn(pc.p), pinv = as_f64(pc.pinv_f64);
#pragma unroll 1
    for (int d = 0, slot = 0; d < nd; ++d) {
        if (d == d_own) continue;
        const int lo = d * ctx.alpha, hi = min(lo + ctx.alpha - 1, level), cnt = hi - lo + 1;
        const int md = m < n ? (t < lo ? t : t - cnt) : (n - cnt) + (m - n);
        const uint64_t* src = a.dig + boff + ((size_t)d * a.dig_stride + md) * ctx.N + base + rl * G::C;
        uint64_t* sw = s_tile + (size_t)slot * G::SW;
        ++slot;
        uint64_t x[16];
#pragma unroll
        for (int k = 0; k < 16; ++k) x[k] = src[th + (k << (LC - 4))];
        if (fp)
            rf.run_fp(x, sw, s_tw, lane, th, rl, p, pinv, kRint);
        else
            rf.run_int(x, sw, s_tw, twg, row0 + rl, lane, th, rl, pc);
        __syncwarp(G::MASK);
#pragma unroll
        for (int k = 0; k < 16; ++k) sw[17 * lane + k] = x[k];
    }
    __syncwarp(G::MASK);

    const bool fpk = a.fp_sums && pc.p < kFpPrimeBound;
    uint64_t* xb = a.xb + boff + (size_t)m * ctx.N + base;
    uint64_t* xa = a.xa + boff + (size_t)m * ctx.N + base;
    auto word = [&](const uint64_t* q, int i) { return *reinterpret_cast<const ulonglong2*>(q + limb_off + i); };
    for (int i = 2 * lane; i < G::GW; i += 2 * G::WL) {
        const int wi = padi(i);
        ulonglong2 ob, oa;
        ulonglong2 ta0, ta1, tb0, tb1;  // the inputs of the tensor product
        if (tensor) {
            ta0 = word(a.a0[bi], i);
            ta1 = word(a.a1[bi], i);
            tb0 = word(a.b0[bi], i);
            tb1 = word(a.b1[bi], i);
        }
        if (fpk) {
            double sb0 = 0, sb1 = 0, sa0 = 0, sa1 = 0;
            auto conv = [](uint64_t u) { return as_f64(fp_from_u(u)); };
            auto prod = [&](uint64_t u, uint64_t v) { return fp_mulmod(conv(u), conv(v), p, pinv); };
#pragma unroll
            for (int d = 0; d < 6; ++d) {
                if (d < nd) {
                    const ulonglong2 kb2 = *reinterpret_cast<const ulonglong2*>(a.kb + d * kstride + limb_off + i);
                    const ulonglong2 ka2 = *reinterpret_cast<const ulonglong2*>(a.ka + d * kstride + limb_off + i);
                    double x0, x1;
                    if (d == d_own) {
                        x0 = prod(ta1.x, tb1.x);
                        x1 = prod(ta1.y, tb1.y);
                    } else {
                        const uint64_t* tile = s_tile + (size_t)(d_own >= 0 && d > d_own ? d - 1 : d) * G::SW;
                        if (fp) {
                            x0 = as_f64(tile[wi]);
                            x1 = as_f64(tile[wi + 1]);
                        } else {
                            x0 = as_f64(fp_from_u(reduce_fwd(tile[wi], pc)));
                            x1 = as_f64(fp_from_u(reduce_fwd(tile[wi + 1], pc)));
                        }
                    }
                    sb0 = __dadd_rn(sb0, fp_mulmod(x0, as_f64(fp_from_u(kb2.x)), p, pinv));
                    sb1 = __dadd_rn(sb1, fp_mulmod(x1, as_f64(fp_from_u(kb2.y)), p, pinv));
                    sa0 = __dadd_rn(sa0, fp_mulmod(x0, as_f64(fp_from_u(ka2.x)), p, pinv));
                    sa1 = __dadd_rn(sa1, fp_mulmod(x1, as_f64(fp_from_u(ka2.y)), p, pinv));
                }
            }
            if (tensor) {
                // P^-1 times the centred sum (< 0.54p) plus one or two products
                // (<= 0.875p each)
                const double2 ci = *reinterpret_cast<const double2*>(ctx.md_pinvf + 2 * t);
                auto down = [&](double s) { return fp_mulw(fp_center(s, p, pinv), ci.x, ci.y, p); };
                sb0 = __dadd_rn(down(sb0), prod(ta0.x, tb0.x));
                sb1 = __dadd_rn(down(sb1), prod(ta0.y, tb0.y));
                sa0 = __dadd_rn(__dadd_rn(down(sa0), prod(ta0.x, tb1.x)), prod(ta1.x, tb0.x));
                sa1 = __dadd_rn(__dadd_rn(down(sa1), prod(ta0.y, tb1.y)), prod(ta1.y, tb0.y));
            }
            ob.x = fp_sum_to_u(sb0, p, pinv);
            ob.y = fp_sum_to_u(sb1, p, pinv);
            oa.x = fp_sum_to_u(sa0, p, pinv);
            oa.y = fp_sum_to_u(sa1, p, pinv);
        } else {
            Acc128 sb0, sb1, sa0, sa1;
#pragma unroll
            for (int d = 0; d < 6; ++d) {
                if (d < nd) {
                    const ulonglong2 kb2 = *reinterpret_cast<const ulonglong2*>(a.kb + d * kstride + limb_off + i);
                    const ulonglong2 ka2 = *reinterpret_cast<const ulonglong2*>(a.ka + d * kstride + limb_off + i);
                    uint64_t x0, x1;
                    if (d == d_own) {
                        x0 = mul_mod(ta1.x, tb1.x, pc);
                        x1 = mul_mod(ta1.y, tb1.y, pc);
                    } else {
                        const uint64_t* tile = s_tile + (size_t)(d_own >= 0 && d > d_own ? d - 1 : d) * G::SW;
                        if (fp) {
                            x0 = fp_to_u(as_f64(tile[wi]), p, pinv);
                            x1 = fp_to_u(as_f64(tile[wi + 1]), p, pinv);
                        } else {
                            x0 = reduce_fwd(tile[wi], pc);
                            x1 = reduce_fwd(tile[wi + 1], pc);
                        }
                    }
                    sb0.mac(x0, kb2.x);
                    sb1.mac(x1, kb2.y);
                    sa0.mac(x0, ka2.x);
                    sa1.mac(x1, ka2.y);
                }
            }
            ob.x = sb0.reduce(pc);
            ob.y = sb1.reduce(pc);
            oa.x = sa0.reduce(pc);
            oa.y = sa1.reduce(pc);
            if (tensor) {
                const ulonglong2 ci = ldg2(ctx.md_pinv, t);
                auto sum = [&](uint64_t s, uint64_t u0, uint64_t v0, uint64_t u1, uint64_t v1) {
                    Acc128 e;
                    e.mac(u0, v0);
                    e.mac(u1, v1);
                    return add_mod(mul_shoup(s, ci.x, ci.y, pc.p), e.reduce(pc), pc.p);
                };
                ob.x = sum(ob.x, ta0.x, tb0.x, 0, 0);
                ob.y = sum(ob.y, ta0.y, tb0.y, 0, 0);
                oa.x = sum(oa.x, ta0.x, tb1.x, ta1.x, tb0.x);
                oa.y = sum(oa.y, ta0.y, tb1.y, ta1.y, tb0.y);
            }
        }
        *reinterpret_cast<ulonglong2*>(xb + i) = ob;
        *reinterpret_cast<ulonglong2*>(xa + i) = oa;
    }
}

// ---------------------------------------------------------------------------
// inverse, pass A: row stages logN-1..LR (GS), with fused prologue
// ---------------------------------------------------------------------------
// Prologue modes of the inverse row pass (per segment): IL_PLAIN reads `in`,
// IL_MUL the product in*in2.
// ODD: the limbs may start at an odd word, as a caller's of fides_ntt and
// fides_ntt_batch (an odd stride) may; IL_PLAIN, 8-byte loads.  An instance of its own:
// the choice made in the kernel cost an affine step at N = 2^14 0.25 of 68.4 us.
template <int LR, int LC, bool FP, bool WIDE, bool ODD = false>
__global__ void __launch_bounds__(RowGeo<LR, LC>::NT, WIDE ? RowGeo<LR, LC>::MINB_WIDE : RowGeo<LR, LC>::MINB)
    k_ntt_inv_rows(const __grid_constant__ DevCtx ctx, const __grid_constant__ LimbMap map) {
    using G = RowGeo<LR, LC>;
    constexpr int NST2 = LC - 4;
    __shared__ __align__(16) uint64_t sm[G::W * G::SW];
    __shared__ ulonglong2 s_twa[G::W * G::TW];

    pdl_trigger();
    const LimbRef lr = resolve_limb(map, blockIdx.z, blockIdx.y, ctx.N, ctx.L);
    const PrimeConst pc = ctx.pc[lr.prime];
    const bool fp = FP && pc.p < kFpPrimeBound;
    const uint64_t* twg = (fp ? ctx.inv_twf : ctx.inv_tw) + (size_t)lr.prime * 2 * ctx.N;

    const int w = threadIdx.x / G::WL, lane = threadIdx.x % G::WL;
    const int th = lane % G::TPR, rl = lane / G::TPR;
    const int row0 = (blockIdx.x * G::W + w) * G::RW;
    const int row = row0 + rl;
    const size_t base = (size_t)row0 * G::C;
    uint64_t* sw = sm + w * G::SW;
    ulonglong2* s_tw = s_twa + w * G::TW;
    stage_row_tw<LR, LC>(s_tw, twg, row0, lane);
    // this thread's D_s' (see stage_row_tw), by partner bit
    ulonglong2 D[NST2 > 0 ? NST2 : 1];
    if (fp) {
#pragma unroll
        for (int kb = 0; kb < NST2; ++kb)
            D[kb] = ldg2(twg, ((size_t)(G::R + row) << (LC - 1 - kb)) + ((size_t)th << (3 - kb)));
    }
    const double p = __ull2double_rn(pc.p), pinv = as_f64(pc.pinv_f64);
    pdl_wait();
    uint64_t x[16];
    if constexpr (ODD) {
#pragma unroll 1
        for (int i = lane; i < G::GW; i += G::WL) {
            const uint64_t u = lr.in[base + i];
            sw[padi(i)] = fp ? fp_from_u(u) : u;
        }
    } else {
        // all 16 words of the lane are loaded before any is used, so the
        // global loads (twice as many with a second operand) are in flight together
        ulonglong2 v[8];
        const uint64_t* in = lr.in + base + 2 * lane;
#pragma unroll
        for (int q = 0; q < 8; ++q) v[q] = *reinterpret_cast<const ulonglong2*>(in + 2 * G::WL * q);
        if (lr.lmode == IL_PLAIN) {
            if (fp) {
#pragma unroll
                for (int q = 0; q < 8; ++q) {
                    v[q].x = fp_from_u(v[q].x);
                    v[q].y = fp_from_u(v[q].y);
                }
            }
        } else {
            const uint64_t* in2 = lr.in2 + base + 2 * lane;
            // double-precision limbs: exact products, centred (the schedule's entry bound)
            auto one = [&](uint64_t a, uint64_t b) -> uint64_t {
                if (fp)
                    return as_u64(fp_center(fp_mulmod(as_f64(fp_from_u(a)), as_f64(fp_from_u(b)), p, pinv), p, pinv));
                return mul_mod(a, b, pc);
            };
#pragma unroll
            for (int q = 0; q < 8; ++q) {
                const ulonglong2 u = *reinterpret_cast<const ulonglong2*>(in2 + 2 * G::WL * q);
                v[q].x = one(v[q].x, u.x);
                v[q].y = one(v[q].y, u.y);
            }
        }
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            const int wi = padi(2 * lane + 2 * G::WL * q);
            sw[wi] = v[q].x;
            sw[wi + 1] = v[q].y;
        }
    }
    stage_wait();
    __syncwarp(G::MASK);

    if constexpr (NST2 > 0) {
#pragma unroll
        for (int k = 0; k < 16; ++k) x[k] = sw[17 * lane + k];
        if (fp) {
            const ulonglong2* gw = s_tw + G::RW * 15;
            fp_inv<LR, LC, 0, 0, NST2>(
                x, [&](int kb, int g) { return form_tw(D[kb], as_f64(gw[g].x), g, p, pinv); }, p, pinv);
        } else {
            int_stages<0, NST2 - 1, 1, 2>(
                x,
                [&](int kb, int g) {
                    return ldg2(twg, ((size_t)(G::R + row) << (LC - 1 - kb)) + ((size_t)th << (3 - kb)) + g);
                },
                pc.p, pc.two_p);
        }
#pragma unroll
        for (int k = 0; k < 16; ++k) sw[17 * lane + k] = x[k];
        __syncwarp(G::MASK);
    }
#pragma unroll
    for (int k = 0; k < 16; ++k) x[k] = sw[padi(rl * G::C + th + (k << (LC - 4)))];
    const ulonglong2* g1 = s_tw + rl * 15;
    auto getb = [&](int kb, int g) { return g1[(8 >> kb) - 1 + g]; };
    if (fp)
        fp_inv<LR, LC, 1, 0, 4>(x, getb, p, pinv);
    else
        int_stages<0, 3, 1, 2>(x, getb, pc.p, pc.two_p);
    // double-precision limbs leave as doubles; the column pass continues on
    // them without converting
    uint64_t* dst = lr.out + base + rl * G::C;
#pragma unroll
    for (int k = 0; k < 16; ++k) dst[th + (k << (LC - 4))] = x[k];
}

// ---------------------------------------------------------------------------
// inverse, pass B: column stages LR-1..0 (GS), N^-1 and CRT scale folded in
// ---------------------------------------------------------------------------
__device__ __forceinline__ const uint64_t* inv_scale_entry(const DevCtx& ctx, const LimbRef& lr) {
    switch (lr.smode) {
        case IS_MODUP: return ctx.modup_scale + ((size_t)lr.level * ctx.L + lr.prime) * 4;
        case IS_MODDOWN: return ctx.md_scale + (size_t)(lr.prime - ctx.L) * 4;
        default: return ctx.intt_scale + (size_t)lr.prime * 4;
    }
}

template <int LR, int LC, bool FP, bool WIDE>
__global__ void __launch_bounds__(ColGeo<LR, LC>::NT, WIDE ? ColGeo<LR, LC>::MINB_WIDE : ColGeo<LR, LC>::MINB)
    k_ntt_inv_cols(const __grid_constant__ DevCtx ctx, const __grid_constant__ LimbMap map) {
    using G = ColGeo<LR, LC>;
    constexpr int C = G::C, TC = G::TC;
    __shared__ __align__(16) uint64_t sm[LR > 4 ? G::R * TC : 1];
    __shared__ ulonglong2 tws[G::R];

    pdl_trigger();
    const LimbRef lr = resolve_limb(map, blockIdx.z, blockIdx.y, ctx.N, ctx.L);
    const PrimeConst pc = ctx.pc[lr.prime];
    const bool fp = FP && pc.p < kFpPrimeBound;
    const ulonglong2* twg = reinterpret_cast<const ulonglong2*>(fp ? ctx.inv_twf : ctx.inv_tw) + (size_t)lr.prime * ctx.N;
    for (int i = threadIdx.x; i < G::R; i += G::NT) stage16(&tws[i], &twg[i]);
    const uint64_t* se = inv_scale_entry(ctx, lr);
    const ulonglong2 s0 = ldg2(se, 0), s1 = ldg2(se, 1);

    const int c = threadIdx.x % TC, th = threadIdx.x / TC;
    const int col = blockIdx.x * TC + c;
    const double p = __ull2double_rn(pc.p), pinv = as_f64(pc.pinv_f64);
    pdl_wait();
    uint64_t x[16];
    if constexpr (LR > 4) {
#pragma unroll
        for (int k = 0; k < 16; ++k) x[k] = lr.out[(size_t)((th << 4) + k) * C + col];
        stage_wait();
        __syncthreads();
        auto ga = [&](int kb, int g) { return tws[(1 << (LR - 1 - kb)) + (th << (3 - kb)) + g]; };
        if (fp)
            fp_inv<LR, LC, 2, 0, LR - 4>(x, ga, p, pinv);
        else
            int_stages<0, LR - 5, 1, 2>(x, ga, pc.p, pc.two_p);
#pragma unroll
        for (int k = 0; k < 16; ++k) sm[((th << 4) + k) * TC + c] = x[k];
        __syncthreads();
#pragma unroll
        for (int k = 0; k < 16; ++k) x[k] = sm[(th + (k << (LR - 4))) * TC + c];
    } else {
#pragma unroll
        for (int k = 0; k < 16; ++k) x[k] = lr.out[(size_t)(th + k) * C + col];
        stage_wait();
        __syncthreads();
    }
    auto gb = [&](int kb, int g) { return tws[(8 >> kb) + g]; };
    // last stage (twiddle index 1) with the N^-1 * scale fold
    if (fp) {
        fp_inv<LR, LC, 3, 0, 3>(x, gb, p, pinv);
        const double a0 = fp_centred_const(s0.x, pc.p), a1 = fp_centred_const(s1.x, pc.p);
        const double a0q = __dmul_rn(a0, pinv), a1q = __dmul_rn(a1, pinv);
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const double X = as_f64(x[k]), Y = as_f64(x[k + 8]);
            x[k] = fp_pos_to_u(fp_mulw_sh(__dadd_rn(X, Y), a0, a0q, p, kRint + 2.0), p, pinv);
            x[k + 8] = fp_pos_to_u(fp_mulw_sh(__dsub_rn(X, Y), a1, a1q, p, kRint + 2.0), p, pinv);
        }
    } else {
        int_stages<0, 2, 1, 2>(x, gb, pc.p, pc.two_p);
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const uint64_t X = x[k], Y = x[k + 8];
            x[k] = mul_shoup(X + Y, s0.x, s0.y, pc.p);
            x[k + 8] = mul_shoup(X - Y + pc.two_p, s1.x, s1.y, pc.p);
        }
    }
#pragma unroll
    for (int k = 0; k < 16; ++k) lr.out[(size_t)(th + (k << (LR - 4))) * C + col] = x[k];
}

// ---------------------------------------------------------------------------
// launchers of one ring dimension
// ---------------------------------------------------------------------------
// grid (tiles, batch element, limb): CTAs run x fastest, then y, so the
// elements of a batch that share a prime run together and its twiddle table is
// fetched from HBM once per launch rather than once per element
// Threads up to which a launch takes the wide instances, where the two curves
// cross (back to back, medians of five; 65536 words are 4096 threads).  Forward
// and the short columns' inverse: 640 threads per SM, 23.1 x 65536 words.  us
// narrow / wide: N = 2^16, 50 bits, forward 18 limbs 14.9 / 11.3, 23 limbs 15.0 / 14.4,
// 24 limbs 15.0 / 15.4, 27 limbs 14.8 / 15.6; 59 bits 23 limbs 27.4 / 26.0, 24 limbs
// 27.8 / 27.7, 27 limbs 27.5 / 28.1; N = 2^13 23 x 65536 words forward 13.3 / 12.0 and
// inverse 14.2 / 12.6, 25 x forward 13.2 / 13.4 and inverse 14.2 / 14.4.  The inverse
// with columns of 128 words and more stays ahead up to one narrow wave, 768 threads
// per SM: 2^16 50 bits 24 limbs 16.4 / 16.0, 27 limbs 16.3 / 16.3; 2^15 59 bits 2 x 24
// limbs 28.4 / 26.4, 2 x 27 limbs 28.8 / 26.5.
constexpr size_t wide_threads(bool inverse, int lr) { return (size_t)(inverse && lr >= 7 ? 768 : 640) * 148; }

template <int LR, int LC>
struct NttN {
    using CG = ColGeo<LR, LC>;
    using RG = RowGeo<LR, LC>;
    static dim3 gcols(const LimbMap& m) { return dim3(CG::C / CG::TC, m.nb > 0 ? m.nb : 1, m.total); }
    static dim3 grows(const LimbMap& m) { return dim3(RG::GROUPS / RG::W, m.nb > 0 ? m.nb : 1, m.total); }

    template <bool INV, class K>
    static void launch(K narrow, K wide, dim3 g, int nt, const DevCtx& ctx, const LimbMap& map, cudaStream_t st) {
        launch_pdl((size_t)g.x * g.y * g.z * nt <= wide_threads(INV, LR) ? wide : narrow, g, nt, 0, st, ctx, map);
    }
    static void fwd_cols(const DevCtx& ctx, const LimbMap& map, cudaStream_t st) {
        if (ntt_fwd_is_fp(ctx.ntt_variant))
            launch<false>(k_ntt_fwd_cols<LR, LC, true, false>, k_ntt_fwd_cols<LR, LC, true, true>, gcols(map), CG::NT, ctx, map, st);
        else
            launch<false>(k_ntt_fwd_cols<LR, LC, false, false>, k_ntt_fwd_cols<LR, LC, false, true>, gcols(map), CG::NT, ctx, map, st);
    }
    static void fwd(const DevCtx& ctx, const LimbMap& map, cudaStream_t st) {
        fwd_cols(ctx, map, st);
        if (ntt_fwd_is_fp(ctx.ntt_variant))
            launch<false>(k_ntt_fwd_rows<LR, LC, true, false>, k_ntt_fwd_rows<LR, LC, true, true>, grows(map), RG::NT, ctx, map, st);
        else
            launch<false>(k_ntt_fwd_rows<LR, LC, false, false>, k_ntt_fwd_rows<LR, LC, false, true>, grows(map), RG::NT, ctx, map, st);
    }
    static bool odd_words(const LimbMap& m) {
        bool odd = false;
        for (int s = 0; s < m.nseg; ++s)
            odd = odd || (reinterpret_cast<uintptr_t>(m.seg[s].in) & 15) || (m.nb > 1 && (m.seg[s].bstride & 1));
        return odd;
    }
    static void inv(const DevCtx& ctx, const LimbMap& map, cudaStream_t st) {
        const bool odd = odd_words(map);
        if (ntt_inv_is_fp(ctx.intt_variant)) {
            if (odd)
                launch_pdl(k_ntt_inv_rows<LR, LC, true, false, true>, grows(map), RG::NT, 0, st, ctx, map);
            else
                launch<true>(k_ntt_inv_rows<LR, LC, true, false>, k_ntt_inv_rows<LR, LC, true, true>, grows(map), RG::NT, ctx, map, st);
            launch<true>(k_ntt_inv_cols<LR, LC, true, false>, k_ntt_inv_cols<LR, LC, true, true>, gcols(map), CG::NT, ctx, map, st);
        } else {
            if (odd)
                launch_pdl(k_ntt_inv_rows<LR, LC, false, false, true>, grows(map), RG::NT, 0, st, ctx, map);
            else
                launch<true>(k_ntt_inv_rows<LR, LC, false, false>, k_ntt_inv_rows<LR, LC, false, true>, grows(map), RG::NT, ctx, map, st);
            launch<true>(k_ntt_inv_cols<LR, LC, false, false>, k_ntt_inv_cols<LR, LC, false, true>, gcols(map), CG::NT, ctx, map, st);
        }
    }

    template <bool FP>
    static void rows_ks_v(const DevCtx& ctx, const KsHmultArgs& a, int nb, cudaStream_t st) {
        const int n = a.level + 1, nd = a.level / ctx.alpha + 1;
        auto bytes = [](int tiles) { return ks_warp_words<LR, LC>(tiles) * 8 * RG::W; };
        auto grid = [&](int limbs) { return dim3(RG::GROUPS / RG::W, nb, limbs); };
        KsHmultArgs q = a;
        q.nd = nd;
        q.m0 = 0;
        if (ctx.ks_variant & 8) {
            // split launch: the ciphertext-prime outputs need one tile less
            // (their own digit's value is a product of input limbs) and run at
            // 6 CTAs of four warps per SM; the special-prime outputs, with a
            // tile for every digit, at 4
            KsHmultArgs sp = q;
            sp.m0 = n;
            count_launches(1);
            launch_pdl(k_ntt_fwd_rows_ks<LR, LC, FP, 6>, grid(n), RG::NT, bytes(nd - 1), st, ctx, q, nd - 1);
            launch_pdl(k_ntt_fwd_rows_ks<LR, LC, FP, 4>, grid(ctx.K), RG::NT, bytes(nd), st, ctx, sp, nd);
            return;
        }
        launch_pdl(k_ntt_fwd_rows_ks<LR, LC, FP, 4>, grid(n + ctx.K), RG::NT, bytes(nd), st, ctx, q, nd);
    }
    static void rows_ks(const DevCtx& ctx, const KsHmultArgs& a, int nb, cudaStream_t st) {
        if (ntt_fwd_is_fp(ctx.ntt_variant))
            rows_ks_v<true>(ctx, a, nb, st);
        else
            rows_ks_v<false>(ctx, a, nb, st);
    }
    // Shared-memory opt-in of the fused kernel.  The limit belongs to the process
    // and device, not to a context: it is the most that any context can ask for.
    static cudaError_t prepare() {
        const int bytes = (int)(ks_warp_words<LR, LC>(kMaxFusedDigits) * 8 * RG::W);
        cudaError_t e = cudaSuccess;
        auto opt_in = [&](auto k) {
            const cudaError_t r = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
            if (e == cudaSuccess) e = r;
        };
        opt_in(k_ntt_fwd_rows_ks<LR, LC, true, 6>);
        opt_in(k_ntt_fwd_rows_ks<LR, LC, true, 4>);
        opt_in(k_ntt_fwd_rows_ks<LR, LC, false, 6>);
        opt_in(k_ntt_fwd_rows_ks<LR, LC, false, 4>);
        return e;
    }
};

}  // namespace fides
