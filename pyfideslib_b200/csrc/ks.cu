// ks.cu -- ModUp / ModDown base conversions, the hybrid key-switch inner
// products (with the tensor product) and the element-wise kernels, for sm_100a.
//
// Role in the reference: src/CKKS/Conv.cu (DecompAndModUpConv, ModDown2),
// src/CKKS/ElemenwiseBatchKernels.cu (binomialMult_, fusedDotKSK_2_,
// hoistedRotateDotKSK_2_, element-wise ops) and src/Rotation.cu
// (automorph_multi_).  Same arithmetic (exact 128-bit accumulation of the
// base-conversion sums with one reduction per output), own kernels:
//   * one thread per coefficient; the inputs of a conversion are staged once
//     in shared memory and every output limb of the digit is produced from
//     them, so each input limb is read from HBM once per digit;
//   * the inner product reads each key limb once and accumulates both key
//     halves in 128-bit registers, reducing once per output;
//   * rotations fold the automorphism into the inner product as a gather of
//     the digit values; Galois keys are held permuted to the output order, so
//     key loads and stores stay coalesced and vectorised.
#include "fp64.cuh"
#include "kernels.hpp"

namespace fides {

__device__ __forceinline__ uint32_t brev_bits(uint32_t x, int bits) { return __brev(x) >> (32 - bits); }

// src/Rotation.cuh:14-26 automorph_slot: slot of the image of slot j.
__device__ __forceinline__ uint32_t automorph_slot(int logN, uint32_t k, uint32_t j) {
    const uint32_t e = (brev_bits(j, logN) << 1) + 1;
    const uint32_t r = ((e * k) & ((2u << logN) - 1)) >> 1;
    return brev_bits(r, logN);
}

// ---------------------------------------------------------------------------
// ModUp base conversion (DecompAndModUpConv): for digit d at `level`, with
// inputs xt_i = [x_i * (Q'/q_i)^-1]_{q_i} (produced by the scaled INTT), every
// target prime t outside the digit gets  sum_i xt_i * [Q'/q_i]_t  mod t.
// Digit d's targets are stored at dig + (d*dig_stride + m)*N, m = target index
// (Q primes below the digit, Q primes above it up to `level`, then P).
//
// Each thread owns two adjacent coefficients and keeps the digit's inputs in
// registers; the block stages its slice of the conversion matrix and the
// target constants in shared memory.  Sums of up to 16 products of residues
// below 2^62 stay below 2^128, so one reduction per output suffices.
// ---------------------------------------------------------------------------
constexpr int kConvThreads = 128;
constexpr int kConvTargets = 32;  // targets per block
constexpr int kMaxConvIn = 16;    // digit size / special count handled in registers

template <class ACC>
__device__ __forceinline__ void conv_store(uint64_t* out, const ACC& a, const ACC& b, const PrimeConst& pc) {
    ulonglong2 o;
    o.x = a.reduce(pc);
    o.y = b.reduce(pc);
    *reinterpret_cast<ulonglong2*>(out) = o;
}

// MAXIN: the register arrays and unrolled loops cover MAXIN inputs (the digit
// size rounded up to a multiple of 4), so no issue slot goes to inputs that
// do not exist.  ACC: Acc128, or AccSplit when every modulus is below 2^60;
// the autotuner picks per context (identical sums).
template <int MAXIN, class ACC>
__global__ void __launch_bounds__(kConvThreads) k_modup_conv(const __grid_constant__ DevCtx ctx, int level,
                                                             const uint64_t* xt, uint64_t* dig, size_t dig_stride,
                                                             size_t bstride) {
    pdl_trigger();
    pdl_wait();
    __shared__ uint64_t sM[MAXIN][kConvTargets];
    __shared__ PrimeConst sP[kConvTargets];
    const int ndig = level / ctx.alpha + 1;
    const int d = blockIdx.y % ndig;
    const size_t boff = (size_t)(blockIdx.y / ndig) * bstride;
    xt += boff;
    dig += boff;
    const int n = level + 1;
    const int lo = d * ctx.alpha;
    const int hi = min(lo + ctx.alpha - 1, level);
    const int cnt = hi - lo + 1;
    const int ntar = n - cnt + ctx.K;
    const int m0 = blockIdx.z * kConvTargets;
    if (m0 >= ntar) return;
    const int nt = min(kConvTargets, ntar - m0);
    const int NP = ctx.L + ctx.K;
    const uint64_t* mat = ctx.modup_mat + (size_t)level * ctx.L * NP;
    for (int e = threadIdx.x; e < cnt * nt; e += kConvThreads) {
        const int i = e / nt, mm = e % nt, m = m0 + mm;
        const int jj = m < lo ? m : m + cnt;
        const int t = jj < n ? jj : ctx.L + (jj - n);
        sM[i][mm] = mat[(size_t)(lo + i) * NP + t];
        if (i == 0) sP[mm] = ctx.pc[t];
    }
    const size_t j = ((size_t)blockIdx.x * kConvThreads + threadIdx.x) * 2;
    uint64_t x0[MAXIN], x1[MAXIN];
#pragma unroll
    for (int i = 0; i < MAXIN; ++i) {
        if (i < cnt) {
            const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(xt + (size_t)(lo + i) * ctx.N + j);
            x0[i] = v.x;
            x1[i] = v.y;
        }
    }
    __syncthreads();
    uint64_t* out = dig + ((size_t)d * dig_stride + m0) * ctx.N + j;
    // two targets per iteration: four independent 128-bit accumulators
#pragma unroll 1
    for (int mm = 0; mm < nt; mm += 2) {
        const int m2 = mm + 1 < nt ? mm + 1 : mm;
        ACC a, b, c2, d2;
#pragma unroll
        for (int i = 0; i < MAXIN; ++i) {
            if (i < cnt) {
                const uint64_t M = sM[i][mm], M2 = sM[i][m2];
                a.mac(x0[i], M);
                b.mac(x1[i], M);
                c2.mac(x0[i], M2);
                d2.mac(x1[i], M2);
            }
        }
        conv_store(out + (size_t)mm * ctx.N, a, b, sP[mm]);
        if (m2 != mm) conv_store(out + (size_t)m2 * ctx.N, c2, d2, sP[m2]);
    }
}

// One coefficient per thread, four targets per iteration: half the input
// registers of k_modup_conv (twice the resident warps), the same products.
template <int MAXIN>
__global__ void __launch_bounds__(kConvThreads) k_modup_conv_c1(const __grid_constant__ DevCtx ctx, int level,
                                                                const uint64_t* xt, uint64_t* dig, size_t dig_stride,
                                                                size_t bstride) {
    pdl_trigger();
    pdl_wait();
    __shared__ uint64_t sM[MAXIN][kConvTargets];
    __shared__ PrimeConst sP[kConvTargets];
    const int ndig = level / ctx.alpha + 1;
    const int d = blockIdx.y % ndig;
    const size_t boff = (size_t)(blockIdx.y / ndig) * bstride;
    xt += boff;
    dig += boff;
    const int n = level + 1;
    const int lo = d * ctx.alpha;
    const int hi = min(lo + ctx.alpha - 1, level);
    const int cnt = hi - lo + 1;
    const int ntar = n - cnt + ctx.K;
    const int m0 = blockIdx.z * kConvTargets;
    if (m0 >= ntar) return;
    const int nt = min(kConvTargets, ntar - m0);
    const int NP = ctx.L + ctx.K;
    const uint64_t* mat = ctx.modup_mat + (size_t)level * ctx.L * NP;
    for (int e = threadIdx.x; e < cnt * nt; e += kConvThreads) {
        const int i = e / nt, mm = e % nt, m = m0 + mm;
        const int jj = m < lo ? m : m + cnt;
        const int t = jj < n ? jj : ctx.L + (jj - n);
        sM[i][mm] = mat[(size_t)(lo + i) * NP + t];
        if (i == 0) sP[mm] = ctx.pc[t];
    }
    const size_t j = (size_t)blockIdx.x * kConvThreads + threadIdx.x;
    uint64_t x[MAXIN];
#pragma unroll
    for (int i = 0; i < MAXIN; ++i)
        if (i < cnt) x[i] = xt[(size_t)(lo + i) * ctx.N + j];
    __syncthreads();
    uint64_t* out = dig + ((size_t)d * dig_stride + m0) * ctx.N + j;
#pragma unroll 1
    for (int mm = 0; mm < nt; mm += 4) {
        int m[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) m[u] = min(mm + u, nt - 1);
        Acc128 acc[4];
#pragma unroll
        for (int i = 0; i < MAXIN; ++i) {
            if (i < cnt) {
#pragma unroll
                for (int u = 0; u < 4; ++u) acc[u].mac(x[i], sM[i][m[u]]);
            }
        }
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (mm + u < nt) out[(size_t)(mm + u) * ctx.N] = acc[u].reduce(sP[mm + u]);
    }
}

bool conv_supported(const DevCtx& ctx) { return ctx.alpha <= kMaxConvIn && ctx.K <= kMaxConvIn; }

void launch_modup_conv(const DevCtx& ctx, int level, int nb, const uint64_t* xt, uint64_t* dig, size_t dig_stride,
                       size_t bstride, cudaStream_t st) {
    if ((ctx.conv_variant == 3 || ctx.conv_variant == 4) && conv_tc_supported(ctx)) {
        launch_modup_conv_tc(ctx, level, nb, xt, dig, dig_stride, bstride, st, ctx.conv_variant == 3 ? 32 : 16);
        return;
    }
    const int nd = level / ctx.alpha + 1;
    const int maxtar = level + 1 + ctx.K;
    dim3 g(ctx.N / (2 * kConvThreads), nd * nb, (maxtar + kConvTargets - 1) / kConvTargets);
    count_launches(1);
    const dim3 g1(ctx.N / kConvThreads, g.y, g.z);
#define FIDES_MODUP(M)                                                                                       \
    if (ctx.conv_variant == 2)                                                                              \
        launch_pdl(k_modup_conv_c1<M>, g1, kConvThreads, 0, st, ctx, level, xt, dig, dig_stride, bstride);          \
    else if (ctx.conv_variant == 1)                                                                         \
        launch_pdl(k_modup_conv<M, AccSplit>, g, kConvThreads, 0, st, ctx, level, xt, dig, dig_stride, bstride);    \
    else                                                                                                    \
        launch_pdl(k_modup_conv<M, Acc128>, g, kConvThreads, 0, st, ctx, level, xt, dig, dig_stride, bstride);
    if (ctx.alpha <= 4) {
        FIDES_MODUP(4)
    } else if (ctx.alpha <= 8) {
        FIDES_MODUP(8)
    } else if (ctx.alpha <= 12) {
        FIDES_MODUP(12)
    } else {
        FIDES_MODUP(16)
    }
#undef FIDES_MODUP
}

// ---------------------------------------------------------------------------
// key-switch inner product (fusedDotKSK_2_ / hoistedRotateDotKSK_2_)
//   xb[m] = sum_d D_d[t] * kb[d][t] (+ P * c0[t] for Q primes when c0 given)
//   xa[m] = sum_d D_d[t] * ka[d][t]
// over the extended basis m in [0, n+K) (prime t = m or L + m - n).  D_d[t] is
// the original evaluation value e2[t] when t lies in digit d, otherwise the
// ModUp output.  Rotations (galois g != 0): out[j] = sum_d D_d[slot(g, j)] *
// k'_d[j] (+ P * c0[slot(g, j)]), where a Galois key is held permuted,
// k'_d[j] = k_d[slot(g, j)] (the key that switches sigma_g(s) back to s):
// only the digit values and c0 are gathered, the key streams in order.
// ---------------------------------------------------------------------------
// The batch elements of one limb run one after the other (blockIdx.y), so the
// key limb (or hoisted digits) they share is fetched from HBM once and served
// from L2 to the rest of the batch.  (Folding the element into blockIdx.x and
// dividing by the batch size per thread cost 32 hoisted rotations 1.1%.)
// FPK: limbs of primes below 2^50 accumulate on the FP64 pipes (fp64.cuh):
// each product x k is reduced to |r| <= 0.875p, the sum of up to 6 digits (more
// take the integer sums) and of the P c0 term stays below 5.8p < 2^53, and one
// centring plus a floor reduction give the canonical residue -- the same values
// as the 128-bit integer sums.
// SEED: some element's key is seeded (ka null), its a half regenerated per
// coefficient; the instantiation without it carries no generator code (52
// registers; 48 measured the same).  Left free, the unrolled digit loop with
// the generator takes 56-72; the bound holds it at 48 (FP64 sums) or 40 so that
// 5-6 blocks stay resident (not the split-product accumulator, which would
// spill).
template <class ACC>
constexpr bool kIsSplitAcc = false;
template <>
constexpr bool kIsSplitAcc<AccSplit> = true;

template <class ACC, bool FPK, bool GRP, bool SEED>
__global__ void __launch_bounds__(256, SEED ? (FPK ? 5 : (kIsSplitAcc<ACC> ? 0 : 6)) : 0)
    k_ks_inner(const __grid_constant__ DevCtx ctx, int level, int nd, const __grid_constant__ KsArgs args) {
    pdl_trigger();
    pdl_wait();
    const int n = level + 1;
    const int m = blockIdx.z;
    const int bi = blockIdx.y;
    const int bx = blockIdx.x;
    const int t = m < n ? m : ctx.L + (m - n);
    const PrimeConst pc = ctx.pc[t];
    const size_t kstride = (size_t)(ctx.L + ctx.K) * ctx.N;
    const size_t boff = (size_t)bi * args.bstride;
    const uint64_t* kb = args.kb[bi];
    const uint64_t* ka = args.ka[bi];  // null: seeded, digit d's a half is uniform_mod(astream ^ (d+1) << 48, t, j)
    const uint64_t astream = args.a_seed[bi];
    // source limb of each digit for this prime (GRP, grouped hoisting: the
    // element's ModUp is that of its group, a table entry)
    const int gi = GRP ? (int)args.dig_elem[bi] : bi;
    const uint64_t* srcs[8];
#pragma unroll
    for (int d = 0; d < 8; ++d) {
        if (d < nd) {
            const int lo = d * ctx.alpha;
            const int hi = min(lo + ctx.alpha - 1, level);
            const int cnt = hi - lo + 1;
            if (m < n && t >= lo && t <= hi) {
                srcs[d] = args.own[bi] + (size_t)t * ctx.N;
            } else {
                const int md = m < n ? (t < lo ? t : t - cnt) : (n - cnt) + (m - n);
                srcs[d] = args.dig + (size_t)gi * args.dig_bstride + ((size_t)d * args.dig_stride + md) * ctx.N;
            }
        }
    }
    uint64_t* xb = args.xb + boff + (size_t)m * ctx.N;
    uint64_t* xa = args.xa + boff + (size_t)m * ctx.N;
    {
        // rotation: outputs j, j+1 gather the digit values (and c0) at the
        // automorphism's source slots; the key is stored permuted (entry j is
        // the one that pairs with output j), so its loads stay vectorised.
        // Slots 2i and 2i+1 belong to exponents e and e + N, and g (e + N) =
        // g e + N mod 2N for odd g: the sources of an adjacent pair are an
        // adjacent pair, possibly swapped, and are read as one 16-byte word.
        // (With one 8-byte gather per output and integer products by P this
        // branch took 851 us for 32 rotations of 20 limbs at N = 2^16, 70% of
        // the issue slots busy.)
        const size_t j = ((size_t)bx * blockDim.x + threadIdx.x) * 2;
        if (j >= (size_t)ctx.N) return;  // N = 256: half a block
        const uint32_t g = args.galois[bi];
        const uint32_t s0 = g ? automorph_slot(ctx.logN, g, (uint32_t)j) : (uint32_t)j;
        const bool swap = s0 & 1;
        const size_t sp = s0 & ~1u;
        auto gather = [&](const uint64_t* src) {
            const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(src + sp);
            return swap ? make_ulonglong2(v.y, v.x) : v;
        };
        const size_t koff = (size_t)t * ctx.N + j;
        const uint64_t* c0 = args.c0[bi];
        auto key_a = [&](int d) {
            ulonglong2 a;
            if (!SEED || ka) {
                a = *reinterpret_cast<const ulonglong2*>(ka + d * kstride + koff);
            } else {
                a.x = uniform_mod(astream ^ ((uint64_t)(d + 1) << 48), t, (uint32_t)j, pc.p);
                a.y = uniform_mod(astream ^ ((uint64_t)(d + 1) << 48), t, (uint32_t)j + 1, pc.p);
            }
            return a;
        };
        if constexpr (FPK) {
            // up to 6 digits: |sum| <= 6 * 0.875p + 0.54p (the P c0 term) < 8p
            if (pc.p < kFpPrimeBound && nd <= 6) {
                const double p = __ull2double_rn(pc.p), pinv = as_f64(pc.pinv_f64);
                double sb0 = 0, sb1 = 0, sa0 = 0, sa1 = 0;
                if (c0 && m < n) {
                    const double2 pm = __ldg(reinterpret_cast<const double2*>(ctx.md_pmodf) + t);
                    const ulonglong2 c = gather(c0 + (size_t)m * ctx.N);
                    sb0 = fp_mulw(as_f64(fp_from_u(c.x)), pm.x, pm.y, p);
                    sb1 = fp_mulw(as_f64(fp_from_u(c.y)), pm.x, pm.y, p);
                }
#pragma unroll
                for (int d = 0; d < 6; ++d) {
                    if (d < nd) {
                        const ulonglong2 x = gather(srcs[d]);
                        const ulonglong2 b = *reinterpret_cast<const ulonglong2*>(kb + d * kstride + koff);
                        const ulonglong2 a = key_a(d);
                        const double x0 = as_f64(fp_from_u(x.x)), x1 = as_f64(fp_from_u(x.y));
                        sb0 = __dadd_rn(sb0, fp_mulmod(x0, as_f64(fp_from_u(b.x)), p, pinv));
                        sb1 = __dadd_rn(sb1, fp_mulmod(x1, as_f64(fp_from_u(b.y)), p, pinv));
                        sa0 = __dadd_rn(sa0, fp_mulmod(x0, as_f64(fp_from_u(a.x)), p, pinv));
                        sa1 = __dadd_rn(sa1, fp_mulmod(x1, as_f64(fp_from_u(a.y)), p, pinv));
                    }
                }
                ulonglong2 ob, oa;
                ob.x = fp_sum_to_u(sb0, p, pinv);
                ob.y = fp_sum_to_u(sb1, p, pinv);
                oa.x = fp_sum_to_u(sa0, p, pinv);
                oa.y = fp_sum_to_u(sa1, p, pinv);
                *reinterpret_cast<ulonglong2*>(xb + j) = ob;
                *reinterpret_cast<ulonglong2*>(xa + j) = oa;
                return;
            }
        }
        ACC sb0, sb1, sa0, sa1;
#pragma unroll
        for (int d = 0; d < 8; ++d) {
            if (d < nd) {
                const ulonglong2 x = gather(srcs[d]);
                const ulonglong2 b = *reinterpret_cast<const ulonglong2*>(kb + d * kstride + koff);
                const ulonglong2 a = key_a(d);
                sb0.mac(x.x, b.x);
                sb1.mac(x.y, b.y);
                sa0.mac(x.x, a.x);
                sa1.mac(x.y, a.y);
            }
        }
        if (c0 && m < n) {
            const ulonglong2 pm = __ldg(reinterpret_cast<const ulonglong2*>(ctx.md_pmod) + t);
            const ulonglong2 c = gather(c0 + (size_t)m * ctx.N);
            sb0.mac(mul_shoup(c.x, pm.x, pm.y, pc.p), 1);
            sb1.mac(mul_shoup(c.y, pm.x, pm.y, pc.p), 1);
        }
        ulonglong2 ob, oa;
        ob.x = sb0.reduce(pc);
        ob.y = sb1.reduce(pc);
        oa.x = sa0.reduce(pc);
        oa.y = sa1.reduce(pc);
        *reinterpret_cast<ulonglong2*>(xb + j) = ob;
        *reinterpret_cast<ulonglong2*>(xa + j) = oa;
    }
}

template <class ACC, bool FPK, bool GRP>
static void ks_inner_go(const DevCtx& ctx, int level, int nd, const KsArgs& args, bool seeded, dim3 g,
                        cudaStream_t st) {
    if (seeded)
        launch_pdl(k_ks_inner<ACC, FPK, GRP, true>, g, 256, 0, st, ctx, level, nd, args);
    else
        launch_pdl(k_ks_inner<ACC, FPK, GRP, false>, g, 256, 0, st, ctx, level, nd, args);
}

void launch_ks_inner(const DevCtx& ctx, int level, int nb, const KsArgs& args, cudaStream_t st) {
    count_launches(1);
    bool seeded = false;
    for (int b = 0; b < nb; ++b) seeded = seeded || args.ka[b] == nullptr;
    const int nd = level / ctx.alpha + 1;
    const dim3 g((ctx.N + 511) / 512, nb, level + 1 + ctx.K);
    if (args.dig_group > 0) {
        if (ctx.ks_variant & 1)
            ks_inner_go<Acc128, true, true>(ctx, level, nd, args, seeded, g, st);
        else
            ks_inner_go<Acc128, false, true>(ctx, level, nd, args, seeded, g, st);
    } else {
        if (ctx.ks_variant & 1)
            ks_inner_go<Acc128, true, false>(ctx, level, nd, args, seeded, g, st);
        else if (ctx.conv_variant == 1)
            ks_inner_go<AccSplit, false, false>(ctx, level, nd, args, seeded, g, st);
        else
            ks_inner_go<Acc128, false, false>(ctx, level, nd, args, seeded, g, st);
    }
}

// ---------------------------------------------------------------------------
// key-switch inner product of a product (a0, a1)(b0, b1), with the tensor
// product (binomialMult_) formed on the way: the own limb of digit d is a1 b1,
// and the ciphertext limbs leave as e + P^-1 x,
//   XB[m] = a0 b0 + P^-1 sum_d D_d[t] kb[d][t]
//   XA[m] = a0 b1 + a1 b0 + P^-1 sum_d D_d[t] ka[d][t]      (m < n),
// the special limbs as the sums.  FP64 limbs, up to 8 digits: the own digit's
// product is signed, |a1 b1 mod| <= 0.875p, so each digit's product with the key is
// too, the sum is at most 7p < 2^53, and centred, times P^-1 (0.54p) and with the
// one or two products added it stays below 2.3p.  (tests/test_exact_arith.py runs
// these sums on the host.)  Integer sums as in k_ks_inner.
// ---------------------------------------------------------------------------
// Its loads' latency bounds this kernel (8 pairs: 8 of 16 stall cycles per
// instruction, DRAM 53%).
// ModUp's inverse transform takes a1 b1 in its own load, so no limb of the
// tensor product is stored: 8 limbs of traffic per limb of the level instead of
// 13 around the tensor product, that inverse, this kernel and the final row
// pass, and one launch less.  64 registers: 4 CTAs per SM, without spills (left
// free it takes 72, 3 CTAs, one product at N = 2^16 258 us instead of 251).
// N = 2^16, L = 30, with a tensor kernel / this: one product 260 / 248 us, 21
// pairs at uneven levels 6449 / 6072 us.  Large batches form these sums in the
// epilogue of the digits' row pass instead (k_ntt_fwd_rows_ks).
template <bool FPK, bool SEED>
__global__ void __launch_bounds__(256, 4)
    k_ks_hmult(const __grid_constant__ DevCtx ctx, const __grid_constant__ KsHmultArgs args) {
    pdl_trigger();
    pdl_wait();
    const int n = args.level + 1, nd = args.nd;
    const int m = blockIdx.z;
    const int bi = blockIdx.y;  // a limb's elements run together and share its key tiles through L2
    const bool tensor = m < n;
    const int t = tensor ? m : ctx.L + (m - n);
    const PrimeConst pc = ctx.pc[t];
    const size_t kstride = (size_t)(ctx.L + ctx.K) * ctx.N;
    const size_t boff = (size_t)bi * args.bstride;
    const size_t j = ((size_t)blockIdx.x * 256 + threadIdx.x) * 2;
    if (j >= (size_t)ctx.N) return;  // N = 256: half a block
    const size_t koff = (size_t)t * ctx.N + j;
    auto word = [&](const uint64_t* q) { return *reinterpret_cast<const ulonglong2*>(q + koff); };
    auto own_digit = [&](int d) { return tensor && (unsigned)(m - d * ctx.alpha) < (unsigned)ctx.alpha; };
    auto digit_at = [&](int d) {  // ModUp output of digit d: the Q primes outside it, then the special primes
        const int lo = d * ctx.alpha, cnt = min(ctx.alpha, n - lo);
        return args.dig + boff + ((size_t)d * args.dig_stride + (m < lo ? m : m - cnt)) * ctx.N + j;
    };
    auto digit = [&](int d) { return *reinterpret_cast<const ulonglong2*>(digit_at(d)); };
    auto key_a = [&](int d) {
        ulonglong2 a;
        if (!SEED) {
            a = word(args.ka + d * kstride);
        } else {
            a.x = uniform_mod(args.a_seed ^ ((uint64_t)(d + 1) << 48), t, (uint32_t)j, pc.p);
            a.y = uniform_mod(args.a_seed ^ ((uint64_t)(d + 1) << 48), t, (uint32_t)j + 1, pc.p);
        }
        return a;
    };
    // The later digits' words are asked for at the start: left to the loop, each
    // digit waited for HBM in turn (one product at N = 2^16, L = 30 251 us instead of
    // 248, 21 pairs 6094 instead of 6072).  In k_ks_inner, whose digits come from
    // L2, the same for its keys was 0.3-1% slower.
    for (int d = 1; d < nd; ++d) {
        prefetch_l2(args.kb + d * kstride + koff);
        if (!SEED) prefetch_l2(args.ka + d * kstride + koff);
        if (!own_digit(d)) prefetch_l2(digit_at(d));
    }
    ulonglong2 a0, a1, b0, b1;
    if (tensor) {
        a0 = word(args.a0[bi]);
        a1 = word(args.a1[bi]);
        b0 = word(args.b0[bi]);
        b1 = word(args.b1[bi]);
    }
    ulonglong2 ob, oa;
    if (FPK && pc.p < kFpPrimeBound) {
        const double p = __ull2double_rn(pc.p), pinv = as_f64(pc.pinv_f64);
        auto conv = [](uint64_t u) { return as_f64(fp_from_u(u)); };
        auto prod = [&](uint64_t u, uint64_t v) { return fp_mulmod(conv(u), conv(v), p, pinv); };
        double sb0 = 0, sb1 = 0, sa0 = 0, sa1 = 0;
#pragma unroll
        for (int d = 0; d < 8; ++d) {
            if (d < nd) {
                const ulonglong2 b = word(args.kb + d * kstride), a = key_a(d);
                double x0, x1;
                if (own_digit(d)) {
                    x0 = prod(a1.x, b1.x);
                    x1 = prod(a1.y, b1.y);
                } else {
                    const ulonglong2 x = digit(d);
                    x0 = conv(x.x);
                    x1 = conv(x.y);
                }
                sb0 = __dadd_rn(sb0, fp_mulmod(x0, conv(b.x), p, pinv));
                sb1 = __dadd_rn(sb1, fp_mulmod(x1, conv(b.y), p, pinv));
                sa0 = __dadd_rn(sa0, fp_mulmod(x0, conv(a.x), p, pinv));
                sa1 = __dadd_rn(sa1, fp_mulmod(x1, conv(a.y), p, pinv));
            }
        }
        if (tensor) {
            // P^-1 times the centred sum (< 0.54p) plus one or two products (<= 0.875p each)
            const double2 ci = __ldg(reinterpret_cast<const double2*>(ctx.md_pinvf) + t);
            auto down = [&](double s) { return fp_mulw(fp_center(s, p, pinv), ci.x, ci.y, p); };
            sb0 = __dadd_rn(down(sb0), prod(a0.x, b0.x));
            sb1 = __dadd_rn(down(sb1), prod(a0.y, b0.y));
            sa0 = __dadd_rn(__dadd_rn(down(sa0), prod(a0.x, b1.x)), prod(a1.x, b0.x));
            sa1 = __dadd_rn(__dadd_rn(down(sa1), prod(a0.y, b1.y)), prod(a1.y, b0.y));
        }
        ob.x = fp_sum_to_u(sb0, p, pinv);
        ob.y = fp_sum_to_u(sb1, p, pinv);
        oa.x = fp_sum_to_u(sa0, p, pinv);
        oa.y = fp_sum_to_u(sa1, p, pinv);
    } else {
        Acc128 sb0, sb1, sa0, sa1;
#pragma unroll
        for (int d = 0; d < 8; ++d) {
            if (d < nd) {
                const ulonglong2 b = word(args.kb + d * kstride), a = key_a(d);
                const ulonglong2 x = own_digit(d) ? make_ulonglong2(mul_mod(a1.x, b1.x, pc), mul_mod(a1.y, b1.y, pc))
                                                  : digit(d);
                sb0.mac(x.x, b.x);
                sb1.mac(x.y, b.y);
                sa0.mac(x.x, a.x);
                sa1.mac(x.y, a.y);
            }
        }
        ob.x = sb0.reduce(pc);
        ob.y = sb1.reduce(pc);
        oa.x = sa0.reduce(pc);
        oa.y = sa1.reduce(pc);
        if (tensor) {
            const ulonglong2 ci = __ldg(reinterpret_cast<const ulonglong2*>(ctx.md_pinv) + t);
            auto cross = [&](uint64_t u0, uint64_t v0, uint64_t u1, uint64_t v1) {
                Acc128 e;
                e.mac(u0, v0);
                e.mac(u1, v1);
                return e.reduce(pc);
            };
            auto down = [&](uint64_t s, uint64_t e) { return add_mod(mul_shoup(s, ci.x, ci.y, pc.p), e, pc.p); };
            ob.x = down(ob.x, mul_mod(a0.x, b0.x, pc));
            ob.y = down(ob.y, mul_mod(a0.y, b0.y, pc));
            oa.x = down(oa.x, cross(a0.x, b1.x, a1.x, b0.x));
            oa.y = down(oa.y, cross(a0.y, b1.y, a1.y, b0.y));
        }
    }
    const size_t o = boff + (size_t)m * ctx.N + j;
    *reinterpret_cast<ulonglong2*>(args.xb + o) = ob;
    *reinterpret_cast<ulonglong2*>(args.xa + o) = oa;
}

template <bool FPK>
static void ks_hmult_go(const DevCtx& ctx, int nb, const KsHmultArgs& args, cudaStream_t st) {
    const dim3 g((ctx.N + 511) / 512, nb, args.level + 1 + ctx.K);
    if (args.ka == nullptr)
        launch_pdl(k_ks_hmult<FPK, true>, g, 256, 0, st, ctx, args);
    else
        launch_pdl(k_ks_hmult<FPK, false>, g, 256, 0, st, ctx, args);
}

void launch_ks_hmult(const DevCtx& ctx, int nb, const KsHmultArgs& a, cudaStream_t st) {
    count_launches(1);
    KsHmultArgs args = a;
    args.nd = a.level / ctx.alpha + 1;
    if (ctx.ks_variant & 1)
        ks_hmult_go<true>(ctx, nb, args, st);
    else
        ks_hmult_go<false>(ctx, nb, args, st);
}

// ---------------------------------------------------------------------------
// ModDown base conversion (ModDown2), both halves of a key-switch result in
// one launch (blockIdx.z = half).  y = special limbs already scaled by
// (P/p_k)^-1 (scaled INTT).  Without ttop: w_j = sum_k y_k [P/p_k]_{q_j} for
// j = 0..level.  With ttop (fused rescale; ttop = INTT(e_l + P^-1 x_l)):
//   conv_l = sum_k y_k [P/p_k]_{q_l};  tl = ttop - P^-1 conv_l  (mod q_l)
//   w_j = P^-1 conv_j + SwitchModulus(tl, q_l -> q_j)  for j < level.
// ---------------------------------------------------------------------------


template <int MAXIN, class ACC>
__global__ void __launch_bounds__(kConvThreads) k_moddown_conv(const __grid_constant__ DevCtx ctx, int level,
                                                               const __grid_constant__ MdArgs args) {
    pdl_trigger();
    pdl_wait();
    __shared__ uint64_t sM[MAXIN][kConvTargets];
    __shared__ PrimeConst sP[kConvTargets];
    __shared__ ulonglong2 sPinv[kConvTargets];
    const int half = blockIdx.z & 1;
    const size_t boff = (size_t)(blockIdx.z >> 1) * args.bstride;
    const uint64_t* y = args.y[half] + boff;
    uint64_t* w = args.w[half] + boff;
    const uint64_t* ttop = args.ttop[half] ? args.ttop[half] + boff : nullptr;
    const int K = ctx.K, L = ctx.L;
    const int nout = ttop ? level : level + 1;
    const int q0 = blockIdx.y * kConvTargets;
    const int nt = min(kConvTargets, nout - q0);
    if (nt <= 0) return;
    for (int e = threadIdx.x; e < K * nt; e += kConvThreads) {
        const int k = e / nt, qq = e % nt;
        sM[k][qq] = ctx.md_mat[(size_t)k * L + q0 + qq];
        if (k == 0) {
            sP[qq] = ctx.pc[q0 + qq];
            sPinv[qq] = reinterpret_cast<const ulonglong2*>(ctx.md_pinv)[q0 + qq];
        }
    }
    const size_t j = ((size_t)blockIdx.x * kConvThreads + threadIdx.x) * 2;
    uint64_t y0[MAXIN], y1[MAXIN];
#pragma unroll
    for (int k = 0; k < MAXIN; ++k) {
        if (k < K) {
            const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(y + (size_t)k * ctx.N + j);
            y0[k] = v.x;
            y1[k] = v.y;
        }
    }
    uint64_t tl0 = 0, tl1 = 0;
    uint64_t ql = 0;
    if (ttop) {
        const PrimeConst pl = ctx.pc[level];
        const ulonglong2 pinv_l = reinterpret_cast<const ulonglong2*>(ctx.md_pinv)[level];
        ACC a, b;
#pragma unroll
        for (int k = 0; k < MAXIN; ++k) {
            if (k < K) {
                const uint64_t M = ctx.md_mat[(size_t)k * L + level];
                a.mac(y0[k], M);
                b.mac(y1[k], M);
            }
        }
        const ulonglong2 tv = *reinterpret_cast<const ulonglong2*>(ttop + j);
        tl0 = sub_mod(tv.x, mul_shoup(a.reduce(pl), pinv_l.x, pinv_l.y, pl.p), pl.p);
        tl1 = sub_mod(tv.y, mul_shoup(b.reduce(pl), pinv_l.x, pinv_l.y, pl.p), pl.p);
        ql = pl.p;
    }
    __syncthreads();
    auto finish = [&](int qq, const ACC& a, const ACC& b) {
        const PrimeConst pc = sP[qq];
        ulonglong2 o;
        o.x = a.reduce(pc);
        o.y = b.reduce(pc);
        if (ttop) {
            const ulonglong2 pinv = sPinv[qq];
            o.x = add_mod(mul_shoup(o.x, pinv.x, pinv.y, pc.p), switch_modulus(tl0, ql, pc), pc.p);
            o.y = add_mod(mul_shoup(o.y, pinv.x, pinv.y, pc.p), switch_modulus(tl1, ql, pc), pc.p);
        }
        *reinterpret_cast<ulonglong2*>(w + (size_t)(q0 + qq) * ctx.N + j) = o;
    };
#pragma unroll 1
    for (int qq = 0; qq < nt; qq += 2) {
        const int q2 = qq + 1 < nt ? qq + 1 : qq;
        ACC a, b, c2, d2;
#pragma unroll
        for (int k = 0; k < MAXIN; ++k) {
            if (k < K) {
                const uint64_t M = sM[k][qq], M2 = sM[k][q2];
                a.mac(y0[k], M);
                b.mac(y1[k], M);
                c2.mac(y0[k], M2);
                d2.mac(y1[k], M2);
            }
        }
        finish(qq, a, b);
        if (q2 != qq) finish(q2, c2, d2);
    }
}

void launch_moddown_conv(const DevCtx& ctx, int level, int nb, const MdArgs& a, cudaStream_t st) {
    const int nout = a.ttop[0] ? level : level + 1;
    if (nout <= 0) return;
    if ((ctx.conv_variant == 3 || ctx.conv_variant == 4) && conv_tc_supported(ctx)) {
        launch_moddown_conv_tc(ctx, level, nb, a, st, ctx.conv_variant == 3 ? 32 : 16);
        return;
    }
    dim3 g(ctx.N / (2 * kConvThreads), (nout + kConvTargets - 1) / kConvTargets, 2 * nb);
    count_launches(1);
#define FIDES_MODDOWN(M)                                                      \
    if (ctx.conv_variant == 1)                                                \
        launch_pdl(k_moddown_conv<M, AccSplit>, g, kConvThreads, 0, st, ctx, level, a); \
    else                                                                      \
        launch_pdl(k_moddown_conv<M, Acc128>, g, kConvThreads, 0, st, ctx, level, a);
    if (ctx.K <= 4) {
        FIDES_MODDOWN(4)
    } else if (ctx.K <= 8) {
        FIDES_MODDOWN(8)
    } else if (ctx.K <= 12) {
        FIDES_MODDOWN(12)
    } else {
        FIDES_MODDOWN(16)
    }
#undef FIDES_MODDOWN
}

// ---------------------------------------------------------------------------
// element-wise
// ---------------------------------------------------------------------------
__device__ __forceinline__ ulonglong2 ew_apply(int op, const ulonglong2 x, const uint64_t* b, size_t i,
                                               const PrimeConst& pc) {
    ulonglong2 r = x;
    if (op == EW_COPY) return r;
    if (op == EW_NEG) {
        r.x = neg_mod(x.x, pc.p);
        r.y = neg_mod(x.y, pc.p);
        return r;
    }
    const ulonglong2 y = *reinterpret_cast<const ulonglong2*>(b + i);
    if (op == EW_ADD) {
        r.x = add_mod(x.x, y.x, pc.p);
        r.y = add_mod(x.y, y.y, pc.p);
    } else if (op == EW_SUB) {
        r.x = sub_mod(x.x, y.x, pc.p);
        r.y = sub_mod(x.y, y.y, pc.p);
    } else if (pc.p < kFpPrimeBound) {
        const double p = __ull2double_rn(pc.p), pinv = as_f64(pc.pinv_f64);
        r.x = fp_to_u(fp_mulmod(as_f64(fp_from_u(x.x)), as_f64(fp_from_u(y.x)), p, pinv), p, pinv);
        r.y = fp_to_u(fp_mulmod(as_f64(fp_from_u(x.y)), as_f64(fp_from_u(y.y)), p, pinv), p, pinv);
    } else {
        r.x = mul_mod(x.x, y.x, pc);
        r.y = mul_mod(x.y, y.y, pc);
    }
    return r;
}

// One operation per component (grid z): a ciphertext operation is one launch.
__global__ void k_elementwise(const __grid_constant__ DevCtx ctx, int q0, const __grid_constant__ EwArgs args) {
    pdl_trigger();
    pdl_wait();
    const int limb = blockIdx.y, h = blockIdx.z;
    const PrimeConst pc = ctx.pc[q0 + limb];
    const size_t i = (size_t)limb * ctx.N + (size_t)(blockIdx.x * blockDim.x + threadIdx.x) * 2;
    const ulonglong2 x = *reinterpret_cast<const ulonglong2*>(args.a[h] + i);
    *reinterpret_cast<ulonglong2*>(args.o[h] + i) = ew_apply(args.op[h], x, args.b[h], i, pc);
}

void launch_elementwise2(const DevCtx& ctx, int n, int q0, const EwArgs& args, cudaStream_t st) {
    if (n <= 0) return;
    count_launches(1);
    launch_pdl(k_elementwise, dim3(ctx.N / 256, n, args.o[1] ? 2 : 1), 128, 0, st, ctx, q0, args);
}

void launch_elementwise(const DevCtx& ctx, int op, int n, int q0, const uint64_t* a, const uint64_t* b,
                        uint64_t* out, cudaStream_t st) {
    EwArgs e{};
    e.a[0] = a;
    e.b[0] = b;
    e.o[0] = out;
    e.op[0] = op;
    launch_elementwise2(ctx, n, q0, e, st);
}

// Extended-basis sums of key-switch results: for output u, the elements
// start[u] .. start[u+1]-1 of XB and XA (n ciphertext limbs, then K special
// limbs, at bstride) are added into element start[u].  Two coefficients per
// thread.
__global__ void k_ext_sum(const __grid_constant__ DevCtx ctx, const __grid_constant__ ExtSumArgs a) {
    pdl_trigger();
    pdl_wait();
    const int limb = blockIdx.y, u = blockIdx.z;
    const int j = (blockIdx.x * blockDim.x + threadIdx.x) * 2;
    if (j >= ctx.N) return;
    const uint64_t p = ctx.pc[limb < a.n ? limb : ctx.L + (limb - a.n)].p;
    const size_t i = (size_t)limb * ctx.N + j;
    const int b0 = a.start[u], b1 = a.start[u + 1];
    for (int h = 0; h < 2; ++h) {
        ulonglong2* dst = reinterpret_cast<ulonglong2*>(a.x[h] + (size_t)b0 * a.bstride + i);
        ulonglong2 s = *dst;
        for (int b = b0 + 1; b < b1; ++b) {
            const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(a.x[h] + (size_t)b * a.bstride + i);
            s.x = add_mod(s.x, v.x, p);
            s.y = add_mod(s.y, v.y, p);
        }
        *dst = s;
    }
}

void launch_ext_sum(const DevCtx& ctx, const ExtSumArgs& a, cudaStream_t st) {
    if (a.nout <= 0) return;
    count_launches(1);
    launch_pdl(k_ext_sum, dim3((ctx.N + 511) / 512, a.n + ctx.K, a.nout), 256, 0, st, ctx, a);
}

// One constant per limb applied to both components of a ciphertext (grid z =
// component), the constants in the kernel parameters: nothing is uploaded and
// nothing waits.  MUL: both times (c, Shoup companion); else c is added to
// component 0 and component 1 is copied.
template <bool MUL>
__global__ void k_ct_scalar(const __grid_constant__ DevCtx ctx, const __grid_constant__ CtScalarArgs args) {
    pdl_trigger();
    pdl_wait();
    const int limb = blockIdx.y, h = blockIdx.z;
    const uint64_t p = ctx.pc[args.q0 + limb].p;
    const size_t i = (size_t)limb * ctx.N + (size_t)(blockIdx.x * blockDim.x + threadIdx.x) * 2;
    ulonglong2 x = *reinterpret_cast<const ulonglong2*>(args.a[h] + i);
    if constexpr (MUL) {
        x.x = mul_shoup(x.x, args.c[limb][0], args.c[limb][1], p);
        x.y = mul_shoup(x.y, args.c[limb][0], args.c[limb][1], p);
    } else if (h == 0) {
        x.x = add_mod(x.x, args.c[limb][0], p);
        x.y = add_mod(x.y, args.c[limb][0], p);
    }
    *reinterpret_cast<ulonglong2*>(args.o[h] + i) = x;
}

void launch_ct_scalar(const DevCtx& ctx, bool mul, int nlimbs, const CtScalarArgs& args, cudaStream_t st) {
    if (nlimbs <= 0 || nlimbs > kMaxLinLimbs) return;
    const dim3 g(ctx.N / 256, nlimbs, 2);
    count_launches(1);
    if (mul)
        launch_pdl(k_ct_scalar<true>, g, 128, 0, st, ctx, args);
    else
        launch_pdl(k_ct_scalar<false>, g, 128, 0, st, ctx, args);
}

// Sum of n ciphertexts (both components, grid z).
__global__ void k_ct_sum(const __grid_constant__ DevCtx ctx, const __grid_constant__ CtSumArgs args) {
    pdl_trigger();
    pdl_wait();
    const int limb = blockIdx.y, h = blockIdx.z;
    const uint64_t p = ctx.pc[limb].p;
    const size_t i = (size_t)limb * ctx.N + (size_t)(blockIdx.x * blockDim.x + threadIdx.x) * 2;
    ulonglong2 s = *reinterpret_cast<const ulonglong2*>(args.in[h][0] + i);
#pragma unroll 4
    for (int k = 1; k < args.n; ++k) {
        const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(args.in[h][k] + i);
        s.x = add_mod(s.x, v.x, p);
        s.y = add_mod(s.y, v.y, p);
    }
    *reinterpret_cast<ulonglong2*>(args.out[h] + i) = s;
}

void launch_ct_sum(const DevCtx& ctx, int nlimbs, const CtSumArgs& args, cudaStream_t st) {
    if (nlimbs <= 0 || args.n < 1 || args.n > kMaxSum) return;
    count_launches(1);
    launch_pdl(k_ct_sum, dim3(ctx.N / 256, nlimbs, 2), 128, 0, st, ctx, args);
}

// Plaintext dot products (the inner sums of a baby-step giant-step transform,
// one output per giant step): each thread owns two coefficients of both halves
// and reads each plaintext term once for c0 and c1.  The outputs vary fastest
// over the grid, then the tiles of a limb, then the limbs: the giant steps read
// the same baby-step tiles at the same time, so a baby step comes from HBM once
// per transform.  (One launch per giant step read every baby step from HBM
// again: 8 launches of 46 us for 64 diagonals of 20 limbs at N = 2^16, 8 baby
// steps of 21 MB each, 5.5 TB/s.)
// Sums: exact FP64 products for primes below 2^50 (|r| <= 0.875p, centred every
// seven terms, below 7.2p), else 128-bit ones folded every 15 terms (products of
// residues below 2^62 are below 2^124).
// Role in the reference: dotProductPt_ (CKKS/ElemenwiseBatchKernels.cu:651).
__global__ void __launch_bounds__(128) k_dot_pt(const __grid_constant__ DevCtx ctx, const __grid_constant__ DotArgs args) {
    pdl_trigger();
    pdl_wait();
    const int u = blockIdx.x, limb = blockIdx.z;
    const PrimeConst pc = ctx.pc[limb];
    const size_t i = (size_t)limb * ctx.N + (size_t)(blockIdx.y * blockDim.x + threadIdx.x) * 2;
    const int k0 = args.start[u], k1 = args.start[u + 1];
    ulonglong2 r0 = make_ulonglong2(0, 0), r1 = r0;
    if (args.accumulate[u]) {
        r0 = *reinterpret_cast<const ulonglong2*>(args.o0[u] + i);
        r1 = *reinterpret_cast<const ulonglong2*>(args.o1[u] + i);
    }
    auto term = [&](int k, ulonglong2& w, ulonglong2& x, ulonglong2& y) {
        const int b = args.baby[k];
        w = *reinterpret_cast<const ulonglong2*>(args.p[k] + i);
        x = *reinterpret_cast<const ulonglong2*>(args.c0[b] + i);
        y = *reinterpret_cast<const ulonglong2*>(args.c1[b] + i);
    };
    if (pc.p < kFpPrimeBound) {
        const double p = __ull2double_rn(pc.p), pinv = as_f64(pc.pinv_f64);
        auto conv = [](uint64_t v) { return as_f64(fp_from_u(v)); };
        double a0 = conv(r0.x), a1 = conv(r0.y), b0 = conv(r1.x), b1 = conv(r1.y);
        int since = 0;
#pragma unroll 4
        for (int k = k0; k < k1; ++k) {
            ulonglong2 w, x, y;
            term(k, w, x, y);
            const double w0 = conv(w.x), w1 = conv(w.y);
            a0 = __dadd_rn(a0, fp_mulmod(conv(x.x), w0, p, pinv));
            a1 = __dadd_rn(a1, fp_mulmod(conv(x.y), w1, p, pinv));
            b0 = __dadd_rn(b0, fp_mulmod(conv(y.x), w0, p, pinv));
            b1 = __dadd_rn(b1, fp_mulmod(conv(y.y), w1, p, pinv));
            if (++since == 7) {
                a0 = fp_center(a0, p, pinv);
                a1 = fp_center(a1, p, pinv);
                b0 = fp_center(b0, p, pinv);
                b1 = fp_center(b1, p, pinv);
                since = 0;
            }
        }
        r0 = make_ulonglong2(fp_sum_to_u(a0, p, pinv), fp_sum_to_u(a1, p, pinv));
        r1 = make_ulonglong2(fp_sum_to_u(b0, p, pinv), fp_sum_to_u(b1, p, pinv));
    } else {
        Acc128 a0, a1, b0, b1;
        a0.lo = r0.x;
        a1.lo = r0.y;
        b0.lo = r1.x;
        b1.lo = r1.y;
        int since = 0;
#pragma unroll 2
        for (int k = k0; k < k1; ++k) {
            ulonglong2 w, x, y;
            term(k, w, x, y);
            a0.mac(x.x, w.x);
            a1.mac(x.y, w.y);
            b0.mac(y.x, w.x);
            b1.mac(y.y, w.y);
            if (++since == 15) {
                a0.lo = a0.reduce(pc), a0.hi = 0;
                a1.lo = a1.reduce(pc), a1.hi = 0;
                b0.lo = b0.reduce(pc), b0.hi = 0;
                b1.lo = b1.reduce(pc), b1.hi = 0;
                since = 0;
            }
        }
        r0 = make_ulonglong2(a0.reduce(pc), a1.reduce(pc));
        r1 = make_ulonglong2(b0.reduce(pc), b1.reduce(pc));
    }
    *reinterpret_cast<ulonglong2*>(args.o0[u] + i) = r0;
    *reinterpret_cast<ulonglong2*>(args.o1[u] + i) = r1;
}

void launch_dot_pt(const DevCtx& ctx, int nlimbs, const DotArgs& args, cudaStream_t st) {
    if (nlimbs <= 0 || args.nout <= 0) return;
    count_launches(1);
    launch_pdl(k_dot_pt, dim3(args.nout, ctx.N / 256, nlimbs), 128, 0, st, ctx, args);
}

// Integer linear combination (leaf sums of polynomial evaluation, integer
// scalar products): each thread owns two coefficients of both components.
__global__ void k_lincomb(const __grid_constant__ DevCtx ctx, const __grid_constant__ LinArgs args) {
    pdl_trigger();
    pdl_wait();
    const int limb = blockIdx.y;
    const PrimeConst pc = ctx.pc[args.q0 + limb];
    const size_t i = (size_t)limb * ctx.N + (size_t)(blockIdx.x * blockDim.x + threadIdx.x) * 2;
    ulonglong2 r0 = make_ulonglong2(0, 0), r1 = make_ulonglong2(0, 0);
#pragma unroll 1
    for (int k = 0; k < args.n; ++k) {
        const uint64_t z = args.z[k][limb][0], zs = args.z[k][limb][1];
        const ulonglong2 x = *reinterpret_cast<const ulonglong2*>(args.in0[k] + i);
        const ulonglong2 y = *reinterpret_cast<const ulonglong2*>(args.in1[k] + i);
        r0.x = add_mod(r0.x, mul_shoup(x.x, z, zs, pc.p), pc.p);
        r0.y = add_mod(r0.y, mul_shoup(x.y, z, zs, pc.p), pc.p);
        r1.x = add_mod(r1.x, mul_shoup(y.x, z, zs, pc.p), pc.p);
        r1.y = add_mod(r1.y, mul_shoup(y.y, z, zs, pc.p), pc.p);
    }
    if (args.has_add) {
        r0.x = add_mod(r0.x, args.add0[limb], pc.p);
        r0.y = add_mod(r0.y, args.add0[limb], pc.p);
    }
    *reinterpret_cast<ulonglong2*>(args.out0 + i) = r0;
    *reinterpret_cast<ulonglong2*>(args.out1 + i) = r1;
}

void launch_lincomb(const DevCtx& ctx, int nlimbs, const LinArgs& args, cudaStream_t st) {
    if (nlimbs <= 0 || nlimbs > kMaxLinLimbs || args.n < 0 || args.n > kMaxLin) return;
    dim3 g(ctx.N / 256, nlimbs);
    count_launches(1);
    launch_pdl(k_lincomb, g, 128, 0, st, ctx, args);
}

// X^k in evaluation form: slot i of prime j holds psi_j^e, e = (2 brev(i) + 1) k
// mod 2N; psi^m = fwd_tw[j][brev(m)] for m < N and psi^N = -1.
// Role in the reference: Ciphertext::multMonomial (used by Bootstrap.cu:268).
__global__ void k_mult_monomial(const __grid_constant__ DevCtx ctx, const uint64_t* in0, const uint64_t* in1,
                                uint64_t* out0, uint64_t* out1, uint32_t k) {
    pdl_trigger();
    pdl_wait();
    const int limb = blockIdx.y;
    const uint64_t* in = blockIdx.z ? in1 : in0;
    uint64_t* out = blockIdx.z ? out1 : out0;
    const uint64_t p = ctx.pc[limb].p;
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t mask2n = (2u << ctx.logN) - 1;
    const uint32_t e = (((brev_bits(i, ctx.logN) << 1) + 1) * k) & mask2n;
    const uint32_t m = e & ((uint32_t)ctx.N - 1);
    const ulonglong2 w = __ldg(reinterpret_cast<const ulonglong2*>(ctx.fwd_tw) + (size_t)limb * ctx.N +
                               brev_bits(m, ctx.logN));
    const size_t o = (size_t)limb * ctx.N + i;
    const uint64_t v = mul_shoup(in[o], w.x, w.y, p);
    out[o] = (e >= (uint32_t)ctx.N) ? neg_mod(v, p) : v;
}

void launch_mult_monomial(const DevCtx& ctx, int nlimbs, const uint64_t* in0, const uint64_t* in1, uint64_t* out0,
                          uint64_t* out1, uint32_t k, cudaStream_t st) {
    if (nlimbs <= 0) return;
    dim3 g(ctx.N / 256, nlimbs, 2);
    count_launches(1);
    launch_pdl(k_mult_monomial, g, 256, 0, st, ctx, in0, in1, out0, out1, k);
}

__global__ void k_automorph(const __grid_constant__ DevCtx ctx, const uint64_t* in, uint64_t* out,
                            uint32_t galois_inv) {
    pdl_trigger();
    pdl_wait();
    const size_t base = (size_t)blockIdx.y * ctx.N;
    const uint32_t j = blockIdx.x * blockDim.x + threadIdx.x;
    out[base + j] = in[base + automorph_slot(ctx.logN, galois_inv, j)];
}

void launch_automorph(const DevCtx& ctx, int nlimbs, const uint64_t* in, uint64_t* out, uint32_t galois_inv,
                      cudaStream_t st) {
    if (nlimbs <= 0) return;
    dim3 g(ctx.N / 256, nlimbs);
    count_launches(1);
    launch_pdl(k_automorph, g, 256, 0, st, ctx, in, out, galois_inv);
}

}  // namespace fides
