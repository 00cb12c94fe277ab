// conv_tc.cu -- ModUp and ModDown base conversions on the 5th-generation
// tensor cores.
//
// Role in the reference: DecompAndModUpConv and ModDown2 (src/CKKS/Conv.cu),
// the same contractions as k_modup_conv / k_moddown_conv in ks.cu:
//   out[m][j] = sum_i x_i[j] * M[i][m]  (mod p_m),
// with M[i][m] = (Q'/q_i) mod p_m over the cnt limbs i of one digit (ModUp),
// or (P/p_k) mod q_m over the K special limbs (ModDown), for ntar targets m.
//
// Exact int8 split (this file's own design): with x_i = sum_a x_{i,a} 2^{8a}
// (bytes) and the pre-shifted constants M'_{i,m,a} = M[i][m] 2^{8a} mod p_m
// = sum_s M'_{i,m,a,s} 2^{8s} (bytes), the value
//   V'[j][m] = sum_i sum_a x_{i,a} M'_{i,m,a} = sum_{s<8} c_s 2^{8s},
//   c_s = sum_i sum_a x_{i,a} M'_{i,m,a,s},
// is congruent to V mod p_m, and every c_s is one entry of an unsigned 8-bit
// matrix product A[j][(i,a)] = x_{i,a}, B[(i,a)][(m,s)] = M'_{i,m,a,s},
// accumulated exactly in 32 bits (c_s < 16 * 8 * 255^2 < 2^23).  Folding the
// byte position of x into the constants keeps V' below 2^80 and needs 8
// columns per target, against 2^128 and 15 columns for the plain split.
// A tile of 128 coefficients is multiplied by B with tcgen05.mma kind::i8
// (M = 128, N = 8 columns per target, K = 32 bytes per instruction) into
// tensor memory; the epilogue reads each coefficient's column sums with
// tcgen05.ld, reassembles V' and reduces it with one 15-bit quotient
// (reduce_cols).  The tensor cores take the 64x64-bit products off the integer
// pipes; what is left there is a few shifts and adds and three multiplies per
// output.
//
// Operands sit in shared memory in the canonical K-major layout without
// swizzle: core matrices of 8 rows x 16 bytes stored contiguously, 8-row
// groups 128 bytes apart (SBO) and 16-byte K chunks LBO bytes apart.  A is
// rebuilt per tile from coalesced limb loads; every B (per level and digit,
// per level for ModDown) is built once per context and copied in by each
// CTA.  Every wait on the MMA completion barrier is bounded; a timeout sets an
// error flag and the CTA releases its tensor memory and returns.
#include <algorithm>
#include <vector>

#include "kernels.hpp"

namespace fides {

namespace {

constexpr int kTcThreads = 256;     // 8 warps: two per tensor-memory lane quarter
constexpr int kTcRows = 128;        // coefficients per tile (MMA M)
constexpr int kTcCols = 8;          // accumulator columns per target (byte positions 0..7 of V')
constexpr uint32_t kTcLboA = (kTcRows / 8) * 128;  // A: K-chunk stride in bytes
constexpr uint32_t kSpinLimit = 1u << 20;
// smallest modulus of reduce_cols: below it the quotient can be short by two
// (and below 2^16 its constant no longer fits 32 bits)
constexpr uint64_t kTcMinModulus = 1ull << 17;

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// shared-memory matrix descriptor (canonical K-major, no swizzle)
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
    uint64_t d = (uint64_t)((addr >> 4) & 0x3FFF);
    d |= (uint64_t)((lbo >> 4) & 0x3FFF) << 16;
    d |= (uint64_t)((sbo >> 4) & 0x3FFF) << 32;
    d |= (uint64_t)1 << 46;  // descriptor version of sm_100; base offset 0, no swizzle
    return d;
}

// instruction descriptor of kind::i8: unsigned A and B, s32 accumulator,
// both operands K-major, shape M x N
__host__ __device__ constexpr uint32_t idesc_u8(int M, int N) {
    return (2u << 4) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

__device__ __forceinline__ void mma_u8(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                       uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, {%5, %6, %7, %8}, p;\n\t}\n" ::"r"(tmem_d),
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate), "r"(0u), "r"(0u), "r"(0u), "r"(0u));
}

__device__ __forceinline__ bool wait_parity(uint32_t bar, uint32_t phase) {
    for (uint32_t it = 0; it < kSpinLimit; ++it) {
        uint32_t done;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}\n"
            : "=r"(done)
            : "r"(bar), "r"(phase)
            : "memory");
        if (done) return true;
    }
    return false;
}

// 8 and 32 consecutive accumulator columns of this thread's lane (no wait)
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, uint32_t (&c)[8]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];\n"
                 : "=r"(c[0]), "=r"(c[1]), "=r"(c[2]), "=r"(c[3]), "=r"(c[4]), "=r"(c[5]), "=r"(c[6]), "=r"(c[7])
                 : "r"(taddr));
}
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&c)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, "
        "%15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];\n"
        : "=r"(c[0]), "=r"(c[1]), "=r"(c[2]), "=r"(c[3]), "=r"(c[4]), "=r"(c[5]), "=r"(c[6]), "=r"(c[7]), "=r"(c[8]),
          "=r"(c[9]), "=r"(c[10]), "=r"(c[11]), "=r"(c[12]), "=r"(c[13]), "=r"(c[14]), "=r"(c[15]), "=r"(c[16]),
          "=r"(c[17]), "=r"(c[18]), "=r"(c[19]), "=r"(c[20]), "=r"(c[21]), "=r"(c[22]), "=r"(c[23]), "=r"(c[24]),
          "=r"(c[25]), "=r"(c[26]), "=r"(c[27]), "=r"(c[28]), "=r"(c[29]), "=r"(c[30]), "=r"(c[31])
        : "r"(taddr));
}
__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory"); }

// V' mod p for V' = sum_{s<8} c_s 2^{8s}, c_s < 2^23, 2^17 <= p < 2^62 (kTcMinModulus).
// The pairs w_k = c_{2k} + c_{2k+1} 2^8 fit 32 bits, and with
// e = w_0 + w_2 2^32, o = w_1 + w_3 2^32:  V' = e + o 2^16,
// floor(V'/2^16) = floor(e/2^16) + o  and  V' mod 2^64 = e + (o << 16).
// V' < 8 cnt 255 p (cnt input limbs): the quotient has at most 15 bits, so 32
// bits T = floor(V' / 2^s) of V' and one 32-bit high product give it,
//   q = floor(T M / 2^(32+k)),  M = floor(2^(32+k+s) / p) or up to two less,
// with s = max(16, bits(p) + bits(2040 cnt) - 32), k = bits(p) - 1 - s: short of
// V'/p by less than 1 + 2^s / p + 3 T / 2^(32+k) < 2, so V' - q p (formed modulo
// 2^64) lies in [0, 2p).  (A 64-bit Barrett quotient, floor(2^80 / p), took
// eight half-rate multiplies per output against three, and that pipe was 65%
// busy: ModUp of 32 elements 608 us, ModDown 598 us at the HMult shape.)
struct __align__(16) TcMod {
    uint64_t np;   // -p
    uint32_t M;
    uint32_t shk;  // s - 16 in bits 0-4, kTcNear, k << 16
};
constexpr uint32_t kTcNear = 0x100;  // fused ModDown: q_level < 2p
__device__ __forceinline__ TcMod tc_mod(const PrimeConst& pc, int cnt) {
    const int bits = 64 - __clzll((long long)pc.p);
    const int s = max(16, bits + (32 - __clz(2040 * cnt)) - 32);
    const int k = max(0, bits - 1 - s);
    // 1/p is within 2^-52 relative: one less than its floor never exceeds the exact floor
    const double m = ldexp(__longlong_as_double((long long)pc.pinv_f64), 32 + k + s);
    return {0 - pc.p, (uint32_t)(uint64_t)m - 1u, (uint32_t)(s - 16) | (uint32_t)k << 16};
}
__device__ __forceinline__ uint64_t reduce_cols(const uint32_t* c, const TcMod& t) {
    const uint32_t w0 = c[0] + (c[1] << 8), w1 = c[2] + (c[3] << 8);
    const uint32_t w2 = c[4] + (c[5] << 8), w3 = c[6] + (c[7] << 8);
    const uint64_t e = ((uint64_t)w2 << 32) | w0;
    const uint64_t o = ((uint64_t)w3 << 32) | w1;
    const uint64_t h = (e >> 16) + o;
    const uint32_t T = __funnelshift_r((uint32_t)h, (uint32_t)(h >> 32), t.shk);  // shift taken mod 32
    const uint32_t q = __umulhi(T, t.M) >> (t.shk >> 16);
    const uint64_t a = (uint64_t)q * (uint32_t)t.np + e;
    const uint64_t r = a + ((uint64_t)(q * (uint32_t)(t.np >> 32)) << 32) + (o << 16);
    const uint64_t s = r + t.np;
    return (int64_t)s < 0 ? r : s;  // r < 2p < 2^63
}

// target index m of a digit -> prime id (the other Q primes, then the special ones)
__device__ __forceinline__ int target_prime(int m, int lo, int cnt, int n, int L) {
    const int jj = m < lo ? m : m + cnt;
    return jj < n ? jj : L + (jj - n);
}

// Geometry of one conversion: the digit's limbs (ModUp) or the K special
// limbs (ModDown) against the target primes of a level.
struct TcShape {
    int level, n, lo, cnt, ntar, ntar2;
    bool md, fused;
    __device__ TcShape(const DevCtx& ctx, int lev, bool is_md, bool is_fused, int d)
        : level(lev), n(lev + 1), lo(0), md(is_md), fused(is_md && is_fused) {
        if (md) {
            cnt = ctx.K;
            ntar = n;  // level targets (+ the top limb) or level + 1 targets
        } else {
            lo = d * ctx.alpha;
            cnt = min(lo + ctx.alpha - 1, level) - lo + 1;
            ntar = n - cnt + ctx.K;
        }
        ntar2 = (ntar + 1) & ~1;  // MMA widths are multiples of 16 columns
    }
    // prime of target m
    __device__ int tprime(const DevCtx& ctx, int m) const {
        if (md) return fused ? (m == 0 ? level : m - 1) : m;
        return target_prime(m, lo, cnt, n, ctx.L);
    }
    // conversion constant of input limb i for target m; ModDown with the fused
    // rescale converts P^-1 x directly, so its constants carry P^-1 mod q
    __device__ uint64_t matrix(const DevCtx& ctx, int i, int m) const {
        const int t = tprime(ctx, m);
        if (md) {
            const uint64_t M = ctx.md_mat[(size_t)i * ctx.L + t];
            if (!fused) return M;
            const ulonglong2 pinv = reinterpret_cast<const ulonglong2*>(ctx.md_pinv)[t];
            return mul_shoup(M, pinv.x, pinv.y, ctx.pc[t].p);
        }
        return ctx.modup_mat[((size_t)level * ctx.L + lo + i) * (ctx.L + ctx.K) + t];
    }
    __device__ uint32_t lbo_b() const { return (uint32_t)ntar2 * kTcCols / 8 * 128; }
};

// B of a conversion in its shared-memory layout: for K chunk c (limbs 2c,
// 2c+1) and target m, the 16 constants M'_{i,m,a} = M[i][m] 2^{8a} mod p_m;
// column 8m + s of the chunk holds their bytes s (16 bytes: a of limb 2c,
// then a of limb 2c+1), 2*CK chunks lbo_b bytes apart.
template <int CK>
__device__ void tc_build_b(const DevCtx& ctx, const TcShape& sh, uint8_t* dst) {
    const uint32_t lbo_b = sh.lbo_b();
    for (int u = threadIdx.x; u < 2 * CK * sh.ntar2; u += blockDim.x) {
        const int c = u / sh.ntar2, m = u % sh.ntar2;
        uint64_t mp[16];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int i = 2 * c + h;
            const bool live = i < sh.cnt && m < sh.ntar;
            const PrimeConst pc = ctx.pc[live ? sh.tprime(ctx, m) : 0];
            uint64_t v = live ? sh.matrix(ctx, i, m) : 0;
#pragma unroll
            for (int a = 0; a < 8; ++a) {
                mp[8 * h + a] = v;
                if (live && a < 7) v = reduce128(v >> 56, v << 8, pc);  // v 2^8 mod p
            }
        }
#pragma unroll
        for (int sb = 0; sb < kTcCols; ++sb) {
            uint32_t w[4] = {0, 0, 0, 0};
#pragma unroll
            for (int pos = 0; pos < 16; ++pos) w[pos >> 2] |= (uint32_t)((mp[pos] >> (8 * sb)) & 0xFF) << (8 * (pos & 3));
            const int nn = m * kTcCols + sb;
            *reinterpret_cast<uint4*>(dst + (size_t)c * lbo_b + (nn >> 3) * 128 + (nn & 7) * 16) =
                make_uint4(w[0], w[1], w[2], w[3]);
        }
    }
}

// index of a conversion's B in the context table
__host__ __device__ inline int tc_table_index(int L, int dnum, bool md, int level, int d_or_fused) {
    return md ? L * dnum + 2 * level + d_or_fused : level * dnum + d_or_fused;
}

// One CTA per table entry of one kind (blockIdx.x = level, blockIdx.y =
// digit or fused flag); entries that do not exist at a level are skipped.
template <int CK, bool MD>
__global__ void __launch_bounds__(256) k_conv_tc_table(const __grid_constant__ DevCtx ctx, uint8_t* tab,
                                                      const uint64_t* __restrict__ offs) {
    const int level = blockIdx.x, y = blockIdx.y;
    if (!MD && y > level / ctx.alpha) return;
    const TcShape sh(ctx, level, MD, y != 0, y);
    tc_build_b<CK>(ctx, sh, tab + offs[tc_table_index(ctx.L, ctx.dnum, MD, level, y)]);
}

// One conversion launch: ModUp (blockIdx.y = element * digits + digit) or
// ModDown (blockIdx.y = 2 * element + half).
struct TcArgs {
    const uint64_t* xt;  // ModUp: scaled limbs of element 0
    uint64_t* dig;       // ModUp: digit outputs of element 0
    size_t dig_stride;   // ModUp: limbs per digit
    size_t bstride;      // ModUp: words between batch elements
    int nb;              // batch elements
    MdArgs md;           // ModDown
};

// CK: K = 32*CK bytes of A per row, up to 4*CK input limbs.  CHUNK: targets
// per MMA (N = 8*CHUNK), also the tensor-memory columns a CTA holds / 8 (32
// targets: 256 columns, two CTAs per SM; 16 targets: 128 columns, up to three).
// MD: the ModDown conversion, K special limbs -> the Q primes of the level,
// with the fused Rescale of the top limb when md.ttop is set:
//   tl = ttop - P^-1 conv_l (mod q_l),  w_q = P^-1 conv_q + SwitchModulus(tl).
template <int CK, int CHUNK, bool MD>
__global__ void __launch_bounds__(kTcThreads, CHUNK == 16 ? 3 : 2)
    k_conv_tc(const __grid_constant__ DevCtx ctx, int level, const __grid_constant__ TcArgs args) {
    extern __shared__ __align__(1024) uint8_t smem[];
    const int tlog = ctx.logN - 7, ntiles = 1 << tlog;  // tiles of kTcRows = 2^7 coefficients
    // ModDown with the top limb (target 0 = prime `level`); both halves alike
    const bool fused = MD && args.md.ttop[0] != nullptr;
    const int d = MD ? 0 : blockIdx.y;
    const TcShape sh(ctx, level, MD, fused, d);
    const int lo = sh.lo, cnt = sh.cnt, ntar = sh.ntar, ntar2 = sh.ntar2;
    // work items: (element, tile) of digit d (ModUp) or (element, half, tile)
    // (ModDown), split evenly over the CTAs of the row
    const int nitems = (MD ? 2 : 1) * args.nb * ntiles;
    const int it_begin = (int)((long long)blockIdx.x * nitems / gridDim.x);
    const int it_end = (int)((long long)(blockIdx.x + 1) * nitems / gridDim.x);
    // element offset (words) and half of item `it`
    auto item_off = [&](int it, int& half) -> size_t {
        if (MD) {
            const int bh = it >> tlog;
            half = bh & 1;
            return (size_t)(bh >> 1) * args.md.bstride;
        }
        half = 0;
        return (size_t)(it >> tlog) * args.bstride;
    };
    auto item_in = [&](int it) -> const uint64_t* {
        int h;
        const size_t off = item_off(it, h) + (size_t)(it & (ntiles - 1)) * kTcRows;
        return MD ? args.md.y[h] + off : args.xt + off + (size_t)lo * ctx.N;
    };
    const uint32_t lbo_b = sh.lbo_b();

    uint8_t* sA = smem;                                   // 2*CK chunks x kTcLboA
    uint8_t* sB = smem + 2 * CK * kTcLboA;                // 2*CK chunks x lbo_b
    PrimeConst* sP = reinterpret_cast<PrimeConst*>(sB + 2 * CK * lbo_b);
    TcMod* sMod = reinterpret_cast<TcMod*>(sP + ntar2);  // reduction constants per target
    uint64_t* sOm = reinterpret_cast<uint64_t*>(sMod + ntar2);  // ModDown: target - q_level mod target
    uint64_t* sTL = sOm + (MD ? ntar2 : 0);               // ModDown: tl per row
    uint64_t* bar = sTL + (MD ? kTcRows : 0);
    uint32_t* tslot = reinterpret_cast<uint32_t*>(bar + 1);

    for (int m = threadIdx.x; m < ntar2; m += kTcThreads) {  // (the pad target: any constants)
        const PrimeConst pc = ctx.pc[sh.tprime(ctx, min(m, ntar - 1))];
        sP[m] = pc;
        sMod[m] = tc_mod(pc, cnt);
        if (MD) {
            const uint64_t ql = ctx.pc[level].p;
            sOm[m] = pc.p - csub(reduce64_lazy(ql, pc), pc.p);
            if (ql < 2 * pc.p) sMod[m].shk |= kTcNear;
        }
    }
    // A: zero once (limbs cnt..4*CK-1 stay zero)
    for (int i = threadIdx.x; i < 2 * CK * (int)kTcLboA / 16; i += kTcThreads)
        reinterpret_cast<uint4*>(sA)[i] = make_uint4(0, 0, 0, 0);
    // B from the context's table (built once per level and digit)
    {
        const uint4* src = reinterpret_cast<const uint4*>(
            ctx.tc_btab + ctx.tc_boff[tc_table_index(ctx.L, ctx.dnum, MD, level, MD ? (fused ? 1 : 0) : d)]);
        for (int i = threadIdx.x; i < 2 * CK * (int)lbo_b / 16; i += kTcThreads)
            reinterpret_cast<uint4*>(sB)[i] = __ldg(src + i);
    }

    const uint32_t bar_a = smem_u32(bar);
    if (threadIdx.x == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(bar_a), "r"(1u));
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    constexpr uint32_t kTcTmemCols = CHUNK * kTcCols;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(tslot)),
                     "r"(kTcTmemCols));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n");
    }
    asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    const uint32_t tmem = *tslot;
    // The next kernel of the stream may start only now.  A CTA that waits for
    // columns then holds none, and one that holds some and waits (pdl_wait) has only
    // kernels before it whose CTAs all hold theirs: whatever else asks for
    // columns on this SM (a context with 32 targets per MMA beside one with 16 may
    // want more than its 512), every holder ends and gives them back.
    // (Triggered at the start, products and rotations of N = 2^12 and 2^13 take 1-2%
    // less, those of 2^14 3% more, larger ones the same; with the allocation after
    // the wait one product at 2^16 250.8 us instead of 248.7, at 2^12 57.3 instead of 54.1.)
    pdl_trigger();

    const int quarter = warp & 3, wh = warp >> 2;
    const int row = quarter * 32 + lane;
    const uint32_t t_lane = tmem + ((uint32_t)(quarter * 32) << 16);
    const uint32_t a_base = smem_u32(sA), b_base = smem_u32(sB);
    uint32_t phase = 0;
    bool ok = true;
    // this thread's share of an A tile: element e = threadIdx.x + q * kTcThreads
    // is limb e / kTcRows, row e % kTcRows (at most 2*CK elements)
    constexpr int kPer = 2 * CK;
    uint64_t pre[kPer];
    auto fetch = [&](int it) {
        const uint64_t* src = item_in(it);
#pragma unroll
        for (int q = 0; q < kPer; ++q) {
            const int e = threadIdx.x + q * kTcThreads;
            if (e < cnt * kTcRows) pre[q] = src[(size_t)(e / kTcRows) * ctx.N + e % kTcRows];
        }
    };
    // everything up to here (tables, tensor memory, barrier) may run under the
    // previous kernel's tail
    pdl_wait();
    if (it_begin < it_end) fetch(it_begin);
    for (int it = it_begin; it < it_end && ok; ++it) {
        int half;
        const size_t boff = item_off(it, half);
        const size_t j = (size_t)(it & (ntiles - 1)) * kTcRows + row;  // this thread's coefficient
        // this row's outputs: target m at obase + m N (the fused ModDown's target 0
        // is the top limb, which has none)
        uint64_t* obase = MD ? args.md.w[half] + boff + j - (fused ? ctx.N : 0)
                             : args.dig + boff + (size_t)d * args.dig_stride * ctx.N + j;
        uint64_t tl = 0, ql = 0;
        bool up = false;  // tl stands for tl - q_l
#pragma unroll
        for (int q = 0; q < kPer; ++q) {
            const int e = threadIdx.x + q * kTcThreads;
            if (e < cnt * kTcRows) {
                const int i = e / kTcRows, r = e % kTcRows;
                *reinterpret_cast<uint64_t*>(sA + (i >> 1) * kTcLboA + (r >> 3) * 128 + (r & 7) * 16 + (i & 1) * 8) =
                    pre[q];
            }
        }
        asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
        for (int m0 = 0; m0 < ntar2 && ok; m0 += CHUNK) {
            const int nt = min(CHUNK, ntar2 - m0);  // even
            // the A tile is written and the previous chunk's accumulators are read
            asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
            __syncthreads();
            if (threadIdx.x == 0) {
                asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
                const uint32_t idesc = idesc_u8(kTcRows, nt * kTcCols);
#pragma unroll
                for (int k = 0; k < CK; ++k) {
                    const uint64_t ad = smem_desc(a_base + 2 * k * kTcLboA, kTcLboA, 128);
                    const uint64_t bd = smem_desc(b_base + 2 * k * lbo_b + m0 * (kTcCols / 8) * 128, lbo_b, 128);
                    mma_u8(tmem, ad, bd, idesc, k > 0 ? 1u : 0u);
                }
                asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(
                                 bar_a)
                             : "memory");
            }
            const bool got = wait_parity(bar_a, phase);
            phase ^= 1;
            ok = __syncthreads_and(got) != 0;
            if (!ok) break;
            asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
            // the next item's limbs load while this chunk's outputs are formed
            if (m0 + CHUNK >= ntar2 && it + 1 < it_end) fetch(it + 1);
            if (MD && fused) {
                if (m0 == 0) {
                    // target 0 is the top limb: every row's tl first, shared through smem
                    if (wh == 0) {
                        uint32_t c[8];
                        tmem_ld8(t_lane, c);
                        tmem_wait_ld();
                        sTL[row] = sub_mod(args.md.ttop[half][boff + j], reduce_cols(c, sMod[0]), sP[0].p);
                    }
                    __syncthreads();
                }
                tl = sTL[row];
                ql = sP[0].p;
                up = tl > (ql >> 1);
            }
            // four targets share one 32-column load (columns past nt hold old
            // sums, their values are dropped); the warps of half wh take every
            // second group.  The four reductions are independent and run before
            // any store, so that their latencies overlap: with branches between
            // them the epilogue waited two issue slots per instruction at 16
            // warps per SM.  (24 or 32 warps per SM with two targets each were 1-2%
            // slower over a whole HMult.)
#pragma unroll 1
            for (int g = 4 * wh; g < nt; g += 8) {
                uint32_t c[32];
                tmem_ld32(t_lane + (uint32_t)(g * kTcCols), c);
                const int m = m0 + g;
                TcMod md[4];
                uint32_t near = kTcNear;
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    md[u] = sMod[min(m + u, ntar2 - 1)];
                    near &= md[u].shk;
                }
                tmem_wait_ld();
                uint64_t v[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) v[u] = reduce_cols(c + 8 * u, md[u]);
                if (MD && fused) {
                    // v = P^-1 conv_q (folded into the constants) + SwitchModulus(tl, q_l -> q)
                    if (near) {
                        // q_l < 2q, as in any chain of like-sized primes: the centred
                        // tl lies in (-q, q) and one conditional addition does (with a
                        // Barrett step per target of q < q_l one HMult of N = 2^16,
                        // L = 30 took 261 us against 259, 32 of them 6172 against 6112)
                        const uint64_t ctl = up ? tl - ql : tl;
#pragma unroll
                        for (int u = 0; u < 4; ++u) {
                            const uint64_t s = v[u] + ctl + (up ? 0 : md[u].np);  // v + tl' - q or v + tl': [-q, q)
                            v[u] = (int64_t)s < 0 ? s - md[u].np : s;
                        }
                    } else {
#pragma unroll
                        for (int u = 0; u < 4; ++u) {
                            const PrimeConst pc = sP[min(m + u, ntar2 - 1)];
                            uint64_t sw = up ? tl + sOm[min(m + u, ntar2 - 1)] : tl;
                            if (pc.p < ql) sw = csub(reduce64_lazy(sw, pc), pc.p);
                            v[u] = add_mod(v[u], sw, pc.p);
                        }
                    }
                }
                const int lim = min(nt - g, ntar - m);
#pragma unroll
                for (int u = 0; u < 4; ++u)
                    if (u < lim && !(MD && fused && u == 0 && m == 0))
                        obase[(size_t)((uint32_t)(m + u) * (uint32_t)ctx.N)] = v[u];
            }
        }
    }
    // a gave-up wait invalidates this launch's outputs: flagged in the
    // context's error word, which the next synchronising call reports
    if (!ok && threadIdx.x == 0 && ctx.err) atomicOr(ctx.err, kDevErrTensorWait);
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    if (warp == 0) {
        asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(kTcTmemCols));
    }
}

// dynamic shared memory of one CTA for ntar targets
size_t tc_smem_bytes(int ck, int ntar, bool md) {
    const size_t t2 = (size_t)((ntar + 1) & ~1);
    return (size_t)2 * ck * kTcLboA + (size_t)2 * ck * t2 * kTcCols / 8 * 128 + t2 * (sizeof(PrimeConst) + sizeof(TcMod)) +
           (md ? t2 * 8 + (size_t)kTcRows * 8 : 0) + 16;
}

constexpr int kTcMaxTargets = 48;
constexpr size_t kTcSmemCap = 160 * 1024;

template <int CHUNK, bool MD>
void launch_ck(int ck, dim3 g, size_t smem, const DevCtx& ctx, int level, const TcArgs& a, cudaStream_t st) {
    switch (ck) {
        case 1:
            launch_pdl(k_conv_tc<1, CHUNK, MD>, g, kTcThreads, smem, st, ctx, level, a);
            break;
        case 2:
            launch_pdl(k_conv_tc<2, CHUNK, MD>, g, kTcThreads, smem, st, ctx, level, a);
            break;
        case 3:
            launch_pdl(k_conv_tc<3, CHUNK, MD>, g, kTcThreads, smem, st, ctx, level, a);
            break;
        default:
            launch_pdl(k_conv_tc<4, CHUNK, MD>, g, kTcThreads, smem, st, ctx, level, a);
            break;
    }
}

// grid, shared memory and launch; a floor on the shared memory keeps the
// CTAs of an SM within its 512 tensor-memory columns (80 KB: at most two
// CTAs of 256 columns; 58 KB: at most three of 128)
template <bool MD>
void launch_tc(const DevCtx& ctx, int level, int groups, int items, int ck, int ntar, const TcArgs& a,
               cudaStream_t st, int chunk) {
    const size_t floor_bytes = chunk == 32 ? (size_t)80 * 1024 : (size_t)58 * 1024;
    const size_t smem = std::max(tc_smem_bytes(ck, ntar, MD), floor_bytes);
    // one wave: the CTAs of all rows fill the SMs at the occupancy above
    const int ctas = chunk == 32 ? 2 * 148 : 3 * 148;
    const dim3 g(std::max(1, std::min(items, ctas / groups)), groups);
    count_launches(1);
    if (chunk == 32)
        launch_ck<32, MD>(ck, g, smem, ctx, level, a, st);
    else
        launch_ck<16, MD>(ck, g, smem, ctx, level, a, st);
}

}  // namespace

bool conv_tc_eligible(const DevCtx& ctx, uint64_t smallest) {
    if (ctx.alpha > 16 || ctx.K > 16 || smallest < kTcMinModulus) return false;
    const int up = ctx.L - 1 + ctx.K;  // ModUp: at most L-1 other Q primes plus K
    return up <= kTcMaxTargets && ctx.L <= kTcMaxTargets &&
           tc_smem_bytes((ctx.alpha + 3) / 4, up, false) <= kTcSmemCap &&
           tc_smem_bytes((ctx.K + 3) / 4, ctx.L, true) <= kTcSmemCap;
}

// shared-memory opt-in of the instances a context launches, on its device
template <bool MD>
static cudaError_t opt_in(int ck) {
    const int attr = (int)kTcSmemCap;
    auto set = [&](auto k16, auto k32) {
        const cudaError_t e = cudaFuncSetAttribute(k16, cudaFuncAttributeMaxDynamicSharedMemorySize, attr);
        return e != cudaSuccess ? e : cudaFuncSetAttribute(k32, cudaFuncAttributeMaxDynamicSharedMemorySize, attr);
    };
    switch (ck) {
        case 1: return set(k_conv_tc<1, 16, MD>, k_conv_tc<1, 32, MD>);
        case 2: return set(k_conv_tc<2, 16, MD>, k_conv_tc<2, 32, MD>);
        case 3: return set(k_conv_tc<3, 16, MD>, k_conv_tc<3, 32, MD>);
        default: return set(k_conv_tc<4, 16, MD>, k_conv_tc<4, 32, MD>);
    }
}
cudaError_t conv_tc_prepare(const DevCtx& ctx) {
    const cudaError_t e = opt_in<false>((ctx.alpha + 3) / 4);
    return e != cudaSuccess ? e : opt_in<true>((ctx.K + 3) / 4);
}

bool conv_tc_supported(const DevCtx& ctx) { return ctx.tc_btab != nullptr; }

size_t conv_tc_table_layout(const DevCtx& ctx, std::vector<uint64_t>& offs) {
    const int L = ctx.L, K = ctx.K, dn = ctx.dnum;
    offs.assign((size_t)L * dn + 2 * L, 0);
    size_t off = 0;
    auto add = [&](int idx, int ck, int ntar) {
        offs[idx] = off;
        off += (size_t)2 * ck * (size_t)((ntar + 1) & ~1) * kTcCols / 8 * 128;
    };
    for (int level = 0; level < L; ++level) {
        const int n = level + 1;
        for (int d = 0; d <= level / ctx.alpha && d < dn; ++d) {
            const int lo = d * ctx.alpha, cnt = std::min(lo + ctx.alpha - 1, level) - lo + 1;
            add(tc_table_index(L, dn, false, level, d), (ctx.alpha + 3) / 4, n - cnt + K);
        }
        for (int f = 0; f < 2; ++f) add(tc_table_index(L, dn, true, level, f), (K + 3) / 4, n);
    }
    return off;
}

void conv_tc_build_tables(const DevCtx& ctx, cudaStream_t st) {
    const dim3 gu(ctx.L, ctx.dnum), gd(ctx.L, 2);
    uint8_t* tab = const_cast<uint8_t*>(ctx.tc_btab);
    switch ((ctx.alpha + 3) / 4) {
        case 1: k_conv_tc_table<1, false><<<gu, 256, 0, st>>>(ctx, tab, ctx.tc_boff); break;
        case 2: k_conv_tc_table<2, false><<<gu, 256, 0, st>>>(ctx, tab, ctx.tc_boff); break;
        case 3: k_conv_tc_table<3, false><<<gu, 256, 0, st>>>(ctx, tab, ctx.tc_boff); break;
        default: k_conv_tc_table<4, false><<<gu, 256, 0, st>>>(ctx, tab, ctx.tc_boff); break;
    }
    switch ((ctx.K + 3) / 4) {
        case 1: k_conv_tc_table<1, true><<<gd, 256, 0, st>>>(ctx, tab, ctx.tc_boff); break;
        case 2: k_conv_tc_table<2, true><<<gd, 256, 0, st>>>(ctx, tab, ctx.tc_boff); break;
        case 3: k_conv_tc_table<3, true><<<gd, 256, 0, st>>>(ctx, tab, ctx.tc_boff); break;
        default: k_conv_tc_table<4, true><<<gd, 256, 0, st>>>(ctx, tab, ctx.tc_boff); break;
    }
    count_launches(2);
}

void launch_modup_conv_tc(const DevCtx& ctx, int level, int nb, const uint64_t* xt, uint64_t* dig, size_t dig_stride,
                          size_t bstride, cudaStream_t st, int chunk) {
    const int nd = level / ctx.alpha + 1;
    const int n = level + 1, last = n - (nd - 1) * ctx.alpha;
    const int ntar = n - std::min(last, ctx.alpha) + ctx.K;  // largest over the digits
    TcArgs a{};
    a.xt = xt;
    a.dig = dig;
    a.dig_stride = dig_stride;
    a.bstride = bstride;
    a.nb = nb;
    launch_tc<false>(ctx, level, nd, nb * (ctx.N / kTcRows), (ctx.alpha + 3) / 4, ntar, a, st, chunk);
}

void launch_moddown_conv_tc(const DevCtx& ctx, int level, int nb, const MdArgs& md, cudaStream_t st, int chunk) {
    TcArgs a{};
    a.md = md;
    a.nb = nb;
    launch_tc<true>(ctx, level, 1, 2 * nb * (ctx.N / kTcRows), (ctx.K + 3) / 4, level + 1, a, st, chunk);
}

}  // namespace fides
