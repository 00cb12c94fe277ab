// ntt.cu -- host side of the transforms: launch counting, the variants and the
// dispatch on the ring dimension (kernels: ntt_kernels.cuh, ntt_n.cu).
#include <atomic>

#include "kernels.hpp"

namespace fides {

static std::atomic<uint64_t> g_launches{0};
uint64_t launch_count() { return g_launches.load(); }
void count_launches(int n) { g_launches.fetch_add((uint64_t)n); }

bool ntt_supported(int logN) { return logN >= 8 && logN <= 16; }

// Forward variants 0-4 run the integer butterflies on every limb, 5-9 the
// double-precision ones on the limbs of primes below 2^50 (the autotuner times
// one of each); inverse configurations 0-2 and 3-5 likewise.
// ntt_inverse_of(v) pairs each forward variant with an inverse configuration of
// the same arithmetic.  (The numbers once told occupancies and twiddle-fetch
// policies apart; the one kept per arithmetic was the fastest everywhere.)
int ntt_num_variants() { return 10; }
int ntt_num_inverse_variants() { return 6; }
bool ntt_fwd_is_fp(int v) { return v >= 5; }
bool ntt_inv_is_fp(int v) { return v >= 3; }
int ntt_inverse_of(int v) {
    static const int inv[10] = {0, 1, 2, 1, 0, 3, 4, 3, 3, 5};
    return v >= 0 && v < 10 ? inv[v] : 0;
}

template <> const NttOps& ntt_ops<8>();
template <> const NttOps& ntt_ops<9>();
template <> const NttOps& ntt_ops<10>();
template <> const NttOps& ntt_ops<11>();
template <> const NttOps& ntt_ops<12>();
template <> const NttOps& ntt_ops<13>();
template <> const NttOps& ntt_ops<14>();
template <> const NttOps& ntt_ops<15>();
template <> const NttOps& ntt_ops<16>();

static const NttOps* ops_of(int logN) {
    switch (logN) {
        case 8: return &ntt_ops<8>();
        case 9: return &ntt_ops<9>();
        case 10: return &ntt_ops<10>();
        case 11: return &ntt_ops<11>();
        case 12: return &ntt_ops<12>();
        case 13: return &ntt_ops<13>();
        case 14: return &ntt_ops<14>();
        case 15: return &ntt_ops<15>();
        case 16: return &ntt_ops<16>();
        default: return nullptr;
    }
}

void set_modes(LimbMap& map, int lmode, int smode) {
    for (int s = 0; s < map.nseg; ++s) {
        if (lmode >= 0) map.seg[s].lmode = (int8_t)lmode;
        if (smode >= 0) map.seg[s].smode = (int8_t)smode;
    }
}

void ntt_forward(const DevCtx& ctx, const LimbMap& m, int load, int store, cudaStream_t st) {
    if (m.total <= 0) return;
    LimbMap map = m;
    set_modes(map, load, store);
    count_launches(2);
    ops_of(ctx.logN)->fwd(ctx, map, st);
}

cudaError_t ntt_prepare(const DevCtx& ctx) { return ops_of(ctx.logN)->prepare(); }

void ntt_forward_cols(const DevCtx& ctx, const LimbMap& m, int load, cudaStream_t st) {
    if (m.total <= 0) return;
    LimbMap map = m;
    set_modes(map, load, -1);
    count_launches(1);
    ops_of(ctx.logN)->fwd_cols(ctx, map, st);
}

void ntt_rows_keyswitch(const DevCtx& ctx, const KsHmultArgs& a, int nb, cudaStream_t st) {
    count_launches(1);
    ops_of(ctx.logN)->rows_ks(ctx, a, nb, st);
}

bool ntt_rows_keyswitch_supported(const DevCtx& ctx) { return ctx.dnum <= kMaxFusedDigits; }

void ntt_inverse(const DevCtx& ctx, const LimbMap& m, int load, int store, cudaStream_t st) {
    if (m.total <= 0) return;
    LimbMap map = m;
    set_modes(map, load, store);
    count_launches(2);
    ops_of(ctx.logN)->inv(ctx, map, st);
}

}  // namespace fides
