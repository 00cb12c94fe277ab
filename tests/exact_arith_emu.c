/* Host emulation of the exact double-precision arithmetic of the CUDA kernels
 * (pyfideslib_b200/csrc/fp64.cuh) -- test infrastructure only.
 *
 * The device routines are restated with C99 fma() (exactly rounded, like the
 * GPU's __fma_rn) and, for the one round-down FMA, fesetround(FE_DOWNWARD).
 * Built by tests/test_exact_arith.py with -ffp-contract=off so that no other
 * operation is fused.  The drivers run the key-switch sums and the dot products against
 * exact 128-bit integer arithmetic (the transforms: ntt_sched_emu.cpp).
 */
#include <fenv.h>
#include <math.h>
#include <stdint.h>
#include <stdlib.h>
#include <string.h>

typedef unsigned __int128 u128;

static const double kRint = 6755399441055744.0; /* 1.5 * 2^52 */
static const double kTwo52 = 4503599627370496.0;
static const uint64_t kMant52 = (1ull << 52) - 1;

static double fp_mulw(double y, double w, double wq, double p) {
    const double h = y * w;
    const double l = fma(y, w, -h);
    const double q = fma(y, wq, kRint) - kRint;
    return fma(-q, p, h) + l;
}

static double fp_center(double x, double p, double pinv) {
    const double q = fma(x, pinv, kRint) - kRint;
    return fma(-q, p, x);
}

static double fma_rd(double a, double b, double c) {
    fesetround(FE_DOWNWARD);
    volatile double r = fma(a, b, c);
    fesetround(FE_TONEAREST);
    return r;
}

static uint64_t fp_to_u(double v, double p, double pinv_up) {
    const double two_p = p + p;
    const double a = v + two_p;
    const double b = v + (two_p + kTwo52);
    const double q = fma_rd(a, pinv_up, kRint) - kRint;
    const double r = fma(-q, p, b);
    uint64_t u;
    memcpy(&u, &r, 8);
    return u & kMant52;
}

static double fp_mulmod(double x, double y, double p, double pinv) {
    const double h = x * y;
    const double l = fma(x, y, -h);
    const double q = fma(h, pinv, kRint) - kRint;
    return fma(-q, p, h) + l;
}

/* the double nearest above 1/p (context.cpp recip_up) */
static double recip_up(uint64_t p) {
    double x = 1.0 / (double)p;
    int e = 0;
    const double f = frexp(x, &e);
    const uint64_t m = (uint64_t)ldexp(f, 53);
    const int sh = 53 - e;
    if (sh < 128 && (u128)m * p < ((u128)1 << sh)) x = nextafter(x, 1.0);
    return x;
}

static uint64_t mulmod(uint64_t a, uint64_t b, uint64_t p) { return (uint64_t)((u128)a * b % p); }

static uint64_t splitmix(uint64_t* s) {
    uint64_t z = (*s += 0x9E3779B97F4A7C15ull);
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}

/* fp_sum_to_u: canonical residue of |v| < 8p, centred around p first */
static uint64_t fp_sum_to_u(double v, double p, double pinv_up) {
    const double q = fma(v, pinv_up, kRint) - (kRint + 1.0);
    const double w = fma(-q, p, v);
    const double f = fma_rd(w, pinv_up, kRint) - kRint;
    const double r = fma(-f, p, w) + kTwo52;
    uint64_t u;
    memcpy(&u, &r, 8);
    return u & kMant52;
}

/* Rotations' key-switch sums (k_ks_inner): nd products x k reduced by fp_mulmod
 * plus, `c0`, P c0 as a product with a centred constant, reduced from |sum| < 8p,
 * for `trials` random (or, with extreme != 0, maximal) operands.  Returns the
 * number of mismatches. */
int emu_ks_check(uint64_t p, int nd, int c0, uint64_t seed, int trials, int extreme) {
    const double pd = (double)p, pinv = recip_up(p);
    uint64_t s = seed;
    int bad = 0;
    for (int t = 0; t < trials; ++t) {
        double acc = 0;
        uint64_t exact = 0;
        if (c0) {
            const uint64_t c = extreme ? p - 1 : splitmix(&s) % p, m = extreme ? p / 2 + (t & 1) : splitmix(&s) % p;
            const double w = m > p / 2 ? -(double)(p - m) : (double)m;
            acc = fp_mulw((double)c, w, w / pd, pd);
            exact = mulmod(c, m, p);
        }
        for (int dd = 0; dd < nd; ++dd) {
            const uint64_t x = extreme ? p - 1 : splitmix(&s) % p;
            const uint64_t k = extreme ? p - 1 - (uint64_t)(t & 1) : splitmix(&s) % p;
            acc += fp_mulmod((double)x, (double)k, pd, pinv);
            exact = (exact + mulmod(x, k, p)) % p;
        }
        bad += fp_sum_to_u(acc, pd, pinv) != exact;
    }
    return bad;
}

/* Inner product of a product (k_ks_hmult and the form fused into the row pass),
 * double-precision branch, one output of each half: the own digit (own < 0: none,
 * a special limb, whose sums leave as they are) enters as the signed product
 * a1 b1, the others as residues or, `lazy`, as the row pass leaves them (within
 * 1.63p of 0); P^-1 times the centred sum plus the tensor product's one or two
 * products.  extreme: p - 1 and p - 2 operands, and constants at +-p/2.
 * Returns the number of mismatches, -1 when a sum reaches 8p or 2^53. */
int emu_hmult_check(uint64_t p, int nd, int own, int lazy, uint64_t seed, int trials, int extreme) {
    const double pd = (double)p, pinv = recip_up(p);
    uint64_t s = seed;
    int bad = 0;
    for (int t = 0; t < trials; ++t) {
        uint64_t in[4];
        for (int i = 0; i < 4; ++i) in[i] = extreme ? p - 1 - ((uint64_t)t >> i & 1) : splitmix(&s) % p;
        const uint64_t a0 = in[0], a1 = in[1], b0 = in[2], b1 = in[3];
        double acc[2] = {0, 0};
        uint64_t exact[2] = {0, 0};
        for (int d = 0; d < nd; ++d) {
            double x;
            uint64_t xr;
            if (d == own) {
                x = fp_mulmod((double)a1, (double)b1, pd, pinv);
                xr = mulmod(a1, b1, p);
            } else {
                xr = extreme ? p - 1 - ((uint64_t)t >> (d & 3) & 1) : splitmix(&s) % p;
                x = (double)xr;
                if (lazy && extreme) {
                    x = floor(1.63 * pd);
                    xr = (uint64_t)x % p;
                    if (t & 1) x = -x, xr = p - xr;
                } else if (lazy) {
                    if (splitmix(&s) & 1) x -= pd;
                    if (x > 0 && x < 0.63 * pd && splitmix(&s) & 1) x += pd;
                }
            }
            for (int h = 0; h < 2; ++h) {
                const uint64_t k = extreme ? p - 1 - (uint64_t)(h & t) : splitmix(&s) % p;
                acc[h] += fp_mulmod(x, (double)k, pd, pinv);
                exact[h] = (exact[h] + mulmod(xr, k, p)) % p;
                if (fabs(acc[h]) >= 8 * pd || fabs(acc[h]) >= 9007199254740992.0) return -1;
            }
        }
        if (own >= 0) {
            const uint64_t ci = extreme ? (t & 1 ? p / 2 : p / 2 + 1) : splitmix(&s) % p;
            const double c = ci > p / 2 ? -(double)(p - ci) : (double)ci, cq = c / pd;
            for (int h = 0; h < 2; ++h) {
                acc[h] = fp_mulw(fp_center(acc[h], pd, pinv), c, cq, pd);
                exact[h] = mulmod(exact[h], ci, p);
            }
            acc[0] += fp_mulmod((double)a0, (double)b0, pd, pinv);
            acc[1] = (acc[1] + fp_mulmod((double)a0, (double)b1, pd, pinv)) + fp_mulmod((double)a1, (double)b0, pd, pinv);
            exact[0] = (exact[0] + mulmod(a0, b0, p)) % p;
            exact[1] = ((exact[1] + mulmod(a0, b1, p)) % p + mulmod(a1, b0, p)) % p;
        }
        for (int h = 0; h < 2; ++h) bad += fp_sum_to_u(acc[h], pd, pinv) != exact[h];
    }
    return bad;
}

/* Plaintext dot products (k_dot_pt), double-precision branch: n terms, centred
 * every seven, on top of a residue (`accumulate`), and the element-wise product
 * (k_elementwise), floor-reduced without centring. */
int emu_dot_check(uint64_t p, int n, int accumulate, uint64_t seed, int trials, int extreme) {
    const double pd = (double)p, pinv = recip_up(p);
    uint64_t s = seed;
    int bad = 0;
    for (int t = 0; t < trials; ++t) {
        uint64_t exact = accumulate ? (extreme ? p - 1 : splitmix(&s) % p) : 0;
        double acc = (double)exact;
        for (int k = 0, since = 0; k < n; ++k) {
            const uint64_t x = extreme ? p - 1 : splitmix(&s) % p;
            const uint64_t w = extreme ? p - 1 - (uint64_t)(t & 1) : splitmix(&s) % p;
            const double r = fp_mulmod((double)x, (double)w, pd, pinv);
            bad += fp_to_u(r, pd, pinv) != mulmod(x, w, p);
            acc += r;
            exact = (exact + mulmod(x, w, p)) % p;
            if (fabs(acc) >= 8 * pd) return -1;
            if (++since == 7) {
                acc = fp_center(acc, pd, pinv);
                since = 0;
            }
        }
        bad += fp_sum_to_u(acc, pd, pinv) != exact;
    }
    return bad;
}
