/* Host run of the double-precision transforms with the centring schedules of
 * pyfideslib_b200/csrc/ntt_sched.hpp -- test infrastructure only.  The device
 * routines of fp64.cuh are restated with std::fma; every operand is checked
 * against the bound the schedule states for it, and the results against exact
 * integer arithmetic. */
#include <cfenv>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <vector>

#include "../pyfideslib_b200/csrc/ntt_sched.hpp"

using u128 = unsigned __int128;
static const double kRint = 6755399441055744.0, kTwo52 = 4503599627370496.0, k51 = 2251799813685248.0;

static uint64_t mulmod(uint64_t a, uint64_t b, uint64_t p) { return (uint64_t)((u128)a * b % p); }
static uint64_t powmod(uint64_t a, uint64_t e, uint64_t p) {
    uint64_t r = 1;
    for (; e; e >>= 1, a = mulmod(a, a, p))
        if (e & 1) r = mulmod(r, a, p);
    return r;
}
static uint32_t rev(uint32_t x, int n) {
    uint32_t r = 0;
    for (int i = 0; i < n; ++i) r |= (x >> i & 1) << (n - 1 - i);
    return r;
}
static double recip_up(uint64_t p) {
    double x = 1.0 / (double)p;
    int e;
    const double f = std::frexp(x, &e);
    if ((u128)(uint64_t)std::ldexp(f, 53) * p < ((u128)1 << (53 - e))) x = std::nextafter(x, 1.0);
    return x;
}
static bool g_bad;
static double mulw(double y, double w, double wq, double p, double rsub = kRint) {
    const double h = y * w, l = std::fma(y, w, -h);
    if (!(std::fabs(y * wq) < k51)) g_bad = true;
    const double q = std::fma(y, wq, kRint) - rsub;
    return std::fma(-q, p, h) + l;
}
static double center(double x, double p, double pinv, double rsub = kRint) {
    return std::fma(-(std::fma(x, pinv, kRint) - rsub), p, x);
}
static uint64_t pos_to_u(double v, double p, double pinv) {
    if (!(v > 0 && v < 4 * p)) g_bad = true;
    std::fesetround(FE_DOWNWARD);
    volatile double f = std::fma(v, pinv, kRint);
    std::fesetround(FE_TONEAREST);
    const double r = std::fma(-(f - kRint), p, v) + kTwo52;
    uint64_t u;
    std::memcpy(&u, &r, 8);
    return u & ((1ull << 52) - 1);
}
static double mulm(double x, double y, double p, double pinv) {
    const double h = x * y, l = std::fma(x, y, -h);
    return std::fma(-(std::fma(h, pinv, kRint) - kRint), p, h) + l;
}

struct Tab {
    std::vector<uint64_t> w;
    std::vector<double> c, q;
};

/* pattern 0 random, 1 all p - 1, 2 alternating 0 / p - 1, 3 all 0; the inverse runs
 * from canonical residues and from centred ones (what a product in its load
 * leaves).  Returns the number of wrong residues, -1 when a bound is broken */
extern "C" int emu_sched_check(int logn, uint64_t p, uint64_t psi, uint64_t seed, int pattern) {
    using namespace fides;
    const int lr = logn / 2, lc = logn - lr, N = 1 << logn;
    const double pd = (double)p, pinv = recip_up(p);
    g_bad = false;
    const uint64_t ipsi = powmod(psi, p - 2, p);
    Tab f, v;
    for (auto pr : {std::make_pair(&f, psi), std::make_pair(&v, ipsi)}) {
        Tab& t = *pr.first;
        std::vector<uint64_t> a(N, 1);
        for (int j = 1; j < N; ++j) a[j] = mulmod(a[j - 1], pr.second, p);
        for (int j = 0; j < N; ++j) {
            const uint64_t w = a[rev(j, logn)];
            t.w.push_back(w);
            t.c.push_back(w > p / 2 ? -(double)(p - w) : (double)w);
            t.q.push_back(t.c.back() / pd);
        }
    }
    /* twiddle idx of group offset g, formed when asked */
    auto tw = [&](const Tab& t, int idx, int g, bool formed, double& w, double& wq) {
        w = t.c[idx];
        wq = t.q[idx];
        if (formed && g) {
            w = mulm(t.c[idx - g], t.c[g], pd, pinv);
            if (std::fabs(w) > 0.6 * pd) g_bad = true;
            wq = w * pinv;
        }
    };
    std::vector<uint64_t> a(N), e;
    uint64_t s = seed;
    for (int j = 0; j < N; ++j) {
        s = s * 6364136223846793005ull + 1442695040888963407ull;
        a[j] = pattern == 1 ? p - 1 : pattern == 2 ? (j & 1 ? p - 1 : 0) : pattern == 3 ? 0 : (uint64_t)((u128)s * p >> 64);
    }
    e = a;
    for (int m = 1, t = N / 2; m < N; m <<= 1, t >>= 1)
        for (int i = 0; i < m; ++i)
            for (int j = 2 * i * t; j < 2 * i * t + t; ++j) {
                const uint64_t X = e[j], Y = mulmod(e[j + t], f.w[m + i], p);
                e[j] = (X + Y) % p;
                e[j + t] = (X + p - Y) % p;
            }
    std::vector<double> d(a.begin(), a.end());
    const FwdSched sc = fwd_sched(logn, lr);
    for (int m = 1, t = N / 2, st = 0; m < N; m <<= 1, t >>= 1, ++st) {
        const bool formed = st >= lr + 4;
        for (int i = 0; i < m; ++i) {
            double w, wq;
            /* the thread's group offset g < 2^(3 - kb), kb the partner bit */
            const int kb = logn - 1 - st;
            tw(f, m + i, formed ? i & ((1 << (3 - kb)) - 1) : 0, formed, w, wq);
            for (int j = 2 * i * t; j < 2 * i * t + t; ++j) {
                double x = d[j];
                const double y = d[j + t];
                if (std::fabs(x) > sc.bound[st] * pd + 1 || std::fabs(y) > sc.bound[st] * pd + 1) g_bad = true;
                if (sc.red[st]) x = center(x, pd, pinv, st == logn - 1 ? kRint + 2.0 : kRint);
                const double tt = mulw(y, w, wq, pd);
                d[j] = x + tt;
                d[j + t] = x - tt;
            }
        }
    }
    int bad = 0;
    for (int j = 0; j < N; ++j) bad += pos_to_u(d[j], pd, pinv) != e[j];
    if (g_bad) return -1;
    const InvSched iv = inv_sched(lr, lc);
    const uint64_t ninv = powmod(N, p - 2, p), s1 = mulmod(ninv, v.w[1], p);
    auto group = [&](const InvGroup& G, int bit0, int nst, bool formed) {
        for (int kb = 0; kb < nst; ++kb) {
            const int t = 1 << (bit0 + kb), m = N / (2 * t);
            for (int i = 0; i < m; ++i) {
                double w, wq;
                tw(v, m + i, formed ? i & ((1 << (3 - kb)) - 1) : 0, formed, w, wq);
                for (int j = 2 * i * t; j < 2 * i * t + t; ++j) {
                    const double x = d[j], y = d[j + t];
                    const int k = (j >> bit0) & 15;
                    double sm = x + y;
                    if (G.mask[kb] >> k & 1) sm = center(sm, pd, pinv);
                    if (std::fabs(x - y) > (formed ? kYMaxFormed : kYMaxTable) * pd) g_bad = true;
                    d[j] = sm;
                    d[j + t] = mulw(x - y, w, wq, pd);
                }
            }
        }
    };
    auto cst = [&](uint64_t c) { return c > p / 2 ? -(double)(p - c) : (double)c; };
    const double a0 = cst(ninv), a1 = cst(s1), a0q = a0 * pinv, a1q = a1 * pinv;
    for (int centred = 0; centred < 2; ++centred) {
        for (int j = 0; j < N; ++j) d[j] = centred && e[j] > p / 2 ? -(double)(p - e[j]) : (double)e[j];
        if (lc > 4) group(iv.ra, 0, lc - 4, true);
        group(iv.rb, lc - 4, 4, false);
        if (lr > 4) group(iv.ca, lc, lr - 4, false);
        group(iv.cb, lc + lr - 4, 3, false);
        for (int j = 0; j < N / 2; ++j) {
            const double x = d[j], y = d[j + N / 2];
            bad += pos_to_u(mulw(x + y, a0, a0q, pd, kRint + 2.0), pd, pinv) != a[j];
            bad += pos_to_u(mulw(x - y, a1, a1q, pd, kRint + 2.0), pd, pinv) != a[j + N / 2];
        }
    }
    return g_bad ? -1 : bad;
}
