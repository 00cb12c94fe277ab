// ntt_sched.hpp -- where the double-precision transforms centre their values
// (constants evaluated at compile time; tests/test_ntt_sched.py runs the
// schedules on the host and checks the bounds).
//
// Residues of a prime p < 2^50 are held as integer-valued doubles, bounds below
// are in units of p.  A product y w (fp_mulw, fp64.cuh) is exact while the
// quotient |y w / p| stays below 2^51.  Twiddles are held centred, |w| <= p/2,
// so y may reach 4p; twiddles formed in the kernel by one product (fp_mulmod of
// two centred table entries) satisfy |w| <= 0.594p, so y may reach 3.36p.
// The product's remainder is at most
//   1/2 + |y| |w/p - wq| :  wq the rounded w/p of the table: |y| 2^-55,
//                           wq = fl(w fl(1/p)) of a formed w: |y| 0.6 1.5 2^-52.
// Sums and differences below 8p = 2^53 are exact.  Centring a value
// (x - rint(x/p) p, 3 operations) brings it to 1/2; the schedules apply it only
// where the next product's operand would pass its bound, instead of at
// every other stage (forward) or every stage (inverse): 4 of the forward's 16
// stages at N = 2^16, and about one sum in four of the inverse.
#pragma once

namespace fides {

constexpr double kYMaxTable = 3.99, kYMaxFormed = 3.3;
constexpr double kCentred = 0.501;
constexpr double prod_bound(bool formed, double y) { return formed ? 0.5 + 0.225 * y : 0.5 + y / 32; }
constexpr double y_max(bool formed) { return formed ? kYMaxFormed : kYMaxTable; }

// Forward (Cooley-Tukey) stages: x' = x + t, y' = x - t, t = y w.  Every element
// has the same bound, and red[s] says whether stage s centres x first.  The
// last stage always does (its output is reduced to a canonical residue).
// Stages lr+4 and later (the row pass's second register group) use formed
// twiddles.
struct FwdSched {
    bool red[16];
    double bound[17];  // of every element before stage s; bound[logn] at the end
};
constexpr FwdSched fwd_sched(int logn, int lr) {
    FwdSched r{};
    double b = 1.0;  // canonical residues, or centred ones
    for (int s = 0; s < logn; ++s) {
        r.bound[s] = b;
        const double t = prod_bound(s >= lr + 4, b);
        const bool last = s == logn - 1;
        r.red[s] = last || b + t > y_max(s + 1 >= lr + 4);
        b = (r.red[s] ? kCentred : b) + t;
    }
    r.bound[logn] = b;
    return r;
}

// Inverse (Gentleman-Sande) stages of one register group of 16 elements:
// x' = x + y, y' = (x - y) w over partner bits kb = 0 .. nst-1.  Elements keep
// their own interval; mask[kb] bit k says that stage kb centres the sum left
// in element k.  Before a group every element has the interval [lo, hi] (the
// union over the previous group, whose elements the exchange permutes).
struct InvGroup {
    unsigned mask[4];
    double lo, hi;  // after the group
};
// formed: this group's twiddles; next_max: operand bound of the stage after
// the group (on the difference, and on the sum where `both`)
constexpr InvGroup inv_group_sched(int nst, bool formed, double next_max, double lo0, double hi0, bool both) {
    InvGroup g{};
    double lo[16] = {}, hi[16] = {};
    for (int k = 0; k < 16; ++k) {
        lo[k] = lo0;
        hi[k] = hi0;
    }
    for (int kb = 0; kb < nst; ++kb) {
        const bool end = kb == nst - 1;
        const double lim = end ? next_max : y_max(formed);
        for (int k = 0; k < 16; ++k) {
            if (k & (1 << kb)) continue;
            const double l = lo[k], h = hi[k];  // both partners' interval
            double sl = 2 * l, sh = 2 * h;
            const double mag = sh > -sl ? sh : -sl;
            const double need = (end && both) ? 2 * mag : sh - sl;
            if (need > lim) {
                g.mask[kb] |= 1u << k;
                sl = -kCentred;
                sh = kCentred;
            }
            const double t = prod_bound(formed, h - l);
            lo[k] = sl;
            hi[k] = sh;
            lo[k | (1 << kb)] = -t;
            hi[k | (1 << kb)] = t;
        }
    }
    g.lo = lo[0];
    g.hi = hi[0];
    for (int k = 1; k < 16; ++k) {
        g.lo = lo[k] < g.lo ? lo[k] : g.lo;
        g.hi = hi[k] > g.hi ? hi[k] : g.hi;
    }
    return g;
}

// The inverse transform's groups: row pass A (lc - 4 stages, formed twiddles;
// absent for lc = 4), row pass B (4 stages), column pass A (lr - 4 stages;
// absent for lr = 4), column pass B (3 stages and the scaled last one, whose
// sum is a product operand too).
struct InvSched {
    InvGroup ra, rb, ca, cb;
};
constexpr InvSched inv_sched(int lr, int lc) {
    InvSched s{};
    double lo = -kCentred, hi = 1.0;  // canonical residues, or centred products
    if (lc > 4) {
        s.ra = inv_group_sched(lc - 4, true, kYMaxTable, lo, hi, false);
        lo = s.ra.lo;
        hi = s.ra.hi;
    }
    s.rb = inv_group_sched(4, false, kYMaxTable, lo, hi, false);
    lo = s.rb.lo;
    hi = s.rb.hi;
    if (lr > 4) {
        s.ca = inv_group_sched(lr - 4, false, kYMaxTable, lo, hi, false);
        lo = s.ca.lo;
        hi = s.ca.hi;
    }
    s.cb = inv_group_sched(3, false, kYMaxTable, lo, hi, true);
    return s;
}

}  // namespace fides
