// ntt_sched.hpp -- where the double-precision transforms centre their values
// (constants evaluated at compile time).
//
// Residues of a prime p < 2^50 are held as integer-valued doubles; centring
// (x - rint(x/p) p, 3 operations) keeps every value below 1.7p, so that every
// product's quotient stays below 2^51 and every sum is exact.
#pragma once

namespace fides {

// Forward stages (x' = x + y w, y' = x - y w): red[s] says whether stage s
// centres x first.  The column pass (fed canonical residues) centres on odd
// positions of each register group; the row pass (fed the column pass's
// values) on even ones in its first group and always in its second, whose
// twiddles are formed in the kernel and carry a looser quotient.  The last stage
// always centres (its output is reduced to a canonical residue).
struct FwdSched {
    bool red[16];
};
constexpr FwdSched fwd_sched(int logn, int lr) {
    FwdSched r{};
    for (int s = 0; s < logn; ++s)
        r.red[s] = s == logn - 1 || (s < lr ? (s & 3) % 2 == 1 : s < lr + 4 ? (s - lr) % 2 == 0 : true);
    return r;
}

// Inverse stages (x' = x + y, y' = (x - y) w) of one register group: bit k of
// mask[kb] says that partner bit kb's stage centres the sum left in element k.
struct InvGroup {
    unsigned mask[4];
};
struct InvSched {
    InvGroup ra, rb, ca, cb;  // row pass groups, column pass groups
};
constexpr InvSched inv_sched(int, int) {
    constexpr InvGroup all = {{0xffff, 0xffff, 0xffff, 0xffff}};
    return {all, all, all, all};
}

}  // namespace fides
