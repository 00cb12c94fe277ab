// ntt_n.cu -- the transforms of one ring dimension N = 2^FIDES_LOGN; compiled
// once per dimension (Makefile), so that the dimensions build in parallel.
#include "ntt_kernels.cuh"

namespace fides {

template <>
const NttOps& ntt_ops<FIDES_LOGN>() {
    using T = NttN<FIDES_LOGN / 2, FIDES_LOGN - FIDES_LOGN / 2>;
    static const NttOps ops = {T::fwd, T::inv, T::fwd_cols, T::rows_ks, T::prepare};
    return ops;
}

}  // namespace fides
