// warpsum.cuh -- warp sums of the Krylov reductions.
#pragma once

namespace bsc {

// The warp sums of D values (D a power of two up to 32) at once.  While more
// than one value is left, the two halves of the warp split the values
// between them: at each step a lane keeps half of its values and adds what
// its partner at distance o holds of them, so D values take
// D - 1 + 5 - log2(D) adds instead of 5 D.  An FP64 instruction holds this
// GPU's FP64 pipe for the whole warp however few lanes want its result, and
// the shuffle adds bounded the multi-dot kernels (eight dots: 9 adds, 40
// before).  Every value is summed over the same tree as warp_sum_to_lane0's
// (each addition's operands at most exchanged): the same bits.  Returns value
// `which` in the lanes that hold it (all lanes of a group of 32 / D; the
// group's first lane is 32 / D * which).
template <int D, typename V>
__device__ __forceinline__ V warp_sums(V (&v)[D], int& which) {
    const int lane = threadIdx.x & 31;
    which = 0;
#pragma unroll
    for (int o = 16, m = D; o > 0; o >>= 1) {
        if (m > 1) {
            const bool up = lane & o;
            m >>= 1;
#pragma unroll
            for (int q = 0; q < m; ++q) {
                const V send = up ? v[q] : v[q + m], keep = up ? v[q + m] : v[q];
                v[q] = keep + __shfl_xor_sync(0xffffffffu, send, o);
            }
            which = 2 * which + (up ? 1 : 0);
        } else {
            v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
        }
    }
    return v[0];
}

}  // namespace bsc
