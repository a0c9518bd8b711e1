// lanes.cuh -- several lanes per particle for the FP64 pair sums.
//
// A warp issues one FP64 add, multiply or FMA per 64 clocks on this GPU,
// dependent or not, and an SM one per 19 (measured, one block, clock64): with
// fewer than some four warps an SM that have FP64 work at hand, a pair sum's time
// is the length of a thread's own loop, whatever the particle count.  L lanes of a warp then share a particle: each takes
// every L-th neighbour, and the sums are added up across them.
#pragma once

#include <type_traits>

#include "bsc_internal.cuh"

namespace bsc {

// Lanes per particle for n particles.  Measured, 20 WCSPH steps with 1, 2, 4
// and 8 lanes: 3.59, 3.56, 2.67, 2.42 ms at 3816 particles; 3.99, 4.10, 3.48,
// 3.82 at 15797; 4.35, 4.84, 4.70, 5.39 at 30732: by then the particles alone
// give the SMs their warps, and the sums across lanes cost more than the
// shorter loops save.
inline int lanes_for(int64_t n) { return n <= 10000 ? 8 : n <= 20000 ? 4 : 1; }

// Lanes per row in the fine-level passes and products of an FGMRES iteration.
// Measured, four steps with 1 and 4 lanes: FP64 5.53 and 5.22 ms at 3816 rows,
// 5.83 and 5.66 at 10414, 6.91 and 6.90 at 18322, 6.85 and 7.15 at 25881;
// mixed 5.24 and 5.07, 5.31 and 5.14, 6.40 and 6.16, 5.86 and 5.76, and 8.90
// and 9.47 at 78948.  (Two lanes gain
// less at the smallest, eight less everywhere.)
inline int row_lanes(int64_t n) { return n <= 20000 ? 4 : 1; }

template <int L>
struct Lanes {
    int sub;         // this lane's share of its particle
    unsigned mask;   // the lanes of the particle
    unsigned below;  // those before this one
    __device__ __forceinline__ Lanes() {
        const int lane = threadIdx.x & 31;
        sub = lane & (L - 1);
        mask = (L == 32 ? 0xffffffffu : ((1u << L) - 1u)) << (lane - sub);
        below = mask & ((1u << lane) - 1u);
    }
    static __device__ __forceinline__ int64_t particle() {
        return (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) / L;
    }
    // the sum over the particle's lanes, in each of them
    __device__ __forceinline__ double sum(double x) const {
#pragma unroll
        for (int o = L / 2; o > 0; o >>= 1) x += __shfl_xor_sync(mask, x, o);
        return x;
    }
    // lane u's x, a double-float
    template <typename X>
    __device__ __forceinline__ X from(X x, int u) const {
        if (L > 1) {
            x.hi = __shfl_sync(mask, x.hi, u, L);
            x.lo = __shfl_sync(mask, x.lo, u, L);
        }
        return x;
    }
    // acc[q] += a[q] b[q] over the particle's lanes in turn, in each of them: the
    // bits of one thread's fused sums over the same terms (a lane past the end
    // of the list hands in zeros)
    template <typename R, int N>
    __device__ __forceinline__ void ordered(R (&acc)[N], const R (&a)[N], const R (&b)[N]) const {
#pragma unroll
        for (int u = 0; u < L; ++u)
#pragma unroll
            for (int q = 0; q < N; ++q)
                acc[q] = fma(L == 1 ? a[q] : __shfl_sync(mask, a[q], u, L),
                             L == 1 ? b[q] : __shfl_sync(mask, b[q], u, L), acc[q]);
    }
    // the place of this lane's kept item among the particle's, after `count`
    // of them; count moves past them
    __device__ __forceinline__ int place(bool keep, int& count) const {
        if (L == 1) return keep ? count++ : count;
        const unsigned b = __ballot_sync(mask, keep) & mask;
        const int at = count + __popc(b & below);
        count += __popc(b);
        return at;
    }
    __device__ __forceinline__ void sync() const {
        if (L > 1) __syncwarp(mask);
    }
};

// f with the number of lanes as a compile-time constant
template <typename F>
void with_lanes(int lanes, F f) {
    switch (lanes) {
        case 8: f(std::integral_constant<int, 8>{}); break;
        case 4: f(std::integral_constant<int, 4>{}); break;
        default: f(std::integral_constant<int, 1>{}); break;
    }
}

// The FP64 step's pair sums: four lanes, their terms added up in list order
// (Lanes::ordered).  Measured with one and four lanes at 8967, 16422, 23441 and
// 28635 particles (about 20 neighbours), us:
//   search       53 / 31   54 / 48   67 / 56   67 / 61
//   effpor       41 / 33   39 / 43   57 / 47   57 / 49
//   assembly     70 / 35   70 / 49   85 / 60   87 / 74
//   int_vel      55 / 33   53 / 50   70 / 62   70 / 97: its blocks (86 registers) no longer fit at once
//   comp_vel     31 / 23   31 / 32   39 / 37   40 / 43
//   eddyvis      27 / 23   27 / 33   33 / 37   34 / 43  (12931: 26 / 27)
//   opt2_shift   21 / 19   21 / 31   24 / 37   24 / 45  (12931: 20 / 25)
// With 40 and 70 neighbours the lines lie in the same places.  On the mixed path
// the search and the assembly gain as above, int_vel (29 / 17 at 16422) and
// varts are given the lanes up to PAIR_LANES_LIGHT, eddyvis as in FP64 (19 / 19
// at 8967, 19 / 21 at 16422).
constexpr int64_t PAIR_LANES = 30000, PAIR_LANES_VEL = 24000, PAIR_LANES_LIGHT = 20000, PAIR_LANES_EDDY = 12000,
                  PAIR_LANES_SHIFT = 10000;
// (BSC_PAIR_LANES: one or four at any size, for comparing the two)
inline bool pair_lanes(const Ctx* c, int64_t most = PAIR_LANES) {
    return c->pair_lanes ? c->pair_lanes > 1 : c->n <= most;
}
template <typename F>
void with_pair_lanes(const Ctx* c, F f, int64_t most = PAIR_LANES) {
    if (pair_lanes(c, most)) f(std::integral_constant<int, 4>{});
    else f(std::integral_constant<int, 1>{});
}

}  // namespace bsc
