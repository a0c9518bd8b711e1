// bicg_coop.cuh -- whole batches of BiCGSTAB iterations in one cooperative
// launch, for systems whose rows all have a thread of a resident grid.
//
// Bound: the chain of dependent phases, not the arithmetic.  An iteration is
// three phases that end in dot products (v = A p, t = A s, the update of x
// and r) and two that only form vectors (p, s).  As five kernels each phase
// pays a launch, its loads' latencies, and a last-block reduction through a
// ticket.  Here the grid stays resident, 32 rows a warp, dealt round the SMs:
//  - the matrix rows in shared memory (read once per launch);
//  - a row's own vector entries in its thread's registers;
//  - a grid barrier per phase, after which every block sums the partials
//    itself, so that no block waits for a reducing one.  That sum is read and
//    added up by every SM: its layout (a lane's eight values at a stride, so
//    that a warp reads whole lines) and, in larger systems, partials that
//    stand for four warps are what keep it short;
//  - up to MERGE_ROWS rows, p and s formed where they are gathered instead of
//    in phases of their own, by all warps of the block into shared memory:
//    three barriers an iteration instead of five.
// Per iteration at 7600 rows: 35 us as five kernels in a graph, ~15 us here:
// three barriers ~1.8 us each, two products ~2.5 us each (28 FP64 FMAs
// in turn, 64 clocks or more each), three sums with their quotients ~1.5 us each.
// 125k rows of 21 entries: 48.8 us with a partial per warp and two rows per
// thread, 33.5 us here.
// The grid is launched cooperatively (all blocks resident), and every wait is
// bounded: where one runs out the launch ends without its results, and the host
// goes on with the five kernels from x as it is (rows of blocks that had got to
// the end may be new, the others old: any x will do to restart from).
#pragma once

#include "bsc_internal.cuh"
#include "warpsum.cuh"

namespace bsc {

// ---- grid barrier -------------------------------------------------------------------
// count: arrivals (zero at launch, or out of reach: bicg_coop_launch); err: set to 1 once a wait has run out.
// The arrival releases what the block has written (its threads' writes come
// before it by the block barrier), the polls acquire: with relaxed accesses
// between __threadfence() calls a barrier took ~3000 clocks on 152 blocks, and
// steps of 3.8k to 51k rows 5 to 7 % longer (one fence after relaxed polls:
// the same).  A word per block, each watched by every block, took 14000: the
// watching slows the words' stores.
// a constant: as a kernel parameter it cost an iteration 1 % at 4096 rows
constexpr unsigned GRID_SPIN_LIMIT = 1u << 21;  // polls: a few tenths of a second

struct GridBarrier {
    unsigned* count;
    double* err;
    unsigned target = 0;
    // every thread of every block; false (in all threads of the block) if some
    // block never arrived: the caller returns
    __device__ __forceinline__ bool sync() {
        __syncthreads();
        target += gridDim.x;
        int fine = 1;
        if (threadIdx.x == 0) {
            asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(count) : "memory");
            for (unsigned spins = 0;; ++spins) {
                unsigned v;
                asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(count) : "memory");
                if ((int)(v - target) >= 0) break;
                if (spins >= GRID_SPIN_LIMIT) {
                    *err = 1.0;
                    fine = 0;
                    break;
                }
            }
        }
        return __syncthreads_and(fine);
    }
};

constexpr int COOP_WARPS = 16;                     // warps per block at most
constexpr int COOP_BLOCK = COOP_WARPS * 32;
// Measured, four steps with and without MERGE: 24.5 and 24.9 ms at 10414 rows,
// 33.2 and 34.0 at 18322, 38.2 and 35.5 at 21490, 70.3 and 54.7 at 42138.
constexpr int64_t MERGE_ROWS = 20000;
// shared memory of one entry of a warp's 32 rows: value and column, and with MERGE the formed vector's value
constexpr int coop_entry(bool merge) { return 32 * (int)(sizeof(double) + sizeof(int32_t) + (merge ? sizeof(double) : 0)); }
constexpr int COOP_ITERS = 1024;                   // iterations per launch: tens of milliseconds at the largest sizes
constexpr int COOP_BAR = 64;                       // the barrier's word in the ticket array
constexpr int COOP_SETS = 5;                       // partials of an iteration's three reductions, a set per value
// doubles a set takes at most: a partial per warp of rows
constexpr int coop_part(int64_t n) { return (int)((n + 255) / 256 * 8); }

// the warp sum over the tree of warp_sum_to_lane0, in every lane
__device__ __forceinline__ double warp_sum_all(double x) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    return x;
}

// The D values of `part` summed as block_partials and reduce_partials sum
// them: warps in groups of eight (a 256-row block of those kernels), 256
// threads over the groups, trees over 32 and then 8.  The 32-thread parts of
// the 256 with any group are dealt to this block's warps; sh[d][0..7] receives
// their sums (the rest are exact zeros), which warp 0 adds up in eight_sum.
// Only warps with something to add run FP64 instructions: each holds the SM's
// FP64 pipe for its whole warp, and every idle warp's copy of the sums cost as
// much as a working one's (38 us an iteration at 7600 rows with all 16 warps
// computing all scalars).
// G = 4: a partial stands for four warps, the even or the odd ones of a group,
// which one block holds and adds up first: a quarter of the loads and one
// addition a group instead of seven.  Used without MERGE: the blocks' rows
// come in fours of warps, which below some 20000 rows leaves SMs idle (18322
// rows: 33.2 ms with MERGE and G = 1, 33.3 with G = 4; 7281: 18.7 and 21.8;
// 25881 without MERGE: 43.3 and 40.2; 62118: 76.9 and 73.1).
template <int D, int G>
__device__ __forceinline__ void coop_sum(const double* part, int stride, int nwarps, double (&sh)[D][8]) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, W = blockDim.x >> 5;
    const int groups = (nwarps + 7) / 8, parts = min((groups + 31) / 32, 8);
    if (threadIdx.x < 8 * D && (int)(threadIdx.x % 8) >= parts) sh[threadIdx.x / 8][threadIdx.x % 8] = 0.0;
    for (int z = w; z < D * parts; z += W) {
        const int d = z / parts, vw = z - d * parts;
        double x = 0.0;
        for (int g = 32 * vw + lane; g < groups; g += 256) {
            if (G == 4) {
                const double2 y = __ldcg(reinterpret_cast<const double2*>(part + d * stride) + g);
                x += y.x + y.y;
            } else {
                const double* q = part + d * stride + g;
                double y[8];
#pragma unroll
                for (int k = 0; k < 8; ++k) y[k] = 8 * g + k < nwarps ? __ldcg(q + k * groups) : 0.0;
                x += ((y[0] + y[4]) + (y[2] + y[6])) + ((y[1] + y[5]) + (y[3] + y[7]));
            }
        }
        x = warp_sum_all(x);
        if (lane == 0) sh[d][vw] = x;
    }
    __syncthreads();
}
__device__ __forceinline__ double eight_sum(const double (&q)[8], int nwarps) {
    if (nwarps <= 256) return q[0];  // one part: the others are zero
    return ((q[0] + q[4]) + (q[2] + q[6])) + ((q[1] + q[5]) + (q[3] + q[7]));
}

// Up to `iters` iterations from the state k_bicg_init and k_bicg_setup (or an
// earlier launch) left: x, r, rh, p and the scalars rho, target, it.  The
// update order and every sum are those of k_bicg_1..5: the same bits.  K: rows
// per thread.  p2 and v2 are the second halves of the double-buffered p and v
// (MERGE: gathered by other threads while this iteration's are written).
template <typename Op, bool MERGE, int K, int THREADS, int G>
__global__ void __launch_bounds__(THREADS, 1)
    k_bicg_coop(int64_t n, Op A, double* x, double* r, const double* rh, double* p, double* v, double* s, double* p2,
                double* v2, double* part, Scalars* sc, unsigned* count, int iters, int cap) {
    static_assert(G == 1 || K == 1, "G > 1: one row per thread");
    extern __shared__ __align__(16) unsigned char coop_sm[];
    double* sval = reinterpret_cast<double*>(coop_sm);
    double* sy = sval + (size_t)cap * 32;  // MERGE: the formed vector at the entries' columns
    int32_t* scol = reinterpret_cast<int32_t*>(sval + (size_t)cap * 32 * (MERGE ? 2 : 1));
    __shared__ int used;
    // MERGE: the places, lengths and rows' lengths of the block's units, for the warps that form their entries
    __shared__ int u_off[COOP_WARPS], u_len[COOP_WARPS], u_m[COOP_WARPS][32];
    // scalars: one warp computes each once per block and hands it on
    __shared__ double sh1[1][8], sh2[2][8], sh3[2][8], s_alpha, s_omega, s_q, s_ao, s_rr, s_rho;
    __shared__ int s_brk, s_conv;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, W = blockDim.x >> 5;
    if (sc->done | sc->breakdown) return;  // the same for every block
    if (threadIdx.x == 0) used = 0;
    __syncthreads();
    // units of 32 rows dealt round the blocks: the FP64 work of a phase spreads over the SMs
    const int nwarps = (int)((n + 31) / 32);
    int unit[K], m[K], off[K];  // off < 0: the warp reads these rows from memory
    double xi[K], ri[K], pi[K], vi[K], rhi[K], si[K], ti[K];
#pragma unroll
    for (int q = 0; q < K; ++q) {
        if (G > 1) {  // the units of a partial: every (8 / G)-th of a group of eight
            const int z = (w / G) * (int)gridDim.x + (int)blockIdx.x;
            unit[q] = 8 * (z / (8 / G)) + z % (8 / G) + (8 / G) * (w % G);
        } else {
            unit[q] = (w + q * W) * (int)gridDim.x + (int)blockIdx.x;
        }
        const int64_t i = (int64_t)unit[q] * 32 + lane;
        const bool act = i < n;
        m[q] = act ? A.len(i) : 0;
        const int mw = __reduce_max_sync(0xffffffffu, m[q]);
        int o = 0;
        if (lane == 0) o = mw <= cap ? atomicAdd(&used, mw) : cap;  // (the sum stays far from overflow)
        o = __shfl_sync(0xffffffffu, o, 0);
        off[q] = o + mw <= cap ? o : -1;
        if (MERGE) {
            u_m[w][lane] = m[q];
            if (lane == 0) {
                u_off[w] = off[q];
                u_len[w] = mw;
            }
        }
        if (off[q] >= 0)
            for (int k = 0; k < m[q]; ++k) {
                const int64_t e = A.at(i, k);
                sval[(o + k) * 32 + lane] = A.val_at(e);
                scol[(o + k) * 32 + lane] = A.col_at(e);
            }
        xi[q] = act ? x[i] : 0.0;
        ri[q] = act ? r[i] : 0.0;
        pi[q] = act ? p[i] : 0.0;
        rhi[q] = act ? rh[i] : 0.0;
        vi[q] = si[q] = ti[q] = 0.0;
    }
    auto row = [&](int q) { return (int64_t)unit[q] * 32 + lane; };
    auto busy = [&](int q) { return unit[q] < nwarps; };  // warps without rows run no FP64 for them
    auto act = [&](int q) { return row(q) < n; };
    // this thread's row q of A times the vector `get` yields, summed in the
    // row's entry order, four gathers in flight (more, and a software
    // pipeline over rounds of four, were slower)
    auto product = [&](int q, auto get) -> double {
        const int64_t i = row(q);
        const int o = off[q];
        double acc = Op::UNIT_DIAG ? get((int32_t)i) : 0.0;
        int k = 0;
        for (; k + 4 <= m[q]; k += 4) {
            double a[4], y[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                int32_t j;
                if (o >= 0) {
                    j = scol[(o + k + u) * 32 + lane];
                    a[u] = sval[(o + k + u) * 32 + lane];
                } else {
                    const int64_t e = A.at(i, k + u);
                    j = A.col_at(e);
                    a[u] = A.val_at(e);
                }
                y[u] = get(j);
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) acc += a[u] * y[u];
        }
        for (; k < m[q]; ++k) {
            const int64_t e = o >= 0 ? 0 : A.at(i, k);
            const int32_t j = o >= 0 ? scol[(o + k) * 32 + lane] : A.col_at(e);
            const double a = o >= 0 ? sval[(o + k) * 32 + lane] : A.val_at(e);
            acc += a * get(j);
        }
        return acc;
    };
    // MERGE: the vector `get` yields, at every entry of the block's rows, formed
    // by all warps together
    const int units = G * ((8 / G * ((nwarps + 7) / 8) + (int)gridDim.x - 1) / (int)gridDim.x);  // warps with rows, of any block
    auto form = [&](auto get) {
        int base = 0;  // deal the units' entries to the warps in one sequence
        for (int u = 0; u < units; ++u) {
            const int o = u_off[u], len = u_len[u], mu = u_m[u][lane];
            if (o < 0) continue;
            for (int k = (w - base % W + W) % W; k < len; k += W)
                if (k < mu) sy[(o + k) * 32 + lane] = get(scol[(o + k) * 32 + lane]);
            base += len;
        }
        __syncthreads();
    };
    // its product with this thread's row, the diagonal's term first
    auto formed_product = [&](double diag) -> double {
        const int o = off[0];
        double acc = Op::UNIT_DIAG ? diag : 0.0;
        int k = 0;
        for (; k + 4 <= m[0]; k += 4) {
            double a[4], y[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                a[u] = sval[(o + k + u) * 32 + lane];
                y[u] = sy[(o + k + u) * 32 + lane];
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) acc += a[u] * y[u];
        }
        for (; k < m[0]; ++k) acc += sval[(o + k) * 32 + lane] * sy[(o + k) * 32 + lane];
        return acc;
    };
    // a reduction's partials: a warp's sums of one or two values, and the
    // block's part once every warp has handed them over (before grid.sync)
    const int groups = (nwarps + 7) / 8, stride = 8 / G * groups;
    auto place = [&](int u) { return (u & 7) * groups + (u >> 3); };  // G = 1: a group's eight at a stride, read by a lane
    __shared__ double s_part[2][G > 1 ? THREADS / 32 : 1];
    if ((G > 1) && lane < 2) s_part[lane][w] = 0.0;  // warps without rows leave it so
    auto partial1 = [&](int q, double a) {
        a = warp_sum_all(a);
        if (lane == 0) {
            if (G > 1) s_part[0][w] = a;
            else part[place(unit[q])] = a;
        }
    };
    auto partials2 = [&](int q, double a, double b, double* out) {
        double ab[2] = {a, b};
        int which;
        const double y = warp_sums<2, double>(ab, which);
        if ((lane & 15) == 0) {
            if (G > 1) s_part[which][w] = y;
            else out[which * stride + place(unit[q])] = y;
        }
    };
    auto hand_over = [&](int D, double* out) {
        if (G == 1) return;
        __syncthreads();
        const int d = lane >> 3, h = lane & 7, z = h * (int)gridDim.x + (int)blockIdx.x;
        if (w == 0 && d < D && G * h < W && z < stride) {
            const double* y = &s_part[d][G * h];
            out[d * stride + z] = (y[0] + y[2]) + (y[1] + y[3]);
        }
    };
    double rho = sc->rho, alpha = 0.0, omega = 0.0, beta = 0.0, rr = sc->rr;
    const double target = sc->target;
    int it = sc->it, state = 0;
    bool first = true;
    __syncthreads();  // the units' matrix entries
    GridBarrier grid{count, &sc->tmp[7]};
    double *pold = p, *pnew = p2, *vold = v, *vnew = MERGE ? v2 : v;
    double* part1 = part + stride;      // each reduction its own partials: a block may still
    double* part2 = part + 3 * stride;  // read one while another writes the next
    for (int iter = 0; iter < iters; ++iter) {
        // v = A p
        if (!first) {
#pragma unroll
            for (int q = 0; q < K; ++q)
                if (busy(q)) {
                    pi[q] = ri[q] + beta * (pi[q] - omega * vi[q]);
                    if (!MERGE && act(q)) p[row(q)] = pi[q];
                }
            if (!MERGE && !grid.sync()) return;
        }
        if (MERGE && first) form([&](int32_t j) { return pold[j]; });
        if (MERGE && !first) {
            const double be = s_q * s_ao;
            form([&](int32_t j) { return r[j] + be * (pold[j] - omega * vold[j]); });
        }
#pragma unroll
        for (int q = 0; q < K; ++q)
            if (busy(q)) {
                if (act(q)) {
                    if (MERGE && off[q] >= 0)
                        vi[q] = formed_product(pi[q]);
                    else if (MERGE && !first)
                        vi[q] = product(q, [&](int32_t j) { return r[j] + beta * (pold[j] - omega * vold[j]); });
                    else
                        vi[q] = product(q, [&](int32_t j) { return pold[j]; });
                    if (MERGE) pnew[row(q)] = pi[q];
                    vnew[row(q)] = vi[q];
                }
                partial1(q, rhi[q] * vi[q]);
            }
        hand_over(1, part);
        if (!grid.sync()) return;
        coop_sum<1, G>(part, stride, nwarps, sh1);
        if (w == 0) {
            const double d = eight_sum(sh1[0], nwarps);
            const bool b = d == 0.0 || rho == 0.0;
            if (!b) alpha = rho / d;
            if (lane == 0) {
                s_alpha = alpha;
                s_brk = b;
            }
        }
        __syncthreads();
        if (s_brk) {
            state = 2;
            break;
        }
        alpha = s_alpha;
        // t = A s, s = r - alpha v
#pragma unroll
        for (int q = 0; q < K; ++q)
            if (busy(q)) {
                si[q] = ri[q] - alpha * vi[q];
                if (!MERGE && act(q)) s[row(q)] = si[q];
            }
        if (!MERGE && !grid.sync()) return;
        if (MERGE) form([&](int32_t j) { return r[j] - alpha * vnew[j]; });
#pragma unroll
        for (int q = 0; q < K; ++q)
            if (busy(q)) {
                if (act(q)) {
                    if (MERGE && off[q] >= 0)
                        ti[q] = formed_product(si[q]);
                    else if (MERGE)
                        ti[q] = product(q, [&](int32_t j) { return r[j] - alpha * vnew[j]; });
                    else
                        ti[q] = product(q, [&](int32_t j) { return s[j]; });
                }
                partials2(q, ti[q] * si[q], ti[q] * ti[q], part1);
            }
        hand_over(2, part1);
        if (!grid.sync()) return;
        coop_sum<2, G>(part1, stride, nwarps, sh2);
        if (w == 0) {
            const double d0 = eight_sum(sh2[0], nwarps), d1 = eight_sum(sh2[1], nwarps);
            omega = d1 == 0.0 ? 0.0 : d0 / d1;
            if (lane == 0) s_omega = omega;
        }
        __syncthreads();
        omega = s_omega;
        if (w == W - 1) {  // beta's second quotient, while the others update
            const double ao = alpha / omega;
            if (lane == 0) s_ao = ao;
        }
        // x and r, the residual and rho
#pragma unroll
        for (int q = 0; q < K; ++q)
            if (busy(q)) {
                xi[q] = xi[q] + alpha * pi[q] + omega * si[q];
                ri[q] = si[q] - omega * ti[q];
                if (act(q)) r[row(q)] = ri[q];
                partials2(q, ri[q] * ri[q], rhi[q] * ri[q], part2);
            }
        hand_over(2, part2);
        if (!grid.sync()) return;
        coop_sum<2, G>(part2, stride, nwarps, sh3);
        ++it;
        // beta = (rho' / rho) (alpha / omega) by one warp, the stop by another
        if (w == 0) {
            const double d1 = eight_sum(sh3[1], nwarps), q = d1 / rho;
            rho = d1;
            if (lane == 0) {
                s_q = q;
                s_rho = d1;
                s_brk = omega == 0.0 || d1 == 0.0;
            }
        }
        if (w == W - 1) {
            rr = eight_sum(sh3[0], nwarps);
            if (lane == 0) {
                s_rr = rr;
                s_conv = sqrt(rr) <= target;
            }
        }
        __syncthreads();
        state = s_conv ? 1 : s_brk ? 2 : 0;
        if (!state && busy(0)) beta = s_q * s_ao;
        first = false;
        if (MERGE) {
            double* t = pold; pold = pnew; pnew = t;
            t = vold; vold = vnew; vnew = t;
        }
        if (state) break;
    }
#pragma unroll
    for (int q = 0; q < K; ++q)
        if (act(q)) {
            x[row(q)] = xi[q];
            if (!state) p[row(q)] = ri[q] + beta * (pi[q] - omega * vi[q]);  // the next launch's p
        }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        if (!first) {  // an iteration came to its end
            sc->rr = s_rr;
            sc->rho = s_rho;
        }
        sc->it = it;
        sc->done = state == 1 ? 1 : 0;
        sc->breakdown = state == 2 ? 1 : 0;
    }
}

}  // namespace bsc
