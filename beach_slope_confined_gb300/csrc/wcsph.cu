// wcsph.cu -- the differentiable weakly compressible SPH step and its
// hand-written adjoint (the calibration workload: gradients of a wave-probe
// misfit with respect to the porous-drag coefficients and a porosity grid).
//
// Forward step (FP64, one thread per particle, gathers over the frozen
// neighbour lists of the step):
//   rt = max(rho, rho0) (fluid; the reference's dentopress reset of negative
//        pressure, wcsph.f90:36-62), p = B((rt/rho0)^gamma - 1), B = rho0 c0^2/gamma
//   n_i  = 1 - sum_s (1 - phi_s) V_s W(r_is)           porosity from the solids
//   Drho = sum_j m_j (rt_i/rt_j) (v_i - v_j).gW
//        + c2 sum_j (rt_j - rt_i - rhoH_j + rhoH_i) (x_j - x_i).gW V_j/(r^2+lam)
//                                    (wcsph.f90:66-133, c2 = delta 2h c0; the
//                                     diffusion written with x_j - x_i)
//   a    = -n_i sum_j m_j (p_i/rt_i^2 + p_j/rt_j^2) gW
//        + sum_j 2 nu V_j (x_ij.gW)/(r^2+lam) (v_i - v_j) + n_i g
//   R    = -nu alpha (1-n)^2/(n^3 d^2) - beta |v| (1-n)/(n^3 d)   (Ergun, porous.f90:192-212)
//   v'   = (v + dt a)/(1 - dt R n),  x' = x + dt v'/n,  rho' = rt + dt Drho
// with gW = F(r) (x_i - x_j) the Wendland C2 gradient and rhoH(y) the
// hydrostatic density below the still-water level.  Walls are prescribed
// (fixed hydrostatic density; the piston moves its wall particles).  The
// model carries its own particle masses m = rho_init dl^2, so that every
// volume m/rho starts at the lattice volume dl^2, inside the porous layer too
// (the ISPH masses rho0 n dl^2 would leave the kernel sums there short by n
// and the layer out of hydrostatic balance); v is the superficial velocity,
// the particles move at the pore velocity v/n.
//
// Adjoint: the exact reverse of that map for the fluid state (x, y, vx, vy,
// rho), geometry included (the derivative of gW through F'(r)); lists are
// symmetric, so each particle gathers the terms of its own sums and of its
// neighbours' sums without atomics.  Reverse sweep by segments: each segment
// of `ckpt_every` steps is recomputed from its checkpoint, keeping the
// per-step states, lists, porosities and pressure sums the adjoint reads.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "bsc_internal.cuh"
#include "lanes.cuh"
#include "sph_kernel.cuh"

struct bsc_ctx : bsc::Ctx {};  // the same definition as in api.cu

namespace bsc {

struct WcK {
    double rho0, B, gam, inv_gam, grav_c, ys;  // EOS; rhoH(y) = rho0 (1 + grav_c (ys - y))^(1/gamma)
    int igam;                                  // gamma where it is a whole number of 1..EOS_MAX, else 0
    double binom[8];                           // then binom(gamma, k + 1): (1 + t)^gamma - 1 = t (binom[0] + t (...))
    double c2;                                 // delta 2h c0
    double nu, lam, g, dt, d50, H2;
    double alpha, beta;
    double inv_h, wend_F, wend_W;
    double gx0, gy0, gdx, gdy, por_default;
    bool plain_drag;                           // the drag's parameters are moderate: it vanishes at n = 1
    int gnx, gny, kmax, np, gc;  // gc: grid cells one support can overlap
    double R1, depth;                          // probe kernel radius, probe depth
};

struct WcState {
    WcK K{};
    int64_t n = 0, ns = 0;
    int G = 0;                                 // grid cells
    double t0 = 0.0;
    double* init = nullptr;                    // initial state: x y vx vy rho (5n)
    double* mass = nullptr;                    // particle masses rho_init dl^2
    double *theta = nullptr, *sw = nullptr;    // grid porosities; (1 - phi_s) V_s
    int32_t* sg = nullptr;                     // solid -> grid cell or -1
    double *rt = nullptr, *ex = nullptr, *drh = nullptr;  // per step
    double *vol = nullptr, *pr = nullptr;      // m/rt, p/rt^2 (per step)
    double* dpdr = nullptr;                    // dp/drt (per step)
    double* nxt = nullptr;                     // next state (5n)
    double *xp = nullptr, *eta = nullptr, *part = nullptr;  // probes, eta history, partials
    // forward record
    int nsteps = 0, every = 0;
    bool last_kept = false;                    // the forward run kept its last segment
    std::vector<double> tck;
    double* ck = nullptr;                      // checkpoints (5n each)
    int ck_cap = 0, seg_cap = 0, eta_cap = 0;
    double *seg = nullptr, *segn = nullptr, *segP = nullptr;  // (K+1) states; n; P (2n)
    int32_t *segnbr = nullptr, *segcnt = nullptr, *segpc = nullptr;  // lists, counts, cells
    // what the reverse sweep reads from the recomputation, per step: the
    // per-particle quotients, per-pair kernel values (F, F'/r, G, G'/r), the
    // porosity gradient and the per-grid-cell kernel sums of the porosity
    double *segpre = nullptr, *seggeo = nullptr, *segdn = nullptr, *segpgv = nullptr;
    int32_t* segpgi = nullptr;
    // adjoint
    double *lam = nullptr, *lamn = nullptr;    // 5n each
    double *lD = nullptr, *ln = nullptr, *lvl = nullptr, *lrl = nullptr;
    double2* adj2 = nullptr;                   // 3n: AdjPair
    double *dJ = nullptr, *grad = nullptr;
    std::vector<void*> allocs;
};

namespace {

constexpr int WB = 128;
// The FP64-bound pair kernels take blocks of one warp: a block of four runs as
// long as its slowest SM, and 794 of them over 152 SMs leave some with six
// where 5.2 is the mean (forward step on 101573 particles 4 % faster).
constexpr int WPB = 32;
constexpr int EOS_MAX = 8;  // largest whole gamma evaluated as a polynomial
constexpr int GCMAX = 9;  // grid cells one particle's kernel support can overlap (checked at setup)

template <typename T>
int wc_alloc(Ctx* c, WcState* w, T** p, int64_t count) {
    void* q = nullptr;
    cudaError_t e = cudaMalloc(&q, (size_t)std::max<int64_t>(count, 1) * sizeof(T));
    if (e != cudaSuccess) return cuda_err(c, e, "cudaMalloc (wcsph)");
    w->allocs.push_back(q);
    *p = (T*)q;
    return BSC_OK;
}

// Wendland C2: grad W = F(r) d, F' = dF/dr
__device__ __forceinline__ double wF(const WcK& K, double r) {
    const double a = 1.0 - 0.5 * r * K.inv_h;
    return -K.wend_F * a * a * a;
}
__device__ __forceinline__ double wdF(const WcK& K, double r) {
    const double a = 1.0 - 0.5 * r * K.inv_h;
    return 1.5 * K.wend_F * a * a * K.inv_h;
}
// (each operation rounded as written: the porosity pass has the same bits with
// and without the adjoint's record)
__device__ __forceinline__ double wW(const WcK& K, double r) {
    const double q = __dmul_rn(r, K.inv_h), a = fma(-0.5, q, 1.0), a2 = __dmul_rn(a, a);
    return __dmul_rn(__dmul_rn(__dmul_rn(K.wend_W, fma(2.0, q, 1.0)), a2), a2);
}
// the 1-D Wendland C2 kernel of the probes (radius R1, unit integral)
__device__ __forceinline__ double w1(double q, double R1) {
    const double a = 1.0 - q;
    return (1.25 / R1) * (a * a * a) * (1.0 + 3.0 * q);
}
__device__ __forceinline__ double w1q(double q, double R1) {  // d w1 / dq
    const double a = 1.0 - q;
    return -(15.0 / R1) * q * a * a;
}

__device__ __forceinline__ bool is_fluid(const State& S, int64_t i) { return S.tid[i] == BSC_TID_FLUID; }

// fields of a 5n state block
struct St {
    double *x, *y, *vx, *vy, *rho;
};
__host__ __device__ inline St st_of(double* b, int64_t n) { return {b, b + n, b + 2 * n, b + 3 * n, b + 4 * n}; }

__global__ void k_wc_init(int64_t n, State S, WcK K, double vol0, double* __restrict__ mass) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double s = 1.0 + K.grav_c * (K.ys - S.y[i]);
    // hydrostatic density below the level, rho0 above it
    const double r = S.y[i] < K.ys ? K.rho0 * pow(s, K.inv_gam) : K.rho0;
    S.rho[i] = r;
    mass[i] = r * vol0;
}

__global__ void k_wc_solids(int64_t ns, const double* __restrict__ sx, const double* __restrict__ sy,
                            const double* __restrict__ svol, const double* __restrict__ theta, WcK K,
                            double* __restrict__ sw, int32_t* __restrict__ sg) {
    const int64_t s = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (s >= ns) return;
    const double fx = floor((sx[s] - K.gx0) / K.gdx), fy = floor((sy[s] - K.gy0) / K.gdy);
    int g = -1;
    if (fx >= 0.0 && fx < (double)K.gnx && fy >= 0.0 && fy < (double)K.gny) g = (int)fy * K.gnx + (int)fx;
    const double phi = g >= 0 ? theta[g] : K.por_default;
    sw[s] = (1.0 - phi) * svol[s];
    sg[s] = g;
}

// clamped density, the density's excess over the hydrostatic one and
// that one's slope, and the per-particle quotients the pair loops read (volume
// m/rt, p/rt^2)
struct Pre {
    double *rt, *ex, *drh, *vol, *pr, *dpdr;  // dpdr: dp/drt of the EOS
};

// s^(1/m) for a whole m and s > 0 in FP32's range: an FP32 seed, then two
// Newton steps for y^m = s, y -= (y^m - s) / (m y^(m-1)).  The seed's error
// (~1e-6) squares twice below FP64's rounding, so the divisor, which only
// scales a correction of ~1e-6, may be an FP32 reciprocal.
__device__ __forceinline__ double root_of(double s, int m) {
    const float seed = exp2f(__log2f((float)s) / (float)m);
    double y = (double)seed;
    const double scale = (double)(seed / ((float)m * (float)s));  // 1 / (m y^(m-1))
#pragma unroll
    for (int step = 0; step < 2; ++step) {
        double q = y;
        for (int k = 1; k < m; ++k) q *= y;
        y -= (q - s) * scale;
    }
    return y;
}

// Bound: the FP64 pipe.  For a whole gamma (Tait's 7) the EOS is the binomial
// polynomial in t = (rt - rho0)/rho0, exact where pow(rt/rho0, gamma) - 1
// cancels, and the hydrostatic density a Newton root; two pow() took 49 us on
// 101573 particles, these 18 us (cold caches).
__global__ void k_wc_pre(int64_t n, const int8_t* __restrict__ tid, const double* __restrict__ mass,
                         const double* __restrict__ y, const double* __restrict__ rho, WcK K, Pre o) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double r = tid[i] == BSC_TID_FLUID ? fmax(rho[i], K.rho0) : rho[i];
    double qm;  // (rt/rho0)^gamma - 1
    if (K.igam) {
        const double t = (r - K.rho0) / K.rho0;
        qm = K.binom[K.igam - 1];
        for (int k = K.igam - 2; k >= 0; --k) qm = fma(qm, t, K.binom[k]);
        qm *= t;
    } else {
        qm = pow(r / K.rho0, K.gam) - 1.0;
    }
    double p = K.B * qm;
    if (p < 0.0) p = 0.0;
    const double ir = 1.0 / r;
    o.dpdr[i] = K.B * K.gam * (qm + 1.0) * ir;  // B gamma (rt/rho0)^(gamma-1) / rho0
    o.rt[i] = r;
    o.vol[i] = mass[i] * ir;
    o.pr[i] = p * ir * ir;
    const double s = 1.0 + K.grav_c * (K.ys - y[i]);
    const double q = K.igam && s > 1e-3 ? root_of(s, K.igam) : pow(s, K.inv_gam);
    o.ex[i] = r - K.rho0 * q;
    o.drh[i] = -K.rho0 * K.grav_c * K.inv_gam * q / s;
}

// the five state fields, one launch
__global__ void k_wc_copy(int64_t n, St src, St dst) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= n) return;
    dst.x[i] = src.x[i];
    dst.y[i] = src.y[i];
    dst.vx[i] = src.vx[i];
    dst.vy[i] = src.vy[i];
    dst.rho[i] = src.rho[i];
}

// what the porosity pass keeps for the adjoint
struct PorKeep {
    double* dn;    // grad n_i (2n)
    int32_t* pgi;  // grid cell u of particle i at [u * n + i], -1 past the last
    double* pgv;   // sum over that cell's solids of V_s W(r_is)
};

// Porosity n_i from the solids in the 3x3 cells (fluid; 1 elsewhere).  Bound:
// the FP64 pipe, which an instruction holds for the whole warp however few
// lanes run it.  Testing every candidate in FP64 inside the divergent cell
// loop ran ~60 candidates' offsets a particle and their kernels at half the
// lanes; the FP32 pre-test (sph_kernel.cuh) now compacts the survivors, in
// cell order, into this thread's column of shared memory, and the FP64 terms
// run over those, a column at a time.  A particle far from its binned cell
// takes one pass over all of them, by one lane.
// The particles with solids are few and sit together, so several lanes share
// one at any size.  101573 particles: 236 us with a thread each, 64 us, with the adjoint's
// record 83 us.  (With more survivors than the column holds left to one lane
// of the four, a forward step at 96593 particles took 3590 us where the solids
// are nine times as many, 2110 with a thread per particle, 1010 so; the scan's
// loops are kept rolled for the registers, 80 of them instead of 58.)
constexpr int WP_CAP = 32;
template <bool KEEP, int L>
__global__ void __launch_bounds__(WPB, 8) k_wc_por(int64_t n, State S, KParams KP, WcK K, const int32_t* __restrict__ pcell,
                                               const float2* __restrict__ posf, const int32_t* __restrict__ scs,
                                               const int32_t* __restrict__ scc, const float2* __restrict__ sposf,
                                               const double* __restrict__ sx, const double* __restrict__ sy,
                                               const double* __restrict__ sw, const double* __restrict__ svol,
                                               const int32_t* __restrict__ sg, double* __restrict__ nout, PorKeep kp) {
    constexpr int NP = WPB / L;  // particles of the block
    __shared__ int32_t cand[WP_CAP * NP];
    __shared__ double wval[KEEP && L > 1 ? WP_CAP * NP : 1];  // V W of the survivors, for the per-cell sums
    const Lanes<L> ln;
    const int64_t i = ln.particle();
    if (i >= n) return;
    const int p = threadIdx.x / L;
    // the grid cells met so far and their sums (in shared memory: indexed)
    __shared__ int cg[KEEP ? GCMAX * NP : 1];
    __shared__ double cv[KEEP ? GCMAX * NP : 1];
    int ncell = 0;
    double frac = 0.0, gx = 0.0, gy = 0.0;
    if (is_fluid(S, i)) {
        const double xi = S.x[i], yi = S.y[i];
        const int c = pcell[i], cx = c / KP.ny, cy = c - cx * KP.ny;
        const float H2f = (float)(KP.H2 * (1.0 + PRE_MARGIN)), csf = (float)KP.cs;
        const float2 pi = posf[i];
        const bool pre_i = pre_ok(pi, csf);
        // one solid's part of the per-cell sums
        auto cell = [&](int g, double v) {
            if (g < 0) return;
            int u = 0;
            while (u < ncell && cg[u * NP + p] != g) ++u;
            if (u >= K.gc) return;
            cv[u * NP + p] = u < ncell ? cv[u * NP + p] + v : v;
            if (u == ncell) {
                cg[u * NP + p] = g;
                ++ncell;
            }
        };
        auto cell_of = [&](int s, double W) { return W != 0.0 ? sg[s] : -1; };
        // one solid's part of the sums, W its kernel value and F its gradient factor
        auto add = [&](int s, double W, double F, double dx, double dy) {
            frac = fma(sw[s], W, frac);
            if (KEEP) {
                gx -= sw[s] * F * dx;  // grad n = -sum sw grad W
                gy -= sw[s] * F * dy;
            }
        };
        // U solids at once: independent terms in flight
        auto terms = [&](auto U_, const int* q) {
            constexpr int U = decltype(U_)::value;
            double W[U], F[U], dx[U], dy[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                dx[u] = xi - sx[q[u]];
                dy[u] = yi - sy[q[u]];
                const double d2 = fma(dx[u], dx[u], __dmul_rn(dy[u], dy[u])), r = sqrt(d2);
                const bool in = d2 < K.H2;
                W[u] = in ? wW(K, r) : 0.0;
                F[u] = KEEP && in ? wF(K, r) : 0.0;
            }
#pragma unroll
            for (int u = 0; u < U; ++u) {
                add(q[u], W[u], F[u], dx[u], dy[u]);
                if (KEEP && L == 1) cell(cell_of(q[u], W[u]), svol[q[u]] * W[u]);
            }
            return W[0];
        };
        using One = std::integral_constant<int, 1>;
        // windows of WP_CAP survivors, the scan repeated for each; without the
        // pre-test one scan sums over the cells directly, by one lane
        int nc = 0;
#pragma unroll 1
        for (int w0 = 0; w0 == 0 || w0 < nc; w0 += WP_CAP) {
            nc = 0;
#pragma unroll 1
            for (int ax = cx - 1; ax <= cx + 1; ++ax) {
                if (ax < 0 || ax >= KP.nx) continue;
                const float shx = (float)(ax - cx) * csf;
#pragma unroll 1
                for (int ay = cy - 1; ay <= cy + 1; ++ay) {
                    if (ay < 0 || ay >= KP.ny) continue;
                    const float shy = (float)(ay - cy) * csf;
                    const int cc = ax * KP.ny + ay;
                    const int s0 = scs[cc], s1 = s0 + scc[cc];
                    if (!pre_i) {
#pragma unroll 1
                        for (int s = s0; s < s1 && ln.sub == 0; ++s) {
                            const double W = terms(One{}, &s);
                            if (KEEP && L > 1) cell(cell_of(s, W), svol[s] * W);
                        }
                        continue;
                    }
                    for (int s = s0; s < s1; s += L) {
                        const int q = s + ln.sub;
                        bool keep = q < s1;
                        if (keep) {
                            const float2 ps = sposf[q];
                            if (pre_ok(ps, csf)) {
                                const float fdx = pi.x - (ps.x + shx), fdy = pi.y - (ps.y + shy);
                                keep = !(fdx * fdx + fdy * fdy > H2f);
                            }
                        }
                        const int at = ln.place(keep, nc) - w0;
                        if (keep && (unsigned)at < (unsigned)WP_CAP) cand[at * NP + p] = q;
                    }
                }
            }
            ln.sync();
            const int m = min(nc - w0, WP_CAP);
            if (L == 1) {
                constexpr int U = KEEP ? 2 : 4;
                int k = 0;
                for (; k + U <= m; k += U) {
                    int q[U];
#pragma unroll
                    for (int u = 0; u < U; ++u) q[u] = cand[(k + u) * NP + p];
                    terms(std::integral_constant<int, U>{}, q);
                }
                for (; k < m; ++k) terms(One{}, &cand[k * NP + p]);
            } else {
                for (int k = ln.sub; k < m; k += L) {
                    const double W = terms(One{}, &cand[k * NP + p]);
                    if (KEEP) {
                        const int s = cand[k * NP + p];
                        wval[k * NP + p] = svol[s] * W;
                        cand[k * NP + p] = cell_of(s, W);  // read by this lane only
                    }
                }
                ln.sync();
                if (KEEP && ln.sub == 0)
                    for (int k = 0; k < m; ++k) cell(cand[k * NP + p], wval[k * NP + p]);
                ln.sync();
            }
        }
    }
    frac = ln.sum(frac);
    if (KEEP) {
        gx = ln.sum(gx);
        gy = ln.sum(gy);
    }
    if (ln.sub != 0) return;
    nout[i] = is_fluid(S, i) ? 1.0 - frac : 1.0;
    if (KEEP) {
        kp.dn[i] = gx;
        kp.dn[n + i] = gy;
        for (int u = 0; u < K.gc; ++u) {
            kp.pgi[u * n + i] = u < ncell ? cg[u * NP + p] : -1;
            kp.pgv[u * n + i] = u < ncell ? cv[u * NP + p] : 0.0;
        }
    }
}

// one step: next state; the porosity (in nbuf) and the pressure sum P
// (2 per particle, for the adjoint) are kept
template <int L>
__global__ void __launch_bounds__(WPB) k_wc_step(int64_t n, State S, WcK K, const int32_t* __restrict__ nbr,
                                                const int32_t* __restrict__ cnt, Pre pq,
                                                const double* __restrict__ nbuf, St out, double* __restrict__ Pbuf,
                                                double* __restrict__ geo, int64_t slots) {
    const double* __restrict__ rt = pq.rt;
    const double* __restrict__ ex = pq.ex;
    const double* __restrict__ vol = pq.vol;
    const double* __restrict__ pr = pq.pr;
    const Lanes<L> ln;
    const int64_t i = ln.particle();
    if (i >= n) return;
    const double xi = S.x[i], yi = S.y[i], vxi = S.vx[i], vyi = S.vy[i];
    if (!is_fluid(S, i)) {
        if (ln.sub != 0) return;
        out.x[i] = xi;
        out.y[i] = yi;
        out.vx[i] = vxi;
        out.vy[i] = vyi;
        out.rho[i] = S.rho[i];
        Pbuf[i] = Pbuf[n + i] = 0.0;
        return;
    }
    const double rti = rt[i], exi = ex[i], ni = nbuf[i];
    const double pri = pr[i];
    // factors common to a sum (rt_i, c2, 2 nu) are applied after the loop
    double Da = 0.0, Dd = 0.0, Px = 0.0, Py = 0.0, vx = 0.0, vy = 0.0;
    const int m = cnt[i];
    for (int k = ln.sub; k < m; k += L) {
        const int64_t e = ell(i, k, K.kmax);
        const int j = nbr[e];
        const double dx = xi - S.x[j], dy = yi - S.y[j];
        const double r2 = dx * dx + dy * dy, r = sqrt(r2);
        const double iden = rcp_nr(r2 + K.lam);
        const double F = wF(K, r), G = F * r2 * iden;
        if (geo) {  // F, F'/r, G, G'/r for the reverse sweep
            const double ir = rcp_nr(r), dF = wdF(K, r);
            geo[e] = F;
            geo[slots + e] = dF * ir;
            geo[2 * slots + e] = G;
            geo[3 * slots + e] = (dF * r2 + F * 2.0 * r * K.lam * iden) * iden * ir;
        }
        const double Vj = vol[j], VG = Vj * G;
        const double dvx = vxi - S.vx[j], dvy = vyi - S.vy[j];
        Da += Vj * F * (dvx * dx + dvy * dy);  // m_j (rt_i / rt_j) F (v_ij . x_ij) / rt_i
        Dd += (exi - ex[j]) * VG;
        const double pc = S.mass[j] * (pri + pr[j]) * F;
        Px += pc * dx;
        Py += pc * dy;
        vx += VG * dvx;
        vy += VG * dvy;
    }
    Da = ln.sum(Da);
    Dd = ln.sum(Dd);
    Px = ln.sum(Px);
    Py = ln.sum(Py);
    vx = ln.sum(vx);
    vy = ln.sum(vy);
    if (ln.sub != 0) return;
    const double Dr = rti * Da + K.c2 * Dd;
    vx *= 2.0 * K.nu;
    vy *= 2.0 * K.nu;
    const double ax = -ni * Px + vx, ay = -ni * Py + vy + ni * K.g;
    // outside the porous layer (whole warps of it) the drag's quotients and
    // roots, a tenth of this kernel's FP64 work, leave the values as they are
    const bool clear = ni == 1.0 && K.plain_drag && moderate(vxi) && moderate(vyi);
    double vxn = vxi + K.dt * ax, vyn = vyi + K.dt * ay, sxn, syn;
    if (clear) {  // n = 1: no drag, and quotients by 1
        sxn = K.dt * vxn;
        syn = K.dt * vyn;
    } else {
        const double vm = sqrt(vxi * vxi + vyi * vyi), on = 1.0 - ni, n3 = ni * ni * ni;
        const double R = -K.nu * K.alpha * on * on / (n3 * K.d50 * K.d50) - K.beta * vm * on / (n3 * K.d50);
        const double D = 1.0 - K.dt * R * ni;
        vxn /= D;
        vyn /= D;
        sxn = K.dt * vxn / ni;
        syn = K.dt * vyn / ni;
    }
    out.vx[i] = vxn;
    out.vy[i] = vyn;
    out.x[i] = xi + sxn;
    out.y[i] = yi + syn;
    out.rho[i] = rti + K.dt * Dr;
    Pbuf[i] = Px;
    Pbuf[n + i] = Py;
}

// Probe elevations of a state: per-block partials of sum_i V_i w1(x_i - x_p),
// one thread per particle.  Almost every block is out of every probe's reach:
// an FP32 test of the distance (widened past its rounding) keeps the divisions
// and the block sums to the blocks that have a particle in reach, the others
// write their exact zero.  101573 particles, four probes: 27 us before, 8 us.
__global__ void __launch_bounds__(WB) k_wc_eta(int64_t n, const int8_t* __restrict__ tid, const double* __restrict__ mass,
                                               St s, WcK K, const double* __restrict__ xp, double* __restrict__ part) {
    __shared__ double sh[WB];
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    const bool fluid = i < n && tid[i] == BSC_TID_FLUID;
    const double xi = fluid ? s.x[i] : 0.0;
    const float xf = (float)xi, reach = (float)K.R1 * 1.001f;
    for (int p = 0; p < K.np; ++p) {
        const double xpp = xp[p];
        const float xpf = (float)xpp;
        const bool near = fluid && !(fabsf(xf - xpf) > reach + 4e-7f * (fabsf(xf) + fabsf(xpf)));
        if (!__syncthreads_or(near)) {
            if (threadIdx.x == 0) part[blockIdx.x * K.np + p] = 0.0;
            continue;
        }
        double a = 0.0;
        if (near) {
            const double V = mass[i] / s.rho[i], q = fabs(xi - xpp) / K.R1;
            if (q < 1.0) a = V * w1(q, K.R1);
        }
        sh[threadIdx.x] = a;
        __syncthreads();
        for (int o = WB / 2; o > 0; o >>= 1) {
            if (threadIdx.x < o) sh[threadIdx.x] += sh[threadIdx.x + o];
            __syncthreads();
        }
        if (threadIdx.x == 0) part[blockIdx.x * K.np + p] = sh[0];
        __syncthreads();
    }
}

// one block per probe, fixed summation order
__global__ void k_wc_eta_fin(int nb, WcK K, const double* __restrict__ part, double* __restrict__ eta) {
    __shared__ double sh[WB];
    const int p = blockIdx.x;
    double s = 0.0;
    for (int b = threadIdx.x; b < nb; b += WB) s += part[b * K.np + p];
    sh[threadIdx.x] = s;
    __syncthreads();
    for (int o = WB / 2; o > 0; o >>= 1) {
        if (threadIdx.x < o) sh[threadIdx.x] += sh[threadIdx.x + o];
        __syncthreads();
    }
    if (threadIdx.x == 0) eta[p] = sh[0] - K.depth;
}

// ---- adjoint ---------------------------------------------------------------------
// the loss's direct dependence on a state: lam += dJ/deta . d eta/d(x, rho)
__global__ void k_wc_adj_probe(int64_t n, const int8_t* __restrict__ tid, const double* __restrict__ mass, St s,
                               WcK K, const double* __restrict__ xp, const double* __restrict__ dJ, St lam) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= n || tid[i] != BSC_TID_FLUID) return;
    const double V = mass[i] / s.rho[i];
    double gx = 0.0, gr = 0.0;
    for (int p = 0; p < K.np; ++p) {
        const double d = s.x[i] - xp[p], q = fabs(d) / K.R1;
        if (q >= 1.0) continue;
        gx += dJ[p] * V * w1q(q, K.R1) * (d >= 0.0 ? 1.0 : -1.0) / K.R1;
        gr += dJ[p] * (-V / s.rho[i]) * w1(q, K.R1);
    }
    lam.x[i] += gx;
    lam.rho[i] += gr;
}

// block sum of two values into part[block][0..1]
__device__ __forceinline__ void block_sum2(double a, double b, double* __restrict__ part) {
    __shared__ double sa[WB], sb[WB];
    sa[threadIdx.x] = a;
    sb[threadIdx.x] = b;
    __syncthreads();
    for (int o = WB / 2; o > 0; o >>= 1) {
        if (threadIdx.x < o) {
            sa[threadIdx.x] += sa[threadIdx.x + o];
            sb[threadIdx.x] += sb[threadIdx.x + o];
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        part[0] = sa[0];
        part[1] = sb[0];
    }
}

// what the pair sums read of a particle's own adjoint: lam_a times 2 nu and
// times n, and (lam_Drho rt, c2 lam_Drho)
struct AdjPair {
    double2 *vla, *nla, *ab;
};

// the per-particle part of the reverse step: position update, drag, the
// porosity's direct roles; writes lam_a and lam_Drho as the pair sums read them,
// lam_n, and the particle's
// own contributions to lam_v and lam_rt; drag-coefficient partials per block
__global__ void __launch_bounds__(WB) k_wc_adj_local(int64_t n, const int8_t* __restrict__ tid, WcK K, St s0, St s1,
                                                     const double* __restrict__ nbuf, const double* __restrict__ Pbuf,
                                                     const double* __restrict__ rt, St lam, AdjPair ap,
                                                     double* __restrict__ lD, double* __restrict__ ln,
                                                     double* __restrict__ lvl, double* __restrict__ lrl,
                                                     double* __restrict__ part, int pstride) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    double ga = 0.0, gb = 0.0;
    if (i < n && tid[i] == BSC_TID_FLUID) {
        // the quotients by n, n^3, d and D as products with reciprocals taken once
        const double ni = nbuf[i], vx = s0.vx[i], vy = s0.vy[i], vxn = s1.vx[i], vyn = s1.vy[i];
        const double in = 1.0 / ni, in3 = in * in * in, in4 = in3 * in, id = 1.0 / K.d50;
        const double vm = sqrt(vx * vx + vy * vy), on = 1.0 - ni;
        const double cA = K.nu * on * on * in3 * id * id, cB = vm * on * in3 * id;  // dR/dalpha, dR/dbeta (negated)
        const double R = -K.alpha * cA - K.beta * cB;
        const double iD = 1.0 / (1.0 - K.dt * R * ni);
        const double lx = lam.x[i], ly = lam.y[i];
        const double lpx = lam.vx[i] + K.dt * lx * in, lpy = lam.vy[i] + K.dt * ly * in;
        double lni = -K.dt * (lx * vxn + ly * vyn) * in * in;
        const double lax = K.dt * lpx * iD, lay = K.dt * lpy * iD;
        const double lDD = -(lpx * vxn + lpy * vyn) * iD;
        const double lR = -K.dt * ni * lDD;
        lni += -K.dt * R * lDD;
        const double dRdn = -K.nu * K.alpha * id * id * (-2.0 * on * in3 - 3.0 * on * on * in4) -
                            K.beta * vm * id * (-in3 - 3.0 * on * in4);
        lni += lR * dRdn;
        double lvx = lpx * iD, lvy = lpy * iD;
        if (vm > 0.0) {
            const double cv = lR * (-K.beta * on * in3 * id) / vm;
            lvx += cv * vx;
            lvy += cv * vy;
        }
        ga = lR * (-cA);
        gb = lR * (-cB);
        // a = -n P + visc + n g: d a / d n = -P + g
        lni += lax * (-Pbuf[i]) + lay * (-Pbuf[n + i] + K.g);
        const double lDi = K.dt * lam.rho[i];
        ap.vla[i] = make_double2(2.0 * K.nu * lax, 2.0 * K.nu * lay);
        ap.nla[i] = make_double2(ni * lax, ni * lay);
        ap.ab[i] = make_double2(lDi * rt[i], K.c2 * lDi);
        lD[i] = lDi;
        ln[i] = lni;
        lvl[i] = lvx;
        lvl[n + i] = lvy;
        lrl[i] = lam.rho[i];
    } else if (i < n) {
        // a wall has no sums of its own: its products with them vanish
        ap.vla[i] = ap.nla[i] = ap.ab[i] = make_double2(0.0, 0.0);
        lD[i] = ln[i] = 0.0;
    }
    block_sum2(ga, gb, part + (int64_t)blockIdx.x * pstride);
}

// The pair part: for fluid particle k, the terms of its own sums (k as i) and
// of its neighbours' sums (k as j), with the per-pair kernel values and the
// porosity's gradient and per-grid-cell sums that the recomputation kept;
// writes the state adjoint lam_out for the state before the step and the
// block's porosity-grid partials.
// Bound: the FP64 pipe.  The two roles' terms differ by exchanging k and j and
// the sign of the offset, so each kind of term is one expression in a
// (anti)symmetric pair weight:
//   continuity     Q = lamD_k rt_k V_j + lamD_j rt_j V_k
//   diffusion      D = c2 (lamD_k V_j - lamD_j V_k),   del = ex_j - ex_k
//   pressure       M = m_j n_k lam_a,k - m_k n_j lam_a,j
//   viscosity      N = 2 nu (V_j lam_a,k - V_k lam_a,j)
//   d/dx_k:  Q F dv - (p_k/rt_k^2 + p_j/rt_j^2) F M
//            + [F'/r (Q dv.d - ps M.d) + G'/r (N.dv - del D)] d
// and the factors that belong to k alone are applied after the loop: 55 FP64
// operations a pair instead of about 130.  A wall's weights are zero.
// 14600 particles: 134 us before, 70 us.
template <int L>
__global__ void __launch_bounds__(WPB) k_wc_adj_pair(
    int64_t n, State S, WcK K, St s0, const int32_t* __restrict__ nbr, const int32_t* __restrict__ cnt, Pre pq,
    const double* __restrict__ geo, int64_t slots, AdjPair ap,
    const double* __restrict__ lD, const double* __restrict__ ln, const double* __restrict__ lvl,
    const double* __restrict__ lrl, St lam_in, St lam_out, const double* __restrict__ dn,
    const int32_t* __restrict__ pgi, const double* __restrict__ pgv, double* __restrict__ part, int pstride) {
    // grid-porosity partials of the block's warp
    __shared__ double wb[BSC_WCSPH_MAX_GRID];
    const int G = K.gnx * K.gny;
    for (int e = threadIdx.x; e < G; e += WPB) wb[e] = 0.0;
    __syncwarp();
    const Lanes<L> ls;
    const int64_t k = ls.particle();
    const bool act = k < n && S.tid[k] == BSC_TID_FLUID, first = ls.sub == 0;
    double lnk = 0.0;
    if (act) {
        const double xk = s0.x[k], yk = s0.y[k], vxk = s0.vx[k], vyk = s0.vy[k];
        const double exk = pq.ex[k], mk = S.mass[k], Vk = pq.vol[k], prk = pq.pr[k];
        const double irk = 1.0 / pq.rt[k], Vk_rt = Vk * irk;
        const double lDk = lD[k];
        const double2 vlak = ap.vla[k], nlak = ap.nla[k], abk = ap.ab[k];
        double lvx = 0.0, lvy = 0.0, lrt = 0.0, lxx = 0.0, lyy = 0.0;
        if (first) {
            lvx = lvl[k];
            lvy = lvl[n + k];
            lrt = lrl[k];
            lxx = lam_in.x[k];
            lyy = lam_in.y[k];
        }
        double SD = 0.0, S2 = 0.0, SP = 0.0, SV = 0.0;  // sum G D, G c2 lamD_j del, F M.d, G 2 nu lam_a,j.dv
        const int m = cnt[k];
        for (int q = ls.sub; q < m; q += L) {
            const int64_t e = ell(k, q, K.kmax);
            const int j = nbr[e];
            const double F = geo[e], Fr = geo[slots + e], G_ = geo[2 * slots + e], Gr = geo[3 * slots + e];
            const double Vj = pq.vol[j], mj = S.mass[j], ps = prk + pq.pr[j], del = pq.ex[j] - exk;
            const double2 vlaj = ap.vla[j], nlaj = ap.nla[j], abj = ap.ab[j];
            const double dx = xk - s0.x[j], dy = yk - s0.y[j];
            const double dvx = vxk - s0.vx[j], dvy = vyk - s0.vy[j], dvd = dvx * dx + dvy * dy;
            const double Q = abk.x * Vj + abj.x * Vk, QF = Q * F;
            const double D = abk.y * Vj - abj.y * Vk;
            const double Mx = mj * nlak.x - mk * nlaj.x, My = mj * nlak.y - mk * nlaj.y, Md = Mx * dx + My * dy;
            const double Nx = Vj * vlak.x - Vk * vlaj.x, Ny = Vj * vlak.y - Vk * vlaj.y;
            lvx += QF * dx + G_ * Nx;
            lvy += QF * dy + G_ * Ny;
            lrt += (F * dvd) * (lDk * Vj - abj.x * Vk_rt);
            SD += G_ * D;
            S2 += G_ * abj.y * del;
            SP += F * Md;
            SV += G_ * (vlaj.x * dvx + vlaj.y * dvy);
            const double C = Fr * (Q * dvd - ps * Md) + Gr * (Nx * dvx + Ny * dvy - del * D);
            const double psF = ps * F;
            lxx += QF * dvx - psF * Mx + C * dx;
            lyy += QF * dvy - psF * My + C * dy;
        }
        lvx = ls.sum(lvx);
        lvy = ls.sum(lvy);
        lrt = ls.sum(lrt);
        lxx = ls.sum(lxx);
        lyy = ls.sum(lyy);
        SD = ls.sum(SD);
        S2 = ls.sum(S2);
        SP = ls.sum(SP);
        SV = ls.sum(SV);
        if (first) {
            lrt += SD - Vk_rt * S2 + 2.0 * prk * irk * SP + mk * irk * irk * SV;
            lyy -= pq.drh[k] * SD;
            const double lp = -irk * irk * SP;
            // porosity n_k = 1 - sum_s (1 - phi_s) V_s W(r_ks)
            lnk = ln[k];
            lxx += lnk * dn[k];
            lyy += lnk * dn[n + k];
            // pressure and the clamp
            lrt += lp * pq.dpdr[k];
            lam_out.x[k] = lxx;
            lam_out.y[k] = lyy;
            lam_out.vx[k] = lvx;
            lam_out.vy[k] = lvy;
            lam_out.rho[k] = s0.rho[k] >= K.rho0 ? lrt : 0.0;
        }
    } else if (k < n && first) {
        lam_out.x[k] = lam_out.y[k] = lam_out.vx[k] = lam_out.vy[k] = lam_out.rho[k] = 0.0;
    }
    __syncwarp();
    // d n_k / d phi_g = sum over cell g's solids of V_s W(r_ks): lanes with the
    // same cell are summed in lane order by the lowest of them
    const int lane = threadIdx.x;
    for (int u = 0; u < K.gc; ++u) {
        int g = -1;
        double v = 0.0;
        if (act && first) {
            g = pgi[u * n + k];
            v = lnk * pgv[u * n + k];
        }
        if (__all_sync(0xffffffffu, g < 0)) continue;
        const unsigned grp = __match_any_sync(0xffffffffu, g);
        double acc = 0.0;
        for (int src = 0; src < 32; ++src) {
            const double t = __shfl_sync(0xffffffffu, v, src);
            if ((grp >> src) & 1u) acc += t;
        }
        if (g >= 0 && lane == __ffs(grp) - 1) wb[g] += acc;
        __syncwarp();
    }
    for (int g = lane; g < G; g += WPB) part[(int64_t)blockIdx.x * pstride + 2 + g] = wb[g];
}

// grad[q] += sum over blocks of part[block][q]: one block per q, fixed order;
// the drag coefficients (q < 2) have nbl blocks, the porosities nbp
__global__ void k_wc_grad(int nbl, int nbp, int pstride, const double* __restrict__ part, double* __restrict__ grad) {
    __shared__ double sh[WB];
    const int q = blockIdx.x, nb = q < 2 ? nbl : nbp;
    double s = 0.0;
    for (int b = threadIdx.x; b < nb; b += WB) s += part[(int64_t)b * pstride + q];
    sh[threadIdx.x] = s;
    __syncthreads();
    for (int o = WB / 2; o > 0; o >>= 1) {
        if (threadIdx.x < o) sh[threadIdx.x] += sh[threadIdx.x + o];
        __syncthreads();
    }
    if (threadIdx.x == 0) grad[q] += sh[0];
}

}  // namespace

void wc_free(Ctx* c) {
    WcState* w = c->wc;
    if (!w) return;
    if (c->stream) cudaStreamSynchronize(c->stream);
    for (void* p : w->allocs) cudaFree(p);
    delete w;
    c->wc = nullptr;
}

namespace {

int wc_params(Ctx* c, WcState* w, double alpha, double beta, const double* grid) {
    w->K.alpha = alpha;
    w->K.beta = beta;
    w->K.plain_drag = std::fabs(alpha) < 1e15 && std::fabs(beta) < 1e15 && std::fabs(w->K.nu) < 1e15 &&
                      std::fabs(w->K.d50) > 1e-15 && std::fabs(w->K.d50) < 1e15;
    if (grid) BSC_CUDA(c, cudaMemcpyAsync(w->theta, grid, sizeof(double) * w->G, cudaMemcpyHostToDevice, c->stream));
    if (w->ns > 0) {
        k_wc_solids<<<blocks_for(w->ns, 256), 256, 0, c->stream>>>(w->ns, c->sx, c->sy, c->svol, w->theta, w->K, w->sw,
                                                                 w->sg);
        BSC_LAUNCH(c);
    }
    BSC_CUDA(c, cudaStreamSynchronize(c->stream));
    return BSC_OK;
}

// one forward step on c->S; keeps n and P in nbuf, Pbuf
Pre wc_pre(WcState* w) { return {w->rt, w->ex, w->drh, w->vol, w->pr, w->dpdr}; }

// the context's state with the model's masses
State wc_view(Ctx* c, WcState* w) {
    State S = c->S;
    S.mass = w->mass;
    return S;
}

int launch_check(Ctx* c) {
    c->launches++;
    const cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? BSC_OK : cuda_err(c, e, "wcsph step");
}

St st_ctx(Ctx* c) { return {c->S.x, c->S.y, c->S.vx, c->S.vy, c->S.rho}; }

int wc_copy(Ctx* c, St src, St dst) {
    k_wc_copy<<<blocks_for(c->n, 256), 256, 0, c->stream>>>(c->n, src, dst);
    BSC_LAUNCH(c);
    return BSC_OK;
}
int wc_save(Ctx* c, double* dst) { return wc_copy(c, st_ctx(c), st_of(dst, c->n)); }
int wc_load(Ctx* c, const double* src) { return wc_copy(c, st_of(const_cast<double*>(src), c->n), st_ctx(c)); }

// what the recomputation of a segment keeps of one step for the reverse sweep
struct Keep {
    int32_t *nbr, *cnt, *cell;  // neighbour lists, counts, particle cells
    Pre pre;                    // per-particle quotients
    double* geo;                // per-pair kernel values (4 x slots)
    PorKeep por;                // porosity gradient and per-grid-cell sums
};

int64_t list_slots(const Ctx* c) { return ((c->n + 31) / 32) * 32 * (int64_t)c->K.kmax; }

Keep seg_keep(WcState* w, int q, int64_t n, int64_t slots) {
    double* pre = w->segpre + (int64_t)q * 6 * n;
    const int gc = w->K.gc;
    return {w->segnbr + (int64_t)q * slots,
            w->segcnt + (int64_t)q * n,
            w->segpc + (int64_t)q * n,
            {pre, pre + n, pre + 2 * n, pre + 3 * n, pre + 4 * n, pre + 5 * n},
            w->seggeo + (int64_t)q * 4 * slots,
            {w->segdn + (int64_t)q * 2 * n, w->segpgi + (int64_t)q * gc * n, w->segpgv + (int64_t)q * gc * n}};
}

// One step on c->S; keeps the porosity and the pressure sum in nbuf and Pbuf.
// With `keep`, the step's lists, counts and cells are built straight into the
// kept buffers (the context's own are pointed there for the step), and the
// per-particle quotients, per-pair kernel values and porosity derivatives
// are kept too.  The step reads the lists only; `last` (the last step that a
// call runs) takes the full search, and its lists and cells are copied to the
// context's own buffers: the lists, grad W, L and flags that a call leaves are
// those of its last step's search.
int wc_step(Ctx* c, WcState* w, double* nbuf, double* Pbuf, const Keep* keep, bool last) {
    const int64_t n = c->n;
    c->t += w->K.dt;
    int32_t *own_nbr = c->nbr, *own_cnt = c->cnt, *own_cell = c->pcell;
    if (keep) {
        c->nbr = keep->nbr;
        c->cnt = keep->cnt;
        c->pcell = keep->cell;
    }
    const Pre pre = keep ? keep->pre : wc_pre(w);
    int rc = op_piston(c);
    if (!rc) rc = cells_build(c, false);
    if (!rc) rc = last ? op_neighbour(c) : op_neighbour_lists(c);
    if (!rc) {
        const unsigned g = blocks_for(n, WB);
        const int lanes = lanes_for(n);
        const State S = wc_view(c, w);
        k_wc_pre<<<g, WB, 0, c->stream>>>(n, S.tid, S.mass, S.y, S.rho, w->K, pre);
        rc = launch_check(c);
        if (!rc) {
            with_lanes(std::max(lanes, 4), [&](auto L) {
                constexpr int l = decltype(L)::value;
                const unsigned gp = blocks_for(n * l, WPB);
                if (keep)
                    k_wc_por<true, l><<<gp, WPB, 0, c->stream>>>(n, S, c->K, w->K, c->pcell, c->posf, c->scell_start,
                                                                 c->scell_count, c->sposf, c->sx, c->sy, w->sw,
                                                                 c->svol, w->sg, nbuf, keep->por);
                else
                    k_wc_por<false, l><<<gp, WPB, 0, c->stream>>>(n, S, c->K, w->K, c->pcell, c->posf,
                                                                  c->scell_start, c->scell_count, c->sposf, c->sx,
                                                                  c->sy, w->sw, c->svol, w->sg, nbuf, PorKeep{});
            });
            rc = launch_check(c);
        }
        if (!rc) {
            with_lanes(lanes, [&](auto L) {
                constexpr int l = decltype(L)::value;
                k_wc_step<l><<<blocks_for(n * l, WPB), WPB, 0, c->stream>>>(
                    n, S, w->K, c->nbr, c->cnt, pre, nbuf, st_of(w->nxt, n), Pbuf, keep ? keep->geo : nullptr,
                    list_slots(c));
            });
            rc = launch_check(c);
        }
    }
    c->nbr = own_nbr;
    c->cnt = own_cnt;
    c->pcell = own_cell;
    c->have_csr = false;  // the lists that an earlier PPE matrix was laid out on are gone
    if (rc) {
        c->have_lists = false;
        return rc;
    }
    if (keep && last) {  // into the context's own buffers: have_lists speaks for those
        BSC_CUDA(c, cudaMemcpyAsync(own_nbr, keep->nbr, sizeof(int32_t) * list_slots(c), cudaMemcpyDeviceToDevice,
                                    c->stream));
        BSC_CUDA(c, cudaMemcpyAsync(own_cnt, keep->cnt, sizeof(int32_t) * n, cudaMemcpyDeviceToDevice, c->stream));
        BSC_CUDA(c, cudaMemcpyAsync(own_cell, keep->cell, sizeof(int32_t) * n, cudaMemcpyDeviceToDevice, c->stream));
    }
    // the next state becomes the state
    return wc_copy(c, st_of(w->nxt, n), st_ctx(c));
}

}  // namespace
}  // namespace bsc

using namespace bsc;

extern "C" {

int bsc_wcsph_setup(bsc_ctx* c, const bsc_wcsph_params* p) {
    if (!c || !p) return BSC_E_INVALID;
    if (!c->have_state) return set_err(c, BSC_E_INVALID, "wcsph_setup before upload_state");
    if (c->mixed || c->K.kernel != BSC_KERNEL_WENDLAND_C2)
        return set_err(c, BSC_E_INVALID, "wcsph: an FP64 context with the Wendland C2 kernel");
    const int G = p->grid_nx * p->grid_ny;
    if (p->grid_nx < 1 || p->grid_ny < 1 || G > BSC_WCSPH_MAX_GRID || !p->grid_por || !(p->grid_dx > 0) ||
        !(p->grid_dy > 0) || p->nprobe < 1 || p->nprobe > BSC_WCSPH_MAX_PROBES || !(p->c0 > 0) || !(p->gamma > 0))
        return set_err(c, BSC_E_INVALID, "wcsph_setup: bad parameters");
    wc_free(c);
    WcState* w = new (std::nothrow) WcState();
    if (!w) return BSC_E_NOMEM;
    c->wc = w;
    const int64_t n = c->n;
    w->n = n;
    w->ns = c->ns;
    w->G = G;
    WcK& K = w->K;
    const KParams& KP = c->K;
    K.rho0 = KP.rho0;
    K.gam = p->gamma;
    K.inv_gam = 1.0 / p->gamma;
    K.igam = p->gamma == std::floor(p->gamma) && p->gamma <= EOS_MAX ? (int)p->gamma : 0;
    double bin = 1.0;
    for (int k = 0; k < K.igam; ++k) K.binom[k] = bin = bin * (K.igam - k) / (k + 1);
    K.B = KP.rho0 * p->c0 * p->c0 / p->gamma;
    K.grav_c = std::fabs(KP.g) * p->gamma / (p->c0 * p->c0);
    K.ys = p->surface_y;
    K.c2 = p->delta * 2.0 * KP.h * p->c0;
    K.nu = p->nu;
    K.lam = KP.lam;
    K.g = KP.g;
    K.dt = c->dt;
    K.d50 = KP.d50;
    K.H2 = KP.H2;
    K.inv_h = KP.inv_h;
    K.wend_F = KP.wend_F;
    K.wend_W = KP.wend_W;
    K.gx0 = p->grid_x0;
    K.gy0 = p->grid_y0;
    K.gdx = p->grid_dx;
    K.gdy = p->grid_dy;
    K.gnx = p->grid_nx;
    K.gny = p->grid_ny;
    K.por_default = KP.por;
    K.kmax = KP.kmax;
    K.np = p->nprobe;
    K.R1 = 2.0 * KP.h;
    K.depth = p->probe_depth;
    // grid cells a kernel support (diameter 4h) can overlap
    const int ncx = std::min(p->grid_nx, (int)std::floor(4.0 * KP.h / p->grid_dx) + 2);
    const int ncy = std::min(p->grid_ny, (int)std::floor(4.0 * KP.h / p->grid_dy) + 2);
    K.gc = ncx * ncy;
    if (K.gc > GCMAX) return set_err(c, BSC_E_INVALID, "wcsph_setup: porosity grid cells smaller than 2h");
    int rc;
    if ((rc = wc_alloc(c, w, &w->init, 5 * n)) || (rc = wc_alloc(c, w, &w->mass, n)) ||
        (rc = wc_alloc(c, w, &w->theta, G)) ||
        (rc = wc_alloc(c, w, &w->sw, w->ns)) || (rc = wc_alloc(c, w, &w->sg, w->ns)) ||
        (rc = wc_alloc(c, w, &w->rt, n)) || (rc = wc_alloc(c, w, &w->ex, n)) ||
        (rc = wc_alloc(c, w, &w->drh, n)) || (rc = wc_alloc(c, w, &w->vol, n)) || (rc = wc_alloc(c, w, &w->pr, n)) ||
        (rc = wc_alloc(c, w, &w->dpdr, n)) ||
        (rc = wc_alloc(c, w, &w->nxt, 5 * n)) ||
        (rc = wc_alloc(c, w, &w->xp, BSC_WCSPH_MAX_PROBES)) ||
        (rc = wc_alloc(c, w, &w->part, (int64_t)std::max(blocks_for(n * lanes_for(n), WPB), blocks_for(n, WB)) * (2 + BSC_WCSPH_MAX_GRID))) ||
        (rc = wc_alloc(c, w, &w->lam, 5 * n)) || (rc = wc_alloc(c, w, &w->lamn, 5 * n)) ||
        (rc = wc_alloc(c, w, &w->adj2, 3 * n)) || (rc = wc_alloc(c, w, &w->lD, n)) || (rc = wc_alloc(c, w, &w->ln, n)) ||
        (rc = wc_alloc(c, w, &w->lvl, 2 * n)) || (rc = wc_alloc(c, w, &w->lrl, n)) ||
        (rc = wc_alloc(c, w, &w->grad, 2 + BSC_WCSPH_MAX_GRID)))
        return rc;
    BSC_CUDA(c, cudaMemcpyAsync(w->xp, p->probe_x, sizeof(double) * p->nprobe, cudaMemcpyHostToDevice, c->stream));
    // hydrostatic densities, then the initial state
    k_wc_init<<<blocks_for(n, 256), 256, 0, c->stream>>>(n, c->S, K, KP.dl * KP.dl, w->mass);
    BSC_LAUNCH(c);
    if ((rc = wc_save(c, w->init))) return rc;
    w->t0 = c->t;
    return wc_params(c, w, p->alpha, p->beta, p->grid_por);
}

int bsc_wcsph_set_params(bsc_ctx* c, double alpha, double beta, const double* grid_por) {
    if (!c || !c->wc) return c ? set_err(c, BSC_E_INVALID, "wcsph_set_params before wcsph_setup") : BSC_E_INVALID;
    return wc_params(c, c->wc, alpha, beta, grid_por);
}

int bsc_wcsph_forward(bsc_ctx* c, int32_t nsteps, int32_t every, double* eta) {
    if (!c || !c->wc) return c ? set_err(c, BSC_E_INVALID, "wcsph_forward before wcsph_setup") : BSC_E_INVALID;
    if (nsteps < 1 || every < 1 || !eta) return set_err(c, BSC_E_INVALID, "wcsph_forward: bad arguments");
    WcState* w = c->wc;
    const int64_t n = c->n;
    int rc;
    const int nck = (nsteps + every - 1) / every;
    if (nck > w->ck_cap) {
        if ((rc = wc_alloc(c, w, &w->ck, (int64_t)nck * 5 * n))) return rc;
        w->ck_cap = nck;
    }
    if (nsteps > w->eta_cap) {
        if ((rc = wc_alloc(c, w, &w->eta, (int64_t)nsteps * w->K.np)) ||
            (rc = wc_alloc(c, w, &w->dJ, (int64_t)nsteps * w->K.np)))
            return rc;
        w->eta_cap = nsteps;
    }
    if (every > w->seg_cap) {
        const int64_t slots = list_slots(c), gc = w->K.gc;
        if ((rc = wc_alloc(c, w, &w->seg, (int64_t)(every + 1) * 5 * n)) ||
            (rc = wc_alloc(c, w, &w->segn, (int64_t)every * n)) || (rc = wc_alloc(c, w, &w->segP, (int64_t)every * 2 * n)) ||
            (rc = wc_alloc(c, w, &w->segnbr, (int64_t)every * slots)) ||
            (rc = wc_alloc(c, w, &w->segcnt, (int64_t)every * n)) ||
            (rc = wc_alloc(c, w, &w->segpc, (int64_t)every * n)) ||
            (rc = wc_alloc(c, w, &w->segpre, (int64_t)every * 6 * n)) ||
            (rc = wc_alloc(c, w, &w->seggeo, (int64_t)every * 4 * slots)) ||
            (rc = wc_alloc(c, w, &w->segdn, (int64_t)every * 2 * n)) ||
            (rc = wc_alloc(c, w, &w->segpgi, (int64_t)every * gc * n)) ||
            (rc = wc_alloc(c, w, &w->segpgv, (int64_t)every * gc * n)))
            return rc;
        w->seg_cap = every;
    }
    w->nsteps = nsteps;
    w->every = every;
    w->tck.assign(nck, 0.0);
    // the last segment keeps what the reverse sweep reads as it runs, so the
    // adjoint recomputes one segment fewer
    const int last0 = (nck - 1) * every;
    const int64_t slots = list_slots(c);
    w->last_kept = false;
    if ((rc = wc_load(c, w->init))) return rc;
    c->t = w->t0;
    const unsigned nb = blocks_for(n, WB);
    for (int s = 0; s < nsteps; ++s) {
        if (s % every == 0) {
            if ((rc = wc_save(c, w->ck + (int64_t)(s / every) * 5 * n))) return rc;
            w->tck[s / every] = c->t;
        }
        if (s >= last0) {
            const int q = s - last0;
            const Keep kq = seg_keep(w, q, n, slots);
            if ((rc = wc_save(c, w->seg + (int64_t)q * 5 * n)) ||
                (rc = wc_step(c, w, w->segn + (int64_t)q * n, w->segP + (int64_t)q * 2 * n, &kq, s == nsteps - 1)))
                return rc;
            if (s == nsteps - 1 && (rc = wc_save(c, w->seg + (int64_t)(q + 1) * 5 * n))) return rc;
        } else if ((rc = wc_step(c, w, w->segn, w->segP, nullptr, false))) {
            return rc;
        }
        k_wc_eta<<<nb, WB, 0, c->stream>>>(n, c->S.tid, w->mass, st_of(w->nxt, n), w->K, w->xp, w->part);
        BSC_LAUNCH(c);
        k_wc_eta_fin<<<w->K.np, WB, 0, c->stream>>>(nb, w->K, w->part, w->eta + (int64_t)s * w->K.np);
        BSC_LAUNCH(c);
    }
    BSC_CUDA(c, cudaMemcpyAsync(eta, w->eta, sizeof(double) * nsteps * w->K.np, cudaMemcpyDeviceToHost, c->stream));
    int32_t flag = 0;
    BSC_CUDA(c, cudaMemcpyAsync(&flag, c->d_flag, sizeof(int32_t), cudaMemcpyDeviceToHost, c->stream));
    BSC_CUDA(c, cudaStreamSynchronize(c->stream));
    if (flag) {
        BSC_CUDA(c, cudaMemsetAsync(c->d_flag, 0, 4 * sizeof(int32_t), c->stream));
        return set_err(c, BSC_E_CAPACITY, "wcsph_forward: neighbour-list capacity or cell grid exceeded");
    }
    w->last_kept = true;
    return BSC_OK;
}

int bsc_wcsph_adjoint(bsc_ctx* c, const double* dJ_deta, double* grad) {
    if (!c || !c->wc) return c ? set_err(c, BSC_E_INVALID, "wcsph_adjoint before wcsph_setup") : BSC_E_INVALID;
    WcState* w = c->wc;
    if (w->nsteps < 1 || !dJ_deta || !grad) return set_err(c, BSC_E_INVALID, "wcsph_adjoint: run wcsph_forward first");
    const int64_t n = c->n;
    const int nsteps = w->nsteps, every = w->every, np = w->K.np, G = w->G;
    const unsigned nb = blocks_for(n, WB);
    const int pstride = 2 + BSC_WCSPH_MAX_GRID;
    const int64_t slots = list_slots(c);
    int rc;
    BSC_CUDA(c, cudaMemcpyAsync(w->dJ, dJ_deta, sizeof(double) * nsteps * np, cudaMemcpyHostToDevice, c->stream));
    BSC_CUDA(c, cudaMemsetAsync(w->lam, 0, sizeof(double) * 5 * n, c->stream));
    BSC_CUDA(c, cudaMemsetAsync(w->grad, 0, sizeof(double) * (2 + BSC_WCSPH_MAX_GRID), c->stream));
    const int nseg = (nsteps + every - 1) / every;
    for (int sgi = nseg - 1; sgi >= 0; --sgi) {
        const int s0 = sgi * every, s1 = std::min(nsteps, s0 + every);
        // recompute the segment, keeping states, lists, porosities, pressure
        // sums (the last one the forward run kept)
        const bool kept = sgi == nseg - 1 && w->last_kept;
        if (!kept && (rc = wc_load(c, w->ck + (int64_t)sgi * 5 * n))) return rc;
        c->t = w->tck[sgi];
        for (int s = s0; s < s1 && !kept; ++s) {
            const int q = s - s0;
            if ((rc = wc_save(c, w->seg + (int64_t)q * 5 * n))) return rc;
            const Keep kq = seg_keep(w, q, n, slots);
            if ((rc = wc_step(c, w, w->segn + (int64_t)q * n, w->segP + (int64_t)q * 2 * n, &kq, s == s1 - 1 && sgi == 0)))
                return rc;
        }
        if (!kept && (rc = wc_save(c, w->seg + (int64_t)(s1 - s0) * 5 * n))) return rc;
        // reverse through the segment
        for (int s = s1 - 1; s >= s0; --s) {
            const int q = s - s0;
            const St st0 = st_of(w->seg + (int64_t)q * 5 * n, n), st1 = st_of(w->seg + (int64_t)(q + 1) * 5 * n, n);
            St lam = st_of(w->lam, n), lamn = st_of(w->lamn, n);
            // the loss at the state after step s
            k_wc_adj_probe<<<nb, WB, 0, c->stream>>>(n, c->S.tid, w->mass, st1, w->K, w->xp,
                                                     w->dJ + (int64_t)s * np, lam);
            BSC_LAUNCH(c);
            const State S = wc_view(c, w);
            const Keep kq = seg_keep(w, q, n, slots);
            const double* nq = w->segn + (int64_t)q * n;
            const AdjPair ap{w->adj2, w->adj2 + n, w->adj2 + 2 * n};
            const int lanes = lanes_for(n);
            const unsigned nbp = blocks_for(n * lanes, WPB);
            k_wc_adj_local<<<nb, WB, 0, c->stream>>>(n, c->S.tid, w->K, st0, st1, nq, w->segP + (int64_t)q * 2 * n,
                                                     kq.pre.rt, lam, ap, w->lD, w->ln, w->lvl, w->lrl, w->part,
                                                     pstride);
            BSC_LAUNCH(c);
            with_lanes(lanes, [&](auto L) {
                k_wc_adj_pair<decltype(L)::value><<<nbp, WPB, 0, c->stream>>>(
                    n, S, w->K, st0, kq.nbr, kq.cnt, kq.pre, kq.geo, slots, ap, w->lD, w->ln, w->lvl, w->lrl, lam,
                    lamn, kq.por.dn, kq.por.pgi, kq.por.pgv, w->part, pstride);
            });
            BSC_LAUNCH(c);
            k_wc_grad<<<2 + G, WB, 0, c->stream>>>((int)nb, (int)nbp, pstride, w->part, w->grad);
            BSC_LAUNCH(c);
            std::swap(w->lam, w->lamn);
        }
    }
    // the segment buffers now hold the first segment
    if (nseg > 1) w->last_kept = false;
    BSC_CUDA(c, cudaMemcpyAsync(grad, w->grad, sizeof(double) * (2 + G), cudaMemcpyDeviceToHost, c->stream));
    BSC_CUDA(c, cudaStreamSynchronize(c->stream));
    return BSC_OK;
}

}  // extern "C"
