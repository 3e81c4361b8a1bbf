// step_exact.cuh -- strain-rate and momentum gathers of the FP64-exact step.
//
// The reference adds a particle's pair terms one after the other in the order
// of its neighbour list, and so do these kernels; but the terms themselves,
// which hold nearly all of the work (a square root and the divisions of the
// kernel gradient), do not depend on one another.  Small bodies give eight
// lanes to a particle: each forms the terms of every eighth neighbour, writes
// them to shared memory, and then every lane adds up one of the sums in list
// order.  A thread that owns a particle alone walks a chain of 80 square roots
// and divisions, 62 us at the least however few particles there are.
//
// Bound: the latency of the FP64 chain and then the FP64 pipe.  Divisions by a
// number that several quotients share (h, the gradient's denominator, the
// corrected form's sum squared) multiply by its reciprocal and correct the
// quotient (quotient.cuh), so every quotient is the one that the division gives.
#pragma once
#include "nbr_iter.cuh"
#include "physics.cuh"
#include "quotient.cuh"

namespace mcm {
namespace MCM_FLAVOUR_NS {

// Lanes per particle L: eight for bodies that leave the chip idle with one
// thread per particle, one for the others, which then spend no instructions on
// handing terms over.  Measured (us, strain / momentum, 8 lanes and 1; the
// walk before, one thread per particle with a division per quotient, in
// brackets): 2 080 particles 19/22 and 62/64 (83/88), 16 848: 37/40 and 66/66
// (93/102), 35 192: 64/69 and 68/72, 41 360: 76/81 and 72/77, 131 544: 209/238
// and 151/181 (177/206), 685 824: 1092/1180 and 602/705 (796/946).  The
// corrected form meets a little later, at the same line for all that: 35 192:
// 184/206 and 213/229, 41 360: 223/238 and 228/247, 47 328: 238/256 and
// 229/246, 68 120: 357/395 and 242/265 (339/367).
constexpr int kSeqLanesBelow = 36000;
constexpr int seq_threads(int lanes) { return lanes == 1 ? 128 : 256; }
// Neighbours whose records a lane fetches ahead, and the blocks an SM is to hold.
constexpr int seq_ahead(int lanes) { return lanes == 1 ? 1 : 2; }
constexpr int seq_blocks(int disc, int lanes) { return lanes == 1 ? (disc ? 4 : 5) : 2; }

// What a particle's own h gives every pair with a neighbour of the same h.
struct OwnH {
    double h, inv, const1;   // 1/h, 1/(pi h^3) as MCM/mcm_gradw.f90 forms them
};
__device__ __forceinline__ OwnH own_h(double h) { return {h, 1.0 / h, 1.0 / (kPi * h * h * h)}; }

// MCM/mcm_gradw.f90:41-103 (and mcm_kernel.f90:42-95 when WITH_W), the
// expressions of gradw and kernelw.
template <bool WITH_W>
__device__ __forceinline__ void pair_kernel(double x0, double x1, double x2, const OwnH &o, double hj, double (&d)[3],
                                            double &w) {
    double havg = o.h, inv = o.inv, const1 = o.const1;
    if (hj != o.h) {
        havg = 0.5 * (o.h + hj);
        inv = 1.0 / havg;
        const1 = 1.0 / (kPi * havg * havg * havg);
    }
    const double const2 = const1 * 0.25;
    double rad = x0 * x0;
    rad = rad + x1 * x1;
    rad = rad + x2 * x2;
    rad = sqrt(rad);
    const double z = divide(rad, havg, inv);
    double dw = 0.0;
    if (WITH_W) w = 0.0;
    if (z < 1.0) {
        dw = const1 * ((9.0 / 4.0 * z - 3.0) * z);
        if (WITH_W) w = const1 * (((0.75 * z - 1.5) * z) * z + 1.0);
    } else if (z < 2.0) {
        const double t = 2.0 - z;
        dw = -3.0 * const2 * (t * t);
        if (WITH_W) w = const2 * (t * t * t);
    }
    if (rad == 0.0) {
        d[0] = d[1] = d[2] = 0.0;
        return;
    }
    const double den = rad * havg;
    const double n0 = dw * x0, n1 = dw * x1, n2 = dw * x2;
    if (divisor_in_range(den) && dividend_in_range(n0) && dividend_in_range(n1) && dividend_in_range(n2)) {
        const double y = 1.0 / den;
        d[0] = quotient(n0, den, y);
        d[1] = quotient(n1, den, y);
        d[2] = quotient(n2, den, y);
    } else {
        d[0] = n0 / den;
        d[1] = n1 / den;
        d[2] = n2 / den;
    }
}

// Entry k of the particle at position t: its real neighbours in list order,
// itself (disctype 1), its ghosts; past the end itself.
struct Listed {
    int idx;
    bool ghost, self;
};
struct Walk {
    const unsigned *list;
    int t, nreal, nself, total;
};
__device__ __forceinline__ Walk walk_of(const StepArgs &a, int t, bool live) {
    Walk w;
    w.t = live ? t : 0;
    w.nself = a.prm.disctype == 1 ? 1 : 0;
    w.nreal = live ? stored_neighbours(a, t) : 0;
    w.total = live ? w.nreal + w.nself + a.gnnbr[t] : 0;
    w.list = a.nidx + (size_t)w.t * a.nstride;
    return w;
}
__device__ __forceinline__ Listed listed(const StepArgs &a, const Walk &w, int k) {
    if (k < w.nreal) return {(int)(w.list[k] & kPosMask), false, false};
    if (k < w.nreal + w.nself || k >= w.total) return {w.t, false, true};
    return {a.gnbr[(size_t)(k - w.nreal - w.nself) * a.npad + w.t], true, false};
}

// Adds NP terms of every neighbour of the walk to acc, in list order.
// load(entry) fetches a neighbour's records, terms(records, entry, out) forms
// its terms.  U neighbours per lane and round, whose records are fetched before
// the first is used (past the end: the particle's own).  L == 8: sum c of the
// particle in lane c % 8, slot c / 8; buf: the warp's own shared memory,
// 32 U seq_pitch(NP) doubles (an odd pitch, so that neither the lanes that
// write a term nor those that read one meet in a bank).  L == 1: the thread's
// own sums.
constexpr int seq_pitch(int np) { return np | 1; }
template <int L, int NP>
struct Sums {
    static constexpr int S = L == 1 ? NP : (NP + 7) / 8;
    double v[S];
    __device__ __forceinline__ Sums() {
#pragma unroll
        for (int s = 0; s < S; ++s) v[s] = 0.0;
    }
    // sum c of the lane's particle, in every lane
    __device__ __forceinline__ double all(int c) const {
        if (L == 1) return v[c];
        double r = v[0];
#pragma unroll
        for (int s = 1; s < S; ++s)
            if (c / 8 == s) r = v[s];
        return __shfl_sync(0xffffffffu, r, c & 7, 8);
    }
};
template <int L, int U, int NP, typename FL, typename F>
__device__ __forceinline__ void sum_in_order(const StepArgs &a, const Walk &w, double *buf, Sums<L, NP> &acc, FL &&load,
                                             F &&terms) {
    constexpr unsigned kAll = 0xffffffffu;
    constexpr int P = seq_pitch(NP), S = Sums<L, NP>::S;
    const int lane = threadIdx.x & (L - 1);
    double *mine = buf + ((threadIdx.x & 31) / L) * (L * U * P);   // the particle's L U rows
    Listed e[U];
#pragma unroll
    for (int u = 0; u < U; ++u) e[u] = listed(a, w, L * u + lane);
    for (int k0 = 0; L == 1 ? k0 < w.total : __any_sync(kAll, k0 < w.total); k0 += L * U) {
        decltype(load(e[0])) rec[U];
#pragma unroll
        for (int u = 0; u < U; ++u) rec[u] = load(e[u]);
        Listed next[U];
#pragma unroll
        for (int u = 0; u < U; ++u) next[u] = listed(a, w, k0 + L * U + L * u + lane);
        if (L == 1) {
#pragma unroll
            for (int u = 0; u < U; ++u) {
                double out[NP];
                terms(rec[u], e[u], out);
                if (U == 1 || k0 + u < w.total)
#pragma unroll
                    for (int c = 0; c < NP; ++c) acc.v[c] = acc.v[c] + out[c];
                e[u] = next[u];
            }
            continue;
        }
        __syncwarp();
#pragma unroll
        for (int u = 0; u < U; ++u) {
            double out[NP];
            terms(rec[u], e[u], out);
#pragma unroll
            for (int c = 0; c < NP; ++c) mine[(L * u + lane) * P + c] = out[c];
            e[u] = next[u];
        }
        __syncwarp();
        const int m = w.total - k0;
        if (m >= L * U) {
#pragma unroll
            for (int j = 0; j < L * U; ++j)
#pragma unroll
                for (int s = 0; s < S; ++s)
                    if (lane + L * s < NP) acc.v[s] = acc.v[s] + mine[j * P + lane + L * s];
        } else {
            for (int j = 0; j < m; ++j)
#pragma unroll
                for (int s = 0; s < S; ++s)
                    if (lane + L * s < NP) acc.v[s] = acc.v[s] + mine[j * P + lane + L * s];
        }
    }
}

// The corrected form's first two walks (MCM/mcm_corr_strain.f90:51-104,
// mcm_corr_acceleration.f90:63-118): sum of V W and V grad W, then the
// inverse of the gradient correction.  SIGN 1: kernel centred at i (x_i - x_j),
// -1 at j.  vol(entry), pos(entry): a neighbour's V and (x, h).
struct Correction {
    double sw, sg[3], sw2, inv_sw2, invB[3][3];
    __device__ __forceinline__ void corrected(const double (&d)[3], double w, double (&cg)[3]) const {
#pragma unroll
        for (int m = 0; m < 3; ++m) cg[m] = divide(d[m] * sw - w * sg[m], sw2, inv_sw2);
    }
};
struct PosVol {
    double4 x;   // x, h
    double v;
};
template <int L, int SIGN, typename FX, typename FV>
__device__ __forceinline__ void correction_of(const StepArgs &a, const Walk &w, double *buf, const double4 xi,
                                              const OwnH &o, Correction &C, FX &&pos, FV &&vol) {
    auto load = [&](const Listed &e) { return PosVol{pos(e), vol(e)}; };
    auto kernel = [&](const PosVol &r, double (&xr)[3], double (&d)[3], double &wt) {
        xr[0] = r.x.x - xi.x; xr[1] = r.x.y - xi.y; xr[2] = r.x.z - xi.z;
        if (SIGN > 0) pair_kernel<true>(xi.x - r.x.x, xi.y - r.x.y, xi.z - r.x.z, o, r.x.w, d, wt);
        else pair_kernel<true>(xr[0], xr[1], xr[2], o, r.x.w, d, wt);
    };
    Sums<L, 4> s4;
    sum_in_order<L, seq_ahead(L)>(a, w, buf, s4, load, [&](const PosVol &r, const Listed &, double (&out)[4]) {
        double xr[3], d[3], wt;
        kernel(r, xr, d, wt);
        out[0] = r.v * wt;
        out[1] = r.v * d[0];
        out[2] = r.v * d[1];
        out[3] = r.v * d[2];
    });
    C.sw = s4.all(0);
#pragma unroll
    for (int l = 0; l < 3; ++l) C.sg[l] = s4.all(1 + l);
    C.sw2 = C.sw * C.sw;
    C.inv_sw2 = 1.0 / C.sw2;
    Sums<L, 9> b9;
    sum_in_order<L, seq_ahead(L)>(a, w, buf, b9, load, [&](const PosVol &r, const Listed &, double (&out)[9]) {
        double xr[3], d[3], wt, cg[3];
        kernel(r, xr, d, wt);
        C.corrected(d, wt, cg);
#pragma unroll
        for (int n = 0; n < 3; ++n)
#pragma unroll
            for (int m = 0; m < 3; ++m) out[3 * n + m] = r.v * xr[n] * cg[m];
    });
    double B[3][3];
#pragma unroll
    for (int c = 0; c < 9; ++c) B[c / 3][c % 3] = b9.all(c);
    inverse3(B, C.invB);
}

// ------------------------------------------------------------ strain rate
// MCM/mcm_oldstrain.f90 / mcm_corr_strain.f90: rod, spin and trace go to the
// state's diagnostic arrays, which the constitutive kernel reads.
template <int DISC, int L>
__global__ void __launch_bounds__(seq_threads(L), seq_blocks(DISC, L)) k_strain_seq(StepArgs a) {
    chain_wait();
    constexpr int kSeqThreads = seq_threads(L), kPer = kSeqThreads / L;   // particles per block
    __shared__ double bufs[kSeqThreads / 32][L == 1 ? 1 : 64 * seq_pitch(9)];
    __shared__ double grad[9][L == 1 ? 1 : kPer + 1];
    if (skip_step(a)) return;
    double *buf = bufs[threadIdx.x >> 5];
    const int t0 = blockIdx.x * kPer, t = t0 + threadIdx.x / L;
    const bool live = t < a.n;
    const Walk w = walk_of(a, t, live);
    const double4 xi = ld4(a.rec0 + w.t), vi = ld4(a.rec1 + w.t);
    const OwnH o = own_h(xi.w);
    Sums<L, 9> acc;
    auto pos = [&](const Listed &e) { return ld4((e.ghost ? a.grec0 : a.rec0) + e.idx); };
    auto vel = [&](const Listed &e) { return ld4((e.ghost ? a.grec1 : a.rec1) + e.idx); };
    struct PosVel {
        double4 x, v;
    };
    auto load = [&](const Listed &e) { return PosVel{pos(e), vel(e)}; };
    if (DISC == 0) {
        // MCM/mcm_oldstrain.f90:34-54
        sum_in_order<L, seq_ahead(L)>(a, w, buf, acc, load, [&](const PosVel &r, const Listed &, double (&out)[9]) {
            const double4 xj = r.x, vj = r.v;
            double d[3], wt;
            pair_kernel<false>(xi.x - xj.x, xi.y - xj.y, xi.z - xj.z, o, xj.w, d, wt);
            const double dv[3] = {vj.x - vi.x, vj.y - vi.y, vj.z - vi.z};
#pragma unroll
            for (int n = 0; n < 3; ++n) {
                const double tt = vj.w * dv[n];
#pragma unroll
                for (int m = 0; m < 3; ++m) out[3 * n + m] = tt * d[m];
            }
        });
    } else {
        // MCM/mcm_corr_strain.f90:51-134 (kernel centred at i)
        Correction C;
        correction_of<L, 1>(a, w, buf, xi, o, C, pos, [&](const Listed &e) { return vel(e).w; });
        sum_in_order<L, seq_ahead(L)>(a, w, buf, acc, load, [&](const PosVel &r, const Listed &, double (&out)[9]) {
            const double4 xj = r.x, vj = r.v;
            double d[3], wt, cg[3], c2[3];
            pair_kernel<true>(xi.x - xj.x, xi.y - xj.y, xi.z - xj.z, o, xj.w, d, wt);
            C.corrected(d, wt, cg);
#pragma unroll
            for (int n = 0; n < 3; ++n) c2[n] = C.invB[n][0] * cg[0] + C.invB[n][1] * cg[1] + C.invB[n][2] * cg[2];
            const double vv[3] = {vj.x, vj.y, vj.z};
#pragma unroll
            for (int n = 0; n < 3; ++n) {
                const double tt = vj.w * vv[n];
#pragma unroll
                for (int m = 0; m < 3; ++m) out[3 * n + m] = tt * c2[m];
            }
        });
    }
    double *const *f = a.F.f;
    auto put = [&](int q, int i, auto g) {
        const double r11 = 0.5 * (g(0, 0) + g(0, 0)), r22 = 0.5 * (g(1, 1) + g(1, 1)), r33 = 0.5 * (g(2, 2) + g(2, 2));
        switch (q) {
            case 0: f[FR11][i] = r11; break;
            case 1: f[FR22][i] = r22; break;
            case 2: f[FR33][i] = r33; break;
            case 3: f[FR12][i] = 0.5 * (g(0, 1) + g(1, 0)); break;
            case 4: f[FR13][i] = 0.5 * (g(0, 2) + g(2, 0)); break;
            case 5: f[FR23][i] = 0.5 * (g(1, 2) + g(2, 1)); break;
            case 6: f[FW12][i] = 0.5 * (g(0, 1) - g(1, 0)); break;
            case 7: f[FW13][i] = 0.5 * (g(0, 2) - g(2, 0)); break;
            case 8: f[FW23][i] = 0.5 * (g(1, 2) - g(2, 1)); break;
            default: f[FTR][i] = r11 + r22 + r33; break;
        }
    };
    if (L == 1) {
        if (!live) return;
        const int i = a.cell_list[t];
#pragma unroll
        for (int q = 0; q < 10; ++q) put(q, i, [&](int n, int m) { return acc.v[(3 * n + m) % Sums<L, 9>::S]; });
    } else {
        // the block's gradients, then its fields in runs of particles
        const int lane = threadIdx.x & 7;
        grad[lane][threadIdx.x >> 3] = acc.v[0];
        if (lane == 0) grad[8][threadIdx.x >> 3] = acc.v[1];
        __syncthreads();
        const int p = threadIdx.x % kPer;
        if (t0 + p >= a.n) return;
        const int i = a.cell_list[t0 + p];
        for (int q = threadIdx.x / kPer; q < 10; q += kSeqThreads / kPer)
            put(q, i, [&](int n, int m) { return grad[3 * n + m][p]; });
    }
}

// ----------------------------------------------- momentum + integration
__device__ __forceinline__ void sym_from_rec(const double4 &r1, const double4 &r2, double A[3][3]) {
    A[0][0] = r1.x; A[1][1] = r1.y; A[2][2] = r1.z;
    A[0][1] = A[1][0] = r1.w;
    A[0][2] = A[2][0] = r2.x;
    A[1][2] = A[2][1] = r2.y;
}
// The lower triangle from the asymmetric record (cap model).
__device__ __forceinline__ void lower_from_rec(const double4 &r3, double A[3][3]) {
    A[1][0] = r3.x;
    A[2][0] = r3.y;
    A[2][1] = r3.z;
}

// The momentum sums, then per particle (L == 8: by one warp of the block for
// its 32 particles, another warp each round): a (split path), base
// accelerations and displacement BCs (MCM/mcm_boundcond.f90:23-62), block
// partial energy sums (MCM/mcm_calctotale.f90:33-51) and, when integrate is
// set and the run has not terminated, the velocity and position update with
// block bbox partials.  ASYM: the cap model's lower triangle in the fourth
// record.
template <int DISC, bool ASYM, int L>
__global__ void __launch_bounds__(seq_threads(L), seq_blocks(DISC, L)) k_momentum_seq(StepArgs a, int integrate) {
    chain_wait();
    constexpr unsigned kAll = 0xffffffffu;
    constexpr int kSeqThreads = seq_threads(L), kPer = kSeqThreads / L, kWarps = kSeqThreads / 32;
    __shared__ double bufs[kWarps][L == 1 ? 1 : (DISC == 0 ? 64 * seq_pitch(3) : 32 * seq_pitch(18))];
    __shared__ double forces[2][3][L == 1 ? 1 : kPer + 1];
    __shared__ double esum[kWarps][kMaxMat][5], blo[kWarps][3], bhi[kWarps][3];
    if (skip_step(a)) return;
    const int lane = threadIdx.x & (L - 1), sub = threadIdx.x / L, wid = threadIdx.x >> 5, l32 = threadIdx.x & 31;
    double *buf = bufs[wid];
    const int nm = a.nmat;
    double *const *f = a.F.f;
    double x[3] = {1.0e20, 1.0e20, 1.0e20}, xmax[3] = {-1.0e20, -1.0e20, -1.0e20};
    const bool do_int = integrate && !a.time->ended;
    for (int k = l32; k < 5 * nm; k += 32) esum[wid][k / 5][k % 5] = 0.0;
    __syncwarp();
    const int rounds = (a.n + kPer * gridDim.x - 1) / (kPer * gridDim.x);
#pragma unroll 1
    for (int round = 0; round < rounds; ++round) {
        const int t0 = (round * gridDim.x + blockIdx.x) * kPer, t = t0 + sub;
        const bool live = t < a.n;
        const Walk w = walk_of(a, t, live);
        const double4 xi = ld4(a.rec0 + w.t), r2i = ld4(a.rec2 + w.t);
        double Ai[3][3];
        sym_from_rec(ld4(a.rec1 + w.t), r2i, Ai);
        if (ASYM) lower_from_rec(ld4(a.rec3 + w.t), Ai);
        // MCM/mcm_oldacceleration.f90:49-51, mcm_corr_acceleration.f90:45-49
        Sums<L, 3> acc;
        if (a.prm.contact && live) {
            const int i = a.cell_list[t];
            if (L == 1) {
#pragma unroll
                for (int j = 0; j < Sums<L, 3>::S; ++j) acc.v[j] = acc.v[j] + f[FRPX + j][i];
            } else if (lane < 3) {
                acc.v[0] = acc.v[0] + f[FRPX + lane][i];
            }
        }
        const OwnH o = own_h(xi.w);
        auto pos = [&](const Listed &e) { return ld4((e.ghost ? a.grec0 : a.rec0) + e.idx); };
        struct Stress {
            double4 x, r1, r2, r3;
        };
        auto load = [&](const Listed &e) {
            Stress r;
            r.x = pos(e);
            r.r1 = ld4((e.ghost ? a.grec1 : a.rec1) + e.idx);
            r.r2 = ld4((e.ghost ? a.grec2 : a.rec2) + e.idx);
            if (ASYM) r.r3 = ld4((e.ghost ? a.grec3 : a.rec3) + e.idx);
            return r;
        };
        double ac[3];
        if (DISC == 0) {
            // MCM/mcm_oldacceleration.f90:66-89; sigma(m,n) is read as stored,
            // both triangles (they differ for the cap model)
            sum_in_order<L, 1>(a, w, buf, acc, load, [&](const Stress &r, const Listed &, double (&out)[3]) {
                const double4 xj = r.x, r2 = r.r2;
                double d[3], wt;
                pair_kernel<false>(xi.x - xj.x, xi.y - xj.y, xi.z - xj.z, o, xj.w, d, wt);
                double Aj[3][3];
                sym_from_rec(r.r1, r2, Aj);
                if (ASYM) lower_from_rec(r.r3, Aj);
#pragma unroll
                for (int n = 0; n < 3; ++n) {
                    double ds = 0.0;
#pragma unroll
                    for (int m = 0; m < 3; ++m) ds = ds + (Aj[m][n] + Ai[m][n]) * d[m];
                    out[n] = r2.z * ds;
                }
            });
            if (L == 1) {
#pragma unroll
                for (int n = 0; n < 3; ++n) ac[n] = acc.v[n % Sums<L, 3>::S];
            } else {
                ac[0] = acc.v[0];   // lane n: component n
            }
        } else {
            // MCM/mcm_corr_acceleration.f90:63-161 (kernel centred at j; the self
            // slot is zeroed; the final sum uses the last neighbour's mass)
            Correction C;
            correction_of<L, -1>(a, w, buf, xi, o, C, pos,
                                 [&](const Listed &e) { return (e.ghost ? a.grec2 : a.rec2)[e.idx].w; });
            // deltasig(m,n,l) is symmetric in (m,n): 6 x 3 sums
            Sums<L, 18> ds;
            sum_in_order<L, 1>(a, w, buf, ds, load, [&](const Stress &r, const Listed &e, double (&out)[18]) {
                const double4 xj = r.x;
                double d[3], wt, cg[3];
                pair_kernel<true>(xj.x - xi.x, xj.y - xi.y, xj.z - xi.z, o, xj.w, d, wt);
                C.corrected(d, wt, cg);
                double Aj[3][3];
                sym_from_rec(r.r1, r.r2, Aj);
#pragma unroll
                for (int u = 0; u < 6; ++u) {
                    const int m = (u < 3) ? u : (u == 5 ? 1 : 0);
                    const int n = (u < 3) ? u : (u == 3 ? 1 : 2);
                    double dsig = Aj[m][n] + Ai[m][n];
                    if (e.self) dsig = 0.0;
#pragma unroll
                    for (int l = 0; l < 3; ++l) out[3 * u + l] = dsig * cg[l];
                }
            });
            double massj = r2i.z;
            const int ng = w.total - w.nreal - w.nself;
            if (ng > 0) massj = a.grec2[a.gnbr[(size_t)(ng - 1) * a.npad + w.t]].z;
            double S[18];
#pragma unroll
            for (int c = 0; c < 18; ++c) S[c] = ds.all(c);
#pragma unroll
            for (int n = 0; n < 3; ++n) {
                double r = acc.all(n);
#pragma unroll
                for (int m = 0; m < 3; ++m)
#pragma unroll
                    for (int l = 0; l < 3; ++l) r = r + massj * S[3 * sym_index(n, m) + l] * C.invB[l][m];
                if (L == 1) ac[n] = r;
                else if (lane == n) ac[0] = r;
            }
        }
        int tp = t;
        if (L > 1) {
            // the block's sums to one warp, a particle per lane
            if (lane < 3) forces[round & 1][lane][sub] = ac[0];
            __syncthreads();
            if (wid != round % kWarps) continue;
            tp = t0 + l32;
#pragma unroll
            for (int n = 0; n < 3; ++n) ac[n] = forces[round & 1][n][l32 % (L == 1 ? 1 : kPer)];
        }
        int mati = 0;
        double vals[5] = {0.0, 0.0, 0.0, 0.0, 0.0};
        if (tp < a.n) {
            const int i = a.cell_list[tp];
            if (a.prm.baseaccel)
#pragma unroll
                for (int j = 0; j < 3; ++j) ac[j] = ac[j] + a.prm.base_a[j];
            switch (a.F.dispbc[i]) {
                case 1: ac[0] = 0.0; break;
                case 2: ac[1] = 0.0; break;
                case 3: ac[2] = 0.0; break;
                case 4: ac[0] = 0.0; ac[1] = 0.0; break;
                case 5: ac[1] = 0.0; ac[2] = 0.0; break;
                case 6: ac[0] = 0.0; ac[2] = 0.0; break;
                case 7: ac[0] = 0.0; ac[1] = 0.0; ac[2] = 0.0; break;
                default: break;
            }
            if (a.split_mode || a.prm.diag || a.prm.veloc_opt) { f[FAX][i] = ac[0]; f[FAY][i] = ac[1]; f[FAZ][i] = ac[2]; }
            mati = a.F.mat[i];
            const double mass = f[FMASS][i], vabs = f[FVABS][i];
            vals[0] = 0.5 * mass * (vabs * vabs);
            vals[1] = f[FE][i];
            vals[2] = mass * fabs(f[FVX][i]);
            vals[3] = mass * fabs(f[FVY][i]);
            vals[4] = mass * fabs(f[FVZ][i]);
            if (do_int) {
                double xn[3];
                integrate_particle(a, i, ac, a.time->dt, a.time->dtold, xn);
#pragma unroll
                for (int d = 0; d < 3; ++d) { x[d] = fmin(x[d], xn[d]); xmax[d] = fmax(xmax[d], xn[d]); }
            }
        }
        // the warp's sums, round after round
        for (int m = 1; m <= nm; ++m) {
            if (!__any_sync(kAll, mati == m)) continue;
#pragma unroll
            for (int c = 0; c < 5; ++c) {
                double v = mati == m ? vals[c] : 0.0;
#pragma unroll
                for (int s = 16; s > 0; s >>= 1) v += __shfl_xor_sync(kAll, v, s);
                if (l32 == 0) esum[wid][m - 1][c] += v;
            }
        }
    }
    if (do_int) {
#pragma unroll
        for (int d = 0; d < 3; ++d) {
#pragma unroll
            for (int s = 16; s > 0; s >>= 1) {
                x[d] = fmin(x[d], __shfl_xor_sync(kAll, x[d], s));
                xmax[d] = fmax(xmax[d], __shfl_xor_sync(kAll, xmax[d], s));
            }
            if (l32 == 0) { blo[wid][d] = x[d]; bhi[wid][d] = xmax[d]; }
        }
    }
    __syncthreads();
    // per-block partials, the warps' in order: [5*nmat energies][6 bbox]
    double *out = a.red + (size_t)blockIdx.x * (5 * nm + 6);
    for (int k = threadIdx.x; k < 5 * nm; k += kSeqThreads) {
        double v = esum[0][k / 5][k % 5];
        for (int q = 1; q < kWarps; ++q) v += esum[q][k / 5][k % 5];
        out[k] = v;
    }
    if (do_int && threadIdx.x < 3) {
        double lo = blo[0][threadIdx.x], hi = bhi[0][threadIdx.x];
        for (int q = 1; q < kWarps; ++q) { lo = fmin(lo, blo[q][threadIdx.x]); hi = fmax(hi, bhi[q][threadIdx.x]); }
        out[5 * nm + threadIdx.x] = lo;
        out[5 * nm + 3 + threadIdx.x] = hi;
    }
}

}  // namespace MCM_FLAVOUR_NS
}  // namespace mcm
