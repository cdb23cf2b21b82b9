// k_group_adjoint.cu -- reverse sweeps of the solves by groups of degrees.
//
// The adjoint of the group solves (k_solve_group.cu): from the adjoints of
// the uu / vv / ww coefficients of every (omega, l) pair to dL/dc[i][p][k],
// the gradient with respect to the power-form spline segments.  No
// reference counterpart: the reference has no derivatives.  The same
// discrete adjoint as the per-thread sweep (ysg_pair_adjoint.cuh, which
// states the conventions), organised by the shared radial walk:
//   - the coefficient matrices of a stage come from a point (ysg_group.cuh)
//     that depends on (r, omega) alone.  So the sweep contracts a stage's
//     matrix adjoint over the degrees first, to the 7 to 18 numbers of the
//     point's adjoint, and carries that to the spline values once per point
//     and block instead of once per lane (a lane did 60 of these
//     evaluations per step, each with 13 x 4 moment sums in local memory and
//     one atomic add per moment and interval);
//   - the response rows a pair uses (two or three) are obtained from the
//     transposed b-vector integration, as in the solve: row k needs one
//     forward integration of the b-vector started from the row's adjoint and
//     one reverse pass, in place of four forward and four reverse ones;
//   - the l = 0 sweep runs a warp per frequency on step matrices
//     (ysg_radial.cuh), each lane reversing its own piece.
// What bounds it: a stage of the reverse has the right-hand side again, the
// contraction with the coefficients and the transposed product, about four
// forward solves in all, at 8 warps per SM.  Of the cycles between two
// instructions of a warp (31,003 pairs) 2.8 wait for the block's other warps
// (the degrees that start deeper walk on alone), 2.0 for the logged states
// and the stage inputs (6 x 14 components per lane: local memory, held by
// the L2), 1.8 for the FP64 pipe's latency and 0.8 for instructions.
// Measured: 31,003 pairs 173 ms with a thread per pair, 11.9 ms here; their
// l = 0 sweep 64 ms with a thread per frequency, 1.06 ms here; the gradient
// call of a 200-knot ocean deck with 121 degrees 89 -> 5.7 ms.
// Kernels:
//   k_gadj_sph   spheroidal pairs, a degree per lane, NL warps per item
//   k_gadj_tor   toroidal pairs
//   k_gadj_rad   l = 0
#define YSG_LOOPED_STEP 1
#define YSG_CPLX_CALLS
#include <algorithm>

#include "ysg_kernels.h"
#include "ysg_pair_adjoint.cuh"
#include "ysg_group_sph.cuh"
#include "ysg_radial.cuh"

namespace ysg {
inline namespace YSG_VARIANT {
namespace {

// ---------------------------------------------------------------------------
// Adjoints of the points: lane() contracts a matrix adjoint to the lane's
// share of the point's adjoint (NV numbers), values() carries the sum over
// the lanes to the spline values at the point.
// ---------------------------------------------------------------------------
__device__ __forceinline__ double re2(cd a, cd b) { return a.x * b.x - a.y * b.y; }    // Re(a b)

template <int KIND>
struct SolidPointAdj {
    using Point = SolidPoint<KIND>;
    using Bar = SolidCoefBar;
    static constexpr int NV = KIND == 2 ? 18 : 16;
    __device__ static __forceinline__ SolidCoef amat(const LaneCtx& c) { return solid_amat<KIND>(c, 0.0); }
    __device__ static __forceinline__ void lane(const LaneCtx& c, const Bar& s, double* v)
    {
        v[0] = s.t11.x; v[1] = s.t11.y;
        v[2] = c.zeta * s.t12.x; v[3] = c.zeta * s.t12.y;
        v[4] = s.s11.x; v[5] = s.s11.y;
        v[6] = c.zeta * s.s12.x; v[7] = c.zeta * s.s12.y;
        v[8] = s.s22.x; v[9] = s.s22.y;
        v[10] = c.zeta2 * s.s22.x; v[11] = c.zeta2 * s.s22.y;
        v[12] = s.k11.x; v[13] = s.k11.y;
        v[14] = s.k22.x; v[15] = s.k22.y;
        if (KIND == 2) {
            v[16] = c.zeta * s.s23.x - c.flp1 * s.s13.x;
            v[17] = s.t31.x;
        }
    }
    __device__ static __noinline__ void values(const Ctx& c, int il, double rr, const double* v, double* vb)
    {
        const Seg& g = c.sg[il];
        const double u = rr - g.r0;
        const double rrho = seg(g, u, P_RHO), racon = seg(g, u, P_ACON), rccon = seg(g, u, P_CCON);
        const double rfcon = seg(g, u, P_FCON), rncon = seg(g, u, P_NCON), rlcon = seg(g, u, P_LCON);
        const double rqmu = seg(g, u, P_QMU), rxlam = seg(g, u, P_XLAM), rxa2 = seg(g, u, P_XA2);
        const cd qaa = 1.0 + rxa2 * c.lno, qff = 1.0 + rxlam * c.lno, qll = 1.0 + rqmu * c.lno;
        const cd cf = rfcon * qff;
        const cd k11 = 1.0 / (rccon * qaa), k22 = 1.0 / (rlcon * qll);
        const double ri = 1.0 / rr, ri2 = ri * ri;
        const cd t11 = mk(v[0], v[1]), fb = mk(v[2], v[3]), s11 = mk(v[4], v[5]), gb = mk(v[6], v[7]);
        const cd a22 = mk(v[8], v[9]), b22 = mk(v[10], v[11]);
        // t11 = (1 - 2 fc) ri, fb: ri fc; s11 = -w^2 rho + 4 (gamma - rho g r) ri^2,
        // gb: (rho g r - 2 gamma) ri^2; a22 = -w^2 rho - 2 cn ri^2, b22 = (gamma + cn) ri^2
        double rb = -re2(s11 + a22, c.omega2);
        if (KIND != 0) {
            const double gg = seg(g, u, P_GRAV);
            const double rg = (gb.x - 4.0 * s11.x) * ri;           // adjoint of rho g
            rb += rg * gg;
            vb[P_GRAV] = rg * rrho;
        }
        if (KIND == 2) rb += v[16] * ri + v[17] * (-4.0 * c.pib);
        vb[P_RHO] = rb;
        const cd gamb = (4.0 * s11 - 2.0 * gb + b22) * ri2;
        const cd cnb = (b22 - 2.0 * a22) * ri2 - gamb;
        const cd fcb = (fb - 2.0 * t11) * ri;
        // gamma = A qaa - N qll - cf^2 k11, fc = cf k11
        const cd cfb = gamb * (-2.0 * (cf * k11)) + fcb * k11;
        const cd k11b = gamb * (-(cf * cf)) + fcb * cf + mk(v[12], v[13]);
        const cd k22b = mk(v[14], v[15]);
        const cd ck = k11b * k11, lk = k22b * k22;
        vb[P_CCON] = -ck.x / rccon;
        vb[P_LCON] = -lk.x / rlcon;
        const cd qab = gamb * racon - ck / qaa;
        const cd qlb = cnb * rncon - lk / qll;
        vb[P_ACON] = re2(gamb, qaa);
        vb[P_FCON] = re2(cfb, qff);
        vb[P_NCON] = re2(cnb, qll);
        vb[P_XA2] = re2(qab, c.lno);
        vb[P_XLAM] = rfcon * re2(cfb, c.lno);
        vb[P_QMU] = re2(qlb, c.lno);
    }
};

template <int KIND>
struct FluidPointAdj {
    using Point = FluidPoint<KIND>;
    using Bar = FluidCoefBar;
    static constexpr int NV = 7;
    __device__ static __forceinline__ FluidCoef amat(const LaneCtx& c) { return fluid_amat<KIND>(c, 0.0); }
    // cccon | -w^2 rho (- 4 rho g ri) | rho, g, 1/rho
    __device__ static __forceinline__ void lane(const LaneCtx& c, const Bar& s, double* v)
    {
        const cd z = c.zeta2 * got(c.p, 1);
        const cd rr = got(c.p, 3), gr = got(c.p, 4);   // ri, rho; g, 1/rho
        v[0] = s.k11.x; v[1] = s.k11.y;
        v[2] = s.s11.x; v[3] = s.s11.y;
        v[4] = v[5] = 0.0;
        v[6] = -re2(s.k11, z);
        if (KIND == 0) return;                         // s11 = -w^2 rho
        const cd gz = gr.x * z;
        cd gzb = cmac(s.t11, rr.y * gr.x, s.s11);
        v[4] = gr.x * re2(s.s11, gz);
        v[5] = rr.y * re2(s.s11, gz);
        if (KIND == 2) {
            gzb = cmac(gzb, rr.y, s.s12);
            v[4] += s.t21.x * (-c.pib4) + re2(s.s12, gz - c.flp1 * rr.x) + re2(s.s22, z);
        }
        v[5] += re2(gzb, z);
    }
    __device__ static __noinline__ void values(const Ctx& c, int il, double rr, const double* v, double* vb)
    {
        const Seg& g = c.sg[il];
        const double u = rr - g.r0;
        const double rrho = seg(g, u, P_RHO), rccon = seg(g, u, P_CCON), rxa2 = seg(g, u, P_XA2);
        const double gg = seg(g, u, P_GRAV);
        const cd qaa = 1.0 + rxa2 * c.lno;
        const cd k = 1.0 / (rccon * qaa);
        const double ri = 1.0 / rr;
        const cd ub = mk(v[2], v[3]);
        vb[P_RHO] = v[4] - v[6] / (rrho * rrho) - re2(ub, c.omega2);
        if (KIND != 0) {
            vb[P_RHO] += -4.0 * gg * ri * ub.x;
            vb[P_GRAV] = v[5] - 4.0 * rrho * ri * ub.x;
        }
        const cd ck = mk(v[0], v[1]) * k;
        vb[P_CCON] = -ck.x / rccon;
        vb[P_XA2] = -re2(ck / qaa, c.lno);
    }
};

struct TorPointAdj {
    using Point = TorPoint;
    using Bar = TorCoefBar;
    static constexpr int NV = 6;
    __device__ static __forceinline__ TorCoef amat(const LaneCtx& c) { return tor_amat(c, 0.0); }
    __device__ static __forceinline__ void lane(const LaneCtx& c, const Bar& s, double* v)
    {
        v[0] = s.k.x; v[1] = s.k.y;
        v[2] = s.s.x; v[3] = s.s.y;
        v[4] = (c.zeta2 - 2.0) * s.s.x; v[5] = (c.zeta2 - 2.0) * s.s.y;
    }
    __device__ static __noinline__ void values(const Ctx& c, int il, double rr, const double* v, double* vb)
    {
        const Seg& g = c.sg[il];
        const double u = rr - g.r0;
        const double rlcon = seg(g, u, P_LCON), rncon = seg(g, u, P_NCON), rqmu = seg(g, u, P_QMU);
        const cd qll = 1.0 + rqmu * c.lno;
        const cd k = 1.0 / (rlcon * qll);
        const double ri = 1.0 / rr;
        const cd cnb = mk(v[4], v[5]) * (ri * ri), lk = mk(v[0], v[1]) * k;
        vb[P_RHO] = -re2(mk(v[2], v[3]), c.omega2);
        vb[P_NCON] = re2(cnb, qll);
        vb[P_LCON] = -lk.x / rlcon;
        vb[P_QMU] = re2(cnb * rncon - lk / qll, c.lno);
    }
};

// The systems of a reverse sweep: right-hand side, generated transposes and
// point adjoint.
struct RevMinorSolidG {
    using Sys = MinorSolidG;
    using A = MinorSolidGAdj;
    using P = SolidPointAdj<2>;
};
struct RevBvecSolidG {
    using Sys = BvecSolidG;
    using A = BvecSolidGAdj;
    using P = SolidPointAdj<2>;
};
struct RevMinorFluidG {
    using Sys = MinorFluidG;
    using A = MinorFluidGAdj;
    using P = FluidPointAdj<2>;
};
template <int KIND>
struct RevMinorSolidNC {
    using Sys = MinorSolidNC<KIND>;
    using A = MinorSolidNCAdj;
    using P = SolidPointAdj<KIND>;
};
template <int KIND>
struct RevBvecSolidNC {
    using Sys = BvecSolidNC<KIND>;
    using A = BvecSolidNCAdj;
    using P = SolidPointAdj<KIND>;
};
template <int KIND>
struct RevMinorFluidNC {
    using Sys = MinorFluidNC<KIND>;
    using A = MinorFluidNCAdj;
    using P = FluidPointAdj<KIND>;
};
struct RevTor {
    using Sys = TorSys;
    using A = TorSysAdj;
    using P = TorPointAdj;
};

// Warps (of 32 degrees) per item, 8 warps per SM either way (255 registers).
// Sweeps of all kinds in ms with 4 / 2 / 1: 151 x 60 pairs 5.9 / 6.0 / 6.4,
// 31,003 pairs 14.4 / 14.5 / 18.9, 1.1 million 123 / 165 / 268: warps of an
// item fetch the same instructions at nearly the same time.
constexpr int GADJ_NL = 4;
// Shared memory of a sweep's block: batches of SB steps, per warp the
// points' adjoints (summed over its lanes), per point the spline values'.
constexpr int ADJ_NV = 18;
template <int NL_, int NMAX, int SLOTS_>
struct AdjMem {
    static constexpr int NW = 1, NL = NL_, SLOTS = SLOTS_, NT = 32 * NL_;
    static constexpr int SB = NT / 6 < 8 ? NT / 6 : 8;
    static constexpr bool KEEP_R = true;
    static constexpr int LOG_N = NMAX;
    static constexpr int ROWS = NMAX, OWN = NMAX;
    double pt[SB * 6][PT];
    cd slot[SLOTS > 0 ? SLOTS : 1][SLOTS > 0 ? NMAX : 1][SLOTS > 0 ? NT : 1];
    double pb[NL][SB * 6][ADJ_NV];
    double vb[SB * 6][NPARAM];
    double vu[SB * 6];
    double pr[SB * 6];
    double sh[SB];
    int sil[SB];
    int i1[32];
    double rt[32];
    unsigned long long item;
};

// Sums v[0 .. NV-1] over the lanes of the warp: each round halves the list a
// lane keeps and adds its partner's; the sum of number i ends on one lane.
template <int NV, int BIT>
__device__ __forceinline__ void warp_fold(double* v, int lane, int base, int n, double* out)
{
    if constexpr (BIT == 0) {
        if (n > 0) out[base] = v[0];
    } else {
        constexpr int H = (NV + 1) / 2;
        const bool hi = lane & BIT;
        double w[H];
#pragma unroll
        for (int i = 0; i < H; i++) {
            const double lo_v = v[i], hi_v = H + i < NV ? v[H + i] : 0.0;
            const double keep = hi ? hi_v : lo_v, send = hi ? lo_v : hi_v;
            w[i] = keep + __shfl_xor_sync(FULL, send, BIT);
        }
        // entries this lane keeps that exist
        const int m = hi ? max(n - H, 0) : min(n, H);
        warp_fold<H, BIT / 2>(w, lane, base + (hi ? H : 0), m, out);
    }
}

// The spline-value adjoints of the batch's points to the segments: moments
// v u^k summed over the points of an interval, one atomic add per moment.
// Called by the whole block after the points' adjoints are complete.
template <class P, class Mem>
__device__ __noinline__ void point_flush(const Group& g, int nb, double* grad)
{
    Mem& M = group_mem<Mem>();
    const int t = (int)threadIdx.x;
    for (int e = t; e < nb * 6; e += Mem::NT) {
        double v[P::NV], vb[NPARAM];
#pragma unroll
        for (int i = 0; i < P::NV; i++) {
            double s = M.pb[0][e][i];
            for (int w = 1; w < Mem::NL; w++) s += M.pb[w][e][i];
            v[i] = s;
        }
        for (int p = 0; p < NPARAM; p++) vb[p] = 0.0;
        const int il = M.sil[e / 6];
        P::values(g.c, il, M.pr[e], v, vb);
        for (int p = 0; p < NPARAM; p++) M.vb[e][p] = vb[p];
        M.vu[e] = M.pr[e] - g.c.sg[il].r0;
    }
    __syncthreads();
    for (int e = t; e < nb * NPARAM * 4; e += Mem::NT) {
        const int s = e / (NPARAM * 4), p = (e >> 2) % NPARAM, k = e & 3;
        const int il = M.sil[s];
        if (s > 0 && M.sil[s - 1] == il) continue;            // not the first step of its interval
        int s1 = s + 1;
        while (s1 < nb && M.sil[s1] == il) s1++;
        double sum = 0.0;
        for (int q = s * 6; q < s1 * 6; q++) {
            const double u = M.vu[q];
            double m = M.vb[q][p];
            for (int i = 0; i < k; i++) m *= u;
            sum += m;
        }
        if (sum != 0.0) atomicAdd(&grad[((size_t)il * NPARAM + p) * 4 + k], sum);
    }
    __syncthreads();
}

// The reverse of a logged walk (n steps from entry `at`): y holds the
// adjoint of its result on entry and of its start on exit.  `on`: the lane
// took part in the walk; a lane that joined it (`joined`) did so at step
// g.jq, and its adjoint there goes to stb, with y zero from there on.
template <class T, class Mem>
__device__ __noinline__ void group_rev(Group& g, const GroupLog& lg, int at, int n, int i1, int i2, double r1,
                                       double r2, cd* yio, bool on, bool joined, cd* stb, double* grad)
{
    using Sys = typename T::Sys;
    using P = typename T::P;
    constexpr int N = Sys::N, NV = P::NV;
    Mem& M = group_mem<Mem>();
    const int lane = g.lane, wl = threadIdx.x >> 5;
    const int jq = joined ? g.jq : at;
    bool live = on;
    cd y[N];
#pragma unroll
    for (int k = 0; k < N; k++) y[k] = yio[k];
    if (n > 0) {
        Walk w;
        walk_init(w, i1, i2, r1, r2, true);
        int q = at + n, nb;
        while ((nb = walk_fill<typename P::Point, Mem>(g, w)) > 0) {
#pragma unroll 1
            for (int s = 0; s < nb; s++) {
                q--;
                if (live && q < jq) {
#pragma unroll
                    for (int k = 0; k < N; k++) {
                        stb[k] = y[k];
                        y[k] = mk(0.0);
                    }
                    live = false;
                }
                if (!__any_sync(FULL, live)) {
                    for (int e = lane; e < 6 * NV; e += 32) M.pb[wl][s * 6 + e / NV][e % NV] = 0.0;
                    continue;
                }
                const double(*p)[PT] = M.pt + s * 6;
                LaneCtx lc = g.lc;
                cd Y[6][N], yt[N];
                StageVec<Mem, N, (Mem::SLOTS > 0), 0> v1;
                StageVec<Mem, N, (Mem::SLOTS > 1), 1> v2;
#pragma unroll
                for (int k = 0; k < N; k++) {
                    cd v = mk(0.0);
                    if (live) v = lg.y[((size_t)q * Mem::LOG_N + k) * lg.stride];
                    yt[k] = v;
                    Y[0][k] = v;
                }
                if (live) {
                    const double f = lg.f[(size_t)q * lg.stride];
                    if (f != 1.0)
#pragma unroll
                        for (int k = 0; k < N; k++) y[k] = f * y[k];
                }
                // the stage inputs again (group_walk's combinations)
#pragma unroll 1
                for (int st = 0; st < 5; st++) {
                    const double h = *(volatile double*)&M.sh[s];
                    cd d[N];
                    lc.p = p[st];
                    Sys::f(lc, 0.0, yt, d);
                    if (st == 0) {
#pragma unroll
                        for (int k = 0; k < N; k++) {
                            v1.set(k, d[k]);
                            yt[k] = cmac(yt[k], 0.2 * h, d[k]);
                        }
                    } else if (st == 1) {
#pragma unroll
                        for (int k = 0; k < N; k++) {
                            v2.set(k, d[k]);
                            yt[k] = cmac(cmac(Y[0][k], (3.0 / 40.0) * h, v1.get(k)), (9.0 / 40.0) * h, d[k]);
                        }
                    } else if (st == 2) {
#pragma unroll
                        for (int k = 0; k < N; k++) {
                            const cd k1 = v1.get(k), k2 = v2.get(k), y0 = Y[0][k];
                            yt[k] = cmac(cmac(cmac(y0, 0.3 * h, k1), -0.9 * h, k2), 1.2 * h, d[k]);
                            v1.set(k, cmac(cmac(cmac(y0, (1631.0 / 55296.0) * h, k1), (175.0 / 512.0) * h, k2),
                                           (575.0 / 13824.0) * h, d[k]));
                            v2.set(k, cmac(cmac(cmac(y0, (-11.0 / 54.0) * h, k1), 2.5 * h, k2), (-70.0 / 27.0) * h,
                                           d[k]));
                        }
                    } else if (st == 3) {
#pragma unroll
                        for (int k = 0; k < N; k++) {
                            yt[k] = cmac(v2.get(k), (35.0 / 27.0) * h, d[k]);
                            v1.set(k, cmac(v1.get(k), (44275.0 / 110592.0) * h, d[k]));
                        }
                    } else {
#pragma unroll
                        for (int k = 0; k < N; k++) yt[k] = cmac(v1.get(k), (253.0 / 4096.0) * h, d[k]);
                    }
#pragma unroll
                    for (int k = 0; k < N; k++) Y[st + 1][k] = yt[k];
                }
                // the stages backward: kt the adjoint of the stage's
                // derivative (group_walk's transposed combinations)
                cd kt[N];
                {
                    const double h = *(volatile double*)&M.sh[s];
#pragma unroll
                    for (int k = 0; k < N; k++) kt[k] = ((512.0 / 1771.0) * h) * y[k];
                }
#pragma unroll 1
                for (int st = 5; st >= 0; st--) {
                    lc.p = p[st];
                    {
                        typename P::Bar sb;
                        sb.zero();
                        T::A::cgrad(kt, Y[st], sb);
                        double v[NV];
                        P::lane(lc, sb, v);
                        warp_fold<NV, 16>(v, lane, 0, NV, M.pb[wl][s * 6 + st]);
                    }
                    const double h = *(volatile double*)&M.sh[s];
                    cd d[N];
                    T::A::tr(P::amat(lc), kt, d);
                    if (st == 5) {
#pragma unroll
                        for (int k = 0; k < N; k++) {
                            v1.set(k, d[k]);
                            kt[k] = ((253.0 / 4096.0) * h) * d[k];
                        }
                    } else if (st == 4) {
#pragma unroll
                        for (int k = 0; k < N; k++) {
                            v2.set(k, d[k]);
                            kt[k] = cmac(cmac(((125.0 / 594.0) * h) * y[k], (44275.0 / 110592.0) * h, v1.get(k)),
                                         (35.0 / 27.0) * h, d[k]);
                        }
                    } else if (st == 3) {
#pragma unroll
                        for (int k = 0; k < N; k++) {
                            const cd w0 = y[k], g6 = v1.get(k), g5 = v2.get(k);
                            kt[k] = cmac(cmac(cmac(((250.0 / 621.0) * h) * w0, (575.0 / 13824.0) * h, g6),
                                              (-70.0 / 27.0) * h, g5), 1.2 * h, d[k]);
                            v1.set(k, cmac(cmac(((175.0 / 512.0) * h) * g6, 2.5 * h, g5), -0.9 * h, d[k]));
                            v2.set(k, cmac(cmac(cmac(((37.0 / 378.0) * h) * w0, (1631.0 / 55296.0) * h, g6),
                                                (-11.0 / 54.0) * h, g5), 0.3 * h, d[k]));
                            y[k] = (w0 + g6) + (g5 + d[k]);
                        }
                    } else if (st == 2) {
#pragma unroll
                        for (int k = 0; k < N; k++) {
                            kt[k] = cmac(v1.get(k), (9.0 / 40.0) * h, d[k]);
                            v2.set(k, cmac(v2.get(k), (3.0 / 40.0) * h, d[k]));
                            y[k] = y[k] + d[k];
                        }
                    } else if (st == 1) {
#pragma unroll
                        for (int k = 0; k < N; k++) {
                            kt[k] = cmac(v2.get(k), 0.2 * h, d[k]);
                            y[k] = y[k] + d[k];
                        }
                    } else {
#pragma unroll
                        for (int k = 0; k < N; k++) y[k] = y[k] + d[k];
                    }
                }
            }
            __syncthreads();
            point_flush<P, Mem>(g, nb, grad);
        }
    }
    if (joined && live) {
#pragma unroll
        for (int k = 0; k < N; k++) {
            stb[k] = y[k];
            y[k] = mk(0.0);
        }
    }
#pragma unroll
    for (int k = 0; k < N; k++) yio[k] = y[k];
}

// Contributions at one radius (start and source vectors, the receiver's
// gravity) straight to the segments: per lane, or (UNIFORM) for a segment and
// radius all lanes share, summed over the warp first.
template <bool UNIFORM>
struct PointGrad {
    double* g;
    bool on;
    __device__ void add(int i, double u, const double* vb)
    {
        for (int p = 0; p < NPARAM; p++) {
            double v = on ? vb[p] : 0.0;
            if (UNIFORM) {
                for (int d = 16; d > 0; d >>= 1) v += __shfl_xor_sync(FULL, v, d);
                if ((threadIdx.x & 31) != 0) v = 0.0;
            }
            if (v == 0.0) continue;
            double m = v;
            for (int k = 0; k < 4; k++) {
                grad_add(&g[((size_t)i * NPARAM + p) * 4 + k], m);
                m *= u;
            }
        }
    }
};

struct AdjArgs {
    const Knot* kn;
    const Seg* sg;
    const ModelHdr* mh;
    const EventDev* ev;
    UnitDirs u;
    const cd* coefb;
    const long long* off;         // {0, nitems}
    const int* order;
    long long nitems;
    AdjLogs w;                    // s: the b-vector passes, c: the minors
    double* grad;
    unsigned long long* counter;
    int* status;
};

__device__ __forceinline__ GroupLog thread_log(const AdjStepArrays& a, int nthreads)
{
    const size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    return GroupLog{a.y + t, a.f + t, (size_t)nthreads, a.n};
}

__device__ __forceinline__ void adj_group_ctx(Group& g, const AdjArgs& a)
{
    g.c.kn = a.kn;
    g.c.mh = a.mh;
    g.c.sg = a.sg;
    g.c.pib = a.mh->pibigg;
    g.c.kb = nullptr;
    g.c.il = 0;
    for (int q = 0; q < NSYS; q++) g.c.nst[q] = 0;
    g.lane = threadIdx.x & 31;
    g.warp = 0;
    g.cnt = 0;
    g.jq = 0;
}

// The minor algebra's transposes per gravity setting (ysg_pair_adjoint.cuh).
template <int KIND>
struct SphRev {
    using Solid = RevMinorSolidNC<KIND>;
    using Fluid = RevMinorFluidNC<KIND>;
    using Bvec = RevBvecSolidNC<KIND>;
    static constexpr int NB = 4, NJ = 4, START_SOLID = 4, START_FLUID = 5;
    // sign of the responses: +1 above, -1 below (sph_solver_nc)
    __device__ static double sign(bool up) { return up ? 1.0 : -1.0; }
    __device__ static int jump(int i) { return i; }
    __device__ static void b_start(const cd* m, const cd* s, cd* b) { b_solid_start_ngcow(m, s, b); }
    __device__ static void b_start_T(const cd* m, const cd* w, cd* u) { b_solid_start_T_ngcow(m, w, u); }
    __device__ static void b_start_adj(const cd* s, const cd* bb, cd* mb) { bstart_ngcow_adj(s, bb, mb); }
    __device__ static void det_adj(const cd* a, const cd* b, cd d, cd* ab, cd* bb) { delta_ngcow_adj(a, b, d, ab, bb); }
    __device__ static void to_fluid_adj(const cd* fb, cd* sb) { s2f_ngcow_adj(fb, sb); }
    __device__ static void to_solid_adj(const cd* sb, cd* fb) { f2s_ngcow_adj(sb, fb); }
    __device__ static cd row_dot(const cd* m, int k, const cd* v)
    {
        cd q[4], s = mk(0.0);
        sph_ysol_row_ngcow(m, k, q);
        for (int i = 0; i < 4; i++) s = cmac(s, q[i], v[i]);
        return s;
    }
};
template <>
struct SphRev<2> {
    using Solid = RevMinorSolidG;
    using Fluid = RevMinorFluidG;
    using Bvec = RevBvecSolidG;
    static constexpr int NB = 14, NJ = 6, START_SOLID = 1, START_FLUID = 2;
    __device__ static double sign(bool) { return -1.0; }
    __device__ static int jump(int i) { return i < 2 ? i : i + 1; }
    __device__ static __noinline__ void b_start(const cd* m, const cd* s, cd* b) { b_solid_start(m, s, b); }
    __device__ static __noinline__ void b_start_T(const cd* m, const cd* w, cd* u) { b_solid_start_T(m, w, u); }
    __device__ static __noinline__ void b_start_adj(const cd* s, const cd* bb, cd* mb)
    {
        cd e[14], b[14];
#pragma unroll 1
        for (int j = 0; j < 14; j++) {
            unit(e, 14, j);
            b_solid_start(e, s, b);
            cd t = mb[j];
            for (int k = 0; k < 14; k++) t = cmac(t, bb[k], b[k]);
            mb[j] = t;
        }
    }
    __device__ static __noinline__ void det_adj(const cd* a, const cd* b, cd d, cd* ab, cd* bb)
    {
        cd e[14];
#pragma unroll 1
        for (int j = 0; j < 14; j++) {
            unit(e, 14, j);
            ab[j] = cmac(ab[j], d, delta_solid(e, b));
            bb[j] = cmac(bb[j], d, delta_solid(a, e));
        }
    }
    __device__ static __noinline__ void to_fluid_adj(const cd* fb, cd* sb) { s2f_adj(fb, sb); }
    __device__ static __noinline__ void to_solid_adj(const cd* sb, cd* fb) { f2s_adj(sb, fb); }
    __device__ static __noinline__ cd row_dot(const cd* m, int k, const cd* v)
    {
        cd q[14], s = mk(0.0);
        sph_ysol_row(m, k, q);
        for (int i = 0; i < 14; i++) s = cmac(s, q[i], v[i]);
        return s;
    }
};

template <int KIND, int NL>
using SphAdjMem = AdjMem<NL, KIND == 2 ? 14 : 5, KIND == 2 ? 2 : 0>;

template <int KIND, int NL, int MINB>
__global__ void __launch_bounds__(32 * NL, MINB) k_gadj_sph(AdjArgs a)
{
    using S = SphSys<KIND>;
    using R = SphRev<KIND>;
    using Solid = typename S::Solid;
    using Fluid = typename S::Fluid;
    using Bvec = typename R::Bvec::Sys;
    using Pt = SolidPoint<KIND>;
    using Mem = SphAdjMem<KIND, NL>;
    constexpr int NS = Solid::N, NF = Fluid::N, NB = R::NB;
    const EventDev& ev = *a.ev;
    const GroupLog chain = thread_log(a.w.c, a.w.nthreads), scratch = thread_log(a.w.s, a.w.nthreads);
    Group g;
    adj_group_ctx(g, a);
    for (;;) {
        const unsigned long long it = next_item<Mem>(a.counter);
        if ((long long)it >= a.nitems) break;
        const Item w = item_of(a.ev, a.off, 1, a.order ? a.order[it] : (long long)it, GROUP_SPH0 + KIND, 32 * NL);
        item_ctx(g, ev, w, (int)threadIdx.x);
        const ModelHdr* mh = g.c.mh;
        const Knot* kn = g.c.kn;
        const double rr = ev.rr, rs = ev.rs;
        const int ir = ev.ir, is = ev.is;
        const bool up = rr >= rs, fic = mh->fic != 0;
        const int top = up ? is : ir, l = g.c.ll;
        // adjoints of the coefficients; a pair that does not reach L stays out
        cd cb[10];
        {
            const cd* src = a.coefb + (size_t)(l - ev.lmin) * NCOEF * ev.nw + (w.j - 1);
            bool any = false;
            for (int q = 0; q < 10; q++) {
                cb[q] = src[(size_t)q * ev.nw];
                any = any || cb[q].x != 0.0 || cb[q].y != 0.0;
            }
            g.valid = g.valid && any;
        }
        cd st[NS], ms1[NS], ms2[NS], ms3[NS], mf[NF];
        double rt, rmin;
        int level;
        sph_start<KIND>(g.c, ev, up, &level, &rt, st);
        g.i1 = g.valid ? level : 0x7fffffff;
        g.started = false;
        const int imin = block_min<Mem>(g, g.i1, rt, &rmin);
        if (imin == 0x7fffffff) continue;             // no pair of the block reaches L
        for (int k = 0; k < NS; k++) ms1[k] = mk(0.0);
        for (int k = 0; k < NF; k++) mf[k] = mk(0.0);
        const int nic = mh->nic, noc = mh->noc;
        const bool ic = !fic && imin <= nic, core = imin <= noc;
        // the integrations of the solve, every state logged
        int scale3 = 0, jleg = -1, at[7], n[6];
        bool ok = true;
        at[0] = 0;
#pragma unroll 1
        for (int leg = 0; leg < 6; leg++) {
            n[leg] = 0;
            at[leg + 1] = at[leg];
            if (!ok || (leg == 0 && !ic) || (leg == 1 && !core) || (leg == 3 && !mh->ocean)) continue;
            const Leg q = leg_of(leg, mh, kn, ev, imin, rmin, ic, core, up);
            const bool was = g.started;
            if (leg == 1 || leg == 3) {
                if (leg == 3) {
                    for (int k = 0; k < NF; k++) mf[k] = mk(k == 0 ? 1.0 : 0.0);
                } else if (ic) {
                    S::to_fluid(ms1, mf);
                }
                group_walk<Fluid, FluidPoint<KIND>, false, Mem, true>(g, q.i1, q.i2, q.r1, q.r2, mf, leg == 1 ? st : nullptr,
                                                               &chain, at[leg]);
            } else {
                if (leg == 4 && !mh->ocean)
                    for (int k = 0; k < NS; k++) ms2[k] = mk(k == 0 ? 1.0 : 0.0);
                if (leg == 5)
                    for (int k = 0; k < NS; k++) ms3[k] = ms1[k];
                cd* const y = leg == 5 ? ms3 : (leg == 4 ? ms2 : ms1);
                group_walk<Solid, Pt, false, Mem, true>(g, q.i1, q.i2, q.r1, q.r2, y, leg < 4 ? st : nullptr, &chain,
                                                        at[leg]);
                scale3 = g.scale;
            }
            ok = g.nlog >= 0;
            n[leg] = ok ? g.nlog : 0;
            at[leg + 1] = at[leg] + n[leg];
            if (leg < 3) {
                // lanes whose start is the end of the leg join after its last step
                const bool in = g.started;
                if (leg == 1) group_join_rest<Fluid, Mem>(g, noc, mf, st);
                else group_join_rest<Solid, Mem>(g, leg == 0 ? nic : top, ms1, st);
                if (g.started && !in) g.jq = at[leg + 1];
                if (g.started && !was) jleg = leg;
            }
            if (leg == 1) S::to_solid(mf, ms1);
            if (leg == 3) S::to_solid(mf, ms2);
        }
        const int jq = g.jq;                          // the lane's joining step, in leg jleg
        const cd delta = S::det(ms3, ms2);
        const cd* mq = up ? ms2 : ms1;
        const cd* mb = up ? ms1 : ms2;
        cd yb[3][4], ysph[3][4], ms1b[NS], ms2b[NS], ms3b[NS], deltab = mk(0.0);
        for (int k = 0; k < NS; k++) ms1b[k] = ms2b[k] = ms3b[k] = mk(0.0);
        cd* const mqb = up ? ms2b : ms1b;
        cd* const mbb = up ? ms1b : ms2b;
        spheroidal_resp_adj(g.c, ev, l, g.c.omega, cb, cb + 5, yb);
        const int rows = KIND == 2 ? spheroidal_rows(ev) : 3;
        // Row k of the responses is q_k . Phi b_i / delta (with sign and
        // scale); the adjoint of Phi's transpose applied to q_k is Phi applied
        // to the start vector of the jumps weighted with the row's adjoints.
#pragma unroll 1
        for (int k = 0; k < 3; k++) {
            for (int i = 0; i < 4; i++) ysph[k][i] = mk(0.0);
            if (!ok || k >= S::ROWS || !((rows >> k) & 1)) continue;
            cd s[R::NJ], b[NB], wb[NB], u[R::NJ];
            for (int i = 0; i < R::NJ; i++) s[i] = mk(0.0);
            for (int i = 0; i < 4; i++) s[R::jump(i)] = (R::sign(up) * yb[k][i]) / delta;
            R::b_start(mb, s, b);
            if (!g.valid)
                for (int i = 0; i < NB; i++) b[i] = mk(0.0);
            group_walk<Bvec, Pt, false, Mem, true>(g, is, ir, rs, rr, b, nullptr, &scratch, 0);
            if (g.nlog < 0) {
                ok = false;
                continue;
            }
            const int nbv = g.nlog;
            const double F = huge_pow(scale3 - g.scale);
            // q_k's adjoint F b to the minors it is read from
            for (int j = 0; j < NS; j++) {
                cd e[NS];
                unit(e, NS, j);
                mqb[j] = cmac(mqb[j], F, R::row_dot(e, k, b));
            }
            S::row(mq, k, wb);
            for (int i = 0; i < NB; i++) wb[i] = g.valid ? F * wb[i] : mk(0.0);
            group_rev<typename R::Bvec, Mem>(g, scratch, 0, nbv, is, ir, rs, rr, wb, g.valid, false, nullptr, a.grad);
            R::b_start_adj(s, wb, mbb);
            R::b_start_T(mb, wb, u);
            for (int i = 0; i < 4; i++) {
                const cd ui = u[R::jump(i)];
                ysph[k][i] = (R::sign(up) * ui) / delta;
                deltab = deltab - yb[k][i] * (ysph[k][i] / delta);
            }
        }
        if (!ok) {
            if (threadIdx.x == 0) atomicOr(a.status, 1);
            bsync<Mem>();
            continue;
        }
        R::det_adj(ms3, ms2, deltab, ms3b, ms2b);
        if (!g.valid)
            for (int k = 0; k < NS; k++) ms1b[k] = ms2b[k] = ms3b[k] = mk(0.0);
        // the integrations in reverse: 4 (and 3) from ms2, 5 from ms3, 2 .. 0 the chain
        cd stb[NS], mfb[NF];
        for (int k = 0; k < NS; k++) stb[k] = mk(0.0);
        const int order[6] = {4, 3, 5, 2, 1, 0};
#pragma unroll 1
        for (int o = 0; o < 6; o++) {
            const int leg = order[o];
            if ((leg == 0 && !ic) || (leg == 1 && !core) || (leg == 3 && !mh->ocean)) continue;
            const Leg q = leg_of(leg, mh, kn, ev, imin, rmin, ic, core, up);
            const bool on = g.valid && (leg > 2 || (jleg >= 0 && jleg <= leg));
            const bool joined = leg < 3 && jleg == leg && g.valid;
            g.jq = jq;
            if (leg == 1 || leg == 3) {
                for (int k = 0; k < NF; k++) mfb[k] = mk(0.0);
                R::to_solid_adj(leg == 3 ? ms2b : ms1b, mfb);
                group_rev<typename R::Fluid, Mem>(g, chain, at[leg], n[leg], q.i1, q.i2, q.r1, q.r2, mfb, on, joined,
                                                  stb, a.grad);
                if (leg == 1) {
                    for (int k = 0; k < NS; k++) ms1b[k] = mk(0.0);
                    R::to_fluid_adj(mfb, ms1b);
                }
                continue;
            }
            cd* const y = leg == 4 ? ms2b : (leg == 5 ? ms3b : ms1b);
            group_rev<typename R::Solid, Mem>(g, chain, at[leg], n[leg], q.i1, q.i2, q.r1, q.r2, y, on, joined, stb,
                                              a.grad);
            if (leg == 5)
                for (int k = 0; k < NS; k++) ms1b[k] = ms1b[k] + ms3b[k];
        }
        // start vectors, source vectors and the correction's gravity
        PointGrad<false> gl{a.grad, g.valid};
        if (g.valid) {
            if (jleg == 1 || (fic && level <= noc)) start_adj<R::START_FLUID>(g.c, a.u, level, rt, stb, gl);
            else start_adj<R::START_SOLID>(g.c, a.u, level, rt, stb, gl);
        }
        __syncwarp();
        PointGrad<true> gu{a.grad, g.valid};
        spheroidal_rest_adj(g.c, a.u, ev, l, g.c.omega, cb, cb + 5, ysph, gu);
        bsync<Mem>();
    }
}

// ---------------------------------------------------------------------------
// Toroidal pairs (tor_solver_adj of ysg_pair_adjoint.cuh).
// ---------------------------------------------------------------------------
template <int NL>
using TorAdjMem = AdjMem<NL, 2, 0>;

template <int NL, int MINB>
__global__ void __launch_bounds__(32 * NL, MINB) k_gadj_tor(AdjArgs a)
{
    using Mem = TorAdjMem<NL>;
    const EventDev& ev = *a.ev;
    const GroupLog chain = thread_log(a.w.c, a.w.nthreads), scratch = thread_log(a.w.s, a.w.nthreads);
    Group g;
    adj_group_ctx(g, a);
    for (;;) {
        const unsigned long long it = next_item<Mem>(a.counter);
        if ((long long)it >= a.nitems) break;
        const Item w = item_of(a.ev, a.off, 1, a.order ? a.order[it] : (long long)it, GROUP_TOR, 32 * NL);
        item_ctx(g, ev, w, (int)threadIdx.x);
        const int l = g.c.ll;
        const ModelHdr* mh = g.c.mh;
        const Knot* kn = g.c.kn;
        const double rr = ev.rr, rs = ev.rs;
        const int ir = ev.ir, is = ev.is;
        const bool up = rr >= rs;
        const int top = up ? is : ir;
        cd cb[5];
        {
            const cd* src = a.coefb + ((size_t)(l - ev.lmin) * NCOEF + 10) * ev.nw + (w.j - 1);
            bool any = false;
            for (int q = 0; q < 5; q++) {
                cb[q] = src[(size_t)q * ev.nw];
                any = any || cb[q].x != 0.0 || cb[q].y != 0.0;
            }
            g.valid = g.valid && any;
        }
        int i1 = tor_start_level(g.c, l, g.c.omega.x, top);
        if (i1 == top && i1 > mh->noc + 1) i1 = i1 - 1;
        const bool cmb = i1 == mh->noc + 1;
        cd s[2], yb[2][2], ytor[2][2];
        if (cmb) { s[0] = mk(1.0); s[1] = mk(0.0); }
        else tor_ystart(g.c, i1, kn[i1].r, s);
        g.i1 = g.valid ? i1 : 0x7fffffff;
        g.started = false;
        double rmin;
        const int imin = block_min<Mem>(g, g.i1, kn[i1].r, &rmin);
        if (imin == 0x7fffffff) continue;
        toroidal_resp_adj(g.c, ev, l, g.c.omega, cb, yb);
        // y1 to the source (or a receiver below it), y2 from the surface, y3
        // the source-side one continued: logged one after the other
        cd y1[2] = {mk(0.0), mk(0.0)}, y2[2] = {mk(1.0), mk(0.0)}, y3[2];
        const double rbot = up ? rr : rs, rlow = up ? rs : rr;
        const int ibot = up ? ir : is;
        const bool down = rbot != kn[mh->nsl].r;
        int n1 = 0, n2 = 0, n3 = 0;
        group_walk<TorSys, TorPoint, false, Mem, true>(g, imin, top, rmin, rlow, y1, s, &chain, 0);
        n1 = g.nlog;
        {
            const bool in = g.started;
            group_join_rest<TorSys, Mem>(g, top, y1, s);
            if (g.started && !in) g.jq = max(n1, 0);
        }
        const int jq = g.jq;
        bool ok = n1 >= 0;
        if (ok && down) {
            group_walk<TorSys, TorPoint, false, Mem, true>(g, mh->nsl - 1, ibot, kn[mh->nsl].r, rbot, y2, nullptr, &chain, n1);
            n2 = g.nlog;
            ok = n2 >= 0;
        }
        y3[0] = up ? y1[0] : y2[0];
        y3[1] = up ? y1[1] : y2[1];
        int scale3 = 0;
        if (ok) {
            group_walk<TorSys, TorPoint, false, Mem, true>(g, is, ir, rs, rr, y3, nullptr, &scratch, 0);
            n3 = g.nlog;
            scale3 = g.scale;
            ok = n3 >= 0;
        }
        if (!ok) {
            if (threadIdx.x == 0) atomicOr(a.status, 1);
            bsync<Mem>();
            continue;
        }
        // D = P[1] Q[0] - P[0] Q[1]: (P, Q) = (y2, y3) above, (y3, y1) below
        const cd* P = up ? y2 : y3;
        const cd* Q = up ? y3 : y1;
        const cd D = P[1] * Q[0] - P[0] * Q[1];
        const cd delta = 1.0 / D;
        const cd* Bs = up ? y1 : y2;
        const cd* Rv = up ? y2 : y1;
        const cd bv[2] = {Bs[1], -Bs[0]};
        const cd dy[2] = {delta * Rv[0], delta * Rv[1]};
        const double F = huge_pow(scale3);
        cd dyb[2] = {mk(0.0), mk(0.0)}, bvb[2] = {mk(0.0), mk(0.0)};
        for (int p = 0; p < 2; p++)
            for (int b = 0; b < 2; b++) {
                ytor[p][b] = F * (-(dy[p] * bv[b]));
                const cd gq = F * yb[p][b];
                dyb[p] = dyb[p] - gq * bv[b];
                bvb[b] = bvb[b] - gq * dy[p];
            }
        cd y1b[2] = {mk(0.0), mk(0.0)}, y2b[2] = {mk(0.0), mk(0.0)}, y3b[2] = {mk(0.0), mk(0.0)};
        cd* Bsb = up ? y1b : y2b;
        cd* Rb = up ? y2b : y1b;
        cd* Pb = up ? y2b : y3b;
        cd* Qb = up ? y3b : y1b;
        Bsb[1] = Bsb[1] + bvb[0];
        Bsb[0] = Bsb[0] - bvb[1];
        const cd deltab = dyb[0] * Rv[0] + dyb[1] * Rv[1];
        Rb[0] = Rb[0] + delta * dyb[0];
        Rb[1] = Rb[1] + delta * dyb[1];
        const cd Db = -(deltab * (delta * delta));
        Pb[1] = Pb[1] + Db * Q[0];
        Pb[0] = Pb[0] - Db * Q[1];
        Qb[0] = Qb[0] + Db * P[1];
        Qb[1] = Qb[1] - Db * P[0];
        if (!g.valid)
            for (int k = 0; k < 2; k++) y1b[k] = y2b[k] = y3b[k] = mk(0.0);
        group_rev<RevTor, Mem>(g, scratch, 0, n3, is, ir, rs, rr, y3b, g.valid, false, nullptr, a.grad);
        cd* y3sb = up ? y1b : y2b;
        y3sb[0] = y3sb[0] + y3b[0];
        y3sb[1] = y3sb[1] + y3b[1];
        group_rev<RevTor, Mem>(g, chain, n1, n2, mh->nsl - 1, ibot, kn[mh->nsl].r, rbot, y2b, g.valid, false, nullptr,
                               a.grad);
        cd stb[2] = {mk(0.0), mk(0.0)};
        g.jq = jq;
        group_rev<RevTor, Mem>(g, chain, 0, n1, imin, top, rmin, rlow, y1b, g.valid, g.valid, stb, a.grad);
        PointGrad<false> gl{a.grad, g.valid};
        if (g.valid && !cmb) start_adj<0>(g.c, a.u, i1, kn[i1].r, stb, gl);
        __syncwarp();
        PointGrad<true> gu{a.grad, g.valid};
        toroidal_rest_adj(g.c, a.u, ev, l, g.c.omega, cb, ytor, gu);
        bsync<Mem>();
    }
}

// ---------------------------------------------------------------------------
// l = 0 (pair_radial_adj of ysg_pair_adjoint.cuh), a warp per frequency.
// ---------------------------------------------------------------------------
// Grid log of a frequency: per point its radius, interval, and the upward
// and downward solutions there; per step of the no-gravity walks its state,
// radius, size, interval and rescaling factor in the same arrays.
struct RadLog {
    cd* y;                        // gmax x 4
    double* r;                    // gmax
    int* i;                       // gmax
    int gmax;
};

// The adjoints of the pieces of a batch: y the adjoint of the last piece's
// result (pieces in reverse order), carried through the transposed
// matrices; the lane keeps the adjoint of its own piece's result.
__device__ __forceinline__ void rad_scan_T(RadMem& M, const RadMat& m, int lane, int n, cd* y, cd* own, int add,
                                           const cd* yadd)
{
    __syncwarp();
    M.m[lane] = m;
    __syncwarp();
    own[0] = own[1] = mk(0.0);
    for (int t = 0; t < n; t++) {
        if (t == add) {
            y[0] = y[0] + yadd[0];
            y[1] = y[1] + yadd[1];
        }
        if (lane == t) {
            own[0] = y[0];
            own[1] = y[1];
        }
        rad_apply_T(M.m[t], y);
    }
}

__device__ __noinline__ bool rad_wg_adj_warp(Ctx& c, const UnitDirs& u, RadMem& M, int lane, double rr, double rs,
                                             const cd* yb, cd* yout, const RadLog& GL, StepLog& L, SegGrad& G)
{
    const RadGrid g = rad_grid(c, rr, rs, M.pre, lane);
    const int iss = g.iss, irr = g.irr, ngrid = g.ngrid;
    if (ngrid + 1 > GL.gmax || iss < 2 || irr < 2) return false;
    unsigned nst = 0;
    cd own[2], ys[2] = {mk(0.0), mk(0.0)}, y1[2] = {mk(0.0), mk(0.0)}, y2[2] = {mk(1.0), mk(0.0)};
    double rt = 0.0;
    for (int k = 1 + lane; k <= ngrid; k += 32) {
        int iv;
        double r;
        rad_point(g, k, &iv, &r);
        GL.r[k] = r;
        GL.i[k] = iv;
    }
    __syncwarp();
    // upward through the points 2 .. iss
    for (int k0 = 2; k0 <= iss; k0 += 32) {
        const int k = k0 + lane, nb = min(32, iss - k0 + 1);
        RadMat m{mk(1.0), mk(0.0), mk(0.0), mk(1.0)};
        if (k0 == 2) {
            rt = fmin(0.1 * g.drr, 0.1 * GL.r[2]);
            rad_ystart<true>(c, 1, rt, ys);
            y1[0] = ys[0];
            y1[1] = ys[1];
        }
        if (lane < nb) m = rad_piece(c, k == 2 ? 1 : GL.i[k - 1], GL.i[k], k == 2 ? rt : GL.r[k - 1], GL.r[k], &nst);
        rad_scan(M, m, lane, nb, y1, own);
        if (lane < nb) {
            GL.y[4 * (size_t)k] = own[0];
            GL.y[4 * (size_t)k + 1] = own[1];
        }
    }
    // downward from point ngrid to iss
    if (lane == 0) {
        GL.y[4 * (size_t)ngrid + 2] = y2[0];
        GL.y[4 * (size_t)ngrid + 3] = y2[1];
    }
    for (int k0 = ngrid - 1; k0 >= iss; k0 -= 32) {
        const int k = k0 - lane, nb = min(32, k0 - iss + 1);
        RadMat m{mk(1.0), mk(0.0), mk(0.0), mk(1.0)};
        if (lane < nb) m = rad_piece(c, GL.i[k + 1], GL.i[k], GL.r[k + 1], GL.r[k], &nst);
        rad_scan(M, m, lane, nb, y2, own);
        if (lane < nb) {
            GL.y[4 * (size_t)k + 2] = own[0];
            GL.y[4 * (size_t)k + 3] = own[1];
        }
    }
    __syncwarp();
    const bool rec_up = irr <= iss;               // receiver on the upward walk
    const cd yrec[2] = {GL.y[4 * (size_t)irr + (rec_up ? 0 : 2)], GL.y[4 * (size_t)irr + (rec_up ? 1 : 3)]};
    const cd D = y2[1] * y1[0] - y2[0] * y1[1];
    const cd delta = 1.0 / D;
    const cd* Y = rec_up ? y2 : y1;
    const cd bv[2] = {Y[1], -Y[0]};
    const cd dy0 = delta * yrec[0];
    // yout[b] = -delta yrec[0] bv[b], the first row of the responses; yb its adjoints
    cd dyb = mk(0.0), bvb[2];
    for (int b = 0; b < 2; b++) {
        yout[b] = -(dy0 * bv[b]);
        dyb = dyb - yb[b] * bv[b];
        bvb[b] = -(yb[b] * dy0);
    }
    const cd deltab = dyb * yrec[0];
    const cd yrecb[2] = {dyb * delta, mk(0.0)};
    const cd Db = -(deltab * (delta * delta));
    cd y1b[2] = {Db * y2[1], -(Db * y2[0])};
    cd y2b[2] = {-(Db * y1[1]), Db * y1[0]};
    cd* Yb = rec_up ? y2b : y1b;
    Yb[1] = Yb[1] + bvb[0];
    Yb[0] = Yb[0] - bvb[1];
    bool ok = true;
    // the downward walk reversed: y2(k) = piece(k + 1 -> k) y2(k + 1)
    for (int k0 = iss; k0 < ngrid; k0 += 32) {
        const int k = k0 + lane, nb = min(32, ngrid - k0);
        RadMat m{mk(1.0), mk(0.0), mk(0.0), mk(1.0)};
        if (lane < nb) m = rad_piece(c, GL.i[k + 1], GL.i[k], GL.r[k + 1], GL.r[k], &nst);
        rad_scan_T(M, m, lane, nb, y2b, own, rec_up ? -1 : irr - k0, yrecb);
        if (lane < nb) {
            const cd yin[2] = {GL.y[4 * (size_t)(k + 1) + 2], GL.y[4 * (size_t)(k + 1) + 3]};
            ok = yint_adj<RadT>(c, GL.i[k + 1], GL.i[k], GL.r[k + 1], GL.r[k], yin, own, false, L, G) && ok;
        }
    }
    // the upward walk reversed: y1(k) = piece(k - 1 -> k) y1(k - 1), y1(2) from the start
    for (int k0 = iss; k0 >= 2; k0 -= 32) {
        const int k = k0 - lane, nb = min(32, k0 - 1);
        RadMat m{mk(1.0), mk(0.0), mk(0.0), mk(1.0)};
        if (lane < nb) m = rad_piece(c, k == 2 ? 1 : GL.i[k - 1], GL.i[k], k == 2 ? rt : GL.r[k - 1], GL.r[k], &nst);
        rad_scan_T(M, m, lane, nb, y1b, own, rec_up ? k0 - irr : -1, yrecb);
        if (lane < nb) {
            const cd yin[2] = {k == 2 ? ys[0] : GL.y[4 * (size_t)(k - 1)], k == 2 ? ys[1] : GL.y[4 * (size_t)(k - 1) + 1]};
            ok = yint_adj<RadT>(c, k == 2 ? 1 : GL.i[k - 1], GL.i[k], k == 2 ? rt : GL.r[k - 1], GL.r[k], yin, own, false,
                                L, G) && ok;
        }
    }
    if (lane == 0) start_adj<3>(c, u, 1, rt, y1b, G);
    __syncwarp();
    return __all_sync(FULL, ok);
}

// rad_walk with every step logged from entry `at` on; returns the steps, -1
// if they exceed the log.
__device__ __noinline__ int rad_walk_log(Ctx& c, RadMem& M, int lane, int i1, int i2, double r1, double r2, cd* y,
                                         int* scale, const RadLog& GL, int at)
{
    Walk w;
    walk_init(w, i1, i2, r1, r2, false);
    int q = at;
    while (walk_chunk(c, lane, w)) {
        const int nb = min(32, w.total - w.s0);
        if (q + nb > GL.gmax) return -1;
        int iv;
        double x, h;
        walk_step(w, w.s0 + lane, &iv, &x, &h);
        RadMat m{mk(1.0), mk(0.0), mk(0.0), mk(1.0)};
        if (lane < nb) rad_step(c, iv, x, h, m);
        __syncwarp();
        M.m[lane] = m;
        __syncwarp();
        cd own[2] = {y[0], y[1]};
        double f = 1.0;
        for (int t = 0; t < nb; t++) {
            if (lane == t) {
                own[0] = y[0];
                own[1] = y[1];
            }
            rad_apply(M.m[t], y);
            int sc = 0;
            rescale<2>(y, &sc);
            *scale += sc;
            if (lane == t) f = sc > 0 ? SC_HUGE : (sc < 0 ? SC_TINY : 1.0);
        }
        if (lane < nb) {
            const size_t e = (size_t)(q + lane);
            GL.y[4 * e] = own[0];
            GL.y[4 * e + 1] = own[1];
            GL.y[4 * e + 2] = mk(f, h);
            GL.r[e] = x;
            GL.i[e] = iv;
        }
        w.s0 += nb;
        q += nb;
    }
    __syncwarp();
    return q - at;
}

// The reverse of n logged steps: y the adjoint of the result on entry, of
// the start on exit.
__device__ __noinline__ void rad_walk_rev(Ctx& c, RadMem& M, int lane, const RadLog& GL, int at, int n, cd* y, SegGrad& G)
{
    for (int q0 = at + n - 1; q0 >= at; q0 -= 32) {
        const int nb = min(32, q0 - at + 1);
        const size_t e = (size_t)(q0 - lane);
        RadMat m{mk(1.0), mk(0.0), mk(0.0), mk(1.0)};
        double f = 1.0, x = 0.0, h = 0.0;
        int iv = 1;
        if (lane < nb) {
            const cd fh = GL.y[4 * e + 2];
            f = fh.x;
            h = fh.y;
            x = GL.r[e];
            iv = GL.i[e];
            rad_step(c, iv, x, h, m);
            m = RadMat{f * m.a, f * m.b, f * m.c, f * m.d};
        }
        cd own[2];
        rad_scan_T(M, m, lane, nb, y, own, -1, nullptr);
        if (lane < nb) {
            const cd yin[2] = {GL.y[4 * e], GL.y[4 * e + 1]};
            own[0] = f * own[0];
            own[1] = f * own[1];
            c.il = iv;
            rk_step_adj<RadT>(c, yin, x, h, own, G);
        }
    }
}

__device__ __noinline__ bool rad_ng_adj_warp(Ctx& c, const UnitDirs& u, RadMem& M, int lane, double rr, double rs,
                                             int ir, int is, const cd* yb, cd* yout, const RadLog& GL, SegGrad& G)
{
    const ModelHdr* mh = c.mh;
    const Knot* kn = c.kn;
    const bool up = rr >= rs;
    int sc1 = 0, sc2 = 0, sc3 = 0;
    const double rt = fmin(0.1 * c.dr, 0.1 * kn[2].r);
    cd y1[2], y2[2] = {mk(1.0), mk(0.0)}, y3[2];
    rad_ystart<false>(c, 1, rt, y1);
    const int ilo = up ? is : ir, ihi = up ? ir : is, top = up ? mh->nknot : mh->nsl;
    const double rlo = up ? rs : rr, rhi = up ? rr : rs;
    const int n1 = rad_walk_log(c, M, lane, 1, ilo, rt, rlo, y1, &sc1, GL, 0);
    if (n1 < 0) return false;
    const int n2 = rad_walk_log(c, M, lane, top - 1, ihi, kn[top].r, rhi, y2, &sc2, GL, n1);
    if (n2 < 0) return false;
    y3[0] = y2[0];
    y3[1] = y2[1];
    const int n3 = rad_walk_log(c, M, lane, ihi, ilo, rhi, rlo, y3, &sc3, GL, n1 + n2);
    if (n3 < 0) return false;
    const cd D = y3[1] * y1[0] - y3[0] * y1[1];
    const bool degenerate = cabs(D) < 1.0e-100;
    const cd delta = degenerate ? mk(0.0) : 1.0 / D;
    const cd* ya = up ? y1 : y2;                  // forms b
    const cd* yr = up ? y2 : y1;                  // read at the receiver
    const cd bv[2] = {ya[1], -ya[0]};
    const cd dy0 = delta * yr[0];
    const double F = (up ? sc3 != 0 : sc3 > 0) ? huge_pow(sc3) : 1.0;
    cd dyb = mk(0.0), bvb[2];
    for (int b = 0; b < 2; b++) {
        yout[b] = F * (-(dy0 * bv[b]));
        const cd gq = F * yb[b];
        dyb = dyb - gq * bv[b];
        bvb[b] = -(gq * dy0);
    }
    const cd yab[2] = {-bvb[1], bvb[0]};
    const cd deltab = dyb * yr[0];
    const cd yrb[2] = {delta * dyb, mk(0.0)};
    cd y1b[2], y2b[2], y3b[2] = {mk(0.0), mk(0.0)};
    for (int k = 0; k < 2; k++) {
        y1b[k] = up ? yab[k] : yrb[k];
        y2b[k] = up ? yrb[k] : yab[k];
    }
    if (!degenerate) {
        const cd Db = -(deltab * (delta * delta));
        y3b[0] = -(Db * y1[1]);
        y3b[1] = Db * y1[0];
        y1b[0] = y1b[0] + Db * y3[1];
        y1b[1] = y1b[1] - Db * y3[0];
    }
    rad_walk_rev(c, M, lane, GL, n1 + n2, n3, y3b, G);
    y2b[0] = y2b[0] + y3b[0];
    y2b[1] = y2b[1] + y3b[1];
    rad_walk_rev(c, M, lane, GL, n1, n2, y2b, G);
    rad_walk_rev(c, M, lane, GL, 0, n1, y1b, G);
    if (lane == 0) start_adj<6>(c, u, 1, rt, y1b, G);
    __syncwarp();
    return true;
}

// Block b: frequency nw - b.  GL: the frequencies' grid logs one after the
// other; ws: step logs of the lanes' pieces (a few steps each).
__global__ void __launch_bounds__(32) k_gadj_rad(AdjArgs a, RadLog GL, AdjStepArrays ws)
{
    __shared__ RadMem M;
    const int lane = threadIdx.x;
    const EventDev& ev = *a.ev;
    const int j = ev.nw - (int)blockIdx.x;
    const size_t g0 = (size_t)blockIdx.x * GL.gmax;
    GL.y += 4 * g0;
    GL.r += g0;
    GL.i += g0;
    const size_t t = (size_t)blockIdx.x * 32 + lane;
    StepLog L{ws.y + t, ws.x + t, ws.h + t, ws.il + t, ws.f + t, ws.n, (int)(gridDim.x * 32)};
    Group g;
    adj_group_ctx(g, a);
    Ctx& c = g.c;
    c.ats = (double)ev.ats;
    set_l(c, 0);
    set_omega(c, omega_of(ev, j));
    alpha_steps(c);
    // u3 = f (sr0[0] yrad[0] + sr0[1] yrad[1]) / rr
    cd gq = a.coefb[2 * (size_t)ev.nw + (j - 1)];
    if (gq.x == 0.0 && gq.y == 0.0) return;
    if (ev.out != 0) gq = out_factor(ev.out, c.omega) * gq;
    gq = gq / ev.rr;
    cd sr0[2], yout[2];
    source_vector_rad(c, ev.is, ev.rs, ev.mm, sr0);
    const cd yb[2] = {gq * sr0[0], gq * sr0[1]};
    SegGrad G;
    G.init(a.grad);
    const bool ok = ev.grav == 0
                        ? rad_ng_adj_warp(c, a.u, M, lane, ev.rr, ev.rs, ev.ir, ev.is, yb, yout, GL, G)
                        : rad_wg_adj_warp(c, a.u, M, lane, ev.rr, ev.rs, yb, yout, GL, L, G);
    if (!ok) {
        if (lane == 0) atomicOr(a.status, 1);
        return;
    }
    if (lane == 0) {
        const cd s0b[2] = {gq * yout[0], gq * yout[1]};
        source_rad_adj(c, a.u, ev.is, ev.rs, ev.mm, s0b, G);
    }
    G.flush();
}

using AdjFn = void (*)(AdjArgs);
struct AdjKernel {
    AdjFn f;
    int threads;
    size_t smem;
    int width;
    int states;                   // components of a logged state
};
template <class Mem>
AdjKernel adj_kernel_of(AdjFn f)
{
    return {f, Mem::NT, sizeof(Mem), 32 * Mem::NL, Mem::LOG_N};
}
AdjKernel adj_kernel(int kind)
{
    switch (kind) {
        case GROUP_SPH2: return adj_kernel_of<SphAdjMem<2, GADJ_NL>>(k_gadj_sph<2, GADJ_NL, 8 / GADJ_NL>);
        case GROUP_SPH1: return adj_kernel_of<SphAdjMem<1, GADJ_NL>>(k_gadj_sph<1, GADJ_NL, 8 / GADJ_NL>);
        case GROUP_SPH0: return adj_kernel_of<SphAdjMem<0, GADJ_NL>>(k_gadj_sph<0, GADJ_NL, 8 / GADJ_NL>);
        default: return adj_kernel_of<TorAdjMem<GADJ_NL>>(k_gadj_tor<GADJ_NL, 16 / GADJ_NL>);
    }
}

}  // namespace
}  // inline namespace

int group_adj_width(int kind) { return adj_kernel(kind).width; }

int group_adj_threads(int kind) { return adj_kernel(kind).threads; }

int group_adj_states(int kind) { return adj_kernel(kind).states; }

int group_adj_blocks(int kind)
{
    int dev = 0, nsm = 0, per = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
        return 0;
    const AdjKernel k = adj_kernel(kind);
    if (cudaFuncSetAttribute(k.f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)k.smem) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k.f, k.threads, k.smem) != cudaSuccess)
        return 0;
    return nsm * std::max(per, 1);
}

cudaError_t launch_group_adj(int kind, const Knot* kn, const Seg* sg, const ModelHdr* mh, const EventDev* ev,
                             const UnitDirs& u, const cd* coefb, const long long* off, long long nitems,
                             const double* tt, void* order_buf, const AdjLogs& w, double* grad,
                             unsigned long long* counter, int* status, int nblk, int* launched, cudaStream_t st)
{
    *launched = 0;
    if (nitems <= 0) return cudaSuccess;
    const AdjKernel k = adj_kernel(kind);
    AdjArgs a{kn, sg, mh, ev, u, coefb, off, nullptr, nitems, w, grad, counter, status};
    cudaError_t e = cudaMemsetAsync(counter, 0, sizeof *counter, st);
    if (e != cudaSuccess) return e;
    if (nitems > nblk) {
        e = launch_group_order(kind, k.width, kn, mh, ev, off, 1, nitems, tt, order_buf, &a.order, st);
        if (e != cudaSuccess) return e;
        *launched += 2;
    }
    k.f<<<(unsigned)std::min<long long>(nitems, nblk), k.threads, k.smem, st>>>(a);
    *launched += 1;
    return cudaGetLastError();
}

cudaError_t launch_group_adj_rad(const Knot* kn, const Seg* sg, const ModelHdr* mh, const EventDev* ev,
                                 const UnitDirs& u, const cd* coefb, int nw, cd* gy, double* gr, int* gi, int gmax,
                                 const AdjStepArrays& ws, double* grad, int* status, cudaStream_t st)
{
    AdjArgs a{kn, sg, mh, ev, u, coefb, nullptr, nullptr, nw, AdjLogs{}, grad, nullptr, status};
    k_gadj_rad<<<(unsigned)nw, 32, 0, st>>>(a, RadLog{gy, gr, gi, gmax}, ws);
    return cudaGetLastError();
}

}  // namespace ysg
