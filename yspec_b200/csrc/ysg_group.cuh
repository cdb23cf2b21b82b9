// ysg_group.cuh -- radial integrations of many degrees of one frequency at once.
//
// The step sequence of yint (module_int.f90:1847-1968) -- knot intervals,
// steps per interval, radii -- depends on omega and on the radius where a
// solve starts, not on l.  So consecutive degrees of one frequency walk the
// same radii together, one lane each: the walk runs from the deepest start
// of the group, and a lane joins it at its own start level.  What this buys
// over one independent walk per thread:
//   - the coefficient matrices split into parts that depend on (r, omega)
//     alone, with the spline evaluations and the division, and a few
//     products with zeta or l per lane.  The first parts ("points") of the
//     next SB steps x 6 stages are evaluated one per thread and shared
//     through shared memory, 1/32 or 1/128 of an evaluation per lane and
//     stage, where they were a third of a step's instructions;
//   - there is no divergence between the lanes of a group but before the
//     lanes' own starts;
//   - the warps of a block run the same code at nearly the same place, which
//     the instruction cache needs (k_solve_group.cu);
//   - or the components of a system are split between the warps of a block:
//     a warp holds the stage vectors of its own components in registers, and
//     the warps exchange the stage inputs through shared memory, one barrier
//     per stage, so that a step takes less time where there are too few
//     pairs to fill the GPU.
// The step itself keeps y, the stage input and the derivative in registers
// and two partial sums in shared memory or registers: 154 shared-memory
// accesses per lane and step of a 14-component system, where four slots with
// folds (rkck_step_loop of ysg_ode.cuh) take 420.
// Every integer decision (start levels, step counts) is formed by the same
// rounded operations as in ysg_ode.cuh.
#pragma once
#include "ysg_solvers.cuh"

namespace ysg {
inline namespace YSG_VARIANT {
namespace {

constexpr int PT = 20;            // doubles per point
constexpr unsigned FULL = 0xffffffffu;

// ---------------------------------------------------------------------------
// Points: the l-independent parts of the coefficient matrices at (r, omega)
// (solid_amat, fluid_amat and tor_amat of ysg_ode.cuh, factored).
// ---------------------------------------------------------------------------
__device__ __forceinline__ void put(double* o, int k, cd v)
{
    reinterpret_cast<cd*>(o)[k] = v;
}
__device__ __forceinline__ cd got(const double* o, int k) { return reinterpret_cast<const cd*>(o)[k]; }

// t11 | t12/zeta | s11 | s12/zeta | s22 = [4] + zeta^2 [5] | k11 | k22 | ri, rho ri | t31
template <int KIND>
struct SolidPoint {
    __device__ static __forceinline__ void eval(const Ctx& c, int il, double rr, double* o)
    {
        const Seg& g = c.sg[il];
        const double u = rr - g.r0;
        const double rrho = seg(g, u, P_RHO), racon = seg(g, u, P_ACON), rccon = seg(g, u, P_CCON);
        const double rfcon = seg(g, u, P_FCON), rncon = seg(g, u, P_NCON), rlcon = seg(g, u, P_LCON);
        const double rqmu = seg(g, u, P_QMU), rxlam = seg(g, u, P_XLAM), rxa2 = seg(g, u, P_XA2);
        const cd qaa = 1.0 + rxa2 * c.lno, qff = 1.0 + rxlam * c.lno, qll = 1.0 + rqmu * c.lno;
        const cd cacon = racon * qaa, cfcon = rfcon * qff, cncon = rncon * qll;
        const double dc = rccon * norm2(qaa), dl = rlcon * norm2(qll);
        const double inv = 1.0 / (rr * (dc * dl));
        const cd cccon = conj(qaa) * ((rr * dl) * inv);
        const cd fc = cfcon * cccon;
        const cd gamma = cmsc(cacon - cncon, cfcon, fc);
        const double ri = (dc * dl) * inv, ri2 = ri * ri;
        const cd mw2r = -(c.omega2 * rrho);
        put(o, 0, (1.0 - 2.0 * fc) * ri);
        put(o, 1, ri * fc);
        if (KIND == 0) {
            put(o, 2, mw2r + (4.0 * gamma) * ri2);
            put(o, 3, (-2.0 * gamma) * ri2);
        } else {
            const double rgr = rrho * seg(g, u, P_GRAV) * rr;
            put(o, 2, mw2r + (4.0 * (gamma - rgr)) * ri2);
            put(o, 3, (rgr - 2.0 * gamma) * ri2);
        }
        put(o, 4, mw2r - (2.0 * cncon) * ri2);
        put(o, 5, (gamma + cncon) * ri2);
        put(o, 6, cccon);
        put(o, 7, conj(qll) * ((rr * dc) * inv));
        put(o, 8, mk(ri, rrho * ri));
        o[18] = -(4.0 * c.pib * rrho);
    }
};

// cccon | omega^-2 ri^2 | -omega^2 rho (- 4 rho g ri with gravity) | ri, rho | g (0 without), 1/rho.
// Without gravity no gravity term enters the third number: adding it here and
// taking it out per lane would lose the digits it is larger by (at 0.1 mHz
// some 30 times omega^2 rho).
template <int KIND>
struct FluidPoint {
    __device__ static __forceinline__ void eval(const Ctx& c, int il, double rr, double* o)
    {
        const Seg& g = c.sg[il];
        const double u = rr - g.r0;
        const double rrho = seg(g, u, P_RHO), rccon = seg(g, u, P_CCON), rxa2 = seg(g, u, P_XA2);
        const cd qaa = 1.0 + rxa2 * c.lno;
        const double dc = rccon * norm2(qaa);
        const double inv = 1.0 / (rr * rrho * dc);
        const double ri = (rrho * dc) * inv;
        double gg = 0.0;
        cd s = -(c.omega2 * rrho);
        if (KIND != 0) {
            gg = seg(g, u, P_GRAV);
            s = s - 4.0 * (rrho * gg * ri);
        }
        put(o, 0, conj(qaa) * ((rr * rrho) * inv));
        put(o, 1, c.omegai2 * (ri * ri));
        put(o, 2, s);
        put(o, 3, mk(ri, rrho));
        put(o, 4, mk(gg, (rr * dc) * inv));
    }
};

// k | -omega^2 rho | ri^2 N (1 + qmu lno) | ri
struct TorPoint {
    __device__ static __forceinline__ void eval(const Ctx& c, int il, double rr, double* o)
    {
        const Seg& g = c.sg[il];
        const double u = rr - g.r0;
        const double rrho = seg(g, u, P_RHO), rlcon = seg(g, u, P_LCON);
        const double rncon = seg(g, u, P_NCON), rqmu = seg(g, u, P_QMU);
        const cd qll = 1.0 + rqmu * c.lno;
        const double dl = rlcon * norm2(qll);
        const double inv = 1.0 / (rr * dl);
        const double ri = dl * inv;
        put(o, 0, conj(qll) * (rr * inv));
        put(o, 1, -(c.omega2 * rrho));
        put(o, 2, (ri * ri) * (rncon * qll));
        o[6] = ri;
    }
};

// A lane's coefficient matrices from a point: the context type the
// right-hand sides of ysg_ode.cuh are run with here.
struct LaneCtx {
    const double* p;              // point in shared memory
    double zeta, zeta2, fl, flp1, pib4;
};

template <int KIND>
__device__ __forceinline__ SolidCoef solid_amat(const LaneCtx& c, double)
{
    SolidCoef a;
    const cd rr = got(c.p, 8);                     // ri, rho ri
    a.t11 = got(c.p, 0);
    a.t12 = c.zeta * got(c.p, 1);
    a.t21 = -(c.zeta * rr.x);
    a.t22 = 2.0 * rr.x;
    a.s11 = got(c.p, 2);
    a.s12 = c.zeta * got(c.p, 3);
    a.s22 = cmac(got(c.p, 4), c.zeta2, got(c.p, 5));
    a.k11 = got(c.p, 6);
    a.k22 = got(c.p, 7);
    if (KIND == 2) {
        a.t31 = c.p[18];
        a.t33 = -(c.fl * rr.x);
        a.k33 = c.pib4;
        a.s13 = -(c.flp1 * rr.y);
        a.s23 = c.zeta * rr.y;
    } else {
        a.t31 = a.t33 = a.k33 = a.s13 = a.s23 = 0.0;
    }
    return a;
}

template <int KIND>
__device__ __forceinline__ FluidCoef fluid_amat(const LaneCtx& c, double)
{
    FluidCoef a;
    const cd z = c.zeta2 * got(c.p, 1);            // zeta^2 omega^-2 ri^2
    const cd rr = got(c.p, 3), gr = got(c.p, 4);   // ri, rho; g, 1/rho
    a.k11 = cmsc(got(c.p, 0), gr.y, z);
    a.t12 = a.s12 = a.s22 = mk(0.0);
    a.t21 = a.t22 = a.k22 = 0.0;
    if (KIND == 0) {
        a.t11 = mk(-rr.x);
        a.s11 = got(c.p, 2);
        return a;
    }
    const cd gz = gr.x * z;
    a.t11 = gz - rr.x;
    a.s11 = cmac(got(c.p, 2), rr.y * gr.x, gz);
    if (KIND == 2) {
        a.t12 = z;
        a.t21 = -(c.pib4 * rr.y);
        a.t22 = -(c.fl * rr.x);
        a.k22 = c.pib4;
        a.s12 = rr.y * (gz - c.flp1 * rr.x);
        a.s22 = rr.y * z;
    }
    return a;
}

__device__ __forceinline__ TorCoef tor_amat(const LaneCtx& c, double)
{
    TorCoef a;
    a.t = 2.0 * c.p[6];
    a.k = got(c.p, 0);
    a.s = cmac(got(c.p, 1), c.zeta2 - 2.0, got(c.p, 2));
    return a;
}

// ---------------------------------------------------------------------------
// A group is a block.  Its warps hold either the components of the same 32
// degrees (NW warps, NL = 1) or 32 degrees each (NL warps, NW = 1).
// ---------------------------------------------------------------------------
// Its shared memory: NMAX components at most, SLOTS of the two stage vectors
// kept here instead of in registers.
template <int NW_, int NL_, int NMAX, int SLOTS_>
struct GroupMem {
    static constexpr int NW = NW_, NL = NL_, SLOTS = SLOTS_;
    static constexpr int NT = 32 * NW * NL;        // threads
    static constexpr int SB = NT / 6;              // steps per batch of points
    static constexpr bool KEEP_R = false;          // the points' radii are not kept
    static constexpr int LOG_N = NMAX;             // components of a logged state
    static constexpr int ROWS = NMAX + (NW > 1 ? 1 : 0);   // the last row takes the empty own slots
    static constexpr int OWN = (NMAX + NW - 1) / NW;
    double pt[SB * 6][PT];                         // points of the batch
    cd ex[NW > 1 ? 2 : 1][NW > 1 ? ROWS : 1][32];  // exchange of the stage inputs (two in turn)
    cd slot[SLOTS > 0 ? SLOTS : 1][SLOTS > 0 ? OWN : 1][SLOTS > 0 ? NT : 1];
    double sh[SB];                                 // step sizes
    int sil[SB];                                   // intervals
    int i1[32];
    double rt[32];
    unsigned flag[NW][2];                          // per warp: lanes with every / any own component out of range
    unsigned long long item;
};

// The block's group, at the start of its dynamic shared memory (looked up in
// every function, so that accesses compile to shared-memory ones).
template <class Mem>
__device__ __forceinline__ Mem& group_mem()
{
    extern __shared__ __align__(16) unsigned char group_smem[];
    return *reinterpret_cast<Mem*>(group_smem);
}

// The lanes' common state.  ll, zeta, ... of c are the lane's own.
struct Group {
    Ctx c;
    LaneCtx lc;
    int lane, warp;
    int i1;                       // the lane's start level
    bool started, valid;
    long long cnt;                // steps of the valid, started lanes
    int jq;                       // logged walks: first step of the lane in the walk it joined
    int nlog;                     // logged walks: steps of the last one, -1 if they exceed the log
    int scale;                    // the lane's rescalings of the last walk
};

// Barrier of the block, and of the warps that hold one lane's components.
template <class Mem>
__device__ __forceinline__ void bsync()
{
    if (Mem::NT == 32) __syncwarp();
    else __syncthreads();
}
template <class Mem>
__device__ __forceinline__ void gsync()
{
    if (Mem::NW == 1) __syncwarp();
    else __syncthreads();
}
template <class Mem>
__device__ __forceinline__ bool gany(bool p)
{
    if (Mem::NW == 1) return __any_sync(FULL, p);
    return __syncthreads_or(p) != 0;
}

// Bits of a 16-bit mask, in closed form so that it folds to a constant in
// unrolled loops; position of component k among a warp's own.
__host__ __device__ __forceinline__ constexpr int cpop(unsigned m)
{
    const unsigned a = m - ((m >> 1) & 0x5555u), b = (a & 0x3333u) + ((a >> 2) & 0x3333u), c = (b + (b >> 4)) & 0x0f0fu;
    return (int)((c + (c >> 8)) & 0x1fu);
}
__host__ __device__ __forceinline__ constexpr int cpos(unsigned mask, int k) { return cpop(mask & ((1u << k) - 1u)); }

// Components of a system over the warps of a group: warp w holds those of
// mask(w) in its NO own slots, in ascending order.  One warp: all of them.
template <class Sys, int NW>
struct Split {
    static constexpr int NO = Sys::N;
    __host__ __device__ static constexpr unsigned mask(int) { return (1u << Sys::N) - 1u; }
};

// The rows of a warp's own slots; empty slots share the row behind the
// system's largest use of the memory (never read as a component).
template <int NO>
struct Own {
    int row[NO];
};
template <class Sys, int NW, class Mem>
__device__ __forceinline__ Own<Split<Sys, NW>::NO> own_rows(int warp)
{
    constexpr int NO = Split<Sys, NW>::NO;
    Own<NO> o;
    if (NW == 1) {
#pragma unroll
        for (int k = 0; k < NO; k++) o.row[k] = k;
        return o;
    }
    unsigned m = warp == 0 ? Split<Sys, NW>::mask(0) : Split<Sys, NW>::mask(1);
#pragma unroll
    for (int k = 0; k < NO; k++) {
        o.row[k] = m ? __ffs(m) - 1 : Mem::ROWS - 1;
        m &= m - 1u;
    }
    return o;
}
template <int NO>
__device__ __forceinline__ void publish(cd (*ex)[32], const Own<NO>& o, int lane, const cd* y)
{
#pragma unroll
    for (int k = 0; k < NO; k++) ex[o.row[k]][lane] = y[k];
}
// An empty slot holds zero.
template <int NO, class Mem>
__device__ __forceinline__ void fetch(const cd (*ex)[32], const Own<NO>& o, int lane, cd* y)
{
#pragma unroll
    for (int k = 0; k < NO; k++)
        y[k] = (Mem::ROWS > NO && o.row[k] == Mem::ROWS - 1) ? mk(0.0) : ex[o.row[k]][lane];
}

// Own outputs of the right-hand side of warp W; the other warps' components
// of the stage input come from the exchange.
template <class Sys, int NW, int W>
__device__ __forceinline__ void rhs_part(const LaneCtx& lc, const cd (*ex)[32], int lane, const cd* yt, cd* d)
{
    constexpr unsigned MASK = Split<Sys, NW>::mask(W);
    // an offset of zero the compiler cannot see through, one per warp's part:
    // it would otherwise load what several parts read before the branch to
    // them, and hold it in registers
    int z = 0;
    if (NW > 1) asm volatile("" : "+r"(z));
    LaneCtx lw = lc;
    lw.p += z;
    const int lz = lane + z;
    cd m[Sys::N], dd[Sys::N];
#pragma unroll
    for (int k = 0; k < Sys::N; k++) m[k] = ((MASK >> k) & 1u) ? yt[cpos(MASK, k)] : ex[k][lz];
    Sys::f(lw, 0.0, m, dd);
#pragma unroll
    for (int k = 0; k < Split<Sys, NW>::NO; k++) d[k] = mk(0.0);
#pragma unroll
    for (int k = 0; k < Sys::N; k++)
        if ((MASK >> k) & 1u) d[cpos(MASK, k)] = dd[k];
}
template <class Sys, int NW>
__device__ __forceinline__ void rhs_own(int warp, const LaneCtx& lc, const cd (*ex)[32], int lane, const cd* yt, cd* d)
{
    static_assert(NW <= 2, "a part of the right-hand side per warp");
    if (NW == 1 || warp == 0) rhs_part<Sys, NW, 0>(lc, ex, lane, yt, d);
    else rhs_part<Sys, NW, NW - 1>(lc, ex, lane, yt, d);
}

__device__ __forceinline__ int hi_abs(double x) { return __double2hiint(x) & 0x7fffffff; }

// The walk of a group along yint's steps: 32 knot intervals at a time, one
// per lane, and the steps of those intervals in batches of SB.
struct Walk {
    bool rev;                     // the steps in reverse order
    int i1, i2;
    double r1, r2;
    int q0, s0, total;            // next chunk of intervals; next step and steps of this chunk
    int iv, n, cum;               // the lane's interval, its steps, steps up to its end
    double x, h;                  // the lane's interval: first radius, step
};

__device__ __forceinline__ void walk_init(Walk& w, int i1, int i2, double r1, double r2, bool rev)
{
    w.rev = rev;
    w.i1 = i1;
    w.i2 = i2;
    w.r1 = r1;
    w.r2 = r2;
    w.q0 = w.s0 = w.total = 0;
}

// The next chunk of intervals with steps in it; false at the end of the walk.
__device__ __forceinline__ bool walk_chunk(const Ctx& c, int lane, Walk& w)
{
    const bool TR = w.rev;
    const bool up = w.r2 > w.r1;
    const int di = up ? 1 : -1;
    const int nint = (up ? w.i2 - w.i1 : w.i1 - w.i2) + 1;
    const Knot* kn = c.kn;
    while (w.s0 >= w.total) {
        if (w.r1 == w.r2 || w.q0 >= nint) return false;
        const int q = w.q0 + lane;
        w.iv = TR ? w.i2 - di * q : w.i1 + di * q;
        w.n = 0;
        w.x = w.h = 0.0;
        if (q < nint) {
            double rr1, rr2;
            if (up) {
                rr1 = (w.iv == w.i1) ? w.r1 : kn[w.iv].r;
                rr2 = (w.iv == w.i2) ? w.r2 : kn[w.iv + 1].r;
            } else {
                rr1 = (w.iv == w.i1) ? w.r1 : kn[w.iv + 1].r;
                rr2 = (w.iv == w.i2) ? w.r2 : kn[w.iv].r;
            }
            if (rr1 != rr2) {
                const double nf = floor(fabs(rr2 - rr1) / steps(c, w.iv));
                w.n = 1 + (int)fmin(nf, 4194304.0);
                w.x = rr1;
                w.h = (rr2 - rr1) / (double)w.n;
            }
        }
        int cum = w.n;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const int v = __shfl_up_sync(FULL, cum, d);
            if (lane >= d) cum += v;
        }
        w.cum = cum;
        w.total = __shfl_sync(FULL, cum, 31);
        w.s0 = 0;
        w.q0 += 32;
    }
    return true;
}

// Step s of the chunk (clamped to its last): interval, radius and size.  The
// lanes of a warp call it together, each with its own s.
__device__ __forceinline__ void walk_step(const Walk& w, int s, int* iv, double* x, double* h)
{
    s = min(s, w.total - 1);
    int L = 0;                        // intervals of the chunk that end at or before step s
#pragma unroll
    for (int b = 16; b > 0; b >>= 1) {
        const int v = __shfl_sync(FULL, w.cum, L + b - 1);
        if (v <= s) L += b;
    }
    const int bn = __shfl_sync(FULL, w.n, L);
    const double bx = __shfl_sync(FULL, w.x, L), bh = __shfl_sync(FULL, w.h, L);
    int j = s - (__shfl_sync(FULL, w.cum, L) - bn);
    if (w.rev) j = bn - 1 - j;
    *iv = __shfl_sync(FULL, w.iv, L);
    *x = __dadd_rn(bx, __dmul_rn((double)j, bh));
    *h = bh;
}

// The points, step sizes and intervals of the next batch of steps (yint's,
// or in reverse order) into shared memory; returns its steps, 0 at
// the end of the walk.  The warps of a group call it together: one copy in
// the code whatever the components they hold.
template <class Point, class Mem>
__device__ __noinline__ int walk_fill(const Group& g, Walk& w)
{
    Mem& M = group_mem<Mem>();
    if (!walk_chunk(g.c, g.lane, w)) return 0;
    const int nb = min(Mem::SB, w.total - w.s0);
    // point t: stage t % 6 of step t / 6 of the batch
    const int t = (int)threadIdx.x;
    const int sl = t / 6, st = t - 6 * sl;
    int iv;
    double x, h;
    walk_step(w, w.s0 + sl, &iv, &x, &h);
    if (sl < nb) {
        const double a = st == 0 ? 0.0 : st == 1 ? 0.2 : st == 2 ? 0.3 : st == 3 ? 0.6 : st == 4 ? 1.0 : 0.875;
        Point::eval(g.c, iv, x + a * h, M.pt[t]);
        if constexpr (Mem::KEEP_R) M.pr[t] = x + a * h;
        if (st == 0) {
            M.sh[sl] = h;
            M.sil[sl] = iv;
        }
    }
    w.s0 += nb;
    bsync<Mem>();
    return nb;
}

// The exchange's buffer b; none where a warp holds all components.
template <class Mem>
__device__ __forceinline__ const cd (*exchange(const Mem& M, int b))[32]
{
    if constexpr (Mem::NW > 1) return M.ex[b];
    else return nullptr;
}

// A stage vector of the own components: in registers, or (SM) in the
// thread's column of a shared-memory slot.
template <class Mem, int NO, bool SM, int WHICH>
struct StageVec {
    cd r[SM ? 1 : NO];
    static constexpr int SLOT = Mem::SLOTS > 1 ? WHICH : 0;
    __device__ __forceinline__ cd get(int k) const
    {
        return SM ? group_mem<Mem>().slot[SLOT][k][threadIdx.x] : r[SM ? 0 : k];
    }
    __device__ __forceinline__ void set(int k, cd v)
    {
        if (SM) group_mem<Mem>().slot[SLOT][k][threadIdx.x] = v;
        else r[SM ? 0 : k] = v;
    }
};

// Log of the states before every step of a walk (and the rescaling factor
// after it), entry (step, component) of the lanes of a launch side by side,
// LOG_N components of the largest system of the kernel; the pointers are the
// thread's own.
struct GroupLog {
    cd* y;
    double* f;
    size_t stride;                // lanes of the launch
    int cap;                      // steps
};

// yint (TR: the transposed integration, yint_T) for the whole group.  On
// entry every warp's own components are in yio and, with more than one
// warp, published in ex[0] (barrier passed); on exit the same holds for the
// result.  With a start vector (`start`, own components), the lane's vector
// is replaced by it when the walk reaches the lane's start level.
//
// After the third derivative the inputs of stages 5 and 6 and the result are
// carried as partial sums, so at most four vectors are live beside the
// derivative: y, the stage input and it in registers, the two partial sums
// (v1, v2) in registers or, with SLOTS, in shared memory.
template <class Sys, class Point, bool TR, class Mem, bool LOG = false>
__device__ __noinline__ void group_walk(Group& g, int i1, int i2, double r1, double r2, cd* yio, const cd* start,
                                        const GroupLog* lg = nullptr, int at = 0)
{
    constexpr int NW = Mem::NW, NO = Split<Sys, NW>::NO;
    Mem& M = group_mem<Mem>();
    g.scale = 0;
    g.nlog = 0;
    if (r2 == r1) return;
    int lq = at;                     // log index of the next step
    const int lane = g.lane, warp = g.warp;
    const Own<NO> own = own_rows<Sys, NW, Mem>(warp);
    Walk w;
    walk_init(w, i1, i2, r1, r2, TR);
    LaneCtx lc = g.lc;
    cd y[NO];
#pragma unroll
    for (int k = 0; k < NO; k++) y[k] = yio[k];
    bool started = start ? g.started : g.valid;
    const int jl = start ? g.i1 : 0x7fffffff;     // without a start vector nothing joins
    int nact = __popc(__ballot_sync(FULL, started));
    int scale = 0;
    long long cnt = 0;
    int nb;
    while ((nb = walk_fill<Point, Mem>(g, w)) > 0) {
        if (LOG && lq + nb > lg->cap) {
            g.nlog = -1;
            bsync<Mem>();
            return;
        }
#pragma unroll 1
        for (int s = 0; s < nb; s++, lq++) {
            if (__any_sync(FULL, !started && jl <= M.sil[s])) {       // the same lanes in every warp
                if (!started && jl <= M.sil[s]) {
#pragma unroll
                    for (int k = 0; k < NO; k++) y[k] = start[k];
                    started = true;
                    if (LOG) g.jq = lq;
                }
                nact = __popc(__ballot_sync(FULL, started));
                if constexpr (NW > 1) {
                    publish(M.ex[0], own, lane, y);
                    gsync<Mem>();
                }
            }
            // a warp none of whose lanes has started waits for the others
            if (Mem::NL > 1 && nact == 0) continue;
            if (LOG) {
                // streaming stores: only the reverse pass reads them back
#pragma unroll
                for (int k = 0; k < NO; k++)
                    __stcs(reinterpret_cast<double2*>(lg->y + ((size_t)lq * Mem::LOG_N + k) * lg->stride),
                           make_double2(y[k].x, y[k].y));
            }
            const double(*p)[PT] = M.pt + s * 6;
            // One copy of the right-hand side in the code, the stage combinations
            // by case: six copies would overflow the instruction cache.  The step
            // size is read again every stage, so that its products with the
            // weights are not all held in registers over the stages.
            StageVec<Mem, NO, TR ? (Mem::SLOTS > 0) : (Mem::SLOTS > 1), 0> v1;
            StageVec<Mem, NO, TR ? (Mem::SLOTS > 1) : (Mem::SLOTS > 0), 1> v2;
            cd yt[NO];
            if (!TR) {
                // v1, v2 = k1, k2; after k3 the partial sums of the
                // inputs of stages 5 (v2) and 6 (v1) and of the result (y)
#pragma unroll
                for (int k = 0; k < NO; k++) yt[k] = y[k];
#pragma unroll 1
                for (int st = 0; st < 6; st++) {
                    const double h = *(volatile double*)&M.sh[s];
                    cd d[NO];
                    lc.p = p[st];
                    rhs_own<Sys, NW>(warp, lc, exchange(M, st & 1), lane, yt, d);
                    if (st == 0) {
#pragma unroll
                        for (int k = 0; k < NO; k++) {
                            v1.set(k, d[k]);
                            yt[k] = cmac(y[k], 0.2 * h, d[k]);
                        }
                    } else if (st == 1) {
#pragma unroll
                        for (int k = 0; k < NO; k++) {
                            v2.set(k, d[k]);
                            yt[k] = cmac(cmac(y[k], (3.0 / 40.0) * h, v1.get(k)), (9.0 / 40.0) * h, d[k]);
                        }
                    } else if (st == 2) {
#pragma unroll
                        for (int k = 0; k < NO; k++) {
                            const cd k1 = v1.get(k), k2 = v2.get(k), yk = y[k];
                            yt[k] = cmac(cmac(cmac(yk, 0.3 * h, k1), -0.9 * h, k2), 1.2 * h, d[k]);
                            v1.set(k, cmac(cmac(cmac(yk, (1631.0 / 55296.0) * h, k1), (175.0 / 512.0) * h, k2),
                                         (575.0 / 13824.0) * h, d[k]));
                            v2.set(k, cmac(cmac(cmac(yk, (-11.0 / 54.0) * h, k1), 2.5 * h, k2), (-70.0 / 27.0) * h, d[k]));
                            y[k] = cmac(cmac(yk, (37.0 / 378.0) * h, k1), (250.0 / 621.0) * h, d[k]);
                        }
                    } else if (st == 3) {
#pragma unroll
                        for (int k = 0; k < NO; k++) {
                            yt[k] = cmac(v2.get(k), (35.0 / 27.0) * h, d[k]);
                            v1.set(k, cmac(v1.get(k), (44275.0 / 110592.0) * h, d[k]));
                            y[k] = cmac(y[k], (125.0 / 594.0) * h, d[k]);
                        }
                    } else if (st == 4) {
#pragma unroll
                        for (int k = 0; k < NO; k++) yt[k] = cmac(v1.get(k), (253.0 / 4096.0) * h, d[k]);
                    } else {
#pragma unroll
                        for (int k = 0; k < NO; k++) y[k] = cmac(y[k], (512.0 / 1771.0) * h, d[k]);
                    }
                    if constexpr (NW > 1) {
                        if (st < 5) {
                            publish(M.ex[(st + 1) & 1], own, lane, yt);
                            gsync<Mem>();
                        }
                    }
                }
            } else {
                // the transposed step (rkck_step_loop_T): stages 6 .. 1,
                // K_s = h (c_s w + sum_{u>s} b_us G_u), G_s = A_s^T K_s, w += sum G_s.
                // v1, v2 = G_6, G_5; after G_4 the partial sums of K_2 (v1),
                // K_1 (v2) and of the result (y)
                {
                    const double h = *(volatile double*)&M.sh[s];
#pragma unroll
                    for (int k = 0; k < NO; k++) yt[k] = ((512.0 / 1771.0) * h) * y[k];
                }
#pragma unroll 1
                for (int st = 5; st >= 0; st--) {
                    if constexpr (NW > 1) {
                        publish(M.ex[st & 1], own, lane, yt);
                        gsync<Mem>();
                    }
                    const double h = *(volatile double*)&M.sh[s];
                    cd d[NO];
                    lc.p = p[st];
                    rhs_own<Sys, NW>(warp, lc, exchange(M, st & 1), lane, yt, d);
                    if (st == 5) {
#pragma unroll
                        for (int k = 0; k < NO; k++) {
                            v1.set(k, d[k]);
                            yt[k] = ((253.0 / 4096.0) * h) * d[k];
                        }
                    } else if (st == 4) {
#pragma unroll
                        for (int k = 0; k < NO; k++) {
                            v2.set(k, d[k]);
                            yt[k] = cmac(cmac(((125.0 / 594.0) * h) * y[k], (44275.0 / 110592.0) * h, v1.get(k)),
                                         (35.0 / 27.0) * h, d[k]);
                        }
                    } else if (st == 3) {
#pragma unroll
                        for (int k = 0; k < NO; k++) {
                            const cd w0 = y[k], g6 = v1.get(k), g5 = v2.get(k);
                            yt[k] = cmac(cmac(cmac(((250.0 / 621.0) * h) * w0, (575.0 / 13824.0) * h, g6),
                                              (-70.0 / 27.0) * h, g5), 1.2 * h, d[k]);
                            v1.set(k, cmac(cmac(((175.0 / 512.0) * h) * g6, 2.5 * h, g5), -0.9 * h, d[k]));
                            v2.set(k, cmac(cmac(cmac(((37.0 / 378.0) * h) * w0, (1631.0 / 55296.0) * h, g6),
                                              (-11.0 / 54.0) * h, g5), 0.3 * h, d[k]));
                            y[k] = (w0 + g6) + (g5 + d[k]);
                        }
                    } else if (st == 2) {
#pragma unroll
                        for (int k = 0; k < NO; k++) {
                            yt[k] = cmac(v1.get(k), (9.0 / 40.0) * h, d[k]);
                            v2.set(k, cmac(v2.get(k), (3.0 / 40.0) * h, d[k]));
                            y[k] = y[k] + d[k];
                        }
                    } else if (st == 1) {
#pragma unroll
                        for (int k = 0; k < NO; k++) {
                            yt[k] = cmac(v2.get(k), 0.2 * h, d[k]);
                            y[k] = y[k] + d[k];
                        }
                    } else {
#pragma unroll
                        for (int k = 0; k < NO; k++) y[k] = y[k] + d[k];
                    }
                }
            }
            cnt += nact;
            // yint's rescaling, decided on the larger of |Re| and |Im| by
            // the high words of the values (against 1e-20 and 1e20): the
            // choice only changes the representation, which the scale
            // count records
            int mx = 0;
#pragma unroll
            for (int k = 0; k < NO; k++) mx = max(mx, max(hi_abs(y[k].x), hi_abs(y[k].y)));
            double factor = 1.0;
            const bool small = started && mx < 0x3BC79CA1, big = started && mx > 0x4415AF1D;
            if constexpr (NW > 1 && !TR) publish(M.ex[0], own, lane, y);
            if (gany<Mem>(small || big)) {
                unsigned sb = __ballot_sync(FULL, small), bb = __ballot_sync(FULL, big);
                if constexpr (NW > 1) {
                    if (lane == 0) {
                        M.flag[g.warp][0] = sb;
                        M.flag[g.warp][1] = bb;
                    }
                    gsync<Mem>();
                    sb = FULL;
                    bb = 0u;
#pragma unroll
                    for (int q = 0; q < NW; q++) {
                        sb &= M.flag[q][0];
                        bb |= M.flag[q][1];
                    }
                }
                const bool s1 = (sb >> lane) & 1u, b1 = (bb >> lane) & 1u;
                if (s1 || b1) {
                    const double f = s1 ? SC_HUGE : SC_TINY;
                    if (LOG) factor = f;
                    scale += s1 ? 1 : -1;
#pragma unroll
                    for (int k = 0; k < NO; k++) y[k] = y[k] * f;
                    if constexpr (NW > 1 && !TR) publish(M.ex[0], own, lane, y);
                }
                gsync<Mem>();
            }
            if (LOG) lg->f[(size_t)lq * lg->stride] = factor;
        }
        // the points are filled again: every warp has read them.  With one
        // lane per degree the warps of a block run free between the batches,
        // yet stay within a few steps of one another: their instruction
        // fetches meet in the cache, which the walk's code would otherwise
        // overflow.
        if (NW == 1) bsync<Mem>();
    }
    if constexpr (NW > 1 && TR) {    // the other form publishes after every step
        publish(M.ex[0], own, lane, y);
        gsync<Mem>();
    }
#pragma unroll
    for (int k = 0; k < NO; k++) yio[k] = y[k];
    if (start) g.started = started;
    g.cnt += cnt;
    g.scale = scale;
    g.nlog = lq - at;
}

// Lanes that start at or below level `last` but have not met it on a walk
// (their start is the end of the leg): their vector becomes the start vector.
template <class Sys, class Mem>
__device__ __forceinline__ void group_join_rest(Group& g, int last, cd* y, const cd* start)
{
    constexpr int NW = Mem::NW;
    const bool jn = !g.started && g.i1 <= last;
    if (!__any_sync(FULL, jn)) return;
    if (jn) {
#pragma unroll
        for (int k = 0; k < Split<Sys, NW>::NO; k++) y[k] = start[k];
        g.started = true;
    }
    if constexpr (NW > 1) {
        publish(group_mem<Mem>().ex[0], own_rows<Sys, NW, Mem>(g.warp), g.lane, y);
        gsync<Mem>();
    }
}

}  // namespace
}  // inline namespace
}  // namespace ysg
