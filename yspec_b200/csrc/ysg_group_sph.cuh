// ysg_group_sph.cuh -- items of the group kernels and the parts of a
// spheroidal solve that the solve (k_solve_group.cu) and its reverse sweep
// (k_group_adjoint.cu) share: contexts, start vectors, the sequence of
// integrations, the minor algebra per gravity setting.
#pragma once
#include "ysg_group.cuh"
#include "ysg_kernels.h"

namespace ysg {
inline namespace YSG_VARIANT {
namespace {

// ---------------------------------------------------------------------------
// Items
// ---------------------------------------------------------------------------
// First degree of an event's items of a kind (l = 0 is the radial mode,
// toroidal motion starts at l = 2).
__host__ __device__ inline int first_l(int lmin, int kind)
{
    const int lo = kind == GROUP_TOR ? 2 : 1;
    return lmin > lo ? lmin : lo;
}

struct Item {
    int e, j, lb;                 // event, frequency (1-based), first degree
};


// Item `it` of a list with per-event offsets off[0..nev]: the degrees of an
// event vary slowest, its frequencies descend.
__device__ __forceinline__ Item item_of(const EventDev* evs, const long long* off, int nev, long long it, int kind, int width)
{
    int lo = 0, hi = nev;
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (off[mid] <= it) lo = mid;
        else hi = mid;
    }
    const EventDev& ev = evs[lo];
    const long long q = it - off[lo];
    const int b = (int)(q / ev.nw);
    return Item{lo, ev.nw - (int)(q - (long long)b * ev.nw), first_l(ev.lmin, kind) + width * b};
}

__device__ __forceinline__ void lane_ctx(Group& g)
{
    g.lc.zeta = g.c.zeta;
    g.lc.zeta2 = g.c.zeta2;
    g.lc.fl = (double)g.c.ll;
    g.lc.flp1 = (double)g.c.llp1;
    g.lc.pib4 = 4.0 * g.c.pib;
}

// The degree of the item's lane `at` and the item's frequency.
__device__ __forceinline__ void item_ctx(Group& g, const EventDev& ev, const Item& w, int at)
{
    const int l = w.lb + at;
    g.valid = l <= ev.lmax;
    g.c.ats = (double)ev.ats;
    set_l(g.c, g.valid ? l : ev.lmax);
    set_omega(g.c, omega_of(ev, w.j));
    alpha_steps(g.c);
    lane_ctx(g);
}

// Start level, its radius and the start vector of the lane (sph_solver_g and
// sph_solver_nc of ysg_solvers.cuh).
template <int KIND>
__device__ __noinline__ void sph_start(const Ctx& c, const EventDev& ev, bool up, int* level, double* radius, cd* m)
{
    const ModelHdr* mh = c.mh;
    const Knot* kn = c.kn;
    const bool fic = mh->fic != 0;
    const int it = up ? ev.is : ev.ir;
    int i1 = sph_start_level(c, c.ll, c.omega.x, it);
    double rt = kn[i1].r;
    if (i1 == 1 && (up || fic)) rt = fmin(0.1 * c.dr, 0.1 * kn[2].r);
    if (i1 >= it) { i1 = it - 1; rt = kn[i1].r; }
    for (int k = 0; k < (KIND == 2 ? 14 : 5); k++) m[k] = mk(0.0);
    const bool fluid = i1 <= mh->nic ? fic : i1 <= mh->noc;
    if (KIND == 2) {
        if (fluid) sph_minor_fluid_start(c, i1, rt, m);
        else sph_minor_solid_start(c, i1, rt, m);
    } else {
        if (fluid) sph_fluid_start_ng(c, i1, rt, m);
        else sph_minor_solid_start_ng(c, i1, rt, m);
    }
    *level = i1;
    *radius = rt;
}

// The integrations of a spheroidal solve: leg 0 inner core, 1 outer core, 2
// mantle to the source (or to a receiver below it) -> ms1; 3 the ocean, 4 the
// mantle from the surface down to the receiver (or the source) -> ms2; 5 ms1
// continued between the source and the receiver -> ms3.  ic / core: some
// lane starts in the inner core / in the core.
struct Leg {
    int i1, i2;
    double r1, r2;
};
__device__ __forceinline__ Leg leg_of(int leg, const ModelHdr* mh, const Knot* kn, const EventDev& ev, int imin,
                                      double rmin, bool ic, bool core, bool up)
{
    const int nic = mh->nic, noc = mh->noc;
    const int lo = up ? ev.is : ev.ir, hi = up ? ev.ir : ev.is;
    const double rlo = up ? ev.rs : ev.rr, rhi = up ? ev.rr : ev.rs;
    switch (leg) {
        case 0: return Leg{imin, nic, rmin, kn[nic].r};
        case 1: return Leg{ic ? nic + 1 : imin, noc, ic ? kn[nic].r : rmin, kn[noc].r};
        case 2: return Leg{core ? noc + 1 : imin, lo, core ? kn[noc + 1].r : rmin, rlo};
        case 3: return Leg{mh->nknot - 1, mh->nsl + 1, kn[mh->nknot].r, kn[mh->nsl + 1].r};
        case 4:
            if (mh->ocean) return Leg{mh->nsl, hi, kn[mh->nsl].r, rhi};
            return Leg{up ? mh->nknot - 1 : mh->nknot, hi, kn[mh->nknot].r, rhi};
        default: return Leg{lo, hi, rlo, rhi};
    }
}

template <int KIND>
struct SphSys {
    using Solid = MinorSolidNC<KIND>;
    using Fluid = MinorFluidNC<KIND>;
    using Bvec = BvecSolidNCTr<KIND>;
    static constexpr int ROWS = 2;                // response rows used (0 .. ROWS - 1)
    __device__ static void to_fluid(const cd* m, cd* f) { s2f_ngcow(m, f); }
    __device__ static void to_solid(const cd* f, cd* m) { f2s_ngcow(f, m); }
    __device__ static cd det(const cd* a, const cd* b) { return delta_solid_ngcow(a, b); }
    __device__ static void row(const cd* mq, int k, cd* q) { sph_ysol_row_ngcow(mq, k, q); }
    // u . (-1)^(up) / delta as sph_solver_nc
    __device__ static void resp(const cd* mb, const cd* w, bool up, cd delta, double f, cd* y4)
    {
        cd u[4];
        b_solid_start_T_ngcow(mb, w, u);
        for (int i = 0; i < 4; i++) y4[i] = ((up ? u[i] : -u[i]) / delta) * f;
    }
};
template <>
struct SphSys<2> {
    using Solid = MinorSolidG;
    using Fluid = MinorFluidG;
    using Bvec = BvecSolidGTr;
    static constexpr int ROWS = 3;
    __device__ static __noinline__ void to_fluid(const cd* m, cd* f) { s2f(m, f); }
    __device__ static __noinline__ void to_solid(const cd* f, cd* m) { f2s(f, m); }
    __device__ static __noinline__ cd det(const cd* a, const cd* b) { return delta_solid(a, b); }
    __device__ static __noinline__ void row(const cd* mq, int k, cd* q) { sph_ysol_row(mq, k, q); }
    __device__ static __noinline__ void resp(const cd* mb, const cd* w, bool, cd delta, double f, cd* y4)
    {
        cd u[6];
        b_solid_start_T(mb, w, u);
        y4[0] = ((-u[0]) / delta) * f;
        y4[1] = ((-u[1]) / delta) * f;
        y4[2] = ((-u[3]) / delta) * f;
        y4[3] = ((-u[4]) / delta) * f;
    }
};

// The deepest start level of the block's lanes and its radius.
template <class Mem>
__device__ __forceinline__ int block_min(const Group& g, int i1, double rt, double* rmin)
{
    Mem& M = group_mem<Mem>();
    int m = __reduce_min_sync(FULL, i1);
    double r = __shfl_sync(FULL, rt, __ffs(__ballot_sync(FULL, i1 == m)) - 1);
    if (Mem::NL > 1) {
        const int wl = threadIdx.x >> 5;
        if (g.lane == 0) {
            M.i1[wl] = m;
            M.rt[wl] = r;
        }
        __syncthreads();
        for (int w = 0; w < Mem::NL; w++)
            if (M.i1[w] < m) {
                m = M.i1[w];
                r = M.rt[w];
            }
        __syncthreads();
    }
    *rmin = r;
    return m;
}

// The next item of the block's list.
template <class Mem>
__device__ __forceinline__ unsigned long long next_item(unsigned long long* counter)
{
    Mem& M = group_mem<Mem>();
    if (threadIdx.x == 0) M.item = atomicAdd(counter, 1ull);
    bsync<Mem>();
    const unsigned long long it = M.item;
    bsync<Mem>();
    return it;
}

}  // namespace
}  // inline namespace
}  // namespace ysg
