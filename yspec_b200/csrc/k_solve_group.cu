// k_solve_group.cu -- solve stage by groups of degrees of one frequency.
//
// The (omega, l) double loop of yspec.f90:250-426 with an item = (event,
// frequency, a run of consecutive degrees), the radial walks shared by the
// degrees (ysg_group.cuh).  One kernel per kind of solve:
//   k_group_lane    spheroidal, a degree per lane, NL warps per item
//   k_group_split   spheroidal with self-gravitation, 32 degrees per item, the
//                   14 components split over NW warps
//   k_group_tor     toroidal, a degree per lane, NL warps per item
//   k_group_rad     l = 0, a warp per frequency
// Events with the source or a receiver in the core, where legs of different
// lanes would run in different directions, take the pair lists of
// k_solve_batched.cu instead.
//
// What bounds k_group_lane with self-gravitation (form 0, 128 degrees per
// item, two blocks of four warps per SM at 255 registers): dependent FP64
// latency with two warps per SM partition, and the instruction cache.  A
// stepping loop of the 14-component systems is 18 KB; with each warp on its
// own item (one warp per block, eight blocks per SM) the loops of the eight
// warps, at different places, overflow the cache (97 misses per step,
// no_instruction 2.2 cycles per issue); four warps on the same walk fetch
// the same lines within a few steps of one another (no_instruction 0.2).
// Measured on one event at scale (615,820 pairs; solve stage, source at 29
// km / 445 km): 32.3 / 56.8 ms with a pair per thread
// (k_solve_batched.cu), 26.6 / 50.8 ms with one warp per item, 18.3 / 33.4
// ms with four; eight warps (one block per SM) 21.6 / 37.0 ms, two 18.5 /
// 33.4 ms.  The largest event (400 knots, lmax 1500, 100 mHz): 195 -> 112 ms.
//
// A list that does not fill the GPU with such items takes form 1, whose
// step takes less time for fewer degrees.  With the 14 components split
// over two warps a step has half the instructions per warp: one event of
// 9,060 pairs, 3.4 -> 0.9 ms; at scale the split form takes 25.9 / 50.6 ms
// (exchange through shared memory, two barriers' worth of waiting), so it
// serves short lists only.
//
// Items of a launch that do not all fit the GPU at once are taken longest
// first from a list ordered by k_group_cost / k_group_order: cost buckets
// of a sixteenth of an octave from the start level of the item's lowest
// degree.
// The start vectors, the minor algebra and the source vectors run once per
// item: one copy of the complex division and roots keeps them from pushing
// the walks out of the instruction cache.
#define YSG_CPLX_CALLS
#include <algorithm>

#include "ysg_kernels.h"
#include "ysg_group_sph.cuh"
#include "ysg_radial.cuh"

namespace ysg {
inline namespace YSG_VARIANT {
namespace {

// ---------------------------------------------------------------------------
// Self-gravitating spheroidal solves: components per warp, chosen for equal
// FP64 work of the warps (160 and 162 instructions per right-hand side and
// stage combination) and few components read from the other warp (6 each).
// ---------------------------------------------------------------------------
__host__ __device__ constexpr unsigned bits(int a, int b, int c, int d = -1)
{
    return (1u << a) | (1u << b) | (1u << c) | (d >= 0 ? 1u << (d < 0 ? 0 : d) : 0u);
}
template <>
struct Split<MinorSolidG, 2> {
    static constexpr int NO = 7;
    __host__ __device__ static constexpr unsigned mask(int w)
    {
        return w == 0 ? (bits(0, 1, 2, 6) | bits(7, 10, 13)) : (bits(3, 4, 5, 8) | bits(9, 11, 12));
    }
};
template <>
struct Split<BvecSolidGTr, 2> {
    static constexpr int NO = 7;
    __host__ __device__ static constexpr unsigned mask(int w)
    {
        return w == 0 ? (bits(0, 3, 5, 6) | bits(7, 8, 11)) : (bits(1, 2, 4, 9) | bits(10, 12, 13));
    }
};
template <>
struct Split<MinorFluidG, 2> {
    static constexpr int NO = 3;
    __host__ __device__ static constexpr unsigned mask(int w) { return w == 0 ? 0x0bu : 0x14u; }
};

template <int NW>
using SphMemOf = GroupMem<NW, 1, 14, 0>;

// A lane's column of the exchange.
template <int NW>
__device__ __forceinline__ void sph_column(int buf, int lane, cd* m)
{
    const SphMemOf<NW>& M = group_mem<SphMemOf<NW>>();
    for (int k = 0; k < 14; k++) m[k] = M.ex[buf][k][lane];
}
__device__ __noinline__ cd sph_delta(const cd* ms3, const cd* ms2) { return delta_solid(ms3, ms2); }
// The start of the backward integration of response row k, and the
// responses of the row from its end w (as sph_solver_g).
template <int NW>
__device__ __noinline__ void sph_row(int lane, const cd* mq, int k)
{
    SphMemOf<NW>& M = group_mem<SphMemOf<NW>>();
    cd q[14];
    sph_ysol_row(mq, k, q);
    for (int i = 0; i < 14; i++) M.ex[0][i][lane] = q[i];
}
template <int NW>
__device__ __noinline__ void sph_resp(int lane, const cd* mb, cd delta, double f, cd* y4)
{
    cd w[14], u[6];
    sph_column<NW>(0, lane, w);
    b_solid_start_T(mb, w, u);
    y4[0] = ((-u[0]) / delta) * f;
    y4[1] = ((-u[1]) / delta) * f;
    y4[2] = ((-u[3]) / delta) * f;
    y4[3] = ((-u[4]) / delta) * f;
}
struct GroupArgs {
    const Knot* kn;
    const Seg* sg;
    const ModelHdr* mh;
    const EventDev* evs;
    cd* const* coefs;
    const long long* off;         // items of the events before e, nev + 1 entries
    const int* order;             // items longest first, or null
    int nev;
    long long nitems;
    unsigned long long* counter;
    unsigned long long* work;
    const int* next;              // per event the next one with the same solves, or -1; null: none
};

// The coefficients of the item's event, and of the events of the batch that
// differ from it in the moment tensor alone (a.next): they have the same
// responses.
__device__ __noinline__ void sph_store(const Group& g, const GroupArgs& a, const Item& w, const cd (*ysph)[4])
{
    const int l = g.c.ll;
    for (int e = w.e; e >= 0; e = a.next ? a.next[e] : -1) {
        const EventDev& ev = a.evs[e];
        cd y[3][4], uu[5], vv[5];                     // the responses are scaled in place
        for (int k = 0; k < 3; k++)
            for (int i = 0; i < 4; i++) y[k][i] = ysph[k][i];
        spheroidal_coefs(g.c, ev, l, g.c.omega, y, uu, vv);
        if (!g.valid) continue;
        cd* dst = a.coefs[e] + (size_t)(l - ev.lmin) * NCOEF * ev.nw + (w.j - 1);
        // streaming stores: not read again in this launch
        for (int q = 0; q < 5; q++) {
            __stcs(reinterpret_cast<double2*>(dst + (size_t)q * ev.nw), make_double2(uu[q].x, uu[q].y));
            __stcs(reinterpret_cast<double2*>(dst + (size_t)(q + 5) * ev.nw), make_double2(vv[q].x, vv[q].y));
            if (l < 2) __stcs(reinterpret_cast<double2*>(dst + (size_t)(q + 10) * ev.nw), make_double2(0.0, 0.0));
        }
    }
}

__device__ __forceinline__ void group_ctx(Group& g, const GroupArgs& a)
{
    g.c.kn = a.kn;
    g.c.mh = a.mh;
    g.c.sg = a.sg;
    g.c.pib = a.mh->pibigg;
    g.c.kb = nullptr;
    g.c.il = 0;
    for (int q = 0; q < NSYS; q++) g.c.nst[q] = 0;
}

__device__ __forceinline__ void count_work(Group& g, unsigned long long* work, int cls)
{
    if (g.lane == 0 && g.warp == 0 && g.cnt) atomicAdd(&work[cls], (unsigned long long)g.cnt);
    g.cnt = 0;
}

__device__ __forceinline__ int lane_min(int v)
{
    return __reduce_min_sync(FULL, v);
}

// The hand-overs at the core boundaries, on the published vector.
template <int NW>
__device__ __noinline__ void sph_s2f(int lane)
{
    using SphMem = SphMemOf<NW>;
    SphMem& M = group_mem<SphMem>();
    cd m1[14], m2[5];
    for (int k = 0; k < 14; k++) m1[k] = M.ex[0][k][lane];
    s2f(m1, m2);
    for (int k = 0; k < 5; k++) M.ex[0][k][lane] = m2[k];
}
template <int NW>
__device__ __noinline__ void sph_f2s(int lane)
{
    using SphMem = SphMemOf<NW>;
    SphMem& M = group_mem<SphMem>();
    cd m1[5], m2[14];
    for (int k = 0; k < 5; k++) m1[k] = M.ex[0][k][lane];
    f2s(m1, m2);
    for (int k = 0; k < 14; k++) M.ex[0][k][lane] = m2[k];
}

// Publish a vector of a system's warps in ex[0].
template <class Sys, int NW>
__device__ __forceinline__ void sph_publish(const Group& g, const cd* y)
{
    using SphMem = SphMemOf<NW>;
    __syncthreads();                                  // the reads of ex[0] end
    publish(group_mem<SphMem>().ex[0], own_rows<Sys, NW, SphMem>(g.warp), g.lane, y);
    __syncthreads();
}
// The first component one, the others zero (the surface).
template <class Sys, int NW>
__device__ __forceinline__ void sph_unit(const Group& g, cd* y)
{
    const auto own = own_rows<Sys, NW, SphMemOf<NW>>(g.warp);
#pragma unroll
    for (int k = 0; k < Split<Sys, NW>::NO; k++) y[k] = mk(own.row[k] == 0 ? 1.0 : 0.0);
}

template <int NW, int MINB>
__global__ void __launch_bounds__(32 * NW, MINB) k_group_split(GroupArgs a)
{
    using MS = MinorSolidG;
    using MF = MinorFluidG;
    using BT = BvecSolidGTr;
    using Pt = SolidPoint<2>;
    using SphMem = SphMemOf<NW>;
    SphMem& M = group_mem<SphMem>();
    const int lane = threadIdx.x & 31;
    Group g;
    g.lane = lane;
    g.warp = threadIdx.x >> 5;
    g.cnt = 0;
    group_ctx(g, a);
    for (;;) {
        if (threadIdx.x == 0) M.item = atomicAdd(a.counter, 1ull);
        __syncthreads();
        const long long it = (long long)M.item;
        if (it >= a.nitems) break;
        const Item w = item_of(a.evs, a.off, a.nev, a.order ? a.order[it] : it, GROUP_SPH2, 32);
        const EventDev& ev = a.evs[w.e];
        const bool serial = (int)(it % NW) == g.warp;  // the warp that does the one-warp parts of this item
        item_ctx(g, ev, w, lane);
        const ModelHdr* mh = g.c.mh;
        const Knot* kn = g.c.kn;
        const double rr = ev.rr, rs = ev.rs;
        const int ir = ev.ir, is = ev.is;
        const bool up = rr >= rs, fic = mh->fic != 0;
        const int top = up ? is : ir;
        if (serial) {
            cd m[14];
            int i1;
            double rt;
            sph_start<2>(g.c, ev, up, &i1, &rt, m);
            for (int k = 0; k < 14; k++) M.ex[0][k][lane] = m[k];
            M.i1[lane] = i1;
            M.rt[lane] = rt;
        }
        __syncthreads();
        g.i1 = M.i1[lane];
        g.started = false;
        // own components of the start vectors: as solid and as fluid minors
        // (a lane uses the one of its level)
        cd s14[Split<MS, NW>::NO], s5[Split<MF, NW>::NO];
        fetch<Split<MS, NW>::NO, SphMem>(M.ex[0], own_rows<MS, NW, SphMem>(g.warp), lane, s14);
        fetch<Split<MF, NW>::NO, SphMem>(M.ex[0], own_rows<MF, NW, SphMem>(g.warp), lane, s5);
        if (!g.valid) g.i1 = 0x7fffffff;
        const int imin = lane_min(g.i1);
        // the first radius of the walk: that of the deepest lanes
        const double rmin = __shfl_sync(FULL, M.rt[lane], __ffs(__ballot_sync(FULL, g.i1 == imin)) - 1);
        constexpr int NS = Split<MS, NW>::NO, NF = Split<MF, NW>::NO;
        cd y[NS], yf[NF];
#pragma unroll
        for (int k = 0; k < NS; k++) y[k] = mk(0.0);
#pragma unroll
        for (int k = 0; k < NF; k++) yf[k] = mk(0.0);
        const int nic = mh->nic, noc = mh->noc;
        const bool ic = !fic && imin <= nic, core = imin <= noc;
        int scale3 = 0;
        cd ms1[NS], ms2[NS];
#pragma unroll 1
        for (int leg = 0; leg < 6; leg++) {
            if (leg == 0 && !ic) continue;
            if (leg == 1 && !core) continue;
            if (leg == 3 && !mh->ocean) continue;
            const Leg q = leg_of(leg, mh, kn, ev, imin, rmin, ic, core, up);
            if (leg == 1 || leg == 3) {
                // fluid: from the inner core's solid minor, the start vectors or the surface
                if (leg == 1 && ic) {
                    if (serial) sph_s2f<NW>(lane);
                    __syncthreads();
                    fetch<NF, SphMem>(M.ex[0], own_rows<MF, NW, SphMem>(g.warp), lane, yf);
                    __syncthreads();
                } else {
                    if (leg == 3) sph_unit<MF, NW>(g, yf);
                    sph_publish<MF, NW>(g, yf);
                }
                group_walk<MF, FluidPoint<2>, false, SphMem>(g, q.i1, q.i2, q.r1, q.r2, yf, leg == 1 ? s5 : nullptr);
                if (leg == 1) group_join_rest<MF, SphMem>(g, noc, yf, s5);
                count_work(g, a.work, MF::CLS);
                if (serial) sph_f2s<NW>(lane);
                __syncthreads();
                fetch<NS, SphMem>(M.ex[0], own_rows<MS, NW, SphMem>(g.warp), lane, y);
                __syncthreads();
                continue;
            }
            if (leg == 4 && !mh->ocean) sph_unit<MS, NW>(g, y);
            if (leg == 5)
                for (int k = 0; k < NS; k++) y[k] = ms1[k];
            sph_publish<MS, NW>(g, y);
            group_walk<MS, Pt, false, SphMem>(g, q.i1, q.i2, q.r1, q.r2, y, leg < 4 ? s14 : nullptr);
            count_work(g, a.work, MS::CLS);
            if (leg == 0) group_join_rest<MS, SphMem>(g, nic, y, s14);
            if (leg == 2) group_join_rest<MS, SphMem>(g, top, y, s14);
            if (leg == 2)
                for (int k = 0; k < NS; k++) ms1[k] = y[k];
            if (leg == 4)
                for (int k = 0; k < NS; k++) ms2[k] = y[k];
            scale3 = g.scale;
        }
        // the minor algebra, by one warp: ms3 is published in ex[0]
        const auto own = own_rows<MS, NW, SphMem>(g.warp);
        cd delta = mk(1.0), ma[14], mb[14];           // the minors at the receiver's and the source's side
        publish(M.ex[1], own, lane, up ? ms2 : ms1);
        __syncthreads();
        if (serial) {
            sph_column<NW>(0, lane, mb);
            sph_column<NW>(1, lane, ma);
        }
        __syncthreads();
        publish(M.ex[0], own, lane, up ? ms1 : ms2);
        __syncthreads();
        if (serial) {
            if (up) {
                delta = sph_delta(mb, ma);
                sph_column<NW>(0, lane, mb);
            } else {
                cd ms3[14];
                for (int k = 0; k < 14; k++) ms3[k] = mb[k];
                sph_column<NW>(0, lane, mb);
                delta = sph_delta(ms3, mb);
            }
        }
        cd ysph[3][4];
        const int rows = spheroidal_rows(ev);
        for (int k = 0; k < 3; k++) {
            if (!((rows >> k) & 1)) {
                for (int i = 0; i < 4; i++) ysph[k][i] = mk(0.0);
                continue;
            }
            if (serial) sph_row<NW>(lane, ma, k);
            __syncthreads();
            fetch<NS, SphMem>(M.ex[0], own_rows<BT, NW, SphMem>(g.warp), lane, y);
            __syncthreads();
            group_walk<BT, Pt, true, SphMem>(g, is, ir, rs, rr, y, nullptr);
            if (serial) sph_resp<NW>(lane, mb, delta, huge_pow(scale3 - g.scale), ysph[k]);
        }
        count_work(g, a.work, BT::CLS);
        if (serial) sph_store(g, a, w, ysph);
        __syncthreads();
    }
}

// ---------------------------------------------------------------------------
// Spheroidal solves with a degree per lane and NL warps per item, for each
// gravity setting: no gravity (KIND 0), Cowling (1), self-gravitation (2).
// ---------------------------------------------------------------------------
template <int KIND, int NL>
using LaneMem = GroupMem<1, NL, KIND == 2 ? 14 : 5, KIND == 2 ? 2 : 0>;

template <int KIND, int NL, int MINB>
__global__ void __launch_bounds__(32 * NL, MINB) k_group_lane(GroupArgs a)
{
    using S = SphSys<KIND>;
    using Solid = typename S::Solid;
    using Fluid = typename S::Fluid;
    using Bvec = typename S::Bvec;
    using Pt = SolidPoint<KIND>;
    using Mem = LaneMem<KIND, NL>;
    constexpr int NS = Solid::N, NF = Fluid::N;
    Group g;
    g.lane = threadIdx.x & 31;
    g.warp = 0;
    g.cnt = 0;
    group_ctx(g, a);
    for (;;) {
        const unsigned long long it = next_item<Mem>(a.counter);
        if ((long long)it >= a.nitems) break;
        const Item w = item_of(a.evs, a.off, a.nev, a.order ? a.order[it] : (long long)it, GROUP_SPH0 + KIND, 32 * NL);
        const EventDev& ev = a.evs[w.e];
        item_ctx(g, ev, w, (int)threadIdx.x);
        const ModelHdr* mh = g.c.mh;
        const Knot* kn = g.c.kn;
        const double rr = ev.rr, rs = ev.rs;
        const int ir = ev.ir, is = ev.is;
        const bool up = rr >= rs, fic = mh->fic != 0;
        const int top = up ? is : ir;
        cd st[NS], ms1[NS], ms2[NS], ms3[NS], mf[NF];
        double rt, rmin;
        sph_start<KIND>(g.c, ev, up, &g.i1, &rt, st);
        if (!g.valid) g.i1 = 0x7fffffff;
        g.started = false;
        const int imin = block_min<Mem>(g, g.i1, rt, &rmin);
#pragma unroll 1
        for (int k = 0; k < NS; k++) ms1[k] = mk(0.0);
        for (int k = 0; k < NF; k++) mf[k] = mk(0.0);
        const int nic = mh->nic, noc = mh->noc;
        const bool ic = !fic && imin <= nic, core = imin <= noc;
        // legs as in k_group_split
        int scale3 = 0;
#pragma unroll 1
        for (int leg = 0; leg < 6; leg++) {
            if ((leg == 0 && !ic) || (leg == 1 && !core) || (leg == 3 && !mh->ocean)) continue;
            const Leg q = leg_of(leg, mh, kn, ev, imin, rmin, ic, core, up);
            if (leg == 1 || leg == 3) {
                if (leg == 3) {
                    for (int k = 0; k < NF; k++) mf[k] = mk(k == 0 ? 1.0 : 0.0);
                } else if (ic) {
                    S::to_fluid(ms1, mf);
                }
                group_walk<Fluid, FluidPoint<KIND>, false, Mem>(g, q.i1, q.i2, q.r1, q.r2, mf, leg == 1 ? st : nullptr);
                if (leg == 1) group_join_rest<Fluid, Mem>(g, noc, mf, st);
                count_work(g, a.work, Fluid::CLS);
                S::to_solid(mf, leg == 1 ? ms1 : ms2);
                continue;
            }
            if (leg == 4 && !mh->ocean)
                for (int k = 0; k < NS; k++) ms2[k] = mk(k == 0 ? 1.0 : 0.0);
            if (leg == 5)
                for (int k = 0; k < NS; k++) ms3[k] = ms1[k];
            cd* const y = leg == 5 ? ms3 : (leg == 4 ? ms2 : ms1);
            group_walk<Solid, Pt, false, Mem>(g, q.i1, q.i2, q.r1, q.r2, y, leg < 4 ? st : nullptr);
            count_work(g, a.work, Solid::CLS);
            if (leg == 0) group_join_rest<Solid, Mem>(g, nic, y, st);
            if (leg == 2) group_join_rest<Solid, Mem>(g, top, y, st);
            scale3 = g.scale;
        }
        const cd delta = S::det(ms3, ms2);
        const cd* mq = up ? ms2 : ms1;
        const cd* mb = up ? ms1 : ms2;
        cd ysph[3][4];
        const int rows = KIND == 2 ? spheroidal_rows(ev) : 3;
#pragma unroll 1
        for (int k = 0; k < 3; k++) {
            if (k >= S::ROWS || !((rows >> k) & 1)) {
                for (int i = 0; i < 4; i++) ysph[k][i] = mk(0.0);
                continue;
            }
            S::row(mq, k, ms3);
            group_walk<Bvec, Pt, true, Mem>(g, is, ir, rs, rr, ms3, nullptr);
            S::resp(mb, ms3, up, delta, huge_pow(scale3 - g.scale), ysph[k]);
        }
        count_work(g, a.work, Bvec::CLS);
        sph_store(g, a, w, ysph);
        bsync<Mem>();
    }
}

// ---------------------------------------------------------------------------
// Toroidal solves (tor_solver), a degree per lane.
// ---------------------------------------------------------------------------
template <int NL>
using TorMem = GroupMem<1, NL, 2, 0>;

template <int NL, int MINB>
__global__ void __launch_bounds__(32 * NL, MINB) k_group_tor(GroupArgs a)
{
    using Mem = TorMem<NL>;
    Group g;
    g.lane = threadIdx.x & 31;
    g.warp = 0;
    g.cnt = 0;
    group_ctx(g, a);
    for (;;) {
        const unsigned long long it = next_item<Mem>(a.counter);
        if ((long long)it >= a.nitems) break;
        const Item w = item_of(a.evs, a.off, a.nev, a.order ? a.order[it] : (long long)it, GROUP_TOR, 32 * NL);
        const EventDev& ev = a.evs[w.e];
        item_ctx(g, ev, w, (int)threadIdx.x);
        const int l = g.c.ll;
        cd yt[2][2];
        if (!ev.pot) {                                // toroidal motion carries no potential
            const ModelHdr* mh = g.c.mh;
            const Knot* kn = g.c.kn;
            const double rr = ev.rr, rs = ev.rs;
            const int ir = ev.ir, is = ev.is;
            const bool up = rr >= rs;
            const int top = up ? is : ir;
            int i1 = tor_start_level(g.c, l, g.c.omega.x, top);
            if (i1 == top && i1 > mh->noc + 1) i1 = i1 - 1;
            cd s[2];
            if (i1 == mh->noc + 1) { s[0] = mk(1.0); s[1] = mk(0.0); }
            else tor_ystart(g.c, i1, kn[i1].r, s);
            g.i1 = g.valid ? i1 : 0x7fffffff;
            g.started = false;
            double rmin;
            const int imin = block_min<Mem>(g, g.i1, kn[i1].r, &rmin);
            cd y1[2], y2[2], y3[2];
            y1[0] = y1[1] = mk(0.0);
            group_walk<TorSys, TorPoint, false, Mem>(g, imin, top, rmin, up ? rs : rr, y1, s);
            group_join_rest<TorSys, Mem>(g, top, y1, s);
            y2[0] = mk(1.0);
            y2[1] = mk(0.0);
            if ((up ? rr : rs) != kn[mh->nsl].r)
                group_walk<TorSys, TorPoint, false, Mem>(g, mh->nsl - 1, up ? ir : is, kn[mh->nsl].r, up ? rr : rs, y2,
                                                         nullptr);
            // the source-side solution continued from the source to the receiver
            y3[0] = up ? y1[0] : y2[0];
            y3[1] = up ? y1[1] : y2[1];
            group_walk<TorSys, TorPoint, false, Mem>(g, is, ir, rs, rr, y3, nullptr);
            const int scale3 = g.scale;
            cd delta, b0, b1, d0, d1;
            if (up) {
                delta = 1.0 / (y2[1] * y3[0] - y2[0] * y3[1]);
                b0 = y1[1]; b1 = -y1[0];
                d0 = delta * y2[0]; d1 = delta * y2[1];
            } else {
                delta = 1.0 / (y3[1] * y1[0] - y3[0] * y1[1]);
                b0 = y2[1]; b1 = -y2[0];
                d0 = delta * y1[0]; d1 = delta * y1[1];
            }
            yt[0][0] = -(d0 * b0); yt[1][0] = -(d1 * b0);
            yt[0][1] = -(d0 * b1); yt[1][1] = -(d1 * b1);
            if (scale3 != 0) {
                const double f = huge_pow(scale3);
                for (int p = 0; p < 2; p++)
                    for (int q = 0; q < 2; q++) yt[p][q] = yt[p][q] * f;
            }
            count_work(g, a.work, TorSys::CLS);
        }
        for (int e = w.e; e >= 0; e = a.next ? a.next[e] : -1) {       // as sph_store
            const EventDev& em = a.evs[e];
            cd ww[5] = {mk(0.0), mk(0.0), mk(0.0), mk(0.0), mk(0.0)};
            if (!em.pot) {
                cd y[2][2] = {{yt[0][0], yt[0][1]}, {yt[1][0], yt[1][1]}};
                toroidal_coefs(g.c, em, l, g.c.omega, y, ww);
            }
            if (!g.valid) continue;
            cd* dst = a.coefs[e] + ((size_t)(l - em.lmin) * NCOEF + 10) * em.nw + (w.j - 1);
            for (int q = 0; q < 5; q++)
                __stcs(reinterpret_cast<double2*>(dst + (size_t)q * em.nw), make_double2(ww[q].x, ww[q].y));
        }
        bsync<Mem>();
    }
}

// ---------------------------------------------------------------------------
// l = 0 (pair_radial of ysg_solvers.cuh): a warp per frequency (ysg_radial.cuh).
// The chain of steps bounds it: a thread per frequency took 0.94 ms on an
// event of 9,060 pairs (10 mHz), a warp 0.21 ms, beside spheroidal solves of
// 0.92 ms; on one event of 300,000 pairs (220 knots, 40 mHz, deck with an
// ocean) the solve stage went from 9.1 to 5.2 ms with it.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(32) k_group_rad(GroupArgs a)
{
    __shared__ RadMem M;
    const int lane = threadIdx.x;
    const long long it = blockIdx.x;
    int lo = 0, hi = a.nev;
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (a.off[mid] <= it) lo = mid;
        else hi = mid;
    }
    const EventDev& ev = a.evs[lo];
    const int j = ev.nw - (int)(it - a.off[lo]);
    Group g;
    group_ctx(g, a);
    Ctx& c = g.c;
    c.ats = (double)ev.ats;
    set_l(c, 0);
    set_omega(c, omega_of(ev, j));
    alpha_steps(c);
    cd sr0[2], yrad[2][2], ph[2] = {mk(0.0), mk(0.0)};
    unsigned n = 0;
    if (ev.grav != 0) rad_wg_warp(c, M, lane, ev.rr, ev.rs, yrad, ev.pot ? ph : nullptr, &n);
    else if (!ev.pot) rad_ng_warp(c, M, lane, ev.rr, ev.rs, ev.ir, ev.is, yrad, &n);
    for (int e = lo; e >= 0; e = a.next ? a.next[e] : -1) {            // as sph_store
        const EventDev& em = a.evs[e];
        source_vector_rad(c, em.is, em.rs, em.mm, sr0);
        cd u3;
        if (em.pot) u3 = (sr0[0] * ph[0] + sr0[1] * ph[1]) / em.rr;    // no gravity, no potential
        else u3 = (sr0[0] * yrad[0][0] + sr0[1] * yrad[0][1]) / em.rr;
        if (em.out != 0) u3 = out_factor(em.out, c.omega) * u3;
        cd* dst = a.coefs[e] + (j - 1);
        if (lane < NCOEF)
            __stcs(reinterpret_cast<double2*>(dst + (size_t)lane * em.nw),
                   lane == 2 ? make_double2(u3.x, u3.y) : make_double2(0.0, 0.0));
    }
    n = __reduce_add_sync(FULL, n);
    if (lane == 0 && n) atomicAdd(&a.work[RadSys::CLS], (unsigned long long)n);
}

// ---------------------------------------------------------------------------
// Order of the items of a list, longest first.
// ---------------------------------------------------------------------------
constexpr int NBUCKET = 256;

// Cost bucket of every item and the buckets' counts.  The cost is that of
// the item's lowest degree: steps from its start level to the source with
// the walk's per-interval floor, the source-to-receiver steps counted once
// per integration over them; tt[k] = sum over intervals below knot k of
// length / alpha.
__global__ void __launch_bounds__(128) k_group_cost(const Knot* __restrict__ kn, const ModelHdr* __restrict__ mh,
                                                    const EventDev* __restrict__ evs,
                                                    const long long* __restrict__ off, int nev, long long nitems,
                                                    int kind, int width, const double* __restrict__ tt,
                                                    unsigned char* __restrict__ bucket, int* __restrict__ hist)
{
    __shared__ int h[NBUCKET];
    for (int b = threadIdx.x; b < NBUCKET; b += blockDim.x) h[b] = 0;
    __syncthreads();
    for (long long it = (long long)blockIdx.x * blockDim.x + threadIdx.x; it < nitems;
         it += (long long)gridDim.x * blockDim.x) {
        const Item w = item_of(evs, off, nev, it, kind, width);
        const EventDev& ev = evs[w.e];
        Ctx c;
        c.kn = kn;
        c.mh = mh;
        const double om = omega_of(ev, w.j).x;
        const bool up = ev.rr >= ev.rs;
        const int lo = up ? ev.is : ev.ir, hi = up ? ev.ir : ev.is;
        const int i1 = kind == GROUP_TOR ? tor_start_level(c, w.lb, om, lo) : sph_start_level(c, w.lb, om, lo);
        const double f = 4.0 * om;
        const double below = f * (tt[lo] - tt[min(i1, lo)]) + 0.6 * (double)max(lo - i1, 0);
        const double across = f * (tt[hi] - tt[lo]) + 0.6 * (double)(hi - lo);
        const double cost = 20.0 + below + (kind == GROUP_TOR ? 1.0 : 1.0 + (double)__popc(spheroidal_rows(ev))) * across;
        int b = (int)(16.0f * log2f((float)cost));
        b = NBUCKET - 1 - min(max(b, 0), NBUCKET - 1);      // longest first
        bucket[it] = (unsigned char)b;
        atomicAdd(&h[b], 1);
    }
    __syncthreads();
    for (int b = threadIdx.x; b < NBUCKET; b += blockDim.x)
        if (h[b]) atomicAdd(&hist[b], h[b]);
}

// The items by bucket; the order inside a bucket is free (an item's result
// does not depend on when it runs).  hist[NBUCKET ..]: items placed so far.
__global__ void __launch_bounds__(NBUCKET) k_group_order(long long nitems, const unsigned char* __restrict__ bucket,
                                                         int* __restrict__ hist, int* __restrict__ order)
{
    __shared__ int start[NBUCKET];
    const int t = threadIdx.x;
    start[t] = hist[t];
    __syncthreads();
    for (int d = 1; d < NBUCKET; d <<= 1) {
        const int v = t >= d ? start[t - d] : 0;
        __syncthreads();
        start[t] += v;
        __syncthreads();
    }
    for (long long it = (long long)blockIdx.x * NBUCKET + t; it < nitems; it += (long long)gridDim.x * NBUCKET) {
        const int b = bucket[it];
        const int at = (b ? start[b - 1] : 0) + atomicAdd(&hist[NBUCKET + b], 1);
        order[at] = (int)it;
    }
}

using GroupFn = void (*)(GroupArgs);
struct GroupKernel {
    GroupFn f;
    int threads;
    size_t smem;
    int width;                    // degrees per item
};
// The forms of a kind's kernel: 0 for lists that fill the GPU, 1 for short ones.
// The kernels without self-gravitation take 255 registers (eight warps per
// SM) too: with 168 their stepping loops spilled 50 values.  Short lists:
// 0.73 -> 0.55 ms (41 degrees to 6 mHz), 1.33 -> 1.0 ms (Cowling,
// 295 degrees to 20 mHz); long ones: 600 degrees to 43 mHz 3.75 -> 3.16 ms.
GroupKernel group_kernel(int kind, int form)
{
    switch (kind) {
        case GROUP_SPH2:
            if (form == 0) return {k_group_lane<2, 4, 2>, 128, sizeof(LaneMem<2, 4>), 128};
            return {k_group_split<2, 4>, 64, sizeof(SphMemOf<2>), 32};
        case GROUP_SPH1:
            if (form == 0) return {k_group_lane<1, 4, 2>, 128, sizeof(LaneMem<1, 4>), 128};
            return {k_group_lane<1, 1, 8>, 32, sizeof(LaneMem<1, 1>), 32};
        case GROUP_SPH0:
            if (form == 0) return {k_group_lane<0, 4, 2>, 128, sizeof(LaneMem<0, 4>), 128};
            return {k_group_lane<0, 1, 8>, 32, sizeof(LaneMem<0, 1>), 32};
        case GROUP_TOR:
            if (form == 0) return {k_group_tor<4, 4>, 128, sizeof(TorMem<4>), 128};
            return {k_group_tor<1, 16>, 32, sizeof(TorMem<1>), 32};
        default: return {k_group_rad, 32, 0, 1};
    }
}

}  // namespace
}  // inline namespace

int group_form_width(int kind, int form) { return group_kernel(kind, form).width; }

long long group_items(int lmin, int lmax, int nw, int grav, int kind, int width)
{
    if (kind == GROUP_RAD) return lmin == 0 ? nw : 0;
    if (kind != GROUP_TOR && kind != GROUP_SPH0 + grav) return 0;
    const int l0 = first_l(lmin, kind);
    return l0 > lmax ? 0 : (long long)((lmax - l0) / width + 1) * nw;
}

int group_blocks(int kind, int form)
{
    int dev = 0, nsm = 0, per = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
        return 0;
    const GroupKernel k = group_kernel(kind, form);
    if (cudaFuncSetAttribute(k.f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)k.smem) != cudaSuccess ||
        cudaFuncSetAttribute(k.f, cudaFuncAttributePreferredSharedMemoryCarveout, 100) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k.f, k.threads, k.smem) != cudaSuccess)
        return 0;
    return nsm * std::max(per, 1);
}

size_t group_order_bytes(long long nitems)
{
    return 2 * NBUCKET * sizeof(int) + (size_t)nitems * (sizeof(int) + 1);
}

cudaError_t launch_group_order(int kind, int width, const Knot* kn, const ModelHdr* mh, const EventDev* evs,
                               const long long* off, int nev, long long nitems, const double* tt, void* order_buf,
                               const int** order, cudaStream_t st)
{
    int* hist = static_cast<int*>(order_buf);
    int* list = hist + 2 * NBUCKET;
    unsigned char* bucket = reinterpret_cast<unsigned char*>(list + nitems);
    cudaError_t e = cudaMemsetAsync(hist, 0, 2 * NBUCKET * sizeof(int), st);
    if (e != cudaSuccess) return e;
    const long long nb = std::min<long long>((nitems + 127) / 128, 2048);
    k_group_cost<<<(unsigned)nb, 128, 0, st>>>(kn, mh, evs, off, nev, nitems, kind, width, tt, bucket, hist);
    k_group_order<<<(unsigned)std::min<long long>((nitems + NBUCKET - 1) / NBUCKET, 1024), NBUCKET, 0, st>>>(
        nitems, bucket, hist, list);
    *order = list;
    return cudaGetLastError();
}

cudaError_t launch_group(int kind, int form, const Knot* kn, const Seg* sg, const ModelHdr* mh, const EventDev* evs,
                         cd* const* coefs, const long long* off, int nev, long long nitems, const double* tt,
                         void* order_buf, unsigned long long* counter, unsigned long long* work, int resident,
                         const int* next, int* launched, cudaStream_t st)
{
    *launched = 0;
    if (nitems <= 0) return cudaSuccess;
    if (nitems >= (1ll << 31)) return cudaErrorInvalidValue;
    GroupArgs a{kn, sg, mh, evs, coefs, off, nullptr, nev, nitems, counter, work, next};
    const GroupKernel k = group_kernel(kind, form);
    if (kind == GROUP_RAD) {
        k_group_rad<<<(unsigned)nitems, 32, 0, st>>>(a);
        *launched = 1;
        return cudaGetLastError();
    }
    cudaError_t e = cudaMemsetAsync(counter, 0, sizeof *counter, st);
    if (e != cudaSuccess) return e;
    if (nitems > resident) {
        e = launch_group_order(kind, k.width, kn, mh, evs, off, nev, nitems, tt, order_buf, &a.order, st);
        if (e != cudaSuccess) return e;
        *launched += 2;
    }
    k.f<<<(unsigned)std::min<long long>(nitems, resident), k.threads, k.smem, st>>>(a);
    *launched += 1;
    return cudaGetLastError();
}

}  // namespace ysg
