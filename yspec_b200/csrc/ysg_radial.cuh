// ysg_radial.cuh -- the l = 0 solves by a warp per frequency.
//
// rad_solver_wg and rad_solver_ng (module_solver.f90:335-561) integrate a
// 2-component linear system along one long chain of Cash-Karp steps per
// frequency: few solves, each hundreds to thousands of dependent steps.
// The step is linear, so the 32 lanes form the 2 x 2 matrices of 32
// consecutive steps (or pieces between grid points) at once, from two unit
// vectors each, and the solution is carried through them by 2 x 2 products:
// the serial chain holds four dependent multiply-adds per step instead of
// six coefficient matrices with a division each.
#pragma once
#include "ysg_group.cuh"

namespace ysg {
inline namespace YSG_VARIANT {
namespace {

// Matrix of an integration: (y0, y1) -> (a y0 + b y1, c y0 + d y1).
struct RadMat {
    cd a, b, c, d;
};

__device__ __forceinline__ void rad_apply(const RadMat& m, cd* y)
{
    const cd y0 = y[0], y1 = y[1];
    y[0] = cmac(m.a * y0, m.b, y1);
    y[1] = cmac(m.c * y0, m.d, y1);
}
__device__ __forceinline__ void rad_apply_T(const RadMat& m, cd* y)
{
    const cd y0 = y[0], y1 = y[1];
    y[0] = cmac(m.a * y0, m.c, y1);
    y[1] = cmac(m.b * y0, m.d, y1);
}

// One Cash-Karp step (module_int.f90:2016-2064) applied to both columns of m.
__device__ __noinline__ void rad_step(Ctx& c, int iv, double x, double h, RadMat& m)
{
    cd y[4] = {m.a, m.c, m.b, m.d}, k[6][4];
    c.il = iv;
#pragma unroll 1
    for (int s = 0; s < 6; s++) {
        cd v[4] = {y[0], y[1], y[2], y[3]};
#pragma unroll 1
        for (int t = 0; t < s; t++) {
            // ck_in holds the rows of the tableau but the last, whose weights are ck_fold[4] and ck_w[4]
            const double w = h * (s < 5 ? ck_in[s][t] : (t < 4 ? ck_fold[4][t] : ck_w[4]));
#pragma unroll
            for (int q = 0; q < 4; q++) v[q] = cmac(v[q], w, k[t][q]);
        }
        const RadCoef a = rad_amat(c, x + ck_a[s] * h);
        k[s][0] = cmac(a.t * v[0], a.k, v[1]);
        k[s][1] = cmsc(a.s * v[0], a.t, v[1]);
        k[s][2] = cmac(a.t * v[2], a.k, v[3]);
        k[s][3] = cmsc(a.s * v[2], a.t, v[3]);
    }
#pragma unroll
    for (int q = 0; q < 4; q++)
        y[q] = cmac(cmac(cmac(cmac(y[q], (37.0 / 378.0) * h, k[0][q]), (250.0 / 621.0) * h, k[2][q]),
                         (125.0 / 594.0) * h, k[3][q]), (512.0 / 1771.0) * h, k[5][q]);
    m = RadMat{y[0], y[2], y[1], y[3]};
}

// yint without rescaling over (i1, r1) .. (i2, r2) as a matrix; the steps
// are added to *n.
__device__ __noinline__ RadMat rad_piece(Ctx& c, int i1, int i2, double r1, double r2, unsigned* n)
{
    RadMat m{mk(1.0), mk(0.0), mk(0.0), mk(1.0)};
    if (r1 == r2) return m;
    const bool up = r2 > r1;
    const Knot* kn = c.kn;
    for (int i = i1; up ? i <= i2 : i >= i2; i += up ? 1 : -1) {
        double a, b;
        if (up) {
            a = (i == i1) ? r1 : kn[i].r;
            b = (i == i2) ? r2 : kn[i + 1].r;
        } else {
            a = (i == i1) ? r1 : kn[i + 1].r;
            b = (i == i2) ? r2 : kn[i].r;
        }
        if (a == b) continue;
        const double nf = floor(fabs(b - a) / steps(c, i));
        const int ns = 1 + (int)fmin(nf, 4194304.0);
        const double h = (b - a) / (double)ns;
        for (int j = 0; j < ns; j++) rad_step(c, i, __dadd_rn(a, __dmul_rn((double)j, h)), h, m);
        *n += (unsigned)ns;
    }
    return m;
}

// ---------------------------------------------------------------------------
// Grid of module_model.f90:578-787 by index: pre[i] grid points lie below
// interval i.
// ---------------------------------------------------------------------------
constexpr int RAD_KNOTS = 804;    // ysg_model_upload accepts at most 798 knots

struct RadMem {
    RadMat m[32];
    int pre[RAD_KNOTS];
};

struct RadGrid {
    const Knot* kn;
    const int* pre;
    int nknot, ngrid, iss, irr;   // points; indices of the source and the receiver
    double rr, rs, drr;
};

__device__ __forceinline__ RadGrid rad_grid(const Ctx& c, double rr, double rs, int* pre, int lane)
{
    RadGrid g{c.kn, pre, c.mh->nknot, 0, 0, 0, rr, rs, c.dr};
    for (int base = 1; base <= g.nknot - 1; base += 32) {
        const int i = base + lane;
        int cnt = 0, si = 0, ri = 0;
        if (i <= g.nknot - 1 && g.kn[i].r != g.kn[i + 1].r) {
            GridSeg sg[3];
            int sa, ra;
            const int ns = grid_segs(g.kn[i].r, g.kn[i + 1].r, rs, rr, sg, &sa, &ra);
            for (int q = 0; q < ns; q++) {
                cnt += seg_npts(sg[q], g.drr) - (sg[q].first - 1);
                if (q == sa) si = cnt;
                if (q == ra) ri = cnt;
            }
        }
        int incl = cnt;
        for (int d = 1; d < 32; d <<= 1) {
            const int v = __shfl_up_sync(FULL, incl, d);
            if (lane >= d) incl += v;
        }
        const int at = g.ngrid + incl - cnt;
        if (i <= g.nknot) pre[i] = at;
        g.iss = max(g.iss, __reduce_max_sync(FULL, si ? at + si : 0));
        g.irr = max(g.irr, __reduce_max_sync(FULL, ri ? at + ri : 0));
        g.ngrid += __shfl_sync(FULL, incl, 31);
    }
    __syncwarp();
    return g;
}

// Interval and radius of grid point k (1 .. ngrid).
__device__ __forceinline__ void rad_point(const RadGrid& g, int k, int* iv, double* r)
{
    int lo = 1, hi = g.nknot;                 // pre[lo] < k, the last such interval below hi
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (g.pre[mid] < k) lo = mid;
        else hi = mid;
    }
    GridSeg sg[3];
    int sa, ra, m = k - g.pre[lo];
    const int ns = grid_segs(g.kn[lo].r, g.kn[lo + 1].r, g.rs, g.rr, sg, &sa, &ra);
    int q = 0, np = seg_npts(sg[0], g.drr);
    while (q < ns - 1 && m > np - (sg[q].first - 1)) {
        m -= np - (sg[q].first - 1);
        q++;
        np = seg_npts(sg[q], g.drr);
    }
    const double drt = (sg[q].b - sg[q].a) / (double)(np - 1);
    *iv = lo;
    *r = __dadd_rn(sg[q].a, __dmul_rn((double)(sg[q].first + m - 2), drt));
}

// Carries y through the matrices of the lanes 0 .. n - 1 in turn (published
// in shared memory); the lane keeps the result after its own.
__device__ __forceinline__ void rad_scan(RadMem& M, const RadMat& m, int lane, int n, cd* y, cd* own)
{
    __syncwarp();
    M.m[lane] = m;
    __syncwarp();
    own[0] = y[0];
    own[1] = y[1];
    for (int t = 0; t < n; t++) {
        rad_apply(M.m[t], y);
        if (lane == t) {
            own[0] = y[0];
            own[1] = y[1];
        }
    }
}

__device__ __forceinline__ cd warp_sum(cd v)
{
    for (int d = 16; d > 0; d >>= 1) {
        v.x += __shfl_xor_sync(FULL, v.x, d);
        v.y += __shfl_xor_sync(FULL, v.y, d);
    }
    return v;
}
__device__ __forceinline__ cd lane_value(cd v, int lane)
{
    return mk(__shfl_sync(FULL, v.x, lane), __shfl_sync(FULL, v.y, lane));
}

// rad_solver_wg (ysg_solvers.cuh) by a warp: every lane returns the
// responses, and with pot non-null the potentials; n counts the lane's steps.
__device__ __noinline__ void rad_wg_warp(Ctx& c, RadMem& M, int lane, double rr, double rs, cd yout[2][2], cd* pot,
                                         unsigned* n)
{
    const RadGrid g = rad_grid(c, rr, rs, M.pre, lane);
    const int iss = g.iss, irr = g.irr, ngrid = g.ngrid;
    cd yrec[2] = {mk(0.0), mk(0.0)}, own[2];
    cd s1 = mk(0.0), s2 = mk(0.0), g1_iss = mk(0.0), g2_next = mk(0.0);
    double r_iss = 0.0, r_next = 0.0;
    // upward through the points 2 .. iss, piece k from point k - 1
    cd y1[2] = {mk(0.0), mk(0.0)};
    cd gprev = mk(0.0);                          // y1s(1) / r at the batch's previous point
    for (int k0 = 2; k0 <= iss; k0 += 32) {
        const int k = k0 + lane, nb = min(32, iss - k0 + 1);
        RadMat m{mk(1.0), mk(0.0), mk(0.0), mk(1.0)};
        double rk = 0.0, rp = 0.0;
        int ik = 1, ip = 1;
        if (lane < nb) {
            rad_point(g, k, &ik, &rk);
            rad_point(g, k - 1, &ip, &rp);
        }
        double r0 = rp;
        if (k0 == 2) {                           // the first piece starts near the centre
            const double rt = fmin(0.1 * g.drr, 0.1 * __shfl_sync(FULL, rk, 0));
            rad_ystart<true>(c, 1, rt, y1);
            if (lane == 0) {
                r0 = rt;
                ip = 1;
            }
        }
        if (lane < nb) m = rad_piece(c, ip, ik, r0, rk, n);
        rad_scan(M, m, lane, nb, y1, own);
        if (irr >= k0 && irr < k0 + nb) {
            yrec[0] = lane_value(own[0], irr - k0);
            yrec[1] = lane_value(own[1], irr - k0);
        }
        if (pot) {
            const cd gk = lane < nb ? own[0] / rk : mk(0.0);
            cd gp = mk(__shfl_up_sync(FULL, gk.x, 1), __shfl_up_sync(FULL, gk.y, 1));
            if (lane == 0) gp = gprev;
            if (lane < nb && k <= irr) s1 = s1 + (0.5 * (rk - rp)) * (gp + gk);
            gprev = lane_value(gk, nb - 1);
            if (k0 + nb - 1 == iss) {
                g1_iss = gprev;
                r_iss = __shfl_sync(FULL, rk, nb - 1);
            }
        }
    }
    // downward from point ngrid to iss, piece k from point k + 1
    cd y2[2] = {mk(1.0), mk(0.0)};
    cd gabove = mk(0.0);                         // y2s(1) / r at the point above the batch
    if (pot && ngrid > iss) {
        int iv;
        rad_point(g, ngrid, &iv, &r_next);
        gabove = y2[0] / r_next;
        g2_next = gabove;
    }
    for (int k0 = ngrid - 1; k0 >= iss; k0 -= 32) {
        const int k = k0 - lane, nb = min(32, k0 - iss + 1);
        RadMat m{mk(1.0), mk(0.0), mk(0.0), mk(1.0)};
        double rk = 0.0, rp = 0.0;
        int ik = 1, ip = 1;
        if (lane < nb) {
            rad_point(g, k, &ik, &rk);
            rad_point(g, k + 1, &ip, &rp);
            m = rad_piece(c, ip, ik, rp, rk, n);
        }
        rad_scan(M, m, lane, nb, y2, own);
        if (irr > iss && irr <= k0 && irr > k0 - nb) {
            yrec[0] = lane_value(own[0], k0 - irr);
            yrec[1] = lane_value(own[1], k0 - irr);
        }
        if (pot) {
            const cd gk = lane < nb ? own[0] / rk : mk(0.0);
            cd gp = mk(__shfl_up_sync(FULL, gk.x, 1), __shfl_up_sync(FULL, gk.y, 1));
            if (lane == 0) gp = gabove;
            // the segment [k, k + 1], above the source and up to the receiver
            if (lane < nb && k > iss && k + 1 <= irr) s2 = s2 + (0.5 * (rp - rk)) * (gk + gp);
            gabove = lane_value(gk, nb - 1);
            // the lowest point above the source
            const int at = k0 - (iss + 1);
            if (at >= 0 && at < nb) {
                g2_next = lane_value(gk, at);
                r_next = __shfl_sync(FULL, rk, at);
            }
        }
    }
    // a receiver at the surface point above the source's walk
    if (irr > iss && irr == ngrid) {
        yrec[0] = mk(1.0);
        yrec[1] = mk(0.0);
    }
    const cd delta = 1.0 / (y2[1] * y1[0] - y2[0] * y1[1]);
    cd b0, b1;
    if (irr <= iss) { b0 = y2[1]; b1 = -y2[0]; }
    else { b0 = y1[1]; b1 = -y1[0]; }
    const cd d0 = delta * yrec[0], d1 = delta * yrec[1];
    yout[0][0] = -(d0 * b0); yout[1][0] = -(d1 * b0);
    yout[0][1] = -(d0 * b1); yout[1][1] = -(d1 * b1);
    if (pot) {
        s1 = warp_sum(s1);
        s2 = warp_sum(s2);
        // the segment across the source, [iss, iss + 1]
        if (iss + 1 <= irr && iss + 1 <= ngrid) {
            s1 = s1 + (0.5 * (r_next - r_iss)) * g1_iss;
            s2 = s2 + (0.5 * (r_next - r_iss)) * g2_next;
        }
        const cd f = (rr * (4.0 * c.mh->pibigg)) * delta;
        pot[0] = f * (y2[1] * s1 + y1[1] * s2);
        pot[1] = f * (-(y2[0] * s1) - y1[0] * s2);
    }
}

// yint<RadSys> with rescaling by a warp: y and the scale count in every lane.
__device__ __noinline__ void rad_walk(Ctx& c, RadMem& M, int lane, int i1, int i2, double r1, double r2, cd* y,
                                      int* scale, unsigned* n)
{
    Walk w;
    walk_init(w, i1, i2, r1, r2, false);
    while (walk_chunk(c, lane, w)) {
        const int nb = min(32, w.total - w.s0);
        int iv;
        double x, h;
        walk_step(w, w.s0 + lane, &iv, &x, &h);
        RadMat m{mk(1.0), mk(0.0), mk(0.0), mk(1.0)};
        if (lane < nb) {
            rad_step(c, iv, x, h, m);
            *n += 1u;
        }
        __syncwarp();
        M.m[lane] = m;
        __syncwarp();
        for (int t = 0; t < nb; t++) {
            rad_apply(M.m[t], y);
            rescale<2>(y, scale);
        }
        w.s0 += nb;
    }
}

// rad_solver_ng (ysg_solvers.cuh) by a warp.
__device__ __noinline__ void rad_ng_warp(Ctx& c, RadMem& M, int lane, double rr, double rs, int ir, int is,
                                         cd yout[2][2], unsigned* n)
{
    const ModelHdr* mh = c.mh;
    const Knot* kn = c.kn;
    int scale1 = 0, scale2 = 0, scale3 = 0;
    const bool up = rr >= rs;
    cd y1[2], y2[2] = {mk(1.0), mk(0.0)}, y3[2];
    const double rt = fmin(0.1 * c.dr, 0.1 * kn[2].r);
    rad_ystart<false>(c, 1, rt, y1);
    const int ilo = up ? is : ir, ihi = up ? ir : is, top = up ? mh->nknot : mh->nsl;
    const double rlo = up ? rs : rr, rhi = up ? rr : rs;
    rad_walk(c, M, lane, 1, ilo, rt, rlo, y1, &scale1, n);
    rad_walk(c, M, lane, top - 1, ihi, kn[top].r, rhi, y2, &scale2, n);
    y3[0] = y2[0];
    y3[1] = y2[1];
    rad_walk(c, M, lane, ihi, ilo, rhi, rlo, y3, &scale3, n);
    cd delta = y3[1] * y1[0] - y3[0] * y1[1];
    delta = cabs(delta) < 1.0e-100 ? mk(0.0) : 1.0 / delta;
    const cd* ya = up ? y1 : y2;   // source-side solution forming b
    const cd* yb = up ? y2 : y1;   // solution evaluated at the receiver
    const cd b0 = ya[1], b1 = -ya[0];
    const cd d0 = delta * yb[0], d1 = delta * yb[1];
    // the receiver-below branch undoes only a positive scale (module_solver.f90:433-437)
    const double f = (up || scale3 > 0) ? huge_pow(scale3) : 1.0;
    yout[0][0] = (-(d0 * b0)) * f; yout[1][0] = (-(d1 * b0)) * f;
    yout[0][1] = (-(d0 * b1)) * f; yout[1][1] = (-(d1 * b1)) * f;
}

}  // namespace
}  // inline namespace
}  // namespace ysg
