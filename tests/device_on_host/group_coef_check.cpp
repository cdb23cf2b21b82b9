// group_coef_check.cpp -- the coefficient matrices of the group solves
// (ysg_group.cuh: a point shared by the degrees, combined per lane) against
// the same expressions in extended precision, on the CPU.
//
//     group_coef_check <yspec model file> <lowest frequency in mHz>
//
// Every interval of the deck, three radii each, degrees 1, 2, 10 and 100,
// eight frequencies from the lowest one in octaves.  The error of an entry is
// taken in units of 2^-53 of the sum of the magnitudes of its terms, as
// module_int.f90:500-786 states them.  Prints the worst entry of every
// system; exit status 0 if all are within their bounds:
//   -omega^2 rho of a fluid without gravity: 10 (the squared frequency, a
//   cubic in three fused steps, one product: 8 roundings);
//   any other entry: 64 (up to some 40 roundings through the attenuation
//   factors, the fused division and gamma).
#include "block_on_host.h"

#include <complex>

#include "yspec_gpu.h"
#include "yspec_host.h"
#include "ysg_group.cuh"

using namespace ysg;

namespace {

using ld = long double;
using lc = std::complex<long double>;

struct Entry {
    const char* name;
    lc want;
    ld scale;
    cd got;
    double bound;
};

std::vector<Seg> segments(const ysg_model& m)
{
    std::vector<Seg> s((size_t)m.nknot + 1);
    std::memset(static_cast<void*>(s.data()), 0, s.size() * sizeof(Seg));
    for (int i = 1; i < m.nknot; i++) {
        const double h = m.r[i] - m.r[i - 1];
        s[i].r0 = m.r[i - 1];
        for (int p = 0; p < NPARAM; p++) {
            const double y0 = m.val[p][i - 1], y1 = m.val[p][i], c0 = m.cs[p][i - 1], c1 = m.cs[p][i];
            s[i].c[p][0] = y0;
            if (h == 0.0) continue;
            s[i].c[p][1] = (y1 - y0) / h - h * (2.0 * c0 + c1) / 6.0;
            s[i].c[p][2] = 0.5 * c0;
            s[i].c[p][3] = (c1 - c0) / (6.0 * h);
        }
    }
    return s;
}

ld value(const Seg& s, double rr, int p)
{
    const ld t = (ld)rr - (ld)s.r0;
    return s.c[p][0] + t * (s.c[p][1] + t * (s.c[p][2] + t * (ld)s.c[p][3]));
}
lc wide(cd a) { return lc(a.x, a.y); }
lc wide(double a) { return lc(a, 0.0L); }
cd narrow(cd a) { return a; }
cd narrow(double a) { return mk(a); }

template <class T>
void push(std::vector<Entry>& e, const char* name, lc want, ld scale, T got, double bound = 64.0)
{
    e.push_back(Entry{name, want, scale, narrow(got), bound});
}

// the lane's matrices, from the point at rr
LaneCtx lane_of(const Ctx& c, const double* pt)
{
    LaneCtx l;
    l.p = pt;
    l.zeta = c.zeta;
    l.zeta2 = c.zeta2;
    l.fl = (double)c.ll;
    l.flp1 = (double)c.llp1;
    l.pib4 = 4.0 * c.pib;
    return l;
}

template <int KIND>
void solid(const Ctx& c, int il, double rr, std::vector<Entry>& e)
{
    alignas(16) double pt[PT] = {};
    SolidPoint<KIND>::eval(c, il, rr, pt);
    const SolidCoef a = solid_amat<KIND>(lane_of(c, pt), rr);
    auto v = [&](int p) { return value(c.sg[il], rr, p); };
    const ld r = rr, rho = v(P_RHO), g = KIND ? v(P_GRAV) : 0.0L, z = c.zeta, z2 = c.zeta2;
    const lc lno = wide(c.lno), w2 = wide(c.omega) * wide(c.omega);
    const lc A = v(P_ACON) * (1.0L + v(P_XA2) * lno), C = v(P_CCON) * (1.0L + v(P_XA2) * lno);
    const lc F = v(P_FCON) * (1.0L + v(P_XLAM) * lno), N = v(P_NCON) * (1.0L + v(P_QMU) * lno);
    const lc L = v(P_LCON) * (1.0L + v(P_QMU) * lno);
    const lc fc = F / C, gam = A - N - F * fc;
    const ld sgam = std::abs(A) + std::abs(N) + std::abs(F * fc), r2 = r * r, sw = std::abs(w2 * rho);
    push(e, "t11", (1.0L - 2.0L * fc) / r, (1.0L + 2.0L * std::abs(fc)) / r, a.t11);
    push(e, "t12", z * fc / r, std::abs(z * fc) / r, a.t12);
    push(e, "t21", wide(0.0) - z / r, z / r, a.t21);
    push(e, "t22", wide(0.0) + 2.0L / r, 2.0L / r, a.t22);
    push(e, "k11", 1.0L / C, std::abs(1.0L / C), a.k11);
    push(e, "k22", 1.0L / L, std::abs(1.0L / L), a.k22);
    push(e, "s11", -w2 * rho + 4.0L * (gam - rho * g * r) / r2, sw + 4.0L * (sgam + rho * g * r) / r2, a.s11);
    push(e, "s12", z * (rho * g * r - 2.0L * gam) / r2, z * (rho * g * r + 2.0L * sgam) / r2, a.s12);
    push(e, "s22", -w2 * rho + (z2 * (gam + N) - 2.0L * N) / r2,
         sw + (z2 * (sgam + std::abs(N)) + 2.0L * std::abs(N)) / r2, a.s22);
    if (KIND == 2) {
        const ld pib = c.pib, l = c.ll;
        push(e, "t31", wide(0.0) - 4.0L * pib * rho, 4.0L * pib * rho, a.t31);
        push(e, "t33", wide(0.0) - l / r, l / r, a.t33);
        push(e, "s13", wide(0.0) - rho * (l + 1.0L) / r, rho * (l + 1.0L) / r, a.s13);
        push(e, "s23", wide(0.0) + rho * z / r, rho * z / r, a.s23);
    }
}

template <int KIND>
void fluid(const Ctx& c, int il, double rr, std::vector<Entry>& e)
{
    alignas(16) double pt[PT] = {};
    FluidPoint<KIND>::eval(c, il, rr, pt);
    const FluidCoef a = fluid_amat<KIND>(lane_of(c, pt), rr);
    auto v = [&](int p) { return value(c.sg[il], rr, p); };
    const ld r = rr, rho = v(P_RHO), g = KIND ? v(P_GRAV) : 0.0L;
    const lc w2 = wide(c.omega) * wide(c.omega), C = v(P_CCON) * (1.0L + v(P_XA2) * wide(c.lno));
    const lc q = (ld)c.zeta2 / (w2 * r * r);
    const ld sq = std::abs(q), sw = std::abs(w2 * rho);
    push(e, "k11", 1.0L / C - q / rho, std::abs(1.0L / C) + sq / rho, a.k11);
    push(e, "t11", g * q - 1.0L / r, g * sq + 1.0L / r, a.t11);
    push(e, "s11", -w2 * rho + rho * g * (g * q - 4.0L / r), sw + rho * g * (g * sq + 4.0L / r), a.s11,
         KIND ? 64.0 : 10.0);
    if (KIND == 2) {
        const ld pib = c.pib, l = c.ll;
        push(e, "t12", q, sq, a.t12);
        push(e, "t21", wide(0.0) - 4.0L * pib * rho, 4.0L * pib * rho, a.t21);
        push(e, "t22", wide(0.0) - l / r, l / r, a.t22);
        push(e, "s12", rho * (g * q - (l + 1.0L) / r), rho * (g * sq + (l + 1.0L) / r), a.s12);
        push(e, "s22", rho * q, rho * sq, a.s22);
    }
}

void toroidal(const Ctx& c, int il, double rr, std::vector<Entry>& e)
{
    alignas(16) double pt[PT] = {};
    TorPoint::eval(c, il, rr, pt);
    const TorCoef a = tor_amat(lane_of(c, pt), rr);
    auto v = [&](int p) { return value(c.sg[il], rr, p); };
    const ld r = rr, z = (ld)c.zeta2 - 2.0L;
    const lc w2 = wide(c.omega) * wide(c.omega), q = 1.0L + v(P_QMU) * wide(c.lno);
    push(e, "t", wide(0.0) + 2.0L / r, 2.0L / r, a.t);
    push(e, "k", 1.0L / (v(P_LCON) * q), std::abs(1.0L / (v(P_LCON) * q)), a.k);
    push(e, "s", -w2 * v(P_RHO) + z * v(P_NCON) * q / (r * r),
         std::abs(w2 * v(P_RHO)) + z * std::abs(v(P_NCON) * q) / (r * r), a.s);
}

struct Worst {
    double e = 0.0;
    const char* name = "-";
    double r = 0.0, mhz = 0.0;
    int l = 0;
};

}  // namespace

int main(int argc, char** argv)
{
    if (argc < 3) return 2;
    ysh_model* m = nullptr;
    if (ysh_read_model(argv[1], &m)) return 2;
    ysg_model view;
    ysh_model_view(m, &view);
    const std::vector<Seg> sg = segments(view);
    ModelHdr mh{};
    mh.nknot = view.nknot;
    mh.tref = view.tref;
    mh.pibigg = view.pibigg;
    ysh_norms nm;
    ysh_norms_get(&nm);
    bool ok = true;
    const char* systems[7] = {"solid, no gravity", "solid, Cowling", "solid, gravity",
                              "fluid, no gravity", "fluid, Cowling", "fluid, gravity", "toroidal"};
    Worst worst[7];
    for (int f = 0; f < 8; f++) {
        const double mhz = std::atof(argv[2]) * (double)(1 << f), w = 6.283185307179586e-3 * mhz * nm.t_norm;
        for (int l : {1, 2, 10, 100}) {
            Ctx c;
            std::memset(static_cast<void*>(&c), 0, sizeof c);
            c.mh = &mh;
            c.sg = sg.data();
            c.pib = mh.pibigg;
            c.ats = 1.0;
            set_l(c, l);
            set_omega(c, mk(w, -0.05 * w));
            for (int i = 1; i < view.nknot; i++) {
                const double r0 = view.r[i - 1], h = view.r[i] - r0;
                if (h == 0.0) continue;
                const bool is_fluid = view.val[P_LCON][i - 1] == 0.0 && view.val[P_LCON][i] == 0.0;
                for (double x : {r0 + 0.11 * h, r0 + 0.5 * h, r0 + 0.93 * h}) {
                    std::vector<Entry> e[7];
                    if (is_fluid) {
                        fluid<0>(c, i, x, e[3]);
                        fluid<1>(c, i, x, e[4]);
                        fluid<2>(c, i, x, e[5]);
                    } else {
                        solid<0>(c, i, x, e[0]);
                        solid<1>(c, i, x, e[1]);
                        solid<2>(c, i, x, e[2]);
                        toroidal(c, i, x, e[6]);
                    }
                    for (int s = 0; s < 7; s++)
                        for (const Entry& n : e[s]) {
                            const double err = (double)(std::abs(wide(n.got) - n.want) / (n.scale * 0x1p-53L));
                            if (err > worst[s].e) worst[s] = Worst{err, n.name, x, mhz, l};
                            if (!(err <= n.bound)) {
                                if (ok) std::printf("%s %s at r %.6f, l %d, %.2f mHz: %.1f\n", systems[s], n.name, x, l, mhz, err);
                                ok = false;
                            }
                        }
                }
            }
        }
    }
    for (int s = 0; s < 7; s++)
        std::printf("%-18s worst %6.2f  %s, r %.6f, l %d, %.2f mHz\n", systems[s], worst[s].e, worst[s].name, worst[s].r,
                    worst[s].l, worst[s].mhz);
    ysh_free_model(m);
    return ok ? 0 : 1;
}
