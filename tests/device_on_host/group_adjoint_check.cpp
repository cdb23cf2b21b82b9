// group_adjoint_check.cpp -- the reverse sweeps by groups (k_group_adjoint.cu)
// run on the CPU, thread by thread, against the sweep of one pair
// (ysg_pair_adjoint.cuh).
//
//     group_adjoint_check <yspec parameter file>
//
// GROUP_KERNELS is the device part of k_group_adjoint.cu.  Per kernel the first
// and the last item run, with random adjoints for most of their pairs: every
// fifth pair and a warp of 32 degrees do not reach the misfit.  Index checks as
// in group_solve_check.cpp.  Prints the largest difference of the gradient
// relative to the largest entry of the same parameter and power, or to 1e-12 of
// the largest of all for parameters that hardly enter; exit status 0 if all
// are below 1e-10 (the sum of a few hundred steps' terms of either sign).
#include "block_on_host.h"

template <class T> inline T atomicOr(T* p, T v)
{
    const T old = *p;
    *p = old | v;
    return old;
}
#include <random>

#include GROUP_KERNELS
#include "model_tables.h"

namespace ysg {
inline namespace YSG_VARIANT {
namespace {
alignas(16) unsigned char group_smem[1 << 18];
}
}  // namespace
}  // namespace ysg

#if defined(__SANITIZE_ADDRESS__)
#include <sanitizer/asan_interface.h>
#else
#define ASAN_POISON_MEMORY_REGION(p, n) ((void)0)
#define ASAN_UNPOISON_MEMORY_REGION(p, n) ((void)0)
#endif

using namespace ysg;

namespace {

constexpr int CAP = 2500, GRID = 5000, WIDTH = 128;      // logged steps, grid points, degrees per item

struct Kernel {
    const char* name;
    int kind;
    size_t smem;
    int states;
    void (*f)(AdjArgs);
};

}  // namespace

int main(int argc, char** argv)
{
    ysh_params P;
    ysh_model* m = nullptr;
    ysh_event E;
    if (argc < 2 || ysh_read_params(argv[1], &P) || ysh_read_model(P.model_file, &m) || ysh_event_setup(m, &P, &E)) return 2;
    Tables T;
    build_tables(m, T);
    const EventDev ev = event_constants(E.ev, T.view);
    const int n = T.mh.nknot, L = ev.lmax - ev.lmin + 1;
    std::vector<std::vector<Knot>> ukn(NPARAM, std::vector<Knot>(T.kn.size()));
    std::vector<std::vector<Seg>> usg(NPARAM, std::vector<Seg>(T.sg.size()));
    UnitDirs U;
    for (int p = 0; p < NPARAM; p++) {
        std::memset(static_cast<void*>(ukn[p].data()), 0, ukn[p].size() * sizeof(Knot));
        std::memset(static_cast<void*>(usg[p].data()), 0, usg[p].size() * sizeof(Seg));
        for (Knot& k : ukn[p]) k.v[p][0] = 1.0;
        for (Seg& s : usg[p]) s.c[p][0] = 1.0;
        U.kn[p] = ukn[p].data();
        U.sg[p] = usg[p].data();
    }
    const Kernel kernels[3] = {
        ev.grav == 2 ? Kernel{"spheroidal", GROUP_SPH2, sizeof(SphAdjMem<2, 4>), SphAdjMem<2, 4>::LOG_N, k_gadj_sph<2, 4, 2>}
        : ev.grav == 1 ? Kernel{"spheroidal", GROUP_SPH1, sizeof(SphAdjMem<1, 4>), SphAdjMem<1, 4>::LOG_N, k_gadj_sph<1, 4, 2>}
                       : Kernel{"spheroidal", GROUP_SPH0, sizeof(SphAdjMem<0, 4>), SphAdjMem<0, 4>::LOG_N, k_gadj_sph<0, 4, 2>},
        {"toroidal", GROUP_TOR, sizeof(TorAdjMem<4>), TorAdjMem<4>::LOG_N, k_gadj_tor<4, 4>},
        {"radial", GROUP_RAD, 0, 0, nullptr}};
    std::mt19937_64 rng(4);
    std::normal_distribution<double> nd;
    // logs of the single sweeps
    std::vector<cd> ly((size_t)CAP * 14), cy((size_t)CAP * 14), gy((size_t)GRID * 4);
    std::vector<double> lx(CAP), lh(CAP), lf(CAP), cx(CAP), ch(CAP), cf(CAP), gr(GRID);
    std::vector<int> li(CAP), ci(CAP), gi(GRID);
    StepLog SL{ly.data(), lx.data(), lh.data(), li.data(), lf.data(), CAP, 1};
    StepLog CL{cy.data(), cx.data(), ch.data(), ci.data(), cf.data(), CAP, 1};
    GridLog GL{gy.data(), gr.data(), gi.data(), GRID, 1};
    bool good = true;
    for (const Kernel& k : kernels) {
        const bool rad = k.kind == GROUP_RAD;
        const int l0 = rad ? 0 : first_l(ev.lmin, k.kind);
        if (l0 > ev.lmax || (rad && ev.lmin > 0)) continue;
        const long long items = rad ? ev.nw : (long long)((ev.lmax - l0) / WIDTH + 1) * ev.nw;
        std::vector<int> order = some_items(items, 0);
        std::vector<cd> coefb((size_t)L * NCOEF * ev.nw, mk(0.0));
        std::vector<double> got((size_t)(n + 1) * NPARAM * 4, 0.0), want(got.size(), 0.0);
        SegGrad G;
        G.init(want.data());
        for (int it : order) {
            const int b = rad ? 0 : it / ev.nw, j = ev.nw - it % ev.nw, la = l0 + WIDTH * b;
            for (int l = la; l < la + (rad ? 1 : WIDTH) && l <= ev.lmax; l++) {
                if (!rad && ((l - la) % 5 == 3 || ((l - la) >= 32 && (l - la) < 64))) continue;
                cd w[NCOEF] = {};
                const int q0 = k.kind == GROUP_TOR ? 10 : rad ? 2 : 0, q1 = k.kind == GROUP_TOR ? 15 : rad ? 3 : 10;
                for (int q = q0; q < q1; q++) {
                    w[q] = mk(nd(rng), nd(rng));
                    coefb[((size_t)(l - ev.lmin) * NCOEF + q) * ev.nw + (j - 1)] = w[q];
                }
                primal::Ctx c;
                std::memset(static_cast<void*>(&c), 0, sizeof c);
                c.kn = T.kn.data();
                c.sg = T.sg.data();
                c.mh = &T.mh;
                c.pib = T.mh.pibigg;
                c.ats = ev.ats;
                good = (rad ? pair_radial_adj(c, U, ev, j, w, SL, CL, GL, G)
                        : k.kind == GROUP_TOR ? pair_toroidal_adj(c, U, ev, l, j, w + 10, SL, CL, G)
                                              : pair_spheroidal_adj(c, U, ev, l, j, w, w + 5, SL, CL, G)) && good;
            }
        }
        G.flush();
        std::vector<EventDev> evs = {ev};
        std::vector<ModelHdr> mh = {T.mh};
        std::vector<unsigned long long> counter(1, 0);
        std::vector<long long> off = {0, items};
        int status = 0;
        AdjArgs a{T.kn.data(), T.sg.data(), mh.data(), evs.data(), U, coefb.data(), off.data(), order.data(),
                  (long long)order.size(), AdjLogs{}, got.data(), counter.data(), &status};
        if (rad) {
            const size_t nt = (size_t)ev.nw * 32 * RAD_PIECE_STEPS, ng = (size_t)ev.nw * GRID;
            std::vector<cd> wy(nt * 14), wg(ng * 4);
            std::vector<double> wx(nt), wh(nt), wf(nt), wr(ng);
            std::vector<int> wl(nt), wi(ng);
            AdjStepArrays ws{};
            ws.n = RAD_PIECE_STEPS;
            ws.y = wy.data();
            ws.x = wx.data();
            ws.h = wh.data();
            ws.f = wf.data();
            ws.il = wl.data();
            for (int it : order)
                block::run(32, (unsigned)it, (unsigned)ev.nw, [&] { k_gadj_rad(a, RadLog{wg.data(), wr.data(), wi.data(), GRID}, ws); });
        } else {
            const size_t nt = WIDTH;
            std::vector<cd> sy((size_t)CAP * k.states * nt), chain(sy.size());
            std::vector<double> sf((size_t)CAP * nt), cfac(sf.size());
            a.w.nthreads = (int)nt;
            a.w.s.n = a.w.c.n = CAP;
            a.w.s.y = sy.data();
            a.w.s.f = sf.data();
            a.w.c.y = chain.data();
            a.w.c.f = cfac.data();
            ASAN_POISON_MEMORY_REGION(group_smem + k.smem, sizeof group_smem - k.smem);
            block::run(WIDTH, 0, 1, [&] { k.f(a); });
            ASAN_UNPOISON_MEMORY_REGION(group_smem, sizeof group_smem);
        }
        double worst = 0.0;
        for (int r = 0; r < 5; r++) {
            double a0 = 0.0, b0 = 0.0, size = 0.0;
            for (size_t e = 0; e < want.size(); e++) {
                const double d = nd(rng);
                a0 += got[e] * d;
                b0 += want[e] * d;
                size += std::fabs(want[e] * d);
            }
            worst = std::max(worst, size > 0.0 && std::isfinite(a0) ? std::fabs(a0 - b0) / size : INFINITY);
        }
        std::printf("%-10s %zu items, largest difference %.2e, status %d\n", k.name, order.size(), worst, status);
        good = good && status == 0 && worst <= 1e-11;
    }
    ysh_free_event(&E);
    ysh_free_model(m);
    ysh_free_params(&P);
    return good ? 0 : 1;
}
