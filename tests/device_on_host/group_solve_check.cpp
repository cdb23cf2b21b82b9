// group_solve_check.cpp -- the group kernels (k_solve_group.cu) run on the CPU,
// thread by thread, against the solve of one pair (ysg_solvers.cuh).
//
//     group_solve_check <yspec parameter file>
//
// GROUP_KERNELS is the device part of k_solve_group.cu.  Both forms of every
// kernel of the event's gravity setting run on the first, the last and one
// middle item; built with -fsanitize=address,undefined every index is checked,
// and uninitialised locals hold a pattern.  Prints per kernel the largest
// difference of a pair's coefficients relative to the pair's largest one; exit
// status 0 if all are below 2e-12: the two forms take the same steps, a few
// hundred of six stages with ten roundings of 1.1e-16 each.
#include "block_on_host.h"

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

struct Kernel {
    const char* name;
    int kind, width, threads;
    size_t smem;
    void (*f)(GroupArgs);
};

template <int KIND>
void add_spheroidal(std::vector<Kernel>& v)
{
    v.push_back({"wide", GROUP_SPH0 + KIND, 128, 128, sizeof(LaneMem<KIND, 4>), k_group_lane<KIND, 4, 2>});
    if (KIND == 2) v.push_back({"split", GROUP_SPH2, 32, 64, sizeof(SphMemOf<2>), k_group_split<2, 4>});
    else v.push_back({"narrow", GROUP_SPH0 + KIND, 32, 32, sizeof(LaneMem<KIND, 1>), k_group_lane<KIND, 1, 8>});
}

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
    const int L = ev.lmax - ev.lmin + 1;
    std::vector<Kernel> kernels;
    if (ev.grav == 0) add_spheroidal<0>(kernels);
    if (ev.grav == 1) add_spheroidal<1>(kernels);
    if (ev.grav == 2) add_spheroidal<2>(kernels);
    kernels.push_back({"toroidal wide", GROUP_TOR, 128, 128, sizeof(TorMem<4>), k_group_tor<4, 4>});
    kernels.push_back({"toroidal narrow", GROUP_TOR, 32, 32, sizeof(TorMem<1>), k_group_tor<1, 16>});
    kernels.push_back({"radial", GROUP_RAD, 1, 32, 0, k_group_rad});
    double worst = 0.0;
    for (const Kernel& k : kernels) {
        const bool rad = k.kind == GROUP_RAD;
        const int l0 = rad ? 0 : first_l(ev.lmin, k.kind);
        const long long items = rad ? (ev.lmin == 0 ? ev.nw : 0) : l0 > ev.lmax ? 0 : (long long)((ev.lmax - l0) / k.width + 1) * ev.nw;
        if (items == 0) continue;
        std::vector<int> order = some_items(items, 1);
        // exact copies of what the kernel may read and write, so that the next byte is out of bounds
        std::vector<cd> coef((size_t)L * NCOEF * ev.nw, mk(NAN));
        std::vector<cd*> coefs = {coef.data()};
        std::vector<long long> off = {0, items};
        std::vector<unsigned long long> work(NSYS, 0), counter(1, 0);
        std::vector<EventDev> evs = {ev};
        std::vector<ModelHdr> mh = {T.mh};
        const GroupArgs a{T.kn.data(), T.sg.data(), mh.data(), evs.data(), coefs.data(), off.data(), order.data(), 1,
                          (long long)order.size(), counter.data(), work.data(), nullptr};
        ASAN_POISON_MEMORY_REGION(group_smem + k.smem, sizeof group_smem - k.smem);
        if (rad) {
            for (int it : order) block::run(32, (unsigned)it, (unsigned)items, [&] { k.f(a); });
        } else {
            block::run(k.threads, 0, 1, [&] { k.f(a); });
        }
        ASAN_UNPOISON_MEMORY_REGION(group_smem, sizeof group_smem);
        double diff = 0.0;
        for (int it : order) {
            const int b = it / ev.nw, j = ev.nw - it % ev.nw, la = l0 + k.width * b;
            for (int l = la; l < la + k.width && l <= ev.lmax; l++) {
                Ctx c;
                std::memset(static_cast<void*>(&c), 0, sizeof c);
                c.kn = T.kn.data();
                c.sg = T.sg.data();
                c.mh = &T.mh;
                c.pib = T.mh.pibigg;
                c.ats = ev.ats;
                cd want[NCOEF] = {};
                const int q0 = k.kind == GROUP_TOR ? 10 : 0, q1 = k.kind == GROUP_TOR || rad ? 15 : 10;
                if (rad) pair_radial(c, ev, j, want);
                else if (k.kind == GROUP_TOR) pair_toroidal(c, ev, l, j, want + 10);
                else pair_spheroidal(c, ev, l, j, want, want + 5);
                double d = 0.0, big = 0.0;
                for (int q = q0; q < q1; q++) {
                    const double e = cabs(coef[((size_t)(l - ev.lmin) * NCOEF + q) * ev.nw + (j - 1)] - want[q]);
                    d = std::isfinite(e) ? std::max(d, e) : INFINITY;
                    big = std::max(big, cabs(want[q]));
                }
                diff = std::max(diff, d == 0.0 ? 0.0 : d / big);
            }
        }
        std::printf("%-16s %zu items, largest difference %.2e\n", k.name, order.size(), diff);
        worst = std::max(worst, diff);
    }
    ysh_free_event(&E);
    ysh_free_model(m);
    ysh_free_params(&P);
    return worst <= 2e-12 ? 0 : 1;
}
