// model_tables.h -- the device tables of a deck and the constants of an event,
// as the upload forms them, for the CPU checks of the group kernels.
#pragma once
#include <cstring>
#include <vector>

#include "yspec_gpu.h"
#include "yspec_host.h"
#include "ysg_model.cuh"

struct Tables {
    ysg_model view;
    std::vector<ysg::Knot> kn;
    std::vector<ysg::Seg> sg;
    ysg::ModelHdr mh;
};

inline void build_tables(const ysh_model* m, Tables& T)
{
    using namespace ysg;
    ysh_model_view(m, &T.view);
    const ysg_model& v = T.view;
    const int n = v.nknot;
    T.kn.assign((size_t)n + 2, Knot{});
    T.sg.assign((size_t)n + 1, Seg{});
    std::memset(static_cast<void*>(T.kn.data()), 0, T.kn.size() * sizeof(Knot));
    std::memset(static_cast<void*>(T.sg.data()), 0, T.sg.size() * sizeof(Seg));
    for (int i = 0; i < n; i++) {
        Knot& k = T.kn[(size_t)i + 1];
        k.r = v.r[i];
        k.alpha = v.alpha[i];
        k.beta = v.beta[i];
        for (int p = 0; p < NPARAM; p++) {
            k.v[p][0] = v.val[p][i];
            k.v[p][1] = v.cs[p][i];
        }
        knot_derive(k);
    }
    for (int i = 1; i <= n; i++) {
        const Knot &a = T.kn[(size_t)i], &b = T.kn[(size_t)i + 1];
        const double h = i < n ? b.r - a.r : 0.0;
        T.sg[i].r0 = a.r;
        for (int p = 0; p < NPARAM; p++) {
            double* c = T.sg[i].c[p];
            c[0] = a.v[p][0];
            if (h == 0.0) continue;
            c[1] = (b.v[p][0] - a.v[p][0]) / h - h * (2.0 * a.v[p][1] + b.v[p][1]) / 6.0;
            c[2] = 0.5 * a.v[p][1];
            c[3] = (b.v[p][1] - a.v[p][1]) / (6.0 * h);
        }
    }
    ModelHdr& h = T.mh;
    std::memset(&h, 0, sizeof h);
    h.nknot = n;
    h.nic = v.nic;
    h.noc = v.noc;
    h.nsl = v.nsl;
    h.ocean = v.ocean;
    h.fic = v.fic;
    h.imin_alpha = 1;
    for (int i = 2; i <= n; i++)
        if (v.alpha[i - 1] < v.alpha[h.imin_alpha - 1]) h.imin_alpha = i;
    h.imin_beta = v.noc + 1;
    for (int i = v.noc + 2; i <= v.nsl; i++)
        if (v.beta[i - 1] < v.beta[h.imin_beta - 1]) h.imin_beta = i;
    h.tref = v.tref;
    h.pibigg = v.pibigg;
    h.fre_norm = v.fre_norm;
}

inline ysg::EventDev event_constants(const ysg_event& e, const ysg_model& v)
{
    ysg::EventDev d{};
    d.lmin = e.lmin;
    d.lmax = e.lmax;
    d.nw = e.nw;
    d.is = e.is;
    d.ir = e.ir;
    d.ats = e.ats;
    d.grav = e.grav;
    d.out = e.out;
    d.cor = e.cor;
    d.nr = e.nr;
    d.jstride = 1;
    d.rs = e.rs;
    d.rr = e.rr;
    d.ep = e.ep;
    d.wmin = e.wmin;
    d.dw = e.dw;
    d.grav_ir = v.val[ysg::P_GRAV][e.ir - 1];
    for (int i = 0; i < 6; i++) d.mm[i] = e.mm[i];
    return d;
}

// some items of a list of n: the first, the last and `more` between
inline std::vector<int> some_items(long long n, int more)
{
    std::vector<int> v;
    for (int i = 0; i <= more + 1; i++) {
        const int it = (int)((n - 1) * i / (more + 1));
        if (v.empty() || v.back() != it) v.push_back(it);
    }
    return v;
}
