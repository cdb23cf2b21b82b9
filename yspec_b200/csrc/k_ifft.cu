// k_ifft.cu -- time series of yspec.f90:432-486 (module_fourier.f90:55-145).
//
// Per receiver and component the reference builds a length-n row (zero
// outside bins i1..i2, cosine taper, Hermitian extension), runs the
// Numerical-Recipes radix-2 decimation-in-time FFT with isign = +1
// (fourrow_dp, module_fourier.f90:7-50), divides by dt*n, multiplies by
// e^{eps t}, dimensionalises and rotates to Z/N/E.  Its twiddles use the
// single-precision pi of nrtype.f90, so the transform is the same
// butterfly network with angles m*pi_f/mmax; reproducing that network
// (not a DFT with exact pi) is what keeps the traces within 1e-9.
//
// Up to n = 65536 one kernel does all of it (k_series below): a row is held
// in the shared memory of one block or of the blocks of a cluster.
//
// For longer rows the network is split at stage p1 = ceil(log2(n)/2): after
// bit reversal the first p1 stages act inside contiguous blocks of
// b1 = 2^p1 elements (pass A), the remaining stages act on the b1 residue
// classes i mod b1 (pass B), which are independent.  Pass A reads the
// spectra directly and builds the row on the fly; pass B applies the
// post-processing and writes the real traces.  Intermediate rows live in a
// scratch buffer.  Inside a pass each thread runs up to three stages at a
// time in registers (below).
#include <cooperative_groups.h>

#include "ysg_kernels.h"
#include "ysg_tables.cuh"

namespace ysg {

__device__ __forceinline__ unsigned bitrev(unsigned g, int p) { return __brev(g) >> (32 - p); }

// All extents below are powers of two: index arithmetic uses shifts and
// masks (log2 by count of trailing zeros), never integer division.
__device__ __forceinline__ int lg2(int v) { return __ffs(v) - 1; }

// Element i (0-based, natural order) of the filtered Hermitian row.
__device__ __forceinline__ cd row_value(unsigned i, const TraceDev& td, const cd* __restrict__ spec,
                                        const double* __restrict__ filt)
{
    const unsigned n = (unsigned)td.nt, n2 = n / 2;
    bool cj = false;
    if (i > n2) {
        i = n - i;
        cj = true;
    }
    const int I = (int)i + 1;                     // 1-based bin
    if (I < td.i1 || I > td.i2) return mk(0.0);
    cd v = spec[I - td.i1] * filt[i];
    return cj ? conj(v) : v;
}

// ---------------------------------------------------------------------------
// Tables: the twiddles of every stage one after the other (stage s at
// 2^s - 1, entry m: exp(i m pi / 2^s); they do not depend on n), or those of
// the last stage of n alone (tw[m] = exp(i m pi / (n/2)), for the two
// passes); the taper per bin (module_fourier.f90:96-116); e^{eps t} per
// sample.  Null pointers leave a table out.  Every entry is within 0.502 units
// in the last place of the function of its (rounded) argument (ysg_tables.cuh).
// With the library's sincos and exp, within 1.36 and 0.85 units, 400 receivers
// of 16384 samples are 2.2e-16 off 64-bit arithmetic, with these 9.8e-17.  A row of
// blocks per table: the functions are long dependent chains, one after the other
// in a thread they took 2 us more (256.9 against 254.7 us for the whole call).
// ---------------------------------------------------------------------------
__global__ void k_time_tables(int nstage, cd* __restrict__ tws, int nhalf, cd* __restrict__ tw, TaperDev f, int nbin,
                              double* __restrict__ filt, double ep, double dt, int nout, double* __restrict__ expt)
{
    const double pi_d = (double)3.14159265358979323846f;   // nrtype.f90 pi_d (single-precision literal)
    const int i = blockIdx.x * blockDim.x + threadIdx.x, table = blockIdx.y;
    if (table == 0 && tws && i < (1 << nstage) - 1) {
        const int s = 31 - __clz(i + 1), m = i + 1 - (1 << s);
        double sn, c;
        table_sincos((double)m * (pi_d / (double)(1 << s)), &sn, &c);
        tws[i] = mk(c, sn);
    }
    if (table == 0 && tw && i < nhalf) {
        double sn, c;
        table_sincos((double)i * (pi_d / (double)nhalf), &sn, &c);
        tw[i] = mk(c, sn);
    }
    if (table == 1 && filt && i < nbin) {
        double v = 1.0;
        if (!(f.w1 == 0.0 && f.w2 == 0.0 && f.w3 == 0.0 && f.w4 == 0.0)) {
            const double w = __dmul_rn((double)i, f.df);
            double x = -1.0, s, c;                          // angle on the flanks
            if (w < f.w1) v = 0.0;
            else if (w < f.w2) x = pi_d * (w - f.w1) / (f.w2 - f.w1);
            else if (w < f.w3) v = 1.0;
            else if (w < f.w4) x = pi_d * (f.w4 - w) / (f.w4 - f.w3);
            else v = 0.0;
            if (x >= 0.0) {
                table_sincos(x, &s, &c);
                v = 0.5 * (1.0 - c);
            }
        }
        filt[i] = v;
    }
    if (table == 2 && expt && i < nout) expt[i] = table_exp(ep * ((double)i * dt));
}

cudaError_t launch_time_tables(int nstage, cd* tws, int nhalf, cd* tw, const TaperDev& f, int nbin, double* filt,
                               double ep, double dt, int nout, double* expt, cudaStream_t st)
{
    int n = 0;
    if (tws) n = 1 << nstage;
    if (tw && nhalf > n) n = nhalf;
    if (filt && nbin > n) n = nbin;
    if (expt && nout > n) n = nout;
    if (n == 0) return cudaSuccess;
    k_time_tables<<<dim3((n + 127) / 128, 3), 128, 0, st>>>(nstage, tws, nhalf, tw, f, nbin, filt, ep, dt, nout, expt);
    return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// One kernel per transform.  A block holds a tile of 2^ltl positions of a
// row in shared memory and runs stages 0 .. ltl-1 there, up to three at a
// time in registers (a round: each thread takes 8 values that those stages
// never mix with others, works on them and puts them back).  A row of more
// than one tile belongs to a cluster of 2^LCL blocks: the last LCL stages
// pair equal positions of its tiles, read from the other blocks' shared
// memory.  The three components of a receiver are taken in turn (blockDim.y
// = 1) or side by side (3), and the block that wrote a sample rotates it.
//
// What bounds it: shared memory (a row is read and written once per round)
// and the stages' FP64 work, about equal; the rows never leave the SM, where
// two passes over a scratch buffer wrote and read 16 bytes per point.
// Positions are stored at p ^ ((p >> 3) & 7), so that 8 neighbouring threads
// use different banks in every round, also in the first, where each has 8
// consecutive values.  400 receivers, 1200 rows of 16384 and 7202 samples
// kept: 255 us (the two passes in 16 MiB of rows, twiddles by sincos: 1286);
// half the issue slots are used, the rest wait for twiddles from the L2 and
// at the rounds' barriers.  Tiles of 2048 take 5 us more (128 threads) or 100
// (256), 512 threads on a tile 27.
// ---------------------------------------------------------------------------
constexpr int SER_THREADS = 256;         // threads of a component
constexpr int SER_LTILE = 12;            // tiles of 4096 positions, 64 KB: three per SM

struct SerArgs {
    TraceDev td;
    const cd *ur, *ut, *up;
    const double *filt, *expt, *cs, *azep;
    const cd* tws;
    double* out;
};

__device__ __forceinline__ int swz(int p) { return p ^ ((p >> 3) & 7); }

__device__ __forceinline__ void emit(const SerArgs& a, double* __restrict__ o, int c, int i, double x)
{
    if (i >= a.td.nout) return;
    // data/(dt*n), * e^{eps t}, * amplitude scale (yspec.f90:439-460)
    o[(size_t)(c + 1) * a.td.nout + i] = ((x / a.td.scale) * a.expt[i]) * a.td.amp_norm;
    if (c == 0) o[i] = ((double)i * a.td.dt) * a.td.t_norm;
}

// The product of a butterfly, rounded as the compiler contracts it there.
__device__ __forceinline__ cd twmul(cd w, cd b)
{
    return mk(fma(w.x, b.x, -__dmul_rn(w.y, b.y)), fma(w.y, b.x, __dmul_rn(w.x, b.y)));
}

// Stages 0 .. 2 of a row whose band ends below n/8: of the 8 bins
// r + t n/8 of a thread only t = 0 and t = 7 can be non-zero.  The sums with
// zeros and the products with one of the general round are left out (400
// receivers of 16384 samples: 287 -> 254 us), the rest is the same to the bit.
__device__ __forceinline__ void first_round(const SerArgs& a, int ltl, unsigned base, const cd* __restrict__ spec, cd* buf)
{
    const cd w1 = a.tws[2], w21 = a.tws[4], w22 = a.tws[5], w23 = a.tws[6];
    const unsigned top = 7u * (unsigned)(a.td.nt >> 3);
    for (int e = threadIdx.x; e < (1 << (ltl - 3)); e += blockDim.x) {
        const unsigned r = bitrev(base + 8 * e, a.td.log2n);
        const cd x = row_value(r, a.td, spec, a.filt), b4 = row_value(r + top, a.td, spec, a.filt);
        const cd b5 = twmul(w1, b4), t1 = twmul(w21, b5), t2 = twmul(w22, b4), t3 = twmul(w23, b5);
        buf[swz(8 * e)] = x + b4;
        buf[swz(8 * e + 1)] = x - t1;
        buf[swz(8 * e + 2)] = x - t2;
        buf[swz(8 * e + 3)] = x + t3;
        buf[swz(8 * e + 4)] = x - b4;
        buf[swz(8 * e + 5)] = x + t1;
        buf[swz(8 * e + 6)] = x + t2;
        buf[swz(8 * e + 7)] = x - t3;
    }
    __syncthreads();
}

// Stages s0 .. s0+M-1 of the tile.
template <int M>
__device__ __forceinline__ void series_round(const SerArgs& a, int s0, int ltl, unsigned base, const cd* __restrict__ spec,
                                             cd* buf, bool last, double* __restrict__ o, int c)
{
    const int D = 1 << s0;
    for (int e = threadIdx.x; e < (1 << (ltl - M)); e += blockDim.x) {
        const int j = e & (D - 1), p0 = ((e >> s0) << (s0 + M)) + j;
        cd v[1 << M];
#pragma unroll
        for (int k = 0; k < (1 << M); k++)
            v[k] = s0 == 0 ? row_value(bitrev(base + p0 + k, a.td.log2n), a.td, spec, a.filt) : buf[swz(p0 + D * k)];
#pragma unroll
        for (int st = 0; st < M; st++) {
            const cd* tw = a.tws + ((1 << (s0 + st)) - 1) + j;
#pragma unroll
            for (int k = 0; k < (1 << M); k++) {
                if (k & (1 << st)) continue;
                const cd tmp = tw[D * (k & ((1 << st) - 1))] * v[k + (1 << st)];
                v[k + (1 << st)] = v[k] - tmp;
                v[k] = v[k] + tmp;
            }
        }
#pragma unroll
        for (int k = 0; k < (1 << M); k++) {
            if (last) emit(a, o, c, p0 + D * k, v[k].x);
            else buf[swz(p0 + D * k)] = v[k];
        }
    }
    __syncthreads();
}

template <int LCL>
__global__ void __launch_bounds__(LCL ? SER_THREADS : 3 * SER_THREADS, LCL ? 3 : 1) k_series(SerArgs a)
{
    extern __shared__ __align__(16) unsigned char ser_smem[];
    namespace cg = cooperative_groups;
    constexpr int CL = 1 << LCL;
    const int n = a.td.nt, nout = a.td.nout, ltl = a.td.log2n - LCL, TL = 1 << ltl;
    const int q = LCL ? (int)cg::this_cluster().block_rank() : 0;
    const size_t kr = blockIdx.x >> LCL;          // receiver
    cd* buf = reinterpret_cast<cd*>(ser_smem) + (size_t)threadIdx.y * TL;
    double* o = a.out + (size_t)nout * 4 * kr;
    const int share = TL >> LCL, first = q * share;
    const bool narrow = ltl > 3 && a.td.i2 - 1 < n / 8;
    for (int c = threadIdx.y; c < 3; c += blockDim.y) {
        const cd* spec = (c == 0 ? a.ur : (c == 1 ? a.ut : a.up)) + kr * a.td.nw;
        if (narrow) first_round(a, ltl, (unsigned)(q * TL), spec, buf);
        for (int s0 = narrow ? 3 : 0; s0 < ltl; s0 += 3) {
            const int m = min(3, ltl - s0);
            const bool last = LCL == 0 && s0 + m == ltl;
            if (m == 3) series_round<3>(a, s0, ltl, (unsigned)(q * TL), spec, buf, last, o, c);
            else if (m == 2) series_round<2>(a, s0, ltl, (unsigned)(q * TL), spec, buf, last, o, c);
            else series_round<1>(a, s0, ltl, (unsigned)(q * TL), spec, buf, last, o, c);
        }
        if constexpr (LCL > 0) {
            cg::cluster_group cl = cg::this_cluster();
            const cd* tile[CL];
#pragma unroll
            for (int u = 0; u < CL; u++) tile[u] = cl.map_shared_rank(buf, u);
            cl.sync();
            for (int p = first + threadIdx.x; p < first + share; p += blockDim.x) {
                cd v[CL];
#pragma unroll
                for (int u = 0; u < CL; u++) v[u] = tile[u][swz(p)];
#pragma unroll
                for (int st = 0; st < LCL; st++) {
                    const cd* tw = a.tws + ((1 << (ltl + st)) - 1) + p;
#pragma unroll
                    for (int u = 0; u < CL; u++) {
                        if (u & (1 << st)) continue;
                        const cd tmp = tw[(size_t)TL * (u & ((1 << st) - 1))] * v[u + (1 << st)];
                        v[u + (1 << st)] = v[u] - tmp;
                        v[u] = v[u] + tmp;
                    }
                }
#pragma unroll
                for (int u = 0; u < CL; u++) emit(a, o, c, p + TL * u, v[u].x);
            }
            cl.sync();                            // the tiles are free, for the next component or the end
        }
    }
    __syncthreads();
    // rotation of the block's samples to north / east, yspec.f90:466-473
    double ca, sa;
    if (a.cs) {
        ca = a.cs[2 * kr];
        sa = a.cs[2 * kr + 1];
    } else {
        sincos(a.azep[kr], &sa, &ca);
    }
    const int nth = blockDim.x * blockDim.y;
#pragma unroll 4
    for (int e = threadIdx.y * blockDim.x + threadIdx.x; e < TL; e += nth) {
        const int i = first + (e & (share - 1)) + TL * (e >> (ltl - LCL));
        if (i >= min(nout, n)) continue;
        const double t1 = o[(size_t)2 * nout + i], t2 = o[(size_t)3 * nout + i];
        o[(size_t)2 * nout + i] = -(t1 * ca) + t2 * sa;
        o[(size_t)3 * nout + i] = t1 * sa + t2 * ca;
    }
}

template <int LCL>
cudaError_t launch_series_n(const SerArgs& a, cudaStream_t st)
{
    const int TL = a.td.nt >> LCL;
    const int T = TL / 8 < SER_THREADS ? TL / 8 : SER_THREADS, C = LCL ? 1 : 3;
    const size_t smem = (size_t)C * TL * sizeof(cd);
    cudaError_t e = cudaFuncSetAttribute(k_series<LCL>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)a.td.nr << LCL);
    cfg.blockDim = dim3(T, C);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = 1 << LCL;
    at.val.clusterDim.y = at.val.clusterDim.z = 1;
    cfg.attrs = &at;
    cfg.numAttrs = LCL ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, k_series<LCL>, a);
}

// Rows of up to 65536: tiles of 4096 in clusters of up to 8, at 65536 tiles
// of 8192 (128 KB).  cs: (cos, sin) of the receivers' angles, or null and
// azep the angles.
cudaError_t launch_series(const TraceDev& td, const cd* ur, const cd* ut, const cd* up, const double* filt,
                          const cd* tws, const double* expt, const double* cs, const double* azep, double* out,
                          cudaStream_t st)
{
    SerArgs a{td, ur, ut, up, filt, expt, cs, azep, tws, out};
    // the grid holds 2^31 - 1 blocks
    const int chunk = 1 << 27;
    for (int k0 = 0; k0 < td.nr; k0 += chunk) {
        const size_t so = (size_t)k0 * td.nw;
        a.td.nr = td.nr - k0 < chunk ? td.nr - k0 : chunk;
        a.ur = ur + so;
        a.ut = ut + so;
        a.up = up + so;
        a.cs = cs ? cs + 2 * (size_t)k0 : nullptr;
        a.azep = azep ? azep + k0 : nullptr;
        a.out = out + (size_t)k0 * td.nout * 4;
        const int l = td.log2n - SER_LTILE;
        const cudaError_t e = l <= 0 ? launch_series_n<0>(a, st)
                              : l == 1 ? launch_series_n<1>(a, st)
                              : l == 2 ? launch_series_n<2>(a, st)
                                       : launch_series_n<3>(a, st);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

// ---------------------------------------------------------------------------
// Register-blocked passes.  The butterfly network and
// its twiddle indices are unchanged (stage s pairs i and i + 2^s inside
// groups of 2^(s+1), twiddle tw[(i mod 2^s) << (log2(n/2) - s)]); only the
// work split changes.  Each thread holds 8 values and runs up to three
// consecutive stages on them in registers (a "round"); between rounds the
// values go through shared memory.  A round over stages s0 .. s0+m-1 acts on
// subsets {base + j + 2^s0 k : k < 2^m}, j < 2^s0, which those stages never
// mix with anything else.  Pass A covers stages 0 .. p1-1 inside blocks of
// b1 bit-reversed positions (tiles of 2048 positions per CTA), pass B the
// remaining stages on the residue classes r = i mod b1 (2048 / B2 classes
// per CTA, B2 = n / b1); pass B counts positions in units of b1 (u = i div
// b1), so a subset there is {r + b1 (base + j + 2^s0u k)}.
// ---------------------------------------------------------------------------
constexpr int FT = 2048;                 // values per CTA in either pass

// m stages (M = m) starting at stage s on this thread's values: subset q
// holds v[q 2^M + k], k < 2^M, at positions pos0[q] + dstep k (in units of
// i), so the lower value of a butterfly of stage s+st sits at
// pos0[q] + dstep (k mod 2^st) inside its group.
template <int M>
__device__ __forceinline__ void fft_round(cd (&v)[8], int s, const int (&pos0)[8 >> M], int dstep, int ln2,
                                          const cd* __restrict__ tw)
{
#pragma unroll
    for (int st = 0; st < M; st++) {
        const int sh = ln2 - (s + st);
#pragma unroll
        for (int q = 0; q < (8 >> M); q++)
#pragma unroll
            for (int k = 0; k < (1 << M); k++) {
                if (k & (1 << st)) continue;
                const int pos = pos0[q] + dstep * (k & ((1 << st) - 1));
                const cd w = tw[(size_t)pos << sh];
                cd& a = v[q * (1 << M) + k];
                cd& b = v[q * (1 << M) + k + (1 << st)];
                const cd tmp = w * b;
                b = a - tmp;
                a = a + tmp;
            }
    }
}

// One round of pass A on stages s0 .. s0+M-1: load (from the spectra for
// the first round, else from shared memory), butterflies, store (to the
// scratch row for the last round, else to shared memory).
template <int M>
__device__ __forceinline__ void round_a(cd (&v)[8], int s0, bool first, bool last, const TraceDev& td,
                                       unsigned base, int T, const cd* __restrict__ spec,
                                       const double* __restrict__ filt, const cd* __restrict__ tw,
                                       cd* buf, cd* __restrict__ dst)
{
    const int D = 1 << s0, ln2 = td.log2n - 1;
    int pos0[8 >> M];
#pragma unroll
    for (int q = 0; q < (8 >> M); q++) {
        const int sg = q * T + (int)threadIdx.x;          // subset index
        pos0[q] = ((sg >> s0) << (s0 + M)) + (sg & (D - 1));
    }
#pragma unroll
    for (int q = 0; q < (8 >> M); q++)
#pragma unroll
        for (int k = 0; k < (1 << M); k++) {
            const int pos = pos0[q] + D * k;
            v[q * (1 << M) + k] = first ? row_value(bitrev(base + pos, td.log2n), td, spec, filt) : buf[pos];
        }
    int tp[8 >> M];
#pragma unroll
    for (int q = 0; q < (8 >> M); q++) tp[q] = pos0[q] & (D - 1);   // position inside the group
    fft_round<M>(v, s0, tp, D, ln2, tw);
    if (!last && !first) __syncthreads();
#pragma unroll
    for (int q = 0; q < (8 >> M); q++)
#pragma unroll
        for (int k = 0; k < (1 << M); k++) {
            const int pos = pos0[q] + D * k;
            if (last) dst[pos] = v[q * (1 << M) + k];
            else buf[pos] = v[q * (1 << M) + k];
        }
    if (!last) __syncthreads();
}

__global__ void __launch_bounds__(FT / 8) k_ifft_a2(TraceDev td, const cd* __restrict__ ur,
                                                   const cd* __restrict__ ut, const cd* __restrict__ up,
                                                   const double* __restrict__ filt,
                                                   const cd* __restrict__ tw, cd* __restrict__ scr)
{
    __shared__ cd buf[FT];
    const int n = td.nt;
    const int tile = min(FT, n), T = tile / 8;
    const int p1 = lg2(td.b1);
    const int row = blockIdx.y;                   // 3 k + c
    const int k = row / 3, c = row - 3 * k;
    const cd* spec = (c == 0 ? ur : (c == 1 ? ut : up)) + (size_t)k * td.nw;
    const unsigned base = (unsigned)blockIdx.x * tile;
    cd* dst = scr + (size_t)row * n + base;
    cd v[8];
    for (int s0 = 0; s0 < p1; s0 += 3) {
        const int m = min(3, p1 - s0);
        const bool first = s0 == 0, last = s0 + m >= p1;
        if (m == 3) round_a<3>(v, s0, first, last, td, base, T, spec, filt, tw, buf, dst);
        else if (m == 2) round_a<2>(v, s0, first, last, td, base, T, spec, filt, tw, buf, dst);
        else round_a<1>(v, s0, first, last, td, base, T, spec, filt, tw, buf, dst);
    }
}

// One round of pass B on stages p1 + s0 .. p1 + s0 + M - 1 (s0 counted in
// units of b1).  Values of residue class r0 + g at u sit in buf[u G + g].
template <int M>
__device__ __forceinline__ void round_b(cd (&v)[8], int s0, bool first, bool last, const TraceDev& td,
                                        int G, int lG, int r0, int T, const cd* __restrict__ src,
                                        const cd* __restrict__ tw, const double* __restrict__ expt,
                                        cd* buf, double* __restrict__ o, int c)
{
    const int D = 1 << s0, ln2 = td.log2n - 1, b1 = td.b1;
    const int p1 = lg2(b1);
    int up0[8 >> M], gq[8 >> M];
#pragma unroll
    for (int q = 0; q < (8 >> M); q++) {
        const int sg = q * T + (int)threadIdx.x;
        gq[q] = sg & (G - 1);
        const int su = sg >> lG;                          // subset index in u
        up0[q] = ((su >> s0) << (s0 + M)) + (su & (D - 1));
    }
#pragma unroll
    for (int q = 0; q < (8 >> M); q++)
#pragma unroll
        for (int k = 0; k < (1 << M); k++) {
            const int u = up0[q] + D * k;
            v[q * (1 << M) + k] = first ? src[(size_t)(r0 + gq[q]) + (size_t)b1 * u] : buf[u * G + gq[q]];
        }
    int tp[8 >> M];
#pragma unroll
    for (int q = 0; q < (8 >> M); q++) tp[q] = r0 + gq[q] + b1 * (up0[q] & (D - 1));
    fft_round<M>(v, p1 + s0, tp, b1 * D, ln2, tw);
    if (!last && !first) __syncthreads();
#pragma unroll
    for (int q = 0; q < (8 >> M); q++)
#pragma unroll
        for (int k = 0; k < (1 << M); k++) {
            const int u = up0[q] + D * k;
            const cd x = v[q * (1 << M) + k];
            if (!last) {
                buf[u * G + gq[q]] = x;
                continue;
            }
            const int i = r0 + gq[q] + b1 * u;
            if (i >= td.nout) continue;
            // data/(dt*n), * e^{eps t}, * amplitude scale (yspec.f90:439-460)
            o[(size_t)(c + 1) * td.nout + i] = ((x.x / td.scale) * expt[i]) * td.amp_norm;
            if (c == 0) o[i] = ((double)i * td.dt) * td.t_norm;
        }
    if (!last) __syncthreads();
}

__global__ void __launch_bounds__(FT / 8) k_ifft_b2(TraceDev td, int G, const cd* __restrict__ tw,
                                                   const double* __restrict__ expt,
                                                   const cd* __restrict__ scr, double* __restrict__ out)
{
    __shared__ cd buf[FT];
    const int n = td.nt, b1 = td.b1, B2 = n / b1;
    const int pB = lg2(B2), lG = lg2(G), T = G * B2 / 8;
    const int row = blockIdx.y;
    const int k = row / 3, c = row - 3 * k;
    const int r0 = blockIdx.x * G;
    const cd* src = scr + (size_t)row * n;
    double* o = out + (size_t)td.nout * 4 * k;
    cd v[8];
    for (int s0 = 0; s0 < pB; s0 += 3) {
        const int m = min(3, pB - s0);
        const bool first = s0 == 0, last = s0 + m >= pB;
        if (m == 3) round_b<3>(v, s0, first, last, td, G, lG, r0, T, src, tw, expt, buf, o, c);
        else if (m == 2) round_b<2>(v, s0, first, last, td, G, lG, r0, T, src, tw, expt, buf, o, c);
        else round_b<1>(v, s0, first, last, td, G, lG, r0, T, src, tw, expt, buf, o, c);
    }
}

// Rotation to north / east, yspec.f90:466-473.
__global__ void k_rotate(int nout, int nr, const double* __restrict__ cs, const double* __restrict__ azep,
                         double* __restrict__ out)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int k = blockIdx.y;
    if (i >= nout || k >= nr) return;
    double* o = out + (size_t)nout * 4 * k;
    double ca, sa;
    if (cs) {
        ca = cs[2 * k];
        sa = cs[2 * k + 1];
    } else {
        sincos(azep[k], &sa, &ca);
    }
    const double t1 = o[(size_t)2 * nout + i], t2 = o[(size_t)3 * nout + i];
    o[(size_t)2 * nout + i] = -(t1 * ca) + t2 * sa;
    o[(size_t)3 * nout + i] = t1 * sa + t2 * ca;
}

size_t ifft_scratch_bytes(int nt, int nr) { return nt <= SERIES_MAX ? 0 : (size_t)3 * nr * nt * sizeof(cd); }

cudaError_t launch_ifft_a(const TraceDev& td, const cd* ur, const cd* ut, const cd* up, const double* filt,
                          const cd* tw, cd* scratch, cudaStream_t s)
{
    const int tile = td.nt < FT ? td.nt : FT;
    k_ifft_a2<<<dim3(td.nt / tile, 3 * td.nr), tile / 8, 0, s>>>(td, ur, ut, up, filt, tw, scratch);
    return cudaGetLastError();
}

cudaError_t launch_ifft_b(const TraceDev& td, const cd* tw, const double* expt, const cd* scratch, double* out,
                          cudaStream_t s)
{
    const int B2 = td.nt / td.b1;
    int G = FT / B2;
    if (G > td.b1) G = td.b1;
    k_ifft_b2<<<dim3(td.b1 / G, 3 * td.nr), G * B2 / 8, 0, s>>>(td, G, tw, expt, scratch, out);
    return cudaGetLastError();
}

cudaError_t launch_ifft_rotate(const TraceDev& td, const double* cs, const double* azep, double* out, cudaStream_t s)
{
    k_rotate<<<dim3((td.nout + 255) / 256, td.nr), 256, 0, s>>>(td.nout, td.nr, cs, azep, out);
    return cudaGetLastError();
}

cudaError_t launch_ifft(const TraceDev& td, const cd* ur, const cd* ut, const cd* up,
                        const double* filt, const cd* tw, const double* expt, const double* cs_azep,
                        cd* scratch, double* out, cudaStream_t s)
{
    if (td.nr <= 0) return cudaSuccess;
    const int n = td.nt;
    if (n < 8 || n > (1 << 20)) return cudaErrorInvalidValue;
    if (n <= SERIES_MAX) return launch_series(td, ur, ut, up, filt, tw, expt, cs_azep, nullptr, out, s);
    // one row per receiver and component in grid.y (at most 65535): receivers
    // go in chunks; each chunk's rows start at the top of the scratch buffer
    const int chunk = 65535 / 3;
    for (int k0 = 0; k0 < td.nr; k0 += chunk) {
        TraceDev sub = td;
        sub.nr = td.nr - k0 < chunk ? td.nr - k0 : chunk;
        const size_t so = (size_t)k0 * td.nw;
        double* sout = out + (size_t)k0 * td.nout * 4;
        cudaError_t e = launch_ifft_a(sub, ur + so, ut + so, up + so, filt, tw, scratch, s);
        if (e == cudaSuccess) e = launch_ifft_b(sub, tw, expt, scratch, sout, s);
        if (e == cudaSuccess) e = launch_ifft_rotate(sub, cs_azep + 2 * (size_t)k0, nullptr, sout, s);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

}  // namespace ysg
