// k_ifft_noalloc.cu -- the time-series stage without any device allocation.
//
// Some callers cannot let the library allocate device memory: a host that
// reserves the whole GPU for its own pool at start-up, a host whose rules
// forbid hidden allocations, or code where a cudaMalloc would synchronise
// the device and stall its other streams.  ysg_traces_noalloc serves them:
// it runs the same filter + Hermitian extension + inverse FFT +
// post-processing as ysg_event_traces, but reads the spectra from and
// writes the traces to device buffers the caller owns, and keeps its
// intermediate rows in one fixed array compiled into the library.
//
// That array (g_trace_scratch, 2^20 complex values = 16 MiB) is held on
// every GPU that loads the library until the process exits.  It takes the
// tables of a call (twiddles, taper, e^{eps t}, formed by its first kernel)
// and, where a row does not fit a cluster's shared memory (nt > 65536), the
// rows, in chunks of whole receivers; one transform row must fit three
// times, so nt <= 262144.  Every call shares the array: nothing in it needs
// to start at zero (tables and rows are written before they are read), and
// two calls whose work overlaps on the GPU (different streams, or different
// host threads on the same device) race on it and must be serialised by the
// caller.
//
// 400 receivers of 16384 samples: 255 us (k_series of k_ifft.cu; rows
// passed through the array, twiddles by sincos in every butterfly: 1286 us).
//
// The device address of the array is looked up with cudaGetSymbolAddress
// on the first call made on each device (with that device current) and
// cached by device ordinal; that first call should come before any stream
// capture.  The cache assumes the device's primary context, the one the
// runtime API uses, for the life of the process: after cudaDeviceReset, or
// from a separate driver-API context on the same device, the cached address
// is stale and this entry point must not be used.  The
// tables and the rotation angles are formed on the
// device, so apart from the launches nothing is allocated or copied.
#include <mutex>

#include <cuda_runtime.h>

#include "yspec_gpu.h"
#include "ysg_kernels.h"

// Records a CUDA failure for ysg_last_cuda_error() (capi.cu).
int ysg_cuda_fail_at(cudaError_t e, const char* file, int line);

namespace {

constexpr size_t kScratchComplex = (size_t)1 << 20;

}  // namespace

static __device__ __align__(256) ysg::cd g_trace_scratch[kScratchComplex];

namespace {

using ysg::cd;

std::mutex g_mu;
cd* g_addr[128] = {};

// Device address of g_trace_scratch on the current device, looked up once.
int scratch_address(cd** p)
{
    int dev = -1;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return ysg_cuda_fail_at(e, "k_ifft_noalloc.cu", __LINE__);
    if (dev < 0 || dev >= 128) return YSG_ERR_CUDA;
    std::lock_guard<std::mutex> lk(g_mu);
    if (!g_addr[dev]) {
        void* ptr = nullptr;
        e = cudaGetSymbolAddress(&ptr, g_trace_scratch);
        if (e != cudaSuccess) return ysg_cuda_fail_at(e, "k_ifft_noalloc.cu", __LINE__);
        if (!ptr) return YSG_ERR_CUDA;
        g_addr[dev] = static_cast<cd*>(ptr);
    }
    *p = g_addr[dev];
    return YSG_OK;
}

}  // namespace

extern "C" int ysg_traces_noalloc(const ysg_time* tm, const double* d_ur, const double* d_ut,
                                  const double* d_up, const double* d_azep, double* d_out,
                                  int* nout, void* stream)
{
    if (!tm) return YSG_ERR_ARG;
    const int n = tm->nt, nr = tm->nr;
    // the same argument rules as the allocating time-series stage (k_ifft.cu)
    if (n < 8 || (n & (n - 1)) || tm->i1 < 1 || tm->i2 < tm->i1 || tm->i2 > n || nr < 0)
        return YSG_ERR_ARG;
    if (nr > 0 && (!d_ur || !d_ut || !d_up || !d_azep || !d_out)) return YSG_ERR_ARG;
    if ((size_t)3 * n > kScratchComplex) return YSG_ERR_LIMIT;   // one receiver must fit
    const int rows_out = ysg_trace_rows(tm);
    if (nout) *nout = rows_out;
    if (nr == 0) return YSG_OK;
    // an error left pending by earlier work on this thread is cleared here,
    // so the check after the launches reports this call's own failures
    (void)cudaGetLastError();
    cd* scr = nullptr;
    int rc = scratch_address(&scr);
    if (rc) return rc;
    cudaStream_t st = (cudaStream_t)stream;
    int p = 0;
    while ((1 << p) < n) p++;
    ysg::TraceDev td{};
    td.nt = n;
    td.i1 = tm->i1;
    td.i2 = tm->i2;
    td.nw = tm->i2 - tm->i1 + 1;
    td.nr = nr;
    td.nout = rows_out;
    td.log2n = p;
    td.b1 = 1 << ((p + 1) / 2);
    td.dt = tm->dt;
    td.scale = tm->dt * (double)n;
    td.t_norm = tm->t_norm;
    td.amp_norm = tm->amp_norm;
    const ysg::TaperDev taper{tm->df, tm->f11, tm->f12, tm->f21, tm->f22};
    const int nbin = n / 2 + 1;
    const cd* ur = reinterpret_cast<const cd*>(d_ur);
    const cd* ut = reinterpret_cast<const cd*>(d_ut);
    const cd* up = reinterpret_cast<const cd*>(d_up);
#define NOALLOC_CK(x)                                                             \
    do {                                                                          \
        const cudaError_t e_ = (x);                                               \
        if (e_ != cudaSuccess) return ysg_cuda_fail_at(e_, "k_ifft_noalloc.cu", __LINE__); \
    } while (0)
    if (n <= ysg::SERIES_MAX) {
        // twiddles (n - 1), taper (n / 2 + 1 doubles), e^{eps t} (at most n doubles)
        cd* tws = scr;
        double* filt = reinterpret_cast<double*>(scr + n);
        double* expt = reinterpret_cast<double*>(scr + 2 * (size_t)n);
        NOALLOC_CK(ysg::launch_time_tables(p, tws, 0, nullptr, taper, nbin, filt, tm->ep, tm->dt, rows_out, expt, st));
        NOALLOC_CK(ysg::launch_series(td, ur, ut, up, filt, tws, expt, nullptr, d_azep, d_out, st));
        return YSG_OK;
    }
    // twiddles (n / 2); the taper, then e^{eps t} in its place (n / 2); rows
    cd* tw = scr;
    double* tab = reinterpret_cast<double*>(scr + n / 2);
    cd* rows = scr + n;
    const int per_chunk = (int)((kScratchComplex - n) / ((size_t)3 * n));   // receivers per chunk
    NOALLOC_CK(ysg::launch_time_tables(0, nullptr, n / 2, tw, taper, 0, nullptr, 0.0, 0.0, 0, nullptr, st));
    for (int k0 = 0; k0 < nr; k0 += per_chunk) {
        td.nr = nr - k0 < per_chunk ? nr - k0 : per_chunk;
        const size_t so = (size_t)k0 * td.nw;
        double* out = d_out + (size_t)k0 * rows_out * 4;
        NOALLOC_CK(ysg::launch_time_tables(0, nullptr, 0, nullptr, taper, nbin, tab, 0.0, 0.0, 0, nullptr, st));
        NOALLOC_CK(ysg::launch_ifft_a(td, ur + so, ut + so, up + so, tab, tw, rows, st));
        NOALLOC_CK(ysg::launch_time_tables(0, nullptr, 0, nullptr, taper, 0, nullptr, tm->ep, tm->dt, rows_out, tab, st));
        NOALLOC_CK(ysg::launch_ifft_b(td, tw, tab, rows, out, st));
        NOALLOC_CK(ysg::launch_ifft_rotate(td, nullptr, d_azep + k0, out, st));
    }
#undef NOALLOC_CK
    return YSG_OK;
}
