// block_on_host.h -- run one thread block of device code on the CPU.
//
// Every thread of the block is a coroutine with a stack of its own; the warp and
// block collectives suspend it until all threads they join have arrived.  Device
// qualifiers become nothing, the explicitly rounded intrinsics the plain
// operations.  A thread that leaves a collective out hangs no GPU here: the
// scheduler sees that nobody advances and aborts.
#pragma once
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <functional>
#include <vector>

#include <cuda_runtime.h>
#undef __device__
#undef __host__
#undef __forceinline__
#undef __global__
#undef __noinline__
#undef __shared__
#undef __launch_bounds__
#undef __align__
#define __device__
#define __host__
#define __forceinline__ inline
#define __global__
#define __noinline__
#define __shared__
#define __launch_bounds__(...)
#define __align__(n) __attribute__((aligned(n)))

namespace block {

constexpr int MAX_THREADS = 128;
constexpr size_t STACK = 1 << 20;

#if !defined(__x86_64__)
#error "the switch between stacks is written for x86-64"
#endif
// Saves the callee-saved registers and the stack pointer, and takes up another stack.
extern "C" void block_switch_stack(void** save, void* to);
asm(R"(
    .text
    .globl block_switch_stack
block_switch_stack:
    pushq %rbp
    pushq %rbx
    pushq %r12
    pushq %r13
    pushq %r14
    pushq %r15
    movq %rsp, (%rdi)
    movq %rsi, %rsp
    popq %r15
    popq %r14
    popq %r13
    popq %r12
    popq %rbx
    popq %rbp
    ret
)");

struct Fiber {
    void* sp;
    std::vector<char> stack;
    bool done;
};
struct Barrier {
    int gen = 0, n = 0;
};
inline Fiber fiber[MAX_THREADS];
inline void* scheduler;
inline int nthreads, cur;
inline unsigned block_id, grid_size;
inline Barrier warp_bar[MAX_THREADS / 32], block_bar;
inline long long votes[MAX_THREADS];
inline long long progress;
inline std::function<void()> body;

inline void yield()
{
    const int me = cur;
    block_switch_stack(&fiber[me].sp, scheduler);
    cur = me;
}
inline void wait(Barrier& b, int need)
{
    const int g = b.gen;
    progress++;
    if (++b.n == need) {
        b.n = 0;
        b.gen++;
        return;
    }
    while (b.gen == g) yield();
}
inline void warp_sync() { wait(warp_bar[cur >> 5], 32); }
inline void block_sync() { wait(block_bar, nthreads); }
inline void entry()
{
    body();
    fiber[cur].done = true;
    progress++;
    for (;;) yield();
}
inline void run(int threads, unsigned id, unsigned grid, std::function<void()> f)
{
    nthreads = threads;
    block_id = id;
    grid_size = grid;
    body = f;
    for (int t = 0; t < threads; t++) {
        fiber[t].stack.resize(STACK);
        // as block_switch_stack leaves it: six registers, the return address, an aligned frame
        void** top = reinterpret_cast<void**>(((size_t)fiber[t].stack.data() + STACK) & ~(size_t)63) - 1;
        *--top = reinterpret_cast<void*>(&entry);
        for (int r = 0; r < 6; r++) *--top = nullptr;
        fiber[t].sp = top;
        fiber[t].done = false;
    }
    for (int left = threads; left;) {
        const long long before = progress;
        left = 0;
        for (int t = 0; t < threads; t++) {
            if (fiber[t].done) continue;
            cur = t;
            block_switch_stack(&scheduler, fiber[t].sp);
            left += !fiber[t].done;
        }
        if (left && progress == before) {
            std::fprintf(stderr, "block %u: %d threads wait for ever\n", id, left);
            std::abort();
        }
    }
}

struct ThreadX {
    operator unsigned() const { return (unsigned)cur; }
};
struct ThreadIdx {
    ThreadX x;
    unsigned y = 0;
};
struct Dim {
    unsigned x, y;
};

}  // namespace block

#define threadIdx (block::ThreadIdx{})
#define blockIdx (block::Dim{block::block_id, 0})
#define blockDim (block::Dim{(unsigned)block::nthreads, 1})
#define gridDim (block::Dim{block::grid_size, 1})

inline double __dmul_rn(double a, double b) { return a * b; }
inline double __dadd_rn(double a, double b) { return a + b; }
inline double __dsub_rn(double a, double b) { return a - b; }
template <class T> inline T __ldg(const T* p) { return *p; }
template <class T> inline void __stcs(T* p, T v) { *p = v; }
inline int __double2hiint(double x)
{
    long long b;
    std::memcpy(&b, &x, sizeof b);
    return (int)(b >> 32);
}
inline int __popc(unsigned v) { return __builtin_popcount(v); }
inline int __ffs(unsigned v) { return __builtin_ffs((int)v); }
inline void __syncwarp() { block::warp_sync(); }
inline void __syncthreads() { block::block_sync(); }
inline int __syncthreads_or(int p)
{
    block::votes[block::cur] = p;
    block::block_sync();
    int r = 0;
    for (int t = 0; t < block::nthreads; t++) r |= block::votes[t] != 0;
    block::block_sync();
    return r;
}
template <class T> inline T lane_exchange(T v, int src)
{
    static T buf[block::MAX_THREADS];
    const int first = block::cur & ~31;
    buf[block::cur] = v;
    block::warp_sync();
    const T r = buf[first + (src & 31)];
    block::warp_sync();
    return r;
}
inline int lane_id() { return block::cur & 31; }
inline double __shfl_sync(unsigned, double v, int s) { return lane_exchange(v, s); }
inline int __shfl_sync(unsigned, int v, int s) { return lane_exchange(v, s); }
inline double __shfl_xor_sync(unsigned, double v, int d) { return lane_exchange(v, lane_id() ^ d); }
inline int __shfl_up_sync(unsigned, int v, int d) { return lane_exchange(v, lane_id() >= d ? lane_id() - d : lane_id()); }
inline double __shfl_up_sync(unsigned, double v, int d) { return lane_exchange(v, lane_id() >= d ? lane_id() - d : lane_id()); }
template <class F> inline long long warp_reduce(long long v, F f)
{
    const int first = block::cur & ~31;
    block::votes[block::cur] = v;
    block::warp_sync();
    long long r = block::votes[first];
    for (int t = 1; t < 32; t++) r = f(r, block::votes[first + t]);
    block::warp_sync();
    return r;
}
inline unsigned __ballot_sync(unsigned, bool p)
{
    return (unsigned)warp_reduce((long long)p << lane_id(), [](long long a, long long b) { return a | b; });
}
inline bool __any_sync(unsigned m, bool p) { return __ballot_sync(m, p) != 0; }
inline bool __all_sync(unsigned m, bool p) { return __ballot_sync(m, p) == 0xffffffffu; }
inline int __reduce_min_sync(unsigned, int v) { return (int)warp_reduce(v, [](long long a, long long b) { return std::min(a, b); }); }
inline int __reduce_max_sync(unsigned, int v) { return (int)warp_reduce(v, [](long long a, long long b) { return std::max(a, b); }); }
inline unsigned __reduce_add_sync(unsigned, unsigned v) { return (unsigned)warp_reduce(v, [](long long a, long long b) { return a + b; }); }
template <class T, class U> inline T atomicAdd(T* p, U v)
{
    const T old = *p;
    *p = old + (T)v;
    return old;
}
inline void sincos(double x, double* s, double* c) noexcept
{
    *s = std::sin(x);
    *c = std::cos(x);
}
using std::max;
using std::min;
