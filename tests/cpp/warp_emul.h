// Runs the library's kernels on the host, for tests of what a GPU run cannot
// show: every thread of a block is a fiber that runs until it meets a warp or
// block collective, so the order in which the lanes of a warp reach their
// atomics is the test's choice (emu::descending), as CUDA leaves it open.
// Included before any kernel source (tests/emulated.py prepares the sources).
// Plain products and sums are not contracted to FMAs here.
#pragma once
#include <cuda_runtime.h>
#include <math.h>
#include <ucontext.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstdlib>
#include <cstring>
#include <functional>
#include <map>
#include <memory>
#include <vector>

#define __CUDACC__ 1
#undef __shared__
#define __shared__ static
#undef __launch_bounds__
#define __launch_bounds__(...)
#undef __align__
#define __align__(n) __attribute__((aligned(n)))
#undef __noinline__
#define __noinline__
#undef __forceinline__
#define __forceinline__ inline

inline uint3 blockIdx, threadIdx;
inline dim3 gridDim, blockDim;

namespace emu {

inline bool descending = false;                       // lanes (and warps) served from the last one down
inline std::function<bool(unsigned)> wanted_block;    // blocks to run (all when empty)

struct Meeting {  // a collective of the lanes in `mask` of one warp, or of the block
    uint32_t arrived = 0;
    uint64_t round = 0;
    uint64_t in[32], out[32];
};
struct Fiber {
    ucontext_t ctx;
    std::unique_ptr<char[]> stack;
    bool done = false;
};
struct Warp {
    uint32_t alive = 0;
    std::map<uint32_t, Meeting> meet;
};
inline std::vector<Fiber> fibers;
inline std::vector<Warp> warps;
inline unsigned current = 0, block_alive = 0, block_arrived = 0;
inline uint64_t block_round = 0;
inline ucontext_t main_ctx;
inline std::function<void()> body;

inline void pass_on() { swapcontext(&fibers[current].ctx, &main_ctx); }

inline void settle(Warp& w)
{
    for (auto& m : w.meet)
        if (m.second.arrived && (m.second.arrived & w.alive) == (m.first & w.alive)) {
            std::memcpy(m.second.out, m.second.in, sizeof(m.second.out));
            m.second.arrived = 0;
            ++m.second.round;
        }
}

// Meets the other lanes of mask: value of every lane that came, and who they are.
inline const uint64_t* meet(uint32_t mask, uint64_t v, uint32_t* who = nullptr)
{
    Warp& w = warps[current >> 5];
    Meeting& m = w.meet[mask];
    const uint64_t round = m.round;
    m.in[current & 31] = v;
    m.arrived |= 1u << (current & 31);
    settle(w);
    while (m.round == round) pass_on();
    if (who) *who = mask & w.alive;
    return m.out;
}

inline void block_barrier()
{
    const uint64_t round = block_round;
    if (++block_arrived == block_alive) {
        block_arrived = 0;
        ++block_round;
    }
    while (block_round == round) pass_on();
}

inline void entry()
{
    body();
    Fiber& f = fibers[current];
    f.done = true;
    warps[current >> 5].alive &= ~(1u << (current & 31));
    settle(warps[current >> 5]);
    if (--block_alive && block_arrived == block_alive) {
        block_arrived = 0;
        ++block_round;
    }
    for (;;) pass_on();
}

inline void run_block(unsigned threads)
{
    fibers.resize(std::max<size_t>(fibers.size(), threads));
    warps.assign((threads + 31) / 32, Warp());
    block_alive = threads;
    block_arrived = 0;
    for (unsigned t = 0; t < threads; ++t) {
        Fiber& f = fibers[t];
        if (!f.stack) f.stack.reset(new char[256 << 10]);
        f.done = false;
        warps[t >> 5].alive |= 1u << (t & 31);
        getcontext(&f.ctx);
        f.ctx.uc_stack.ss_sp = f.stack.get();
        f.ctx.uc_stack.ss_size = 256 << 10;
        f.ctx.uc_link = nullptr;
        makecontext(&f.ctx, entry, 0);
    }
    while (block_alive) {
        for (unsigned i = 0; i < threads; ++i) {
            const unsigned t = descending ? threads - 1 - i : i;
            if (fibers[t].done) continue;
            current = t;
            threadIdx.x = t;
            swapcontext(&main_ctx, &fibers[t].ctx);
        }
    }
}

template <class... P, class... A>
cudaError_t launch(const cudaLaunchConfig_t* cfg, void (*kernel)(P...), A&&... args)
{
    body = [&] { kernel(static_cast<P>(args)...); };
    gridDim = cfg->gridDim;
    blockDim = cfg->blockDim;
    for (unsigned b = 0; b < gridDim.x; ++b) {
        if (wanted_block && !wanted_block(b)) continue;
        blockIdx.x = b;
        run_block(blockDim.x);
    }
    return cudaSuccess;
}

template <class T>
uint64_t bits(T v)
{
    uint64_t b = 0;
    std::memcpy(&b, &v, sizeof(T));
    return b;
}
template <class T>
T value(uint64_t b)
{
    T v;
    std::memcpy(&v, &b, sizeof(T));
    return v;
}
template <class T, class Fn>
T reduce(uint32_t mask, T v, Fn fn)
{
    uint32_t who;
    const uint64_t* out = meet(mask, bits(v), &who);
    bool any = false;
    T r{};
    for (int l = 0; l < 32; ++l)
        if ((who >> l) & 1u) {
            r = any ? fn(r, value<T>(out[l])) : value<T>(out[l]);
            any = true;
        }
    return r;
}
template <class T>
T from_lane(uint32_t mask, T v, int src)
{
    return value<T>(meet(mask, bits(v))[src & 31]);
}
inline int lane() { return (int)(current & 31); }

}  // namespace emu

#define cudaLaunchKernelEx emu::launch
#define cudaFuncSetAttribute(...) cudaSuccess
#define cudaGetLastError() cudaSuccess
#define cudaMemsetAsync(p, v, n, ...) (std::memset((p), (v), (n)), cudaSuccess)
#define cudaMemcpyToSymbolAsync(dst, src, n, ...) std::memcpy(&(dst), (src), (n))
inline void cudaGridDependencySynchronize() {}

inline void __syncthreads() { emu::block_barrier(); }
inline void __syncwarp(unsigned m = 0xffffffffu) { emu::meet(m, 0); }
inline unsigned __activemask() { return emu::warps[emu::current >> 5].alive; }
template <class T> T __shfl_sync(unsigned m, T v, int src) { return emu::from_lane(m, v, src); }
template <class T> T __shfl_xor_sync(unsigned m, T v, int o) { return emu::from_lane(m, v, emu::lane() ^ o); }
template <class T> T __shfl_up_sync(unsigned m, T v, unsigned o)
{
    const int l = emu::lane();
    return emu::from_lane(m, v, l >= (int)o ? l - (int)o : l);
}
inline unsigned __ballot_sync(unsigned m, bool p)
{
    return emu::reduce(m, p ? 1u << emu::lane() : 0u, [](unsigned a, unsigned b) { return a | b; });
}
inline bool __any_sync(unsigned m, bool p) { return __ballot_sync(m, p) != 0; }
inline bool __all_sync(unsigned m, bool p) { return __ballot_sync(m, !p) == 0; }
template <class T> T __reduce_add_sync(unsigned m, T v) { return emu::reduce(m, v, [](T a, T b) { return a + b; }); }
template <class T> T __reduce_min_sync(unsigned m, T v) { return emu::reduce(m, v, [](T a, T b) { return std::min(a, b); }); }
template <class T> T __reduce_max_sync(unsigned m, T v) { return emu::reduce(m, v, [](T a, T b) { return std::max(a, b); }); }
template <class T> T __reduce_or_sync(unsigned m, T v) { return emu::reduce(m, v, [](T a, T b) { return a | b; }); }
inline unsigned __match_any_sync(unsigned m, unsigned v)
{
    uint32_t who, r = 0;
    const uint64_t* out = emu::meet(m, v, &who);
    for (int l = 0; l < 32; ++l)
        if (((who >> l) & 1u) && (unsigned)out[l] == v) r |= 1u << l;
    return r;
}

template <class T> T atomicAdd(T* p, T v) { T o = *p; *p = o + v; return o; }
inline uint32_t atomicAdd(uint32_t* p, int v) { uint32_t o = *p; *p = o + (uint32_t)v; return o; }
inline float4 atomicAdd(float4* p, float4 v)
{
    float4 o = *p;
    *p = make_float4(o.x + v.x, o.y + v.y, o.z + v.z, o.w + v.w);
    return o;
}
template <class T> T atomicOr(T* p, T v) { T o = *p; *p = o | v; return o; }
template <class T> T atomicMax(T* p, T v) { T o = *p; *p = std::max(o, v); return o; }
template <class T> T atomicMin(T* p, T v) { T o = *p; *p = std::min(o, v); return o; }
template <class T> T atomicExch(T* p, T v) { T o = *p; *p = v; return o; }

template <class T> T __ldg(const T* p) { return *p; }
inline int __popc(unsigned v) { return __builtin_popcount(v); }
inline int __ffs(int v) { return __builtin_ffs(v); }
inline int __clz(int v) { return v ? __builtin_clz((unsigned)v) : 32; }
inline unsigned __float_as_uint(float v) { return emu::value<unsigned>(emu::bits(v)); }
inline int __float_as_int(float v) { return emu::value<int>(emu::bits(v)); }
inline float __uint_as_float(unsigned v) { return emu::value<float>(emu::bits(v)); }
inline float __int_as_float(int v) { return emu::value<float>(emu::bits(v)); }
inline float __fadd_rn(float a, float b) { return a + b; }
inline float __fsub_rn(float a, float b) { return a - b; }
inline float __fmul_rn(float a, float b) { return a * b; }
inline float __fdiv_rn(float a, float b) { return a / b; }
inline float __fsqrt_rn(float a) { return std::sqrt(a); }
inline float __fmaf_rn(float a, float b, float c) { return std::fma(a, b, c); }
inline double __dmul_rn(double a, double b) { return a * b; }
inline float __double2float_rn(double a) { return (float)a; }
inline float __uint2float_rn(unsigned v) { return (float)v; }
inline int __float2int_rz(float v) { return v != v ? 0 : (int)std::fmin(std::fmax(std::trunc(v), -2147483648.f), 2147483520.f); }
inline int __float2int_rd(float v) { return __float2int_rz(std::floor(v)); }
inline int __float2int_ru(float v) { return __float2int_rz(std::ceil(v)); }
inline float2 __fadd2_rn(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
inline float2 __fmul2_rn(float2 a, float2 b) { return make_float2(a.x * b.x, a.y * b.y); }
inline float2 __ffma2_rn(float2 a, float2 b, float2 c) { return make_float2(std::fma(a.x, b.x, c.x), std::fma(a.y, b.y, c.y)); }
inline float rsqrtf(float v) { return 1.0f / std::sqrt(v); }
inline int min(int a, int b) { return a < b ? a : b; }
inline int max(int a, int b) { return a > b ? a : b; }
inline unsigned min(unsigned a, unsigned b) { return a < b ? a : b; }
inline unsigned max(unsigned a, unsigned b) { return a > b ? a : b; }
