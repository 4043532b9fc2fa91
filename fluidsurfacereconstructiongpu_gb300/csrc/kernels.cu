// Per-frame kernels of the reconstruction path.  Each kernel names the
// reference kernel it replaces (ReconstructionCUDA.cu, "cu").
#include "kernels.h"
#include "primitives.h"
#include "cov_solver.cuh"

#include <algorithm>
#include <cmath>

namespace fsr {

__constant__ McConst c_mc;
thread_local uint64_t g_launches = 0;

void upload_mc_tables(cudaStream_t s)
{
    McConst h;
    for (int i = 0; i < 256; ++i) {
        h.tri[i] = mc::kTriPacked[i];
        h.eflags[i] = mc::kDerived.eflags[i];
        h.nverts[i] = mc::kDerived.nverts[i];
    }
    cudaMemcpyToSymbolAsync(c_mc, &h, sizeof(h), 0, cudaMemcpyHostToDevice, s);
}

namespace {

constexpr int kThreads = 256;

inline unsigned blocks_for(uint64_t n, int threads = kThreads)
{
    return (unsigned)std::max<uint64_t>(1, std::min<uint64_t>((n + threads - 1) / threads, 0x7fffffffULL));
}

// threads per block of the per-item and warp-staged kernels: the context's
// block shape (a multiple of 32 up to kThreads, which their per-warp shared
// arrays are sized for)
inline int bs(const KernelCtx& c) { return (c.block >= 32 && c.block <= kThreads && c.block % 32 == 0) ? c.block : kThreads; }

// grid for grid-stride kernels whose length is read on the device
inline unsigned persistent_blocks(const KernelCtx& c, uint64_t cap, int per_sm = 8)
{
    const uint64_t want = (cap + bs(c) - 1) / bs(c);
    // per_sm counts blocks of kThreads threads: smaller blocks get proportionally more
    per_sm = per_sm * (kThreads / bs(c));
    const uint64_t most = std::max<uint64_t>(1, (uint64_t)c.num_sms * per_sm / std::max(1, c.grid_div));
    return (unsigned)std::max<uint64_t>(1, std::min<uint64_t>(want, most));
}

__device__ __forceinline__ void warp_count(uint32_t* counter, bool pred)
{
    const uint32_t m = __ballot_sync(__activemask(), pred);
    if (pred && (threadIdx.x & 31u) == (uint32_t)(__ffs(m) - 1)) atomicAdd(counter, __popc(m));
}

// ------------------------------------------------------------ hashing
// calcParticlesHashKernel (cu:1379-1396) plus the bounds check the
// reference lacks (cu:1391-1395 writes out of bounds for such particles).
__global__ void k_hash(const float* __restrict__ xyz, uint32_t n, Grid sp, uint32_t* __restrict__ keys,
                       uint32_t* __restrict__ vals, Counters* ctr)
{
    after_launch();
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float p[3] = {xyz[3ull * i], xyz[3ull * i + 1], xyz[3ull * i + 2]};
    bool ok;
    keys[i] = cell_key(p, sp, ok);
    vals[i] = i;
    if (!ok) atomicAdd(&ctr->out_of_grid, 1u);
}

// findCellRangeKernel (cu:1399-1435) fused with the gather of the sorted
// particles (the reference sorts positions and densities in place,
// cu:1461-1466) into one float4 per particle.
__global__ void k_ranges_gather(const uint32_t* __restrict__ skeys, const uint32_t* __restrict__ perm,
                                uint32_t n, const float* __restrict__ xyz, const float* __restrict__ dens,
                                float4* __restrict__ sorted, uint2* __restrict__ ranges,
                                uint8_t* __restrict__ occ)
{
    after_launch();
    const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    const uint32_t key = skeys[k];
    const uint32_t prev = k > 0 ? skeys[k - 1] : kEmpty;
    const uint32_t next = k + 1 < n ? skeys[k + 1] : kEmpty;
    if (key != prev) {
        ranges[key].x = k;
        occ[key] = 1;
    }
    if (key != next) ranges[key].y = k + 1;
    const uint32_t s = perm[k];
    // without densities (computed later by k_density) w is left at 0
    sorted[k] = make_float4(xyz[3ull * s], xyz[3ull * s + 1], xyz[3ull * s + 2], dens ? dens[s] : 0.0f);
}

// SPH density of each sorted particle, for frames without a density column
// (the reference's .xyz files carry the simulator's densities and the
// reference computes none): rho_i = m sigma / h^3 sum_j (1 - |x_i - x_j|^2 /
// h^2)^3 over the particles within h, i itself included, sigma = 315 /
// (64 pi) - the poly6 kernel with the normalisation of the reference's own
// field kernel (anisotropicW, cuh:294-310, at G = I / h).  Each particle's
// sum runs over its window's cells in order, so results are deterministic.
//
// A warp's lanes walk the union of their windows together (sets of lanes as in
// window_mates), the candidates within h of their box staged in shared memory
// and evaluated two at a time with packed FP32x2 operations; a candidate
// outside a lane's window lies beyond h of it.  (Each lane on a window of its
// own: 120k particles 0.25 -> 0.11 ms, 1M 0.92 -> 0.33.)
constexpr int kDensityThreads = 128;
constexpr uint32_t kDensityCap = 64;
struct DensitySlice {
    float x[kDensityCap], y[kDensityCap], z[kDensityCap];
};
__global__ void __launch_bounds__(kDensityThreads) k_density(const float4* __restrict__ sorted, uint32_t n,
                                                      const uint2* __restrict__ ranges, Grid sp, int ext, float h,
                                                      float h2, float inv_h2, float scale, float* __restrict__ rho)
{
    after_launch();
    __shared__ __align__(16) DensitySlice slices[kDensityThreads / 32];
    DensitySlice& S = slices[threadIdx.x >> 5];
    const int lane = threadIdx.x & 31;
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    const bool active = t < n;
    if (__all_sync(0xffffffffu, !active)) return;
    const float4 p = active ? sorted[t] : make_float4(0.f, 0.f, 0.f, 0.f);
    const float reach = cull_radius(h, sp.cs);
    const Window w = narrow(window(cell1(p.x, sp.min[0], sp.cs), cell1(p.y, sp.min[1], sp.cs),
                                   cell1(p.z, sp.min[2], sp.cs), ext, sp),
                            p.x, p.y, p.z, reach, sp);
    auto row_range = [&](int x0, int x1, int yy, int zz, uint32_t& beg, uint32_t& end) {
        // the row's cells are contiguous in the sorted array
        const uint32_t c0 = lin3(x0, yy, zz, sp);
        beg = kEmpty;
        end = 0;
        for (int xx = 0; xx <= x1 - x0; ++xx) {
            const uint2 r = __ldg(&ranges[c0 + xx]);
            if (r.x != kEmpty) {
                beg = min(beg, r.x);
                end = max(end, r.y);
            }
        }
    };
    float sum = 0.f;
    const float2 nx = make_float2(-p.x, -p.x), ny = make_float2(-p.y, -p.y), nz = make_float2(-p.z, -p.z);
    const float2 ninv = make_float2(-inv_h2, -inv_h2), one = make_float2(1.0f, 1.0f);
    auto take = [&](uint32_t fill, bool in_set) {
        if ((fill & 1u) && lane == 0) S.x[fill] = S.y[fill] = S.z[fill] = 1.0e18f;  // beyond h of everything
        __syncwarp();
        if (in_set)
#pragma unroll 4
            for (uint32_t k = 0; k < fill; k += 2) {
                const float2 dx = __fadd2_rn(*reinterpret_cast<const float2*>(S.x + k), nx);
                const float2 dy = __fadd2_rn(*reinterpret_cast<const float2*>(S.y + k), ny);
                const float2 dz = __fadd2_rn(*reinterpret_cast<const float2*>(S.z + k), nz);
                const float2 d2 = __ffma2_rn(dx, dx, __ffma2_rn(dy, dy, __fmul2_rn(dz, dz)));
                const float2 u = __ffma2_rn(d2, ninv, one);
                const float2 uu = __fmul2_rn(u, u);
                if (d2.x < h2) sum = fmaf(uu.x, u.x, sum);
                if (d2.y < h2) sum = fmaf(uu.y, u.y, sum);
            }
        __syncwarp();
    };
    uint32_t left = __ballot_sync(0xffffffffu, active);
    for (int sets = 0; left != 0u && sets < kMaxSets; ++sets) {
        const uint32_t set = window_mates(left, w, 2 * ext + 1, lane);
        left &= ~set;
        const bool in_set = (set >> lane) & 1u;
        int ulo[3], uhi[3];
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            ulo[a] = (int)__reduce_min_sync(0xffffffffu, in_set ? (unsigned)w.lo[a] : 0x7fffffffu);
            uhi[a] = (int)__reduce_max_sync(0xffffffffu, in_set ? (unsigned)(w.hi[a] + 1) : 0u) - 1;
        }
        const WarpBox box = warp_box(in_set, p.x, p.y, p.z, reach);
        uint32_t fill = 0;
        for (int zz = ulo[2]; zz <= uhi[2]; ++zz)
            for (int yy = ulo[1]; yy <= uhi[1]; ++yy) {
                uint32_t beg, end;
                row_range(ulo[0], uhi[0], yy, zz, beg, end);
                for (uint32_t base = beg; base < end; base += 32) {
                    float4 q = make_float4(0.f, 0.f, 0.f, 0.f);
                    bool keep = false;
                    if (base + lane < end) {
                        q = __ldg(&sorted[base + lane]);
                        keep = box.keeps(q);
                    }
                    const uint32_t m = __ballot_sync(0xffffffffu, keep);
                    if (keep) {
                        const uint32_t k = fill + __popc(m & ((1u << lane) - 1u));
                        S.x[k] = q.x;
                        S.y[k] = q.y;
                        S.z[k] = q.z;
                    }
                    fill += __popc(m);
                    if (fill + 32u > kDensityCap) {
                        take(fill, in_set);
                        fill = 0;
                    }
                }
            }
        if (fill) take(fill, in_set);
    }
    if ((left >> lane) & 1u)
        for (int zz = w.lo[2]; zz <= w.hi[2]; ++zz)
            for (int yy = w.lo[1]; yy <= w.hi[1]; ++yy) {
                uint32_t beg, end;
                row_range(w.lo[0], w.hi[0], yy, zz, beg, end);
                for (uint32_t i = beg; i < end; ++i) {
                    const float4 q = __ldg(&sorted[i]);
                    const float dx = q.x - p.x, dy = q.y - p.y, dz = q.z - p.z;
                    const float d2 = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
                    const float u = fmaf(-d2, inv_h2, 1.0f);
                    if (d2 < h2) sum = fmaf(u * u, u, sum);
                }
            }
    if (active) rho[t] = scale * sum;
}

__global__ void k_set_density(float4* __restrict__ sorted, const float* __restrict__ rho, uint32_t n)
{
    after_launch();
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t < n) sorted[t].w = rho[t];
}

// ------------------------------------------------------------ surface
// Whether a cell of the window's plane z passes the test.  The plane's loads
// are in flight together; one after the other each was a trip to the L2 (surface
// and involved cells: 150k particles 23 -> 11 us, 8M 27 -> 15).
template <int kExt, class Test>
__device__ __forceinline__ uint8_t plane_any(const Window& w, int x, int y, int z, const Grid& sp, Test test)
{
    bool any = false;
#pragma unroll
    for (int dy = -kExt; dy <= kExt; ++dy)
#pragma unroll
        for (int dx = -kExt; dx <= kExt; ++dx)
            any |= test(lin3(clampi(x + dx, w.lo[0], w.hi[0]), clampi(y + dy, w.lo[1], w.hi[1]), z, sp));
    return any ? 1 : 0;
}

// extractionOfSurfaceParticles (cu:70-120): an occupied cell with an empty
// cell in its clamped 3x3x3 neighbourhood is a surface cell; the last cell
// layer of each axis is never tested (cu:81).
__global__ void k_surface_cells(Grid sp, const uint8_t* __restrict__ occ, uint8_t* __restrict__ surf)
{
    after_launch();
    const uint64_t C = (uint64_t)sp.res[0] * sp.res[1] * sp.res[2];
    const uint64_t t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= C) return;
    uint32_t x, y, z;
    unlin3((uint32_t)t, sp, x, y, z);
    uint8_t s = 0;
    if (x < sp.res[0] - 1 && y < sp.res[1] - 1 && z < sp.res[2] - 1 && occ[t]) {
        const Window w = window((int)x, (int)y, (int)z, 1, sp);
        for (int zz = w.lo[2]; zz <= w.hi[2] && !s; ++zz)
            s = plane_any<1>(w, (int)x, (int)y, zz, sp, [&](uint32_t c) { return occ[c] == 0; });
    }
    surf[t] = s;
}

// The involved cells of extractionOfSurfaceAndInvolveParticles (cu:519-550),
// gathered instead of scattered: an occupied cell is involved when a surface
// cell lies within +-2 cells on every axis.
__global__ void k_involved_cells(Grid sp, const uint8_t* __restrict__ occ, const uint8_t* __restrict__ surf,
                                 uint8_t* __restrict__ invol)
{
    after_launch();
    const uint64_t C = (uint64_t)sp.res[0] * sp.res[1] * sp.res[2];
    const uint64_t t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= C) return;
    uint8_t v = 0;
    if (occ[t]) {
        uint32_t x, y, z;
        unlin3((uint32_t)t, sp, x, y, z);
        const Window w = window((int)x, (int)y, (int)z, 2, sp);
        for (int zz = w.lo[2]; zz <= w.hi[2] && !v; ++zz)
            v = plane_any<2>(w, (int)x, (int)y, zz, sp, [&](uint32_t c) { return surf[c] != 0; });
    }
    invol[t] = v;
}

// The gradient's factor of a neighbour at squared distance d2 (0 < d2 < h^2),
// float(k x x) with x = 1 - d / h, and 1 / d, in the reference's roundings.
template <bool kFast>
__device__ __forceinline__ void colour_gradient(float d2, float h, float h_rcp, float tiny, double k_spiky, float khi,
                                                float klo, float& grad, float& inv)
{
    float ratio;
    if (kFast && d2 >= tiny) {
        const float d = root_exact(d2);
        inv = rcp_exact(d);
        const float q = __fmul_rn(d, h_rcp);
        ratio = fmaf(fmaf(-q, h, d), h_rcp, q);
    } else {
        const float d = __fsqrt_rn(d2);
        inv = __fdiv_rn(1.0f, d);
        ratio = div_exact(d, h, h_rcp);
    }
    // x = float(1.0 - (double)(d / h)): the double difference of 1 and a
    // float is exact, so rounding it to float is the correctly rounded
    // FP32 difference (no FP64 work needed)
    const float x = __fsub_rn(1.0f, ratio);
    // float(k x x) in double (cu:957); in FP32 when |k| is in range (khi > 0)
    grad = khi > 0.f ? spiky_grad(x, khi, klo, k_spiky) : spiky_grad_double(x, k_spiky);
}

// extractionOfSurfaceParticlesUsingColorField (cu:909-971, wSpikyGrad
// cuh:324-334).  The decision |grad c| > 3 depends on a sum, so the sum is
// taken in the reference's order with the reference's roundings (FP64 where
// the source promotes).  Issue-bound on the pairs (16.5 of 32 threads per
// instruction: each lane has its own neighbours); with the root, the division
// and the reciprocal by FMA corrections, the gradient's rounding test halved and
// the window test on sorted indices: 1M particles 1.68 -> 1.29 ms, 262k 0.49 ->
// 0.40.
template <bool kFast>
__global__ void __launch_bounds__(kThreads) k_colorfield(const float4* __restrict__ sorted, uint32_t n,
                                                         const uint2* __restrict__ ranges, Grid sp, float h,
                                                         float h_rcp, float h_lt2, float tiny, double k_spiky, float khi,
                                                         float klo, float mass, uint8_t* __restrict__ psurf)
{
    after_launch();
    __shared__ float4 s_q[kThreads];    // staged candidates, per warp
    __shared__ float s_mr[kThreads];    // their m / rho
    __shared__ uint32_t s_idx[kThreads]; // their sorted index
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    const bool active = t < n;
    if (__all_sync(0xffffffffu, !active)) return;
    const int lane = threadIdx.x & 31;
    const uint32_t wb = threadIdx.x & ~31u;
    const float4 p = active ? sorted[t] : make_float4(0.f, 0.f, 0.f, 1.f);
    const Window w = window(cell1(p.x, sp.min[0], sp.cs), cell1(p.y, sp.min[1], sp.cs),
                            cell1(p.z, sp.min[2], sp.cs), 1, sp);
    float sx = 0.f, sy = 0.f, sz = 0.f;
    // a neighbour at squared distance 0 < d2 < h^2 (the gradient is 0 at d >= h,
    // and +0 / -0 terms leave the sums, never -0, unchanged)
    auto add = [&](float4 q, float d2, float m_rho) {
        float rx = __fsub_rn(p.x, q.x), ry = __fsub_rn(p.y, q.y), rz = __fsub_rn(p.z, q.z);
        float grad, inv;
        colour_gradient<kFast>(d2, h, h_rcp, tiny, k_spiky, khi, klo, grad, inv);
        rx = __fmul_rn(rx, inv);
        ry = __fmul_rn(ry, inv);
        rz = __fmul_rn(rz, inv);
        const float coef = __fmul_rn(m_rho, grad);
        sx = __fadd_rn(sx, __fmul_rn(coef, rx));
        sy = __fadd_rn(sy, __fmul_rn(coef, ry));
        sz = __fadd_rn(sz, __fmul_rn(coef, rz));
    };
    auto dist2 = [&](const float4& q) {
        return dot3_rn(__fsub_rn(p.x, q.x), __fsub_rn(p.y, q.y), __fsub_rn(p.z, q.z));
    };
    auto row_range = [&](int x0, int x1, int yy, int zz, uint32_t& beg, uint32_t& end, uint32_t& cnt) {
        // the particles of a row of x-adjacent cells are contiguous in sorted order
        const uint32_t c0 = lin3(x0, yy, zz, sp);
        beg = kEmpty;
        end = 0;
        cnt = 0;
        for (int xx = 0; xx <= x1 - x0; ++xx) {
            const uint2 r = __ldg(&ranges[c0 + xx]);
            if (r.x != kEmpty) {
                beg = min(beg, r.x);
                end = max(end, r.y);
                cnt += r.y - r.x;
            }
        }
    };
    // nn: the particles of the window at a distance > 0 (the reference counts
    // every particle of the 27 cells, cu:930-950) = the window's particles
    // minus those at distance 0 (the particle itself and exact duplicates)
    uint32_t nn = 0;
    int ulo[3], uhi[3];
    bool compact = true;
#pragma unroll
    for (int ax = 0; ax < 3; ++ax) {
        ulo[ax] = (int)__reduce_min_sync(0xffffffffu, active ? (unsigned)w.lo[ax] : 0x7fffffffu);
        uhi[ax] = (int)__reduce_max_sync(0xffffffffu, active ? (unsigned)(w.hi[ax] + 1) : 0u) - 1;
        compact = compact && uhi[ax] - ulo[ax] <= 4;
    }
    if (compact) {
        // the warp walks the union of its windows; staging drops what lies
        // beyond h of every lane's particle (zero gradient, and such a
        // particle is at a distance > 0, counted through the cell counts);
        // each lane takes the staged particles of its own window in window
        // order (rows from the loop, x from the cell index)
        uint32_t in_window = 0, zeros = 0;
        const WarpBox box = warp_box(active, p.x, p.y, p.z, cull_radius(h, sp.cs));
        for (int zz = ulo[2]; zz <= uhi[2]; ++zz)
            for (int yy = ulo[1]; yy <= uhi[1]; ++yy) {
                const bool row_in = active && zz >= w.lo[2] && zz <= w.hi[2] && yy >= w.lo[1] && yy <= w.hi[1];
                if (!__any_sync(0xffffffffu, row_in)) continue;
                // the run of sorted particles that the row has in this lane's window
                uint32_t beg, end, own = 0, own_end = 0, len = 0;
                if (row_in) row_range(w.lo[0], w.hi[0], yy, zz, own, own_end, len);
                in_window += len;
                uint32_t c;
                row_range(ulo[0], uhi[0], yy, zz, beg, end, c);
                for (uint32_t b = beg; b < end; b += 32) {
                    float4 q = make_float4(0.f, 0.f, 0.f, 0.f);
                    bool keep = false;
                    if (b + lane < end) {
                        q = __ldg(&sorted[b + lane]);
                        keep = box.keeps(q);
                    }
                    const uint32_t mk = __ballot_sync(0xffffffffu, keep);
                    if (keep) {
                        const uint32_t slot = wb + __popc(mk & ((1u << lane) - 1u));
                        s_q[slot] = q;
                        s_mr[slot] = __fdiv_rn(mass, q.w);
                        s_idx[slot] = b + lane;
                    }
                    __syncwarp();
                    const uint32_t cnt = __popc(mk);
                    if (row_in)
                        for (uint32_t k = 0; k < cnt; ++k) {
                            if (s_idx[wb + k] - own >= len) continue;
                            const float4 q2 = s_q[wb + k];
                            const float d2 = dist2(q2);
                            if (!(d2 > 0.0f)) {
                                ++zeros;
                                continue;
                            }
                            if (d2 < h_lt2) add(q2, d2, s_mr[wb + k]);
                        }
                    __syncwarp();
                }
            }
        nn = in_window - zeros;
    } else if (active) {
        for (int zz = w.lo[2]; zz <= w.hi[2]; ++zz)
            for (int yy = w.lo[1]; yy <= w.hi[1]; ++yy) {
                uint32_t beg, end, c;
                row_range(w.lo[0], w.hi[0], yy, zz, beg, end, c);
                for (uint32_t i = beg; i < end; ++i) {
                    const float4 q = __ldg(&sorted[i]);
                    const float d2 = dist2(q);
                    if (!(d2 > 0.0f)) continue;
                    ++nn;
                    if (d2 < h_lt2) add(q, d2, __fdiv_rn(mass, q.w));
                }
            }
    }
    if (!active) return;
    const bool s = nn < 25u || __fsqrt_rn(dot3_rn(sx, sy, sz)) > 3.0f;
    psurf[t] = s ? 1 : 0;
}

// Small frames: four lanes per particle, eight particles per warp.  The
// particles walk the union of their windows row by row; candidates within h of
// their box are staged, each particle's lanes test 32 of them at a time (a bit
// per hit), share its hits out evenly, write the three components of each hit's
// term, and then add one component each in the candidates' order.
constexpr int kColorThreads = 128;
constexpr uint32_t kColorCap = 96;  // staged candidates of a warp
constexpr uint32_t kHitRow = 36;    // pitch of a particle's 32 hits

struct ColorSlice {
    float x[kColorCap], y[kColorCap], z[kColorCap], mr[kColorCap];  // staged candidates, m / rho
    uint32_t idx[kColorCap];                                      // their sorted index
    uint32_t hit[8][kHitRow];                                     // per particle: its hits among 32 candidates
    float term[8][3][kHitRow];                                    // and their terms
};

template <bool kFast>
__global__ void __launch_bounds__(kColorThreads, 8) k_colorfield_quads(const float4* __restrict__ sorted, uint32_t n,
                                                         const uint2* __restrict__ ranges, Grid sp, float h,
                                                         float h_rcp, float h_lt2, float tiny, double k_spiky, float khi,
                                                         float klo, float mass, uint8_t* __restrict__ psurf)
{
    after_launch();
    __shared__ __align__(16) ColorSlice slices[kColorThreads / 32];
    ColorSlice& S = slices[threadIdx.x >> 5];
    const int lane = threadIdx.x & 31, part = lane >> 2;
    const uint32_t sub = lane & 3u;
    const uint32_t t = (blockIdx.x * blockDim.x + threadIdx.x) >> 2;
    const bool active = t < n;
    if (__all_sync(0xffffffffu, !active)) return;
    const float4 p = active ? sorted[t] : make_float4(0.f, 0.f, 0.f, 1.f);
    const Window w = window(cell1(p.x, sp.min[0], sp.cs), cell1(p.y, sp.min[1], sp.cs),
                            cell1(p.z, sp.min[2], sp.cs), 1, sp);
    auto row_range = [&](int x0, int x1, int yy, int zz, uint32_t& beg, uint32_t& end) {
        // the particles of a row of x-adjacent cells are contiguous in sorted order
        const uint32_t c0 = lin3(x0, yy, zz, sp);
        beg = kEmpty;
        end = 0;
        for (int xx = 0; xx <= x1 - x0; ++xx) {
            const uint2 r = __ldg(&ranges[c0 + xx]);
            if (r.x != kEmpty) {
                beg = min(beg, r.x);
                end = max(end, r.y);
            }
        }
    };
    auto dist2 = [&](uint32_t k) {
        return dot3_rn(__fsub_rn(p.x, S.x[k]), __fsub_rn(p.y, S.y[k]), __fsub_rn(p.z, S.z[k]));
    };
    float sum = 0.f;         // component `sub` of the gradient (three lanes)
    uint32_t zeros = 0;      // this lane's tested candidates at distance 0
    uint32_t in_window = 0;  // particles of the window
    // the staged candidates [0, fill); own, len: the run of sorted particles
    // that the row has in this particle's window
    auto take = [&](uint32_t fill, uint32_t own, uint32_t len) {
        __syncwarp();
        for (uint32_t b = 0; b < fill; b += 32) {
            const uint32_t lim = min(32u, fill - b);
            uint32_t m = 0;
            for (uint32_t k = sub; k < lim; k += 4)
                if (S.idx[b + k] - own < len) {
                    const float d2 = dist2(b + k);
                    if (!(d2 > 0.0f)) ++zeros;
                    // (the gradient is 0 at d >= h, and +0 / -0 terms leave the
                    // sums, never -0, unchanged)
                    else if (d2 < h_lt2) m |= 1u << k;
                }
            const uint32_t mine = m;
            m |= __shfl_xor_sync(0xffffffffu, m, 1);
            m |= __shfl_xor_sync(0xffffffffu, m, 2);
            const uint32_t cnt = __popc(m);
            for (uint32_t r = mine; r; r &= r - 1u) {
                const uint32_t k = __ffs(r) - 1;
                S.hit[part][__popc(m & ((1u << k) - 1u))] = b + k;
            }
            __syncwarp();
            for (uint32_t r = sub; r < cnt; r += 4) {
                const uint32_t k = S.hit[part][r];
                float rx = __fsub_rn(p.x, S.x[k]), ry = __fsub_rn(p.y, S.y[k]), rz = __fsub_rn(p.z, S.z[k]);
                const float d2 = dot3_rn(rx, ry, rz);
                float grad, inv;
                colour_gradient<kFast>(d2, h, h_rcp, tiny, k_spiky, khi, klo, grad, inv);
                const float coef = __fmul_rn(S.mr[k], grad);
                S.term[part][0][r] = __fmul_rn(coef, __fmul_rn(rx, inv));
                S.term[part][1][r] = __fmul_rn(coef, __fmul_rn(ry, inv));
                S.term[part][2][r] = __fmul_rn(coef, __fmul_rn(rz, inv));
            }
            const uint32_t end = (cnt + 3u) & ~3u;
            if (cnt + sub < end)
                S.term[part][0][cnt + sub] = S.term[part][1][cnt + sub] = S.term[part][2][cnt + sub] = 0.f;
            __syncwarp();
            if (sub < 3u)
                for (uint32_t r = 0; r < end; r += 4) {
                    const float4 v = *reinterpret_cast<const float4*>(&S.term[part][sub][r]);
                    sum = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(sum, v.x), v.y), v.z), v.w);
                }
            __syncwarp();
        }
    };
    // particles whose windows lie apart are walked in sets (window_mates)
    const float reach = cull_radius(h, sp.cs);
    uint32_t left = __ballot_sync(0xffffffffu, active);
    while (left != 0u) {
        const uint32_t set = window_mates(left, w, 4, lane);
        left &= ~set;
        const bool in_set = (set >> lane) & 1u;
        int ulo[3], uhi[3];
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            ulo[a] = (int)__reduce_min_sync(0xffffffffu, in_set ? (unsigned)w.lo[a] : 0x7fffffffu);
            uhi[a] = (int)__reduce_max_sync(0xffffffffu, in_set ? (unsigned)(w.hi[a] + 1) : 0u) - 1;
        }
        // staging drops what lies beyond h of every particle of the set (zero
        // gradient, and such a particle is at a distance > 0, counted through
        // the cell counts)
        const WarpBox box = warp_box(in_set, p.x, p.y, p.z, reach);
        for (int zz = ulo[2]; zz <= uhi[2]; ++zz)
            for (int yy = ulo[1]; yy <= uhi[1]; ++yy) {
                uint32_t beg, end, own = 0, len = 0, fill = 0;
                if (in_set && zz >= w.lo[2] && zz <= w.hi[2] && yy >= w.lo[1] && yy <= w.hi[1]) {
                    row_range(w.lo[0], w.hi[0], yy, zz, own, len);
                    len = len > own ? len - own : 0u;
                    in_window += len;
                }
                if (!__any_sync(0xffffffffu, len != 0u)) continue;
                row_range(ulo[0], uhi[0], yy, zz, beg, end);
                for (uint32_t base = beg; base < end; base += 32) {
                    float4 q = make_float4(0.f, 0.f, 0.f, 0.f);
                    bool keep = false;
                    if (base + lane < end) {
                        q = __ldg(&sorted[base + lane]);
                        keep = box.keeps(q);
                    }
                    const uint32_t m = __ballot_sync(0xffffffffu, keep);
                    if (keep) {
                        const uint32_t k = fill + __popc(m & ((1u << lane) - 1u));
                        S.x[k] = q.x;
                        S.y[k] = q.y;
                        S.z[k] = q.z;
                        S.mr[k] = __fdiv_rn(mass, q.w);
                        S.idx[k] = base + lane;
                    }
                    fill += __popc(m);
                    if (fill + 32u > kColorCap) {
                        take(fill, own, len);
                        fill = 0;
                    }
                }
                if (fill) take(fill, own, len);
            }
    }
    zeros += __shfl_xor_sync(0xffffffffu, zeros, 1);
    zeros += __shfl_xor_sync(0xffffffffu, zeros, 2);
    const int lead = lane & 28;
    const float sx = __shfl_sync(0xffffffffu, sum, lead), sy = __shfl_sync(0xffffffffu, sum, lead + 1),
                sz = __shfl_sync(0xffffffffu, sum, lead + 2);
    if (!active || sub != 0u) return;
    // nn: the particles of the window at a distance > 0 (the reference counts
    // every particle of the 27 cells, cu:930-950) = the window's particles
    // minus those at distance 0 (the particle itself and exact duplicates)
    const uint32_t nn = in_window - zeros;
    const bool s = nn < 25u || __fsqrt_rn(dot3_rn(sx, sy, sz)) > 3.0f;
    psurf[t] = s ? 1 : 0;
}

// ------------------------------------------------------------ band
// estimationOfSurfaceVertices (cu:554-595): vertices in the clamped box
// idx-3 .. idx+3 (x upper bound exclusive) within 1.5h of a surface
// particle.  `thr` is the largest float whose double value is below
// 1.5*h, so dist <= thr reproduces the reference's double comparison; the
// kernel tests the squared distance against thr2 = sqrt_threshold(thr,
// true), the same decision without the square root.
// Each (y,z) row of at most 6 vertices is OR-ed into the bitset with at most
// two atomics.  kLanes lanes share a particle's z planes: one lane walks 49 rows,
// which is most of a tiny frame's kernel; more lanes only cost flag reads in a
// large one.  kCheck: the words are read first (a stale value only costs an
// atomic), since on a surface a vertex is stamped by seven particles or, on
// coarse grids, by fifty; Akinci12's flags on a fine grid keep every other warp
// full of surface particles, and there the reads cost more than the atomics.
// Measured (us; one lane without the check / 8 or 2 lanes with it): 1.5k particles
// on the coarse grid 25 / 10, 32k 27 / 17, 300k on the coarse grid 87 / 49, 1M 102
// / 93, 8M 453 / 336; Akinci12 262k on the fine grid, 2 lanes: 74 without, 88 with.
template <int kLanes, bool kCheck>
__global__ void k_band_stamp(const float4* __restrict__ sorted, const uint32_t* __restrict__ skeys,
                             const uint8_t* __restrict__ surf, const uint8_t* __restrict__ psurf, uint32_t n,
                             Grid sc, float thr2, uint32_t* __restrict__ bits, Counters* ctr)
{
    after_launch();
    // (kLanes n threads: their number may pass 2^32, the particle's does not)
    const uint32_t t = blockIdx.x * (blockDim.x / kLanes) + threadIdx.x / kLanes, plane = threadIdx.x % kLanes;
    bool is_s = false;
    if (t < n) is_s = psurf ? psurf[t] != 0 : surf[skeys[t]] != 0;
    warp_count(&ctr->n_surface, is_s && plane == 0);
    if (!is_s) return;
    const float4 p = sorted[t];
    const Window w = window(cell1(p.x, sc.min[0], sc.cs), cell1(p.y, sc.min[1], sc.cs),
                            cell1(p.z, sc.min[2], sc.cs), 3, sc);
    if (w.hi[0] <= w.lo[0]) return;
    for (int z = w.lo[2] + (int)plane; z <= w.hi[2]; z += kLanes) {
        const float dz = __fsub_rn(vpos1(z, sc.min[2], sc.cs), p.z);
        for (int y = w.lo[1]; y <= w.hi[1]; ++y) {
            const float dy = __fsub_rn(vpos1(y, sc.min[1], sc.cs), p.y);
            const uint32_t v0 = lin3(w.lo[0], y, z, sc);
            const uint32_t word0 = v0 >> 5;
            uint64_t m = 0;
            for (int x = w.lo[0]; x < w.hi[0]; ++x) {
                const float dx = __fsub_rn(vpos1(x, sc.min[0], sc.cs), p.x);
                // sqrt_rn(d2) <= thr  <=>  d2 < thr2 (the smallest float whose root exceeds thr)
                if (dot3_rn(dx, dy, dz) < thr2) m |= 1ull << (x - w.lo[0]);
            }
            m <<= v0 & 31u;
            const uint32_t m0 = (uint32_t)m, m1 = (uint32_t)(m >> 32);
            if (m0 && (!kCheck || (m0 & ~bits[word0]))) atomicOr(bits + word0, m0);
            if (m1 && (!kCheck || (m1 & ~bits[word0 + 1]))) atomicOr(bits + word0 + 1, m1);
        }
    }
}

__device__ __forceinline__ void mark_group(const GroupMark& gm, uint32_t g, Counters* ctr)
{
    const uint32_t flag = atomicOr(gm.gflag + g, kMarkedGroup);
    if (flag & kMarkedGroup) return;
    const uint32_t gend = (gm.sp.res[0] + 1) * (gm.sp.res[1] + 1) * (gm.sp.res[2] + 1);
    if (flag & kDenseGroup) gm.glist[atomicAdd(&ctr->n_groups, 1u)] = g;
    else gm.glist[gend - 1u - atomicAdd(&ctr->n_sparse, 1u)] = g;
}

// What both list kernels do besides: the overflow flag, and the zeros that the
// classification adds the offsets' tile sums to.
__device__ __forceinline__ void band_list_prologue(const GroupMark& gm, uint32_t cap, Counters* ctr)
{
    const uint32_t nb = ctr->n_band;
    if (blockIdx.x == 0 && threadIdx.x == 0 && nb > cap) {
        atomicOr(&ctr->overflow, 1u);
        atomicMax(&ctr->need_band, nb);
    }
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < gm.ntiles; i += gridDim.x * blockDim.x)
        gm.tile_sums[i] = 0u;
}

// compactSurfaceVertex (cu:293-304) over the bitset: every set bit writes
// its vertex id at its rank.  The band vertices also mark their window
// groups (the spatial cell a vertex's FP32 position falls in, as the grouped
// field kernels' group boxes have it); the first mark of a group appends it
// to the group list.  A word is cut into its grid rows; per row the groups
// from the first set bit's to the last's are marked (a superset at worst:
// a marked group without band vertices is found empty).
__global__ void k_band_list(const uint32_t* __restrict__ bits, const uint32_t* __restrict__ prefix,
                            uint32_t nwords, uint32_t* __restrict__ sv, uint32_t cap, GroupMark gm, Counters* ctr)
{
    after_launch();
    const uint32_t kx = gm.sp.res[0] + 1, ky = gm.sp.res[1] + 1;
    const uint32_t rx = gm.sc.res[0], rxy = gm.sc.res[0] * gm.sc.res[1];
    band_list_prologue(gm, cap, ctr);
    const uint32_t lane = threadIdx.x & 31u;
    for (uint32_t i0 = blockIdx.x * blockDim.x + (threadIdx.x & ~31u); i0 < nwords; i0 += gridDim.x * blockDim.x) {
        const uint32_t i = i0 + lane;
        const uint32_t w0 = i < nwords ? bits[i] : 0u;
        const uint32_t r0 = w0 ? prefix[i] : 0u;
        // the warp writes its words' vertices one word at a time, a lane per bit:
        // consecutive lanes on consecutive entries (each lane writing its own
        // word's, 4 bytes at a time, and each new group's cells read here: 1M ZB05
        // frame, scan and list, 119 -> 90 us, 8M 382 -> 257)
        for (uint32_t m = __ballot_sync(0xffffffffu, w0 != 0u); m; m &= m - 1u) {
            const int src = __ffs((int)m) - 1;
            const uint32_t w = __shfl_sync(0xffffffffu, w0, src), r = __shfl_sync(0xffffffffu, r0, src);
            const uint32_t at = r + (uint32_t)__popc(w & ((1u << lane) - 1u));
            if (((w >> lane) & 1u) && at < cap) sv[at] = ((i0 + (uint32_t)src) << 5) | lane;
        }
        if (w0 == 0u) continue;
        // the word's rows: bits [s, e) lie in row (y, z) from column x on
        const uint32_t v0 = i << 5;
        uint32_t z = v0 / rxy, y = (v0 - z * rxy) / rx, x = v0 - z * rxy - y * rx;
        uint32_t last = 0xffffffffu;
        for (uint32_t s = 0; s < 32u;) {
            const uint32_t len = min(32u - s, rx - x);
            const uint32_t seg = w0 & ((len == 32u ? 0xffffffffu : ((1u << len) - 1u)) << s);
            if (seg) {
                const uint32_t xf = x + (uint32_t)(__ffs(seg) - 1) - s, xl = x + (31u - (uint32_t)__clz(seg)) - s;
                const int cf = clampi(cell1(vpos1(xf, gm.sc.min[0], gm.sc.cs), gm.sp.min[0], gm.sp.cs), 0, (int)kx - 1);
                const int cl = clampi(cell1(vpos1(xl, gm.sc.min[0], gm.sc.cs), gm.sp.min[0], gm.sp.cs), 0, (int)kx - 1);
                const int cy = clampi(cell1(vpos1(y, gm.sc.min[1], gm.sc.cs), gm.sp.min[1], gm.sp.cs), 0, (int)ky - 1);
                const int cz = clampi(cell1(vpos1(z, gm.sc.min[2], gm.sc.cs), gm.sp.min[2], gm.sp.cs), 0,
                                      (int)gm.sp.res[2]);
                for (int cx = cf; cx <= cl; ++cx) {
                    const uint32_t g = (uint32_t)cx + kx * ((uint32_t)cy + ky * (uint32_t)cz);
                    if (g != last) {
                        last = g;
                        if (gm.gflag[g] & kMarkedGroup) continue;  // (a stale value only costs the atomic)
                        mark_group(gm, g, ctr);
                    }
                }
            }
            s += len;
            x = 0;
            if (++y == gm.sc.res[1]) {
                y = 0;
                ++z;
            }
        }
    }
}

// The list for few words (small or coarse grids): a warp per word, a lane per
// bit.  On coarse grids a word crosses ten groups or more, whose flags one lane
// fetched one after the other.  A lane marks its vertex's group and, as the kernel
// above, those between it and the vertex before it in its row (the same groups are
// marked by both).
__global__ void k_band_list_words(const uint32_t* __restrict__ bits, const uint32_t* __restrict__ prefix,
                                  uint32_t nwords, uint32_t* __restrict__ sv, uint32_t cap, GroupMark gm, Counters* ctr)
{
    after_launch();
    const int kx = (int)gm.sp.res[0] + 1, ky = (int)gm.sp.res[1] + 1;
    band_list_prologue(gm, cap, ctr);
    const uint32_t lane = threadIdx.x & 31u;
    for (uint32_t i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < nwords; i += (gridDim.x * blockDim.x) >> 5) {
        const uint32_t w = bits[i];
        if (w == 0u) continue;
        const uint32_t below = w & ((1u << lane) - 1u), v = (i << 5) | lane;
        const uint32_t at = prefix[i] + (uint32_t)__popc(below);
        const bool set = (w >> lane) & 1u;
        uint32_t x, y, z;
        unlin3(v, gm.sc, x, y, z);
        const int cx = clampi(cell1(vpos1(x, gm.sc.min[0], gm.sc.cs), gm.sp.min[0], gm.sp.cs), 0, kx - 1);
        const int cy = clampi(cell1(vpos1(y, gm.sc.min[1], gm.sc.cs), gm.sp.min[1], gm.sp.cs), 0, ky - 1);
        const int cz = clampi(cell1(vpos1(z, gm.sc.min[2], gm.sc.cs), gm.sp.min[2], gm.sp.cs), 0, (int)gm.sp.res[2]);
        const int before = below ? 31 - __clz((int)below) : (int)lane;
        const int px = __shfl_sync(0xffffffffu, cx, before);
        // a vertex before it in the word lies in its row when no more columns lie between them than its own
        const bool row = below != 0u && lane - (uint32_t)before <= x;
        if (!set) continue;
        if (at < cap) sv[at] = v;
        for (int c = row ? px + 1 : cx; c <= cx; ++c) mark_group(gm, (uint32_t)(c + kx * (cy + ky * cz)), ctr);
    }
}


// Stages the warp's next chunk of candidates [base, end): the ones within
// the box's reach go to sq in their order; returns how many.  nbox is the
// number inside the grown box itself, which the callers count towards their
// chunk sums exactly as before the reach test was added, so that the sums
// join their totals at the same points.
// kIndexed: with their sorted index in w.
template <bool kIndexed = false>
__device__ __forceinline__ uint32_t stage_in_box(const float4* __restrict__ src, uint32_t base, uint32_t end,
                                                 const WarpBox& box, float4* sq, int lane, uint32_t& nbox)
{
    float4 q = make_float4(0.f, 0.f, 0.f, 0.f);
    bool in = false, keep = false;
    if (base + lane < end) {
        q = __ldg(&src[base + lane]);
        in = box.holds(q);
        keep = in && box.reaches(q);
        if (kIndexed) q.w = __uint_as_float(base + lane);
    }
    nbox = __popc(__ballot_sync(0xffffffffu, in));
    const uint32_t m = __ballot_sync(0xffffffffu, keep);
    if (keep) sq[__popc(m & ((1u << lane) - 1u))] = q;
    return __popc(m);
}

// ------------------------------------------------------------ anisotropic path
// calculationOfMeanAndSmoothParticles (cu:598-658).  Two means per particle:
// * mean32: the reference's FP32 sum sum(w x) / sum(w) in its order with its
//   roundings.  It decides the neighbour counts of the covariance stage, so
//   it must be the reference's bit for bit.
// * mean: the same quantity to near FP64 accuracy, as x_i + sum(w (x_j -
//   x_i)) / sum(w).  The offsets x_j - x_i are exact (Sterbenz) and at most R
//   long, so their sums stay small; they are summed per chunk of 32 to 63
//   candidates and the chunk sums, like the weights, are added with Kahan
//   compensation (neighbouring particles sum nearly the same candidates in
//   the same order, so the rounding errors of long plain sums would be
//   correlated between them and would not average out in the field).  The reference's own FP32 sum of absolute coordinates is
//   off by up to 4.5e-7 (1M-particle frame) and by more with thousands of
//   neighbours; the covariance is taken about this mean, and the smoothed
//   positions are formed from it.  mean.w = its weight sum (the adjoint
//   divides by it); smoothed.w = m / rho.
#ifndef FSR_SMOOTH_MIN_BLOCKS
#define FSR_SMOOTH_MIN_BLOCKS 4  // 64 registers: 4 blocks of 256 threads per SM (measured best of 1, 4, 5, 6)
#endif
template <bool kFast, bool kSets>
__global__ void __launch_bounds__(kThreads, FSR_SMOOTH_MIN_BLOCKS) k_smooth(const float4* __restrict__ sorted, uint32_t n,
                                                     const uint2* __restrict__ ranges, Grid sp, float R,
                                                     float R_rcp, float R_lt2, float tiny, int span,
                                                     float one_minus_lambda, float lambda, float mass, float4* __restrict__ mean,
                                                     float4* __restrict__ mean32, float4* __restrict__ smoothed)
{
    after_launch();
    __shared__ float4 s_q[kThreads];  // 32 staged candidates per warp
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    const bool active = t < n;
    if (__all_sync(0xffffffffu, !active)) return;
    const int lane = threadIdx.x & 31;
    float4* sq = s_q + (threadIdx.x & ~31u);
    const float4 p = active ? sorted[t] : make_float4(0.f, 0.f, 0.f, 1.f);
    // cells beyond R on some axis only hold zero-weight particles, whose +0
    // terms leave the exact sums unchanged: skip them
    const Window w = narrow(window(cell1(p.x, sp.min[0], sp.cs), cell1(p.y, sp.min[1], sp.cs),
                                   cell1(p.z, sp.min[2], sp.cs), 2, sp),
                            p.x, p.y, p.z, cull_radius(R, sp.cs), sp);
    float ws = 0.f, mx = 0.f, my = 0.f, mz = 0.f;
    // chunk sums of w and w (x_j - x_i), and their compensated totals
    float cw = 0.f, cx = 0.f, cy = 0.f, cz = 0.f;
    Kahan tw, tx, ty, tz;
    auto add = [&](const float4& q) {
        const float dx = __fsub_rn(p.x, q.x), dy = __fsub_rn(p.y, q.y), dz = __fsub_rn(p.z, q.z);
        const float d2 = dot3_rn(dx, dy, dz);
        if (!(d2 < R_lt2)) return;  // d >= R: weight 0, and +0 terms leave the sums unchanged
        const float s = dist_over<kFast>(d2, R, R_rcp, tiny);
        const float wt = __fsub_rn(1.0f, __fmul_rn(__fmul_rn(s, s), s));
        ws = __fadd_rn(ws, wt);
        mx = __fadd_rn(mx, __fmul_rn(q.x, wt));
        my = __fadd_rn(my, __fmul_rn(q.y, wt));
        mz = __fadd_rn(mz, __fmul_rn(q.z, wt));
        cw = __fadd_rn(cw, wt);
        cx = __fmaf_rn(-wt, dx, cx);
        cy = __fmaf_rn(-wt, dy, cy);
        cz = __fmaf_rn(-wt, dz, cz);
    };
    // the chunk sums join the totals once at least 32 candidates (staged or
    // walked) have been added since the last time
    uint32_t since = 0;
    auto fold = [&]() {
        tw.add(cw);
        tx.add(cx);
        ty.add(cy);
        tz.add(cz);
        cw = cx = cy = cz = 0.f;
        since = 0;
    };
    auto row_range = [&](int x0, int x1, int yy, int zz, uint32_t& beg, uint32_t& end) {
        const uint32_t c0 = lin3(x0, yy, zz, sp);
        beg = kEmpty;
        end = 0;
        for (int xx = 0; xx <= x1 - x0; ++xx) {
            const uint2 r = __ldg(&ranges[c0 + xx]);
            if (r.x != kEmpty) {
                beg = min(beg, r.x);
                end = max(end, r.y);
            }
        }
    };
    // Lanes whose windows span few cells per axis walk their union together:
    // each chunk of 32 candidates is loaded once (one per lane) and every lane
    // tests all of them, so no lane idles on a window of its own.  Exact: a
    // candidate outside a lane's window lies beyond the cull radius of its
    // particle on some axis (span >= 0: that radius is below 2 cells, so the
    // +-2 cell window never cuts a lane's narrowed window), and the lane's own
    // candidates keep their window order.
    // kSets (R above a cell: windows of up to 5 x 5 x 5 cells, which a lane on
    // its own would take thousands of steps for): a warp whose windows lie
    // apart walks them set by set.  Else the whole warp is one set or none
    // (measured at R = 0.8 cells: in sets, smoothing 0.81 -> 0.87 ms at 1M).
    auto walk = [&](bool in_set) {
        int ulo[3], uhi[3];
        bool compact = true;
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            ulo[a] = (int)__reduce_min_sync(0xffffffffu, in_set ? (unsigned)w.lo[a] : 0x7fffffffu);
            uhi[a] = (int)__reduce_max_sync(0xffffffffu, in_set ? (unsigned)(w.hi[a] + 1) : 0u) - 1;
            compact = compact && uhi[a] - ulo[a] <= span;
        }
        if (!kSets && !compact) return false;
        // candidates beyond R of every lane's particle are dropped at staging
        // (their weights are 0: the sums are unchanged)
        const WarpBox box = warp_box(in_set, p.x, p.y, p.z, cull_radius(R, sp.cs));
        for (int zz = ulo[2]; zz <= uhi[2]; ++zz)
            for (int yy = ulo[1]; yy <= uhi[1]; ++yy) {
                uint32_t beg, end;
                int x0 = ulo[0], x1 = uhi[0];
                if (kSets && !row_reach(box, sp, yy, zz, x0, x1)) continue;
                row_range(x0, x1, yy, zz, beg, end);
                for (uint32_t base = beg; base < end; base += 32) {
                    uint32_t nbox;
                    const uint32_t cnt = stage_in_box(sorted, base, end, box, sq, lane, nbox);
                    __syncwarp();
                    if (!kSets || in_set) {
                        for (uint32_t k = 0; k < cnt; ++k) add(sq[k]);
                        since += nbox;
                        if (since >= 32) fold();
                    }
                    __syncwarp();
                }
            }
        return true;
    };
    uint32_t left = __ballot_sync(0xffffffffu, active);
    if (kSets) {
        for (int sets = 0; left != 0u && span >= 0 && sets < kMaxSets; ++sets) {
            const uint32_t set = window_mates(left, w, span, lane);
            left &= ~set;
            walk((set >> lane) & 1u);
        }
    } else if (walk(active)) {
        left = 0u;
    }
    if ((left >> lane) & 1u) {
        for (int zz = w.lo[2]; zz <= w.hi[2]; ++zz)
            for (int yy = w.lo[1]; yy <= w.hi[1]; ++yy) {
                uint32_t beg, end;
                row_range(w.lo[0], w.hi[0], yy, zz, beg, end);
                for (uint32_t base = beg; base < end; base += 32) {
                    const uint32_t lim = min(end, base + 32u);
                    for (uint32_t i = base; i < lim; ++i) add(__ldg(&sorted[i]));
                    since += lim - base;
                    if (since >= 32) fold();
                }
            }
    }
    if (!active) return;
    fold();
    // ws >= 1: the particle itself has weight 1
    mx = __fdiv_rn(mx, ws);
    my = __fdiv_rn(my, ws);
    mz = __fdiv_rn(mz, ws);
    mean32[t] = make_float4(mx, my, mz, ws);
    const float W = tw.s - tw.c;
    const float ax = p.x + (tx.s - tx.c) / W, ay = p.y + (ty.s - ty.c) / W, az = p.z + (tz.s - tz.c) / W;
    mean[t] = make_float4(ax, ay, az, W);  // w: the weight sum (the adjoint divides by it)
    smoothed[t] = make_float4(__fadd_rn(__fmul_rn(one_minus_lambda, p.x), __fmul_rn(lambda, ax)),
                              __fadd_rn(__fmul_rn(one_minus_lambda, p.y), __fmul_rn(lambda, ay)),
                              __fadd_rn(__fmul_rn(one_minus_lambda, p.z), __fmul_rn(lambda, az)),
                              __fdiv_rn(mass, p.w));
}

//
// Four lanes per particle; a block of four warps takes 32 consecutive sorted
// particles, a warp eight of them.  The sums must run in candidate order, but
// the weights need not: the candidates that reach the warp's box are staged,
// the four lanes of a particle compute the weights of every fourth group of
// four of them, and then each lane adds one component of the sums (the
// weight, x, y or z) over all of them in order.
constexpr int kQuadThreads = 128;
constexpr uint32_t kQuadCap = 96;               // staged candidates of a warp (multiple of 4)
constexpr uint32_t kQuadRow = kQuadCap + 4;   // row pitch in words: rows 4 banks apart
constexpr uint32_t kQuadGroups = 8;             // chunk sums in flight

struct QuadSlice {
    float q[4][kQuadRow];  // 1, x, y, z of the staged candidates
    float w[8][kQuadRow];  // per particle: their weights (0 at and beyond R)
    uint32_t gend[kQuadGroups];  // ends of the closed chunk sums
    uint32_t idx[kQuadRow];      // the staged candidates' sorted index (own_folds)
};

template <bool kFast>
__global__ void __launch_bounds__(kQuadThreads, 6) k_smooth_quads(const float4* __restrict__ sorted, uint32_t n,
                                                     const uint2* __restrict__ ranges, Grid sp, float R,
                                                     float R_rcp, float R_lt2, float tiny, int max_span,
                                                     float one_minus_lambda, float lambda, float mass, float4* __restrict__ mean,
                                                     float4* __restrict__ mean32, float4* __restrict__ smoothed)
{
    after_launch();
    __shared__ __align__(16) QuadSlice slices[kQuadThreads / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    QuadSlice& S = slices[warp];
    const uint32_t first = blockIdx.x * 32u;
    if (first + 8u * warp >= n) return;
    // the block's 32 particles, one per lane: their windows and box decide the
    // walk and the chunk sums (the same for the four warps)
    const bool there = first + lane < n;
    const float4 pl = there ? sorted[first + lane] : make_float4(0.f, 0.f, 0.f, 1.f);
    // cells beyond R on some axis only hold zero-weight particles, whose +0
    // terms leave the exact sums unchanged: skip them
    const Window wl = narrow(window(cell1(pl.x, sp.min[0], sp.cs), cell1(pl.y, sp.min[1], sp.cs),
                                    cell1(pl.z, sp.min[2], sp.cs), 2, sp),
                             pl.x, pl.y, pl.z, cull_radius(R, sp.cs), sp);
    // this lane's particle and component
    const int src = 8 * warp + (lane >> 2), comp = lane & 3, part = lane >> 2;
    const uint32_t t = first + src;
    const bool active = t < n;
    float4 p;
    p.x = __shfl_sync(0xffffffffu, pl.x, src);
    p.y = __shfl_sync(0xffffffffu, pl.y, src);
    p.z = __shfl_sync(0xffffffffu, pl.z, src);
    p.w = __shfl_sync(0xffffffffu, pl.w, src);
    const float pc = comp == 0 ? 0.f : comp == 1 ? p.x : comp == 2 ? p.y : p.z;
    // the reference's FP32 sum of this component, the chunk sum, its
    // compensated total; component 0 sums the weights (q = 1, dx = -1)
    float ref = 0.f, chunk = 0.f;
    Kahan tot;
    auto fold = [&]() {
        tot.add(chunk);
        chunk = 0.f;
    };
    auto weight = [&](float qx, float qy, float qz) {
        const float d2 = dot3_rn(__fsub_rn(p.x, qx), __fsub_rn(p.y, qy), __fsub_rn(p.z, qz));
        // d >= R: weight 0, and +0 terms leave the sums unchanged
        const float s = dist_over<kFast>(d2, R, R_rcp, tiny);
        return d2 < R_lt2 ? __fsub_rn(1.0f, __fmul_rn(__fmul_rn(s, s), s)) : 0.f;
    };
    auto sum = [&](float q, float wt) {
        ref = __fadd_rn(ref, __fmul_rn(q, wt));
        chunk = __fmaf_rn(-wt, __fsub_rn(pc, q), chunk);
    };
    // weights of the staged candidates [0, fill), then this component's sums over [s, e)
    auto weights = [&](uint32_t fill, bool on) {
        __syncwarp();
        for (uint32_t k = 4u * comp; k < fill; k += 16u) {
            const float4 X = *reinterpret_cast<const float4*>(&S.q[1][k]);
            const float4 Y = *reinterpret_cast<const float4*>(&S.q[2][k]);
            const float4 Z = *reinterpret_cast<const float4*>(&S.q[3][k]);
            float4 W;
            W.x = weight(X.x, Y.x, Z.x);
            W.y = weight(X.y, Y.y, Z.y);
            W.z = weight(X.z, Y.z, Z.z);
            W.w = weight(X.w, Y.w, Z.w);
            *reinterpret_cast<float4*>(&S.w[part][k]) = on ? W : make_float4(0.f, 0.f, 0.f, 0.f);
        }
        __syncwarp();
    };
    auto sums = [&](uint32_t s, uint32_t e) {
        for (uint32_t k = s; k < e; k += 4) {
            const float4 Q = *reinterpret_cast<const float4*>(&S.q[comp][k]);
            const float4 W = *reinterpret_cast<const float4*>(&S.w[part][k]);
            sum(Q.x, W.x);
            sum(Q.y, W.y);
            sum(Q.z, W.z);
            sum(Q.w, W.w);
        }
    };
    auto row_range = [&](int x0, int x1, int yy, int zz, uint32_t& beg, uint32_t& end) {
        const uint32_t c0 = lin3(x0, yy, zz, sp);
        beg = kEmpty;
        end = 0;
        for (int xx = 0; xx <= x1 - x0; ++xx) {
            const uint2 r = __ldg(&ranges[c0 + xx]);
            if (r.x != kEmpty) {
                beg = min(beg, r.x);
                end = max(end, r.y);
            }
        }
    };
    // Particles whose windows span few cells per axis walk their union
    // together (window_mates), as in k_smooth; the sets are the block's.
    // The chunk sums end where k_smooth's do, so that both kernels' sums agree
    // bit for bit for radii below a cell (max_span 3): where the whole block is
    // one set, at 32 candidates of its box; else at every 32 of the particle's own
    // window, row by row (own_folds).  k_smooth's totals also take the 0 of a chunk
    // that lies beyond R, which can move a compensated total's last bit; after the
    // first such 0 (s = s - c rounded) the next ones change nothing, so one stands for
    // all.  (Without it 1 of 12,000 means in rows of 64 and more differed; 3k
    // particles 302 -> 304 us, 45k 647 -> 648.)
    bool one_set = max_span >= 0;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const int lo = (int)__reduce_min_sync(0xffffffffu, there ? (unsigned)wl.lo[a] : 0x7fffffffu);
        const int hi = (int)__reduce_max_sync(0xffffffffu, there ? (unsigned)(wl.hi[a] + 1) : 0u) - 1;
        one_set = one_set && hi - lo <= max_span;
    }
    const bool own_folds = max_span == 3 && !one_set;
    Window w;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        w.lo[a] = __shfl_sync(0xffffffffu, wl.lo[a], src);
        w.hi[a] = __shfl_sync(0xffffffffu, wl.hi[a], src);
    }
    for (uint32_t k = lane; k < kQuadRow; k += 32) S.q[0][k] = 1.0f;
    const float r = cull_radius(R, sp.cs);
    uint32_t left = __ballot_sync(0xffffffffu, there);
    uint32_t since = 0;  // candidates taken since the chunk sums last joined the totals
    for (int sets = 0; left != 0u && max_span >= 0 && sets < kMaxSets; ++sets) {
        const uint32_t set = window_mates(left, wl, max_span, lane);
        left &= ~set;
        if (((set >> (8 * warp)) & 0xffu) == 0u) continue;  // none of this warp's particles
        const bool in_set = (set >> lane) & 1u;
        const bool mine_in = (set >> src) & 1u;
        int ulo[3], uhi[3];
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            ulo[a] = (int)__reduce_min_sync(0xffffffffu, in_set ? (unsigned)wl.lo[a] : 0x7fffffffu);
            uhi[a] = (int)__reduce_max_sync(0xffffffffu, in_set ? (unsigned)(wl.hi[a] + 1) : 0u) - 1;
        }
        // candidates beyond R of every particle of the warp are dropped at
        // staging; the chunk sums join the totals once at least 32 candidates
        // of the set's box have passed since the last time
        const WarpBox box = warp_box(in_set, pl.x, pl.y, pl.z, r);
        const WarpBox mine = warp_box(mine_in, p.x, p.y, p.z, r);
        uint32_t fill = 0, ngr = 0;
        uint32_t own = 0, len = 0, chunk_at = 0;  // own_folds: the row's run of this particle's window, its chunk
        since = 0;
        // pads the staged candidates to a multiple of 4 with ones of weight 0
        auto pad = [&]() {
            const uint32_t m = (0u - fill) & 3u;
            if ((uint32_t)lane < m) S.q[1][fill + lane] = S.q[2][fill + lane] = S.q[3][fill + lane] = 1.0e18f;
            fill += m;
        };
        auto flush = [&]() {
            const uint32_t staged = fill;
            pad();
            weights(fill, mine_in);
            if (own_folds) {
                for (uint32_t k = 0; k < staged; ++k) {
                    const float wt = S.w[part][k];  // 0: beyond R, or of another window
                    const uint32_t c = (S.idx[k] - own) >> 5;
                    if (wt != 0.f && c != chunk_at) {
                        fold();
                        if (c - chunk_at > 1u) tot.add(0.f);
                        chunk_at = c;
                    }
                    sum(S.q[comp][k], wt);
                }
                fill = 0;
                __syncwarp();
                return;
            }
            uint32_t s = 0;
            for (uint32_t g = 0; g < ngr; ++g) {
                const uint32_t e = S.gend[g];
                sums(s, e);
                fold();
                s = e;
            }
            sums(s, fill);
            fill = ngr = 0;
            __syncwarp();
        };
        for (int zz = ulo[2]; zz <= uhi[2]; ++zz)
            for (int yy = ulo[1]; yy <= uhi[1]; ++yy) {
                uint32_t beg, end;
                int x0 = ulo[0], x1 = uhi[0];
                if (max_span > 3 && !row_reach(mine, sp, yy, zz, x0, x1)) continue;
                row_range(x0, x1, yy, zz, beg, end);
                if (own_folds) {
                    own = len = chunk_at = 0;
                    if (mine_in && zz >= w.lo[2] && zz <= w.hi[2] && yy >= w.lo[1] && yy <= w.hi[1]) {
                        row_range(w.lo[0], w.hi[0], yy, zz, own, len);
                        len = len > own ? len - own : 0u;
                    }
                }
                float4 next = beg + lane < end ? __ldg(&sorted[beg + lane]) : make_float4(0.f, 0.f, 0.f, 0.f);
                for (uint32_t base = beg; base < end; base += 32) {
                    const float4 q = next;
                    if (base + 32 + lane < end) next = __ldg(&sorted[base + 32 + lane]);
                    const bool in = base + lane < end && box.holds(q);
                    const uint32_t nbox = __popc(__ballot_sync(0xffffffffu, in));
                    if (nbox == 0u) continue;
                    const bool keep = in && mine.reaches(q);
                    const uint32_t m = __ballot_sync(0xffffffffu, keep);
                    if (keep) {
                        const uint32_t k = fill + __popc(m & ((1u << lane) - 1u));
                        S.q[1][k] = q.x;
                        S.q[2][k] = q.y;
                        S.q[3][k] = q.z;
                        if (own_folds) S.idx[k] = base + lane;
                    }
                    fill += __popc(m);
                    since += own_folds ? 0u : nbox;
                    if (since >= 32 && !own_folds) {
                        since = 0;
                        pad();
                        if (lane == 0) S.gend[ngr] = fill;
                        ++ngr;
                    }
                    if (fill + 35u > kQuadCap || ngr == kQuadGroups) flush();
                }
                if (own_folds) {
                    flush();
                    // the row's full chunks have ended, its rest waits for more
                    if (len >= 32u) {
                        if (chunk_at < (len >> 5)) fold();
                        if (chunk_at + 1u < (len >> 5)) tot.add(0.f);
                        since = 0;
                    }
                    since += len & 31u;
                    if (since >= 32u) {
                        fold();
                        since = 0;
                    }
                }
            }
        flush();
    }
    if (left != 0u) {
        // each particle walks its own window, 32 candidates at a time
        since = 0;
        if ((left >> src) & 1u)
            for (int zz = w.lo[2]; zz <= w.hi[2]; ++zz)
                for (int yy = w.lo[1]; yy <= w.hi[1]; ++yy) {
                    uint32_t beg, end;
                    row_range(w.lo[0], w.hi[0], yy, zz, beg, end);
                    const uint32_t quad = 0xfu << (lane & 28);
                    for (uint32_t base = beg; base < end; base += 32) {
                        const uint32_t lim = min(end, base + 32u);
                        for (uint32_t i = base + comp; i < lim; i += 4) {
                            const float4 q = __ldg(&sorted[i]);
                            S.w[part][i - base] = weight(q.x, q.y, q.z);
                        }
                        __syncwarp(quad);
                        for (uint32_t i = base; i < lim; ++i) {
                            const float wt = S.w[part][i - base];
                            if (wt != 0.f)
                                sum(comp == 0 ? 1.0f : __ldg(reinterpret_cast<const float*>(sorted + i) + comp - 1), wt);
                        }
                        __syncwarp(quad);
                        since += lim - base;
                        if (since >= 32) {
                            fold();
                            since = 0;
                        }
                    }
                }
        __syncwarp();
    }
    fold();
    const int lead = lane & 28;  // component 0 holds the weight sums (>= 1: the particle itself has weight 1)
    const float ws = __shfl_sync(0xffffffffu, ref, lead);
    const float val = tot.s - tot.c;
    const float W = __shfl_sync(0xffffffffu, val, lead);
    if (!active) return;
    const uint32_t o = 4u * t + ((comp + 3) & 3);  // x, y, z, weight sum (mean.w: the adjoint divides by it)
    reinterpret_cast<float*>(mean32)[o] = comp == 0 ? ws : __fdiv_rn(ref, ws);
    const float ax = pc + val / W;
    reinterpret_cast<float*>(mean)[o] = comp == 0 ? W : ax;
    reinterpret_cast<float*>(smoothed)[o] =
        comp == 0 ? __fdiv_rn(mass, p.w) : __fadd_rn(__fmul_rn(one_minus_lambda, pc), __fmul_rn(lambda, ax));
}

// calculationOfTransformMatricesForParticles (cu:689-827) for every
// particle of an involved cell.  The neighbour count (dist <= r about the
// FP32 mean, cu:746) is exact; the covariance is accumulated in chunk sums
// joined with Kahan compensation (CovChunkAccum); the eigen-decomposition
// runs in FP32 and is redone in FP64 when the covariance's condition number
// exceeds 1e4.
// Output record per particle: (x,y,z smoothed, r2max) (G row 0, coef)
// (G row 1, 0) (G row 2, 0) with coef = sigma det(G) m / rho.
// Blocks of two warps: a warp without involved particles exits at once, and
// a small block gives its registers back as soon as its two warps are done,
// so the working warps' blocks fill the SM.
// P lanes per particle: each takes every P-th candidate of the particle's
// walk and the lanes' sums and counts are joined at the end (the covariance
// sums may be taken in any order, the count is an integer).  P = 4 for
// small frames, whose particles alone are too few warps to fill the GPU; P
// = 1 otherwise (four lanes measured slower once the GPU is full).  P = 16
// for the smallest frames with wide windows (kSets: thousands of candidates
// per particle; measured with P = 4 / 16 at R = 1.54 cells: 5k particles 0.21 /
// 0.12 ms, 10k 0.29 / 0.21, 20k 0.42 / 0.38, 40k 0.56 / 0.76).  kSets itself, P =
// 4: 40k particles 1.07 -> 0.56 ms, 200k 4.3 -> 2.3 ms.
constexpr int kCovThreads = 64;
constexpr uint32_t kCovSplitBelow = 1u << 17;  // particles below which P = 4
constexpr uint32_t kCovWideBelow = 12288;      // and P = 16 with kSets
#ifndef FSR_COV_MIN_BLOCKS
#define FSR_COV_MIN_BLOCKS 16
#endif

template <int P, bool kFast, bool kSets>
__global__ void __launch_bounds__(kCovThreads, FSR_COV_MIN_BLOCKS) k_cov(CovArgs a, Counters* ctr)
{
    after_launch();
    __shared__ float4 s_q[kCovThreads];  // 32 staged candidates per warp
    const uint32_t t = (blockIdx.x * blockDim.x + threadIdx.x) / P;
    const uint32_t sub = threadIdx.x % P;
    bool act = t < a.n && a.invol[a.skeys[t]];
    warp_count(&ctr->n_involved, act && sub == 0);
    if (__all_sync(0xffffffffu, !act)) return;
    const int lane = threadIdx.x & 31;
    float4* sq = s_q + (threadIdx.x & ~31u);
    const float4 p = act ? a.sorted[t] : make_float4(0.f, 0.f, 0.f, 1.f);
    // m: the compensated mean the covariance is taken about; m32: the
    // reference's FP32 mean, which decides the neighbour count (dist <= r,
    // cu:746).  They differ by the FP32 mean's rounding error, dm.
    const float4 m = act ? a.mean[t] : p;
    float dm;
    {
        const float4 m32 = act ? a.mean32[t] : p;
        dm = sqrtf(fmaf(m.x - m32.x, m.x - m32.x, fmaf(m.y - m32.y, m.y - m32.y, (m.z - m32.z) * (m.z - m32.z))));
    }
    const float cr = cull_radius(a.R, a.sp.cs) + 2.0f * dm;
    // |q - m|^2 below in2 (above out2) puts q within (beyond) R of m32 with a
    // margin far above the roundings of both squared distances: only
    // candidates in the shell between them take the reference's test
    const float rin = (a.R - dm) * (1.0f - 1e-5f), rout = (a.R + dm) * (1.0f + 1e-5f);
    const float in2 = rin > 0.f ? rin * rin : 0.f, out2 = rout * rout;
    // the window is centred on the particle's cell (cu:710-716); only
    // particles within R of the means count or weigh, so cells beyond R of
    // them on some axis are skipped
    const Window w = narrow(window(cell1(p.x, a.sp.min[0], a.sp.cs), cell1(p.y, a.sp.min[1], a.sp.cs),
                                   cell1(p.z, a.sp.min[2], a.sp.cs), 2, a.sp),
                            m.x, m.y, m.z, cr, a.sp);
    CovChunkAccum acc;
    uint32_t since = 0;  // candidates taken since the chunk sums last joined the totals
    auto fold = [&]() {
        acc.fold();
        since = 0;
    };
    uint32_t nn = 0;
    // d > R: neither counted nor weighed (out2 > R^2; a weight of 0 adds nothing)
    auto take = [&](const float4& q) {
        const float vx = __fsub_rn(q.x, m.x), vy = __fsub_rn(q.y, m.y), vz = __fsub_rn(q.z, m.z);
        const float d2 = dot3_rn(vx, vy, vz);
        if (d2 < in2) ++nn;
        else if (d2 < out2) {  // rare: m32 is loaded again (L1) rather than kept in registers
            const float4 m32 = a.mean32[t];
            if (dot3_rn(__fsub_rn(q.x, m32.x), __fsub_rn(q.y, m32.y), __fsub_rn(q.z, m32.z)) < a.R_le2) ++nn;
        }
        const float s = dist_over<kFast>(d2, a.R, a.R_rcp, a.tiny);
        const float wt = 1.0f - s * s * s;
        acc.add(vx, vy, vz, d2 < a.R_lt2 ? wt : 0.f);
    };
    auto near = [&](const float4& q) {
        return dot3_rn(__fsub_rn(q.x, m.x), __fsub_rn(q.y, m.y), __fsub_rn(q.z, m.z)) < out2;
    };
    auto row_range = [&](int x0, int x1, int yy, int zz, uint32_t& beg, uint32_t& end) {
        const uint32_t c0 = lin3(x0, yy, zz, a.sp);
        beg = kEmpty;
        end = 0;
        for (int xx = 0; xx <= x1 - x0; ++xx) {
            const uint2 r = __ldg(&a.ranges[c0 + xx]);
            if (r.x != kEmpty) {
                beg = min(beg, r.x);
                end = max(end, r.y);
            }
        }
    };
    // Compact warps walk the union of their windows with staged candidates,
    // as in k_smooth.  Exact when the +-2 cell window never cuts a lane's
    // window narrowed about its mean (the mean lies within R of the particle:
    // launch_cov checks R + cull radius < 2 cells), so every candidate the
    // union adds lies beyond R of that lane's mean.  kSets (that check fails,
    // R near or above a cell): a lane takes only the staged candidates of its
    // own window, whose cells of a row are one run of the sorted particles,
    // and windows that lie apart are walked set by set.
    auto walk = [&](bool in_set) {
        int ulo[3], uhi[3];
        bool compact = a.coop_ok != 0;
#pragma unroll
        for (int ax = 0; ax < 3; ++ax) {
            ulo[ax] = (int)__reduce_min_sync(0xffffffffu, in_set ? (unsigned)w.lo[ax] : 0x7fffffffu);
            uhi[ax] = (int)__reduce_max_sync(0xffffffffu, in_set ? (unsigned)(w.hi[ax] + 1) : 0u) - 1;
            compact = compact && uhi[ax] - ulo[ax] <= 3;
        }
        if (!kSets && !compact) return false;
        // candidates beyond R of every lane's mean are dropped at staging
        const WarpBox box = warp_box(in_set, m.x, m.y, m.z, cr);
        for (int zz = ulo[2]; zz <= uhi[2]; ++zz)
            for (int yy = ulo[1]; yy <= uhi[1]; ++yy) {
                uint32_t beg, end, own = 0, len = 0;
                int x0 = ulo[0], x1 = uhi[0];
                if (kSets && P < 16 && !row_reach(box, a.sp, yy, zz, x0, x1)) continue;
                row_range(x0, x1, yy, zz, beg, end);
                if (kSets && in_set && zz >= w.lo[2] && zz <= w.hi[2] && yy >= w.lo[1] && yy <= w.hi[1]) {
                    row_range(w.lo[0], w.hi[0], yy, zz, own, len);
                    len = len > own ? len - own : 0u;
                }
                auto mine = [&](const float4& q) { return !kSets || __float_as_uint(q.w) - own < len; };
                for (uint32_t base = beg; base < end; base += 32) {
                    uint32_t nbox;
                    const uint32_t cnt = stage_in_box<kSets>(a.sorted, base, end, box, sq, lane, nbox);
                    __syncwarp();
                    if (in_set) {
                        uint32_t k = sub;
                        for (; k + 3 * P < cnt; k += 4 * P) {
                            const float4 q0 = sq[k], q1 = sq[k + P], q2 = sq[k + 2 * P], q3 = sq[k + 3 * P];
                            const bool n0 = near(q0) && mine(q0), n1 = near(q1) && mine(q1);
                            const bool n2 = near(q2) && mine(q2), n3 = near(q3) && mine(q3);
                            if (n0) take(q0);
                            if (n1) take(q1);
                            if (n2) take(q2);
                            if (n3) take(q3);
                        }
                        for (; k < cnt; k += P) {
                            const float4 q = sq[k];
                            if (near(q) && mine(q)) take(q);
                        }
                        since += kSets ? (nbox + P - 1) / P : nbox / P;
                        if (since >= 32) fold();
                    }
                    __syncwarp();
                }
            }
        return true;
    };
    uint32_t left = __ballot_sync(0xffffffffu, act);
    if (kSets) {
        for (int sets = 0; left != 0u && sets < kMaxSets; ++sets) {
            const uint32_t set = window_mates(left, w, 5, lane);
            left &= ~set;
            walk((set >> lane) & 1u);
        }
    } else if (walk(act)) {
        left = 0u;
    }
    const bool alone = (left >> lane) & 1u;
    if (alone && P > 1) {
        for (int zz = w.lo[2]; zz <= w.hi[2]; ++zz)
            for (int yy = w.lo[1]; yy <= w.hi[1]; ++yy) {
                uint32_t beg, end;
                row_range(w.lo[0], w.hi[0], yy, zz, beg, end);
                for (uint32_t i = beg + sub; i < end; i += P) {
                    const float4 q = __ldg(&a.sorted[i]);
                    if (near(q)) take(q);
                    if (++since >= 32) fold();
                }
            }
    } else if (alone) {
        for (int zz = w.lo[2]; zz <= w.hi[2]; ++zz)
            for (int yy = w.lo[1]; yy <= w.hi[1]; ++yy) {
                uint32_t beg, end;
                row_range(w.lo[0], w.hi[0], yy, zz, beg, end);
                // four candidates per step
                uint32_t i = beg;
                for (; i + 4 <= end; i += 4) {
                    const float4 q0 = __ldg(&a.sorted[i]), q1 = __ldg(&a.sorted[i + 1]);
                    const float4 q2 = __ldg(&a.sorted[i + 2]), q3 = __ldg(&a.sorted[i + 3]);
                    const bool n0 = near(q0), n1 = near(q1), n2 = near(q2), n3 = near(q3);
                    if (n0) take(q0);
                    if (n1) take(q1);
                    if (n2) take(q2);
                    if (n3) take(q3);
                    since += 4;
                    if (since >= 32) fold();
                }
                for (; i < end; ++i) {
                    const float4 q = __ldg(&a.sorted[i]);
                    if (near(q)) take(q);
                }
            }
    }
    fold();
    // join the particle's lanes (every lane of the warp takes part)
#pragma unroll
    for (int o = 1; o < P; o <<= 1) {
        auto join = [&](Kahan& k) {
            const float s = __shfl_xor_sync(0xffffffffu, k.s, o), c = __shfl_xor_sync(0xffffffffu, k.c, o);
            k.add(s - c);
        };
        join(acc.tot.wsum);
        join(acc.tot.c11);
        join(acc.tot.c22);
        join(acc.tot.c33);
        join(acc.tot.c12);
        join(acc.tot.c13);
        join(acc.tot.c23);
        nn += __shfl_xor_sync(0xffffffffu, nn, o);
    }
    if (!act || sub != 0) return;
    const CovAccum& sums = acc.tot;
    float G[9];
    const float rmax = covariance_to_G(sums, nn, a.min_neighbors, a.h, a.h2, a.h_inv, G, &ctr->n_fp64);
    if (a.crec) {  // the normalised covariance for the adjoint (the same expressions as covariance_to_G)
        const bool used = nn >= a.min_neighbors;
        const float iw = used ? 1.0f / sums.wsum.s : 0.f;
        a.crec[2ull * t] = make_float4((a.h2 + sums.c11.s) * iw, sums.c12.s * iw, sums.c13.s * iw, (a.h2 + sums.c22.s) * iw);
        a.crec[2ull * t + 1] = make_float4(sums.c23.s * iw, (a.h2 + sums.c33.s) * iw, sums.wsum.s, used ? 1.f : 0.f);
    }
    const float det = G[0] * G[4] * G[8] + G[1] * G[5] * G[6] + G[2] * G[3] * G[7] - G[0] * G[5] * G[7] -
                      G[1] * G[3] * G[8] - G[2] * G[4] * G[6];
    const float4 sm = a.smoothed[t];
    const float r2 = rmax * rmax * 1.0001f;
    // the cell's reach for the field's cell culling: support radius plus the
    // smoothing displacement (the kernel sits at the smoothed position, which
    // may lie outside the cell's box); positive floats order like their bits
    const float dx = sm.x - p.x, dy = sm.y - p.y, dz = sm.z - p.z;
    const float reach = rmax + sqrtf(fmaf(dx, dx, fmaf(dy, dy, dz * dz))) * 1.0001f;
    atomicMax(reinterpret_cast<int*>(a.cell_rmax) + a.skeys[t], __float_as_int(reach));
    float4* rec = a.grec + 4ull * t;
    rec[0] = make_float4(sm.x, sm.y, sm.z, r2);
    rec[1] = make_float4(G[0], G[1], G[2], a.sigma * det * sm.w);
    rec[2] = make_float4(G[3], G[4], G[5], 0.f);
    rec[3] = make_float4(G[6], G[7], G[8], 0.f);
    // the field's form of the same kernel: q2 = |G d|^2 = d^T (G^T G) d
    const float m00 = G[0] * G[0] + G[3] * G[3] + G[6] * G[6];
    const float m11 = G[1] * G[1] + G[4] * G[4] + G[7] * G[7];
    const float m22 = G[2] * G[2] + G[5] * G[5] + G[8] * G[8];
    const float m01 = G[0] * G[1] + G[3] * G[4] + G[6] * G[7];
    const float m02 = G[0] * G[2] + G[3] * G[5] + G[6] * G[8];
    const float m12 = G[1] * G[2] + G[4] * G[5] + G[7] * G[8];
    float4* q = a.qrec + 3ull * t;
    q[0] = rec[0];
    q[1] = make_float4(m00, 2.0f * m01, 2.0f * m02, rec[1].w);
    q[2] = make_float4(m11, 2.0f * m12, m22, 0.f);
}

// ------------------------------------------------------------ marching cubes
// The field at the grid positions (x0 + k, y, z), k = 0 .. N - 1 (N <= 4): 0
// outside the grid (getValue, cuh:410-416), the fill value off the band.  x0 >= -1
// and x0 + 1 inside.  One or two bitset words and one prefix give the four
// memberships and ranks; the values of neighbouring band vertices follow one
// another.
template <int N>
__device__ __forceinline__ void field_row(const McArgs& a, int x0, int y, int z, float out[N])
{
#pragma unroll
    for (int k = 0; k < N; ++k) out[k] = 0.f;
    if ((uint32_t)y >= a.sc.res[1] || (uint32_t)z >= a.sc.res[2]) return;
    // the first position inside the grid, and the number of those before it
    const int skip = x0 < 0 ? 1 : 0;
    const uint32_t v = lin3((uint32_t)(x0 + skip), (uint32_t)y, (uint32_t)z, a.sc);
    const uint32_t w = v >> 5, sh = v & 31u;
    const uint32_t lo = __ldg(a.band.bits + w), hi = sh + N > 32u ? __ldg(a.band.bits + w + 1) : 0u;
    const uint32_t f = (uint32_t)((((uint64_t)hi << 32) | lo) >> sh) << skip;
    uint32_t r = __ldg(a.band.prefix + w) + __popc(lo & ((1u << sh) - 1u));
#pragma unroll
    for (int k = 0; k < N; ++k) {
        if (x0 + k < 0 || x0 + k >= (int)a.sc.res[0]) continue;
        out[k] = a.fill;
        if ((f >> k) & 1u) {
            if (r < a.cap_band) out[k] = __ldg(a.band.phi + r);  // r >= cap only in a frame that is re-run
            ++r;
        }
    }
}

// The marching-cubes offsets in one reduce-then-scan over the classify
// words (generateTriangles' vertex offsets and compactValidSurfaceCubes:
// cu:367-380 with the scans of cu:1154-1172).  Per band position t: vofs[t]
// = the vertices of the cubes before t, and a cube with vertices is listed
// at valid[its rank among such cubes] = t.  Within a 4096-position tile both
// counts fit 16 bits (at most 15 x 4096 vertices), so each element is one
// word, vertices low and cubes high, and the block scans add such words.  The
// classification adds up the tiles' words; the scan's blocks add up those of the
// tiles before their own, in full words, or for many tiles one block scans them.
__device__ __forceinline__ uint32_t mc_pair(uint32_t info)
{
    const uint32_t nv = info & 0xFFu;
    return nv | (nv != 0u ? 0x10000u : 0u);
}

// detectValidSurfaceCubes (cu:328-364): a band vertex as cube origin is
// valid when all 8 corners are band vertices and the case emits triangles.
__global__ void k_mc_classify(McArgs a, const Counters* ctr, uint32_t* tile_sums)
{
    after_launch();
    const uint32_t nb = min(ctr->n_band, a.cap_band);
    const uint32_t rx = a.sc.res[0], rxy = a.sc.res[0] * a.sc.res[1];
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, nwarps = (gridDim.x * blockDim.x) >> 5;
    // Runs of 128 once the runs of 32 would put too many atomics on a tile's word:
    // 9M band vertices 92 us, 80 with runs of 128, 84 with 256; below a million the
    // shorter runs keep more warps busy (a 32k frame 10 / 12).
    const uint32_t span = nb < 1u << 20 ? 32u : 128u;
    const uint32_t step = span * nwarps;
    for (uint32_t t0 = span * warp; t0 < nb; t0 = next_of(t0, step, nb)) {
        uint32_t sum = 0;
#pragma unroll 1
        for (uint32_t k = lane; k < span; k += 32u) {
            const uint32_t t = t0 + k;
            const uint32_t v = t < nb ? a.sv[t] : 0xffffffffu;
            uint32_t x, y, z;
            unlin3(v, a.sc, x, y, z);
            uint32_t info = 0;
            // the cube's corners as 4 rows of two x-neighbours, (dy, dz) in
            // {0,1}^2: one bitset word (two when the pair straddles a word) and
            // one prefix per row give both memberships and both ranks (the x + 1
            // corner of a row in the band follows its x corner: rank + 1)
            if (t < nb && x < a.sc.res[0] - 1 && y < a.sc.res[1] - 1 && z < a.sc.res[2] - 1) {
                uint32_t vr[4], wd[4];
                bool all = true;
#pragma unroll
                for (int r = 0; r < 4; ++r) {
                    vr[r] = v + (uint32_t)(r & 1) * rx + (uint32_t)(r >> 1) * rxy;
                    const uint32_t w = vr[r] >> 5, b = vr[r] & 31u;
                    wd[r] = __ldg(a.band.bits + w);
                    const uint32_t next = b < 31u ? (wd[r] >> (b + 1)) : __ldg(a.band.bits + w + 1);
                    all = all && ((wd[r] >> b) & 1u) && (next & 1u);
                }
                if (all) {
                    uint32_t cs = 0;
                    bool in_cap = true;
#pragma unroll
                    for (int r = 0; r < 4; ++r) {
                        const uint32_t b = vr[r] & 31u;
                        const uint32_t r0 =
                            r == 0 ? t : __ldg(a.band.prefix + (vr[r] >> 5)) + __popc(wd[r] & ((1u << b) - 1u));
                        // ranks beyond the capacity only occur in a frame that overflowed and is re-run
                        if (r0 + 1 >= a.cap_band) {
                            in_cap = false;
                            break;
                        }
                        const int dy = r & 1, dz = r >> 1;
                        const int i0 = dy ? (dz ? 2 : 3) : (dz ? 1 : 0);  // corner (0, dy, dz); (1, dy, dz) is i0 + 4
                        if (__ldg(a.band.phi + r0) <= a.iso) cs |= 1u << i0;
                        if (__ldg(a.band.phi + r0 + 1) <= a.iso) cs |= 1u << (i0 + 4);
                    }
                    if (in_cap) info = (uint32_t)c_mc.nverts[cs] | (cs << 8);
                }
            }
            if (t < nb) a.mc[t] = info;
            sum += mc_pair(info);
        }
        // the tile's sums for the offsets (a kernel of its own before: offsets of 9M
        // vertices 45 us, 35 without it)
        sum = __reduce_add_sync(0xffffffffu, sum);
        if (lane == 0 && sum != 0u) atomicAdd(tile_sums + t0 / kScanTile, sum);
    }
}

// The frame's vertex and cube counts, and the pool overflow flags.
__device__ __forceinline__ void mc_counts(const McArgs& a, Counters* ctr, uint32_t verts, uint32_t cubes)
{
    ctr->n_mesh_verts = verts;
    ctr->n_valid = cubes;
    if (cubes > a.cap_valid) {
        atomicOr(&ctr->overflow, 2u);
        atomicMax(&ctr->need_valid, cubes);
    }
    if (verts > a.cap_mesh) {
        atomicOr(&ctr->overflow, 4u);
        atomicMax(&ctr->need_mesh, verts);
    }
}

// One block: exclusive scans of both tile totals, over the tiles' words and
// behind them.
__global__ void __launch_bounds__(kScanThreads) k_mc_scan_tile_sums(McArgs a, Counters* ctr, uint32_t* tile_sums,
                                                                    uint32_t ntiles_max)
{
    after_launch();
    __shared__ uint32_t warp_sums[kScanThreads / 32];
    __shared__ uint32_t last[2];
    const uint32_t n = min(ctr->n_band, a.cap_band);
    const uint32_t ntiles = (n + kScanTile - 1) / kScanTile;
    uint32_t carry[2] = {0u, 0u};
    for (uint32_t b = 0; b < ntiles; b += kScanThreads) {
        const uint32_t i = b + threadIdx.x;
        const uint32_t both = i < ntiles ? tile_sums[i] : 0u;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const uint32_t x = h ? both >> 16 : both & 0xFFFFu;
            const uint32_t incl = block_inclusive_scan(x, warp_sums);
            if (i < ntiles) tile_sums[h * ntiles_max + i] = carry[h] + incl - x;
            if (threadIdx.x == kScanThreads - 1) last[h] = incl;
            __syncthreads();
            carry[h] += last[h];
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) mc_counts(a, ctr, carry[0], carry[1]);
}

template <bool kSums>
__global__ void __launch_bounds__(kScanThreads) k_mc_tile_scan(McArgs a, Counters* ctr, const uint32_t* tile_sums,
                                                               uint32_t ntiles_max)
{
    after_launch();
    __shared__ uint32_t warp_sums[kScanThreads / 32];
    __shared__ uint32_t tile_vals[kScanTilePadded];
    const uint32_t n = min(ctr->n_band, a.cap_band);
    const uint32_t ntiles = (n + kScanTile - 1) / kScanTile;
    for (uint32_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        const uint64_t base = (uint64_t)tile * kScanTile;
#pragma unroll
        for (uint32_t k = 0; k < kScanItems; ++k) {
            const uint32_t j = k * kScanThreads + threadIdx.x;
            const uint64_t i = base + j;
            tile_vals[scan_slot(j)] = i < n ? mc_pair(__ldg(a.mc + i)) : 0u;
        }
        __syncthreads();
        // each thread owns kScanItems consecutive positions
        uint32_t local[kScanItems];
        uint32_t s = 0;
#pragma unroll
        for (uint32_t k = 0; k < kScanItems; ++k) {
            local[k] = tile_vals[scan_slot(threadIdx.x * kScanItems + k)];
            s += local[k];
        }
        const uint32_t incl = block_inclusive_scan(s, warp_sums);
        uint32_t run = incl - s;  // packed exclusive prefix within the tile
        uint32_t pv = 0, pq = 0;
        if (kSums) {
            for (uint32_t i = threadIdx.x; i < tile; i += kScanThreads) {
                const uint32_t both = __ldg(tile_sums + i);
                pv += both & 0xFFFFu;
                pq += both >> 16;
            }
            pv = block_sum(pv, warp_sums);
            pq = block_sum(pq, warp_sums);
            if (tile == ntiles - 1 && threadIdx.x == kScanThreads - 1)
                mc_counts(a, ctr, pv + (incl & 0xFFFFu), pq + (incl >> 16));
        } else {
            pv = tile_sums[tile];
            pq = tile_sums[ntiles_max + tile];
        }
#pragma unroll
        for (uint32_t k = 0; k < kScanItems; ++k) {
            const uint64_t t = base + threadIdx.x * kScanItems + k;
            if (local[k] != 0u && t < n) {
                const uint32_t q = pq + (run >> 16);
                if (q < a.cap_valid) a.valid[q] = (uint32_t)t;
            }
            tile_vals[scan_slot(threadIdx.x * kScanItems + k)] = pv + (run & 0xFFFFu);
            run += local[k];
        }
        __syncthreads();
#pragma unroll
        for (uint32_t k = 0; k < kScanItems; ++k) {
            const uint32_t j = k * kScanThreads + threadIdx.x;
            const uint64_t i = base + j;
            if (i < n) a.vofs[i] = tile_vals[scan_slot(j)];
        }
        __syncthreads();
    }
}

__device__ __forceinline__ void normalize_fast(float n[3])
{
    const float inv = rsqrtf(fmaf(n[0], n[0], fmaf(n[1], n[1], n[2] * n[2])));
    n[0] *= inv;
    n[1] *= inv;
    n[2] *= inv;
}

// fVector3::normalize (MathVector.cpp:5-15): scaled only when longer than 1e-7
__device__ __forceinline__ void normalize_guarded(float n[3])
{
    const float len = sqrtf(fmaf(n[0], n[0], fmaf(n[1], n[1], n[2] * n[2])));
    if (len > 1.0e-7f) {
        const float f = 1.0f / len;
        n[0] *= f;
        n[1] *= f;
        n[2] *= f;
    }
}

// generateTriangles (cu:383-463), or with host_mc the host marching cubes
// of Akinci12 (MarchingCubesCPU.cpp:3-72: no normal sign flip, guarded
// normalisation, epsilon test in double).
// The 32 grid positions a cube's corners and central-difference normals
// read: for each corner row (y, z in {0,1}) x = -1..2 (slots 0-15, the
// corners at x = 0, 1), and above/below each corner column y = -1, 2
// (slots 16-23) and z = -1, 2 (slots 24-31).  Each slot outside the cube
// serves one corner's normal, so that normal is written back over its three
// such slots once it is formed.
__device__ __forceinline__ int mc_corner_slot(int cx, int cy, int cz) { return (cz * 2 + cy) * 4 + cx + 1; }
__device__ __forceinline__ int mc_nx_slot(int cx, int cy, int cz) { return (cz * 2 + cy) * 4 + (cx ? 3 : 0); }
__device__ __forceinline__ int mc_ny_slot(int cx, int cy, int cz) { return 16 + (cz * 2 + cx) * 2 + cy; }
__device__ __forceinline__ int mc_nz_slot(int cx, int cy, int cz) { return 24 + (cy * 2 + cx) * 2 + cz; }

__global__ void __launch_bounds__(kThreads) k_mc_generate(McArgs a, const Counters* ctr)
{
    after_launch();
    // per thread: the cube's 32 field values, then corner values and normals
    // ([slot][thread]), so that the cut edges can index them without
    // spilling registers
    __shared__ float s_f[32 * kThreads];
    const uint32_t nq = min(ctr->n_valid, a.cap_valid);
    const uint32_t ntot = ctr->n_mesh_verts;
    if (ntot > a.cap_mesh) return;
    const float sgn = a.host_mc ? 1.0f : (a.iso < 0.0f ? -1.0f : 1.0f);
    const int tid = threadIdx.x, lane = tid & 31, wbase = tid & ~31;
    float* f = s_f + tid;
    auto S = [&](int slot) -> float& { return f[slot * kThreads]; };
    // a warp takes 32 consecutive valid cubes: their vertices are one
    // contiguous run of the output, which the warp then writes with
    // consecutive lanes on consecutive vertices (coalesced stores)
    for (uint32_t q0 = blockIdx.x * blockDim.x + (uint32_t)wbase; q0 < nq; q0 += gridDim.x * blockDim.x) {
        const uint32_t q = q0 + (uint32_t)lane;
        uint32_t cs = 0, nv = 0, base = 0;
        int X = 0, Y = 0, Z = 0;
        if (q < nq) {
            const uint32_t t = a.valid[q];
            const uint32_t info = a.mc[t];
            cs = info >> 8;
            nv = info & 0xFFu;
            base = a.vofs[t];
            uint32_t x, y, z;
            unlin3(a.sv[t], a.sc, x, y, z);
            X = (int)x;
            Y = (int)y;
            Z = (int)z;
            // the 32 positions as 12 rows of x-neighbours (one by one, each
            // with its bitset word, prefix and value in turn, the lookups took
            // longest: 188 -> 119 us for 2.5M triangles, 97 -> 54 us for 0.93M)
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                const int cy = r & 1, cz = r >> 1;
                float row[4], below[2], above[2];
                field_row<4>(a, X - 1, Y + cy, Z + cz, row);
                // (cy as the row's x-independent place: rows at y = -1, 2 for z = cz,
                // rows at z = -1, 2 for y = cz)
                if (cy == 0) {
                    field_row<2>(a, X, Y - 1, Z + cz, below);
                    field_row<2>(a, X, Y + 2, Z + cz, above);
                } else {
                    field_row<2>(a, X, Y + cz, Z - 1, below);
                    field_row<2>(a, X, Y + cz, Z + 2, above);
                }
#pragma unroll
                for (int xi = 0; xi < 4; ++xi) S(r * 4 + xi) = row[xi];
                const int base = cy == 0 ? 16 : 24;
#pragma unroll
                for (int cx = 0; cx < 2; ++cx) {  // slots of (cx, cz) or (cx, cy = cz)
                    S(base + (cz * 2 + cx) * 2) = below[cx];
                    S(base + (cz * 2 + cx) * 2 + 1) = above[cx];
                }
            }
            // corner normals, f(p - e) - f(p + e) per axis, over their slots
            for (int i = 0; i < 8; ++i) {
                const int cx = mc::cornerDx(i), cy = mc::cornerDy(i), cz = mc::cornerDz(i);
                float cn[3] = {cx ? S(mc_corner_slot(0, cy, cz)) - S(mc_nx_slot(1, cy, cz))
                                  : S(mc_nx_slot(0, cy, cz)) - S(mc_corner_slot(1, cy, cz)),
                               cy ? S(mc_corner_slot(cx, 0, cz)) - S(mc_ny_slot(cx, 1, cz))
                                  : S(mc_ny_slot(cx, 0, cz)) - S(mc_corner_slot(cx, 1, cz)),
                               cz ? S(mc_corner_slot(cx, cy, 0)) - S(mc_nz_slot(cx, cy, 1))
                                  : S(mc_nz_slot(cx, cy, 0)) - S(mc_corner_slot(cx, cy, 1))};
                if (a.host_mc) normalize_guarded(cn);
                else normalize_fast(cn);
                S(mc_nx_slot(cx, cy, cz)) = cn[0];
                S(mc_ny_slot(cx, cy, cz)) = cn[1];
                S(mc_nz_slot(cx, cy, cz)) = cn[2];
            }
        }
        // the warp's run: the exclusive prefix of its cubes' vertex counts
        uint32_t ex = nv;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, ex, o);
            if (lane >= o) ex += y;
        }
        const uint32_t total = __shfl_sync(0xffffffffu, ex, 31);
        ex -= nv;
        const uint32_t run0 = __shfl_sync(0xffffffffu, base, 0);  // lane 0 holds a cube (q0 < nq)
        __syncwarp();
        for (uint32_t jb = 0; jb < total; jb += 32) {
            const uint32_t j = jb + (uint32_t)lane;
            // the cube of vertex j: the last lane whose run starts at or before j
            int c = 0;
#pragma unroll
            for (int step = 16; step > 0; step >>= 1) {
                const uint32_t e = __shfl_sync(0xffffffffu, ex, (c + step) & 31);
                if (c + step < 32 && e <= j) c += step;
            }
            const uint32_t k = j - __shfl_sync(0xffffffffu, ex, c);
            const uint32_t ccs = __shfl_sync(0xffffffffu, cs, c);
            const int cX = __shfl_sync(0xffffffffu, X, c), cY = __shfl_sync(0xffffffffu, Y, c),
                      cZ = __shfl_sync(0xffffffffu, Z, c);
            if (j >= total) continue;
            const float* g = s_f + wbase + c;  // that cube's slots
            auto G = [&](int slot) { return g[slot * kThreads]; };
            const int e = (int)((c_mc.tri[ccs] >> (4u * k)) & 0xFu);
            const int i0 = mc::edgeA(e), i1 = mc::edgeB(e);
            const int a0x = mc::cornerDx(i0), a0y = mc::cornerDy(i0), a0z = mc::cornerDz(i0);
            const int a1x = mc::cornerDx(i1), a1y = mc::cornerDy(i1), a1z = mc::cornerDz(i1);
            const float v0 = G(mc_corner_slot(a0x, a0y, a0z)), v1 = G(mc_corner_slot(a1x, a1y, a1z));
            const float d = v1 - v0;
            const float fr = (d > -1.0e-7f && d < 1.0e-7f) ? 0.5f : (a.iso - v0) / d;
            const int c0[3] = {cX + a0x, cY + a0y, cZ + a0z};
            const int c1[3] = {cX + a1x, cY + a1y, cZ + a1z};
            float ip[3], in[3];
#pragma unroll
            for (int kk = 0; kk < 3; ++kk) {
                const float p0 = vpos1(c0[kk], a.sc.min[kk], a.sc.cs), p1 = vpos1(c1[kk], a.sc.min[kk], a.sc.cs);
                ip[kk] = fmaf(fr, p1 - p0, p0);
                const float n0 = G(kk == 0 ? mc_nx_slot(a0x, a0y, a0z) : kk == 1 ? mc_ny_slot(a0x, a0y, a0z)
                                                                       : mc_nz_slot(a0x, a0y, a0z));
                const float n1 = G(kk == 0 ? mc_nx_slot(a1x, a1y, a1z) : kk == 1 ? mc_ny_slot(a1x, a1y, a1z)
                                                                       : mc_nz_slot(a1x, a1y, a1z));
                in[kk] = fmaf(fr, n1 - n0, n0);
            }
            if (a.host_mc) normalize_guarded(in);
            else normalize_fast(in);
            const uint64_t o = 3ull * (run0 + j);
            a.out_pos[o] = ip[0];
            a.out_pos[o + 1] = ip[1];
            a.out_pos[o + 2] = ip[2];
            a.out_nrm[o] = sgn * in[0];
            a.out_nrm[o + 1] = sgn * in[1];
            a.out_nrm[o + 2] = sgn * in[2];
            if (a.out_key) {
                // the edge's lower end point and its axis (the one coordinate
                // in which the two corners differ)
                const uint32_t lx = (uint32_t)min(c0[0], c1[0]), ly = (uint32_t)min(c0[1], c1[1]),
                               lz = (uint32_t)min(c0[2], c1[2]);
                const uint32_t axis = c0[0] != c1[0] ? 0u : (c0[1] != c1[1] ? 1u : 2u);
                const uint64_t lin = (uint64_t)lx + (uint64_t)a.sc.res[0] * ((uint64_t)ly + (uint64_t)a.sc.res[1] * lz);
                a.out_key[run0 + j] = 3ull * lin + axis;
            }
        }
        __syncwarp();  // the next cubes overwrite the slots
    }
}

__global__ void k_particle_flags(const uint32_t* __restrict__ skeys, const uint8_t* __restrict__ surf,
                                 const uint8_t* __restrict__ psurf, uint32_t n, uint32_t* __restrict__ out)
{
    after_launch();
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n) return;
    out[t] = psurf ? psurf[t] : surf[skeys[t]];
}

}  // namespace

// ------------------------------------------------------------ launchers

// Smallest float x >= 0 whose correctly rounded square root is >= R
// (strict = false) or > R (strict = true): for d2 >= 0,
//   sqrt_rn(d2) <  R  <=>  d2 < threshold(R, false)
//   sqrt_rn(d2) <= R  <=>  d2 < threshold(R, true)
// so the kernels test distances without a square root and take the root
// only where the weight needs it.  sqrtf on the host and __fsqrt_rn on the
// device are both the IEEE correctly rounded square root.
float sqrt_threshold(float R, bool strict)
{
    auto ok = [&](float x) { return strict ? std::sqrt(x) > R : std::sqrt(x) >= R; };
    float x = R * R;
    if (!(x > 0.0f) || !std::isfinite(x)) return x;
    while (x > 0.0f && ok(std::nextafterf(x, 0.0f))) x = std::nextafterf(x, 0.0f);
    while (!ok(x)) x = std::nextafterf(x, INFINITY);
    return x;
}

void launch_hash(const KernelCtx& c, const float* xyz, uint32_t n, const Grid& sp, uint32_t* keys,
                 uint32_t* vals, Counters* ctr)
{
    if (!n) return;
    launch_after(k_hash, blocks_for(n, bs(c)), bs(c), 0, c.stream, xyz, n, sp, keys, vals, ctr);
    ++g_launches;
}

void launch_ranges_gather(const KernelCtx& c, const uint32_t* skeys, const uint32_t* perm, uint32_t n,
                          const float* xyz, const float* dens, float4* sorted, uint2* ranges, uint8_t* occ)
{
    if (!n) return;
    launch_after(k_ranges_gather, blocks_for(n, bs(c)), bs(c), 0, c.stream, skeys, perm, n, xyz, dens, sorted, ranges,
                 occ);
    ++g_launches;
}

void launch_density(const KernelCtx& c, float4* sorted, uint32_t n, const uint2* ranges, const Grid& sp, float h,
                    float mass, float* rho)
{
    if (n == 0) return;
    const int ext = std::max(1, (int)std::ceil((double)h * 1.0001 / sp.cs + 1e-4));
    const float h2 = h * h;
    const float sigma = 315.0f / (64.0f * 3.1415926535898f);
    const float scale = mass * sigma / (h * h * h);
    launch_after(k_density, blocks_for(n, kDensityThreads), kDensityThreads, 0, c.stream, sorted, n, ranges, sp, ext, h,
                 h2, 1.0f / h2, scale, rho);
    launch_after(k_set_density, blocks_for(n, bs(c)), bs(c), 0, c.stream, sorted, rho, n);
    g_launches += 2;
}

void launch_surface_cells(const KernelCtx& c, const Grid& sp, const uint8_t* occ, uint8_t* surf)
{
    const uint64_t C = (uint64_t)sp.res[0] * sp.res[1] * sp.res[2];
    launch_after(k_surface_cells, blocks_for(C, bs(c)), bs(c), 0, c.stream, sp, occ, surf);
    ++g_launches;
}

void launch_involved_cells(const KernelCtx& c, const Grid& sp, const uint8_t* occ, const uint8_t* surf,
                           uint8_t* invol)
{
    const uint64_t C = (uint64_t)sp.res[0] * sp.res[1] * sp.res[2];
    launch_after(k_involved_cells, blocks_for(C, bs(c)), bs(c), 0, c.stream, sp, occ, surf, invol);
    ++g_launches;
}

void launch_colorfield(const KernelCtx& c, const float4* sorted, uint32_t n, const uint2* ranges,
                       const uint32_t* skeys, const Grid& sp, float h, float h2, float mass, uint8_t* psurf)
{
    if (!n) return;
    // -45 / (pi h^4) exactly as the reference evaluates it in double
    const double k = -45.0 / (3.1415926535 * (double)h2 * (double)h2);
    // the FP32 form of the gradient needs |k| x^2 (x in (0, 1]) to stay a
    // normal float: |k| within [1e-20, 1e30]; else the double expression
    const double K = -k;
    float khi = 0.f, klo = 0.f;
    if (K >= 1e-20 && K <= 1e30) {
        khi = (float)K;
        klo = (float)(K - (double)khi);
    }
    const bool fast = fast_radius(h);
    // one lane per particle / four (ms): 4k particles 0.17 / 0.06, 20k 0.28 /
    // 0.11, 60k 0.29 / 0.18, 100k 0.20-0.33 / 0.20-0.34, 262k 0.40 / 0.46, 1M
    // 1.29 / 1.75
    if (n < 98304u) {
        const auto kernel = fast ? k_colorfield_quads<true> : k_colorfield_quads<false>;
        launch_after(kernel, blocks_for(4ull * n, kColorThreads), kColorThreads, 0, c.stream, sorted, n, ranges, sp, h,
                     1.0f / h, sqrt_threshold(h, false), tiny_d2(h), k, khi, klo, mass, psurf);
    } else {
        const auto kernel = fast ? k_colorfield<true> : k_colorfield<false>;
        launch_after(kernel, blocks_for(n, bs(c)), bs(c), 0, c.stream, sorted, n, ranges, sp, h, 1.0f / h,
                     sqrt_threshold(h, false), tiny_d2(h), k, khi, klo, mass, psurf);
    }
    ++g_launches;
}

void launch_band_stamp(const KernelCtx& c, const float4* sorted, const uint32_t* skeys, const uint8_t* surf,
                       const uint8_t* psurf, uint32_t n, const Grid& sp, const Grid& sc, float thr, uint32_t* bits,
                       Counters* ctr)
{
    if (!n) return;
    const float thr2 = sqrt_threshold(thr, true);
    auto launch = [&](auto kernel, uint32_t lanes) {
        launch_after(kernel, blocks_for((uint64_t)n * lanes, bs(c)), bs(c), 0, c.stream, sorted, skeys, surf, psurf, n,
                     sc, thr2, bits, ctr);
    };
    const bool check = !psurf || sc.cs * 4.0f >= sp.cs;  // (at most 4 grid vertices per cell)
    if (n < 65536u) launch(check ? k_band_stamp<8, true> : k_band_stamp<8, false>, 8);
    else launch(check ? k_band_stamp<2, true> : k_band_stamp<2, false>, 2);
    ++g_launches;
}

void launch_band_list(const KernelCtx& c, const uint32_t* bits, const uint32_t* prefix, uint32_t nwords,
                      uint32_t* sv, uint32_t cap, const GroupMark& gm, Counters* ctr)
{
    // A warp per word while the words make no more than a few rounds of warps;
    // most words of a large grid are empty.  Measured with the scan, a lane per
    // word / a warp per word (us): coarse grids of 68 words 25 / 12, 2.5k 22 / 12,
    // 19k 51 / 31; fine grids of 24k and of 130k 20.5 / 20.5, 754k 33 / 80.
    if (nwords <= 1u << 17)
        launch_after(k_band_list_words, persistent_blocks(c, 32ull * nwords, 8), bs(c), 0, c.stream, bits, prefix,
                     nwords, sv, cap, gm, ctr);
    else
        launch_after(k_band_list, persistent_blocks(c, nwords, 16), bs(c), 0, c.stream, bits, prefix, nwords, sv, cap,
                     gm, ctr);
    ++g_launches;
}


void launch_smooth(const KernelCtx& c, const float4* sorted, uint32_t n, const uint2* ranges, const Grid& sp,
                   float R, float lambda, float mass, float4* mean, float4* mean32, float4* smoothed)
{
    if (!n) return;
    // (1.0 - lambda) is evaluated in double and rounded (cu:656)
    const float oml = (float)(1.0 - (double)lambda);
    // lanes may walk the union of their windows when the cull radius stays
    // below two cells (see k_smooth); it spans up to one cell more per axis than
    // the windows of particles of one cell
    const bool coop_ok = (R * 1.0001f + 1e-4f * sp.cs) < 2.0f * sp.cs * 0.9999f;
    const int max_span = coop_ok ? 2 * (int)std::ceil(std::max(1.0f, R * 1.0001f / sp.cs)) + 1 : -1;
    // Four lanes per particle while one would leave the SMs with two or three
    // warps per scheduler; more lanes cost more instructions per particle once
    // the GPU is full.  Measured, one lane / four (ms): R = 0.8 cells: 20k
    // particles 0.16 / 0.08, 32k 0.12 / 0.09, 64k 0.11-0.23 / 0.14-0.18, 120k
    // 0.28 / 0.31; R = 1.54 cells: 20k 0.62 / 0.25, 40k 0.80 / 0.46, 100k 0.87 /
    // 1.03.
    const bool wide = max_span > 3, fast = fast_radius(R);
    if (n < (wide ? 81920u : 49152u)) {
        const auto kernel = fast ? k_smooth_quads<true> : k_smooth_quads<false>;
        launch_after(kernel, blocks_for(n, 32), kQuadThreads, 0, c.stream, sorted, n, ranges, sp, R, 1.0f / R,
                     sqrt_threshold(R, false), tiny_d2(R), max_span, oml, lambda, mass, mean, mean32, smoothed);
    } else {
        const auto kernel = wide ? (fast ? k_smooth<true, true> : k_smooth<false, true>)
                                 : (fast ? k_smooth<true, false> : k_smooth<false, false>);
        launch_after(kernel, blocks_for(n, bs(c)), bs(c), 0, c.stream, sorted, n, ranges, sp, R, 1.0f / R,
                     sqrt_threshold(R, false), tiny_d2(R), max_span, oml, lambda, mass, mean, mean32, smoothed);
    }
    ++g_launches;
}

void launch_cov(const KernelCtx& c, const CovArgs& a0, Counters* ctr)
{
    if (!a0.n) return;
    CovArgs a = a0;
    a.R_lt2 = sqrt_threshold(a.R, false);
    a.R_rcp = 1.0f / a.R;
    a.R_le2 = sqrt_threshold(a.R, true);
    a.coop_ok = (a.R + a.R * 1.0001f + 1e-4f * a.sp.cs) < 2.0f * a.sp.cs * 0.9999f ? 1 : 0;
    a.tiny = tiny_d2(a.R);
    const bool fast = fast_radius(a.R);
    const bool sets = a.coop_ok == 0;
    auto launch = [&](auto kernel, uint32_t lanes) {
        launch_after(kernel, blocks_for((uint64_t)a.n * lanes, kCovThreads), kCovThreads, 0, c.stream, a, ctr);
    };
    if (sets && a.n < kCovWideBelow) {
        launch(fast ? k_cov<16, true, true> : k_cov<16, false, true>, 16);
    } else if (a.n < kCovSplitBelow) {
        if (sets) launch(fast ? k_cov<4, true, true> : k_cov<4, false, true>, 4);
        else launch(fast ? k_cov<4, true, false> : k_cov<4, false, false>, 4);
    } else {
        if (sets) launch(fast ? k_cov<1, true, true> : k_cov<1, false, true>, 1);
        else launch(fast ? k_cov<1, true, false> : k_cov<1, false, false>, 1);
    }
    ++g_launches;
}

void launch_mc_classify(const KernelCtx& c, const McArgs& a, Counters* ctr, uint32_t* scratch)
{
    launch_after(k_mc_classify, persistent_blocks(c, a.cap_band, 16), bs(c), 0, c.stream, a, ctr, scratch);
    ++g_launches;
}

uint32_t mc_tiles(uint32_t cap_band) { return (cap_band + kScanTile - 1) / kScanTile; }

size_t mc_offsets_scratch_words(uint32_t cap_band) { return 2 * (size_t)mc_tiles(cap_band) + 2; }

void launch_mc_offsets(const KernelCtx& c, const McArgs& a, Counters* ctr, uint32_t* scratch)
{
    const uint32_t ntiles_max = mc_tiles(a.cap_band);
    const uint32_t g = std::max<uint32_t>(1, std::min<uint32_t>(ntiles_max, 65535));
    if (ntiles_max <= kSumTiles) {
        launch_after(k_mc_tile_scan<true>, g, kScanThreads, 0, c.stream, a, ctr, scratch, ntiles_max);
        ++g_launches;
        return;
    }
    launch_after(k_mc_scan_tile_sums, 1, kScanThreads, 0, c.stream, a, ctr, scratch, ntiles_max);
    launch_after(k_mc_tile_scan<false>, g, kScanThreads, 0, c.stream, a, ctr, scratch, ntiles_max);
    g_launches += 2;
}

void launch_mc_generate(const KernelCtx& c, const McArgs& a, Counters* ctr)
{
    launch_after(k_mc_generate, persistent_blocks(c, a.cap_valid, 16), bs(c), 0, c.stream, a, ctr);
    ++g_launches;
}

void launch_particle_flags(const KernelCtx& c, const uint32_t* skeys, const uint8_t* surf, const uint8_t* psurf,
                           uint32_t n, uint32_t* out)
{
    if (!n) return;
    launch_after(k_particle_flags, blocks_for(n, bs(c)), bs(c), 0, c.stream, skeys, surf, psurf, n, out);
    ++g_launches;
}

}  // namespace fsr
