// Spatial hashing as a counting sort by cell (ReconstructorGPU.cpp:292-313:
// calcParticlesHashKernel, thrust sort_by_key and findCellRangeKernel in the
// reference), for grids whose cells are not many more than the particles:
//   1. each particle's cell, and its arrival number there (one atomic per run
//      of equal cells in a warp);
//   2. an exclusive scan of the cells' counts: the cells' first places;
//   3. particle numbers to first place + arrival number: grouped by cell, in
//      no particular order inside one;
//   4. each particle's place inside its cell is the number of smaller particle
//      numbers there (the sort is stable), which also gathers the particles.
// Five launches with a scan in one block, six or (beyond kSumTiles tiles) seven
// with the tiled one, one fewer for at most kBigCell particles, instead of the
// radix sort's two or three passes of three to five; the radix sort stays
// for sparse grids, whose scan would cost more than its passes.  Cells of more
// than kBigCell particles are left to a block each, which sorts their particle
// numbers by radix (the count in step 4 is quadratic).
// Measured (with the frame's memsets, ms): 1.5k particles 0.049 -> 0.034, 32k
// 0.065 -> 0.047, 300k 0.124 -> 0.057, 1M 0.137 -> 0.075, 8M 0.42 -> 0.34.
#include <algorithm>

#include "fsr_internal.h"
#include "kernels.h"
#include "primitives.h"

namespace fsr {
namespace {

constexpr uint32_t kBigCell = 1024;
constexpr uint32_t kDenseParticles = 16;
constexpr uint32_t kCrowdedParticles = 7 * 256;  // four times the usual 64 a cell (h = 4 spacings)

__global__ void k_hash_count(const float* __restrict__ xyz, uint32_t n, Grid sp, uint32_t* __restrict__ keys,
                             uint32_t* __restrict__ arrival, uint32_t* __restrict__ count, Counters* ctr)
{
    after_launch();
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    const int lane = threadIdx.x & 31;
    const bool there = i < n;
    uint32_t key = kEmpty;  // (no cell has this number)
    if (there) {
        const float p[3] = {xyz[3ull * i], xyz[3ull * i + 1], xyz[3ull * i + 2]};
        bool ok;
        key = cell_key(p, sp, ok);
        keys[i] = key;
        if (!ok) atomicAdd(&ctr->out_of_grid, 1u);
    }
    const uint32_t peers = __match_any_sync(0xffffffffu, key);
    const int lead = __ffs((int)peers) - 1;
    uint32_t base = 0;
    if (there && lane == lead) base = atomicAdd(count + key, (uint32_t)__popc(peers));
    base = __shfl_sync(0xffffffffu, base, lead);
    if (there) arrival[i] = base + (uint32_t)__popc(peers & ((1u << lane) - 1u));
}

// Step 3, and per cell what the frame starts from: its range and occupancy, and
// zeros in the cell-sized arrays of later stages (a memset each before).
// gflag: kDenseGroup for the window groups whose cell and its six neighbours hold
// enough particles for their field to be a long work item (an isolated
// particle's groups: one or two), which k_band_list lists first; kCrowdedGroup
// for those whose adjoint several warps share (k_field_iso_backward).
__global__ void k_group(const uint32_t* __restrict__ keys, const uint32_t* __restrict__ arrival,
                        const uint32_t* __restrict__ first, uint32_t n, Grid sp, uint32_t cells, uint32_t groups,
                        uint32_t* __restrict__ grouped, uint2* __restrict__ ranges, uint8_t* __restrict__ occ,
                        float* __restrict__ cell_rmax, uint32_t* __restrict__ gflag, uint32_t* __restrict__ big,
                        Counters* ctr)
{
    after_launch();
    const uint32_t stride = gridDim.x * blockDim.x, start = blockIdx.x * blockDim.x + threadIdx.x;
    for (uint32_t i = start; i < n; i = next_of(i, stride, n)) grouped[__ldg(first + keys[i]) + arrival[i]] = i;
    const uint32_t kx = sp.res[0] + 1, ky = sp.res[1] + 1;
    for (uint32_t c = start; c < groups; c = next_of(c, stride, groups)) {
        // (groups beyond the last cell of an axis count as that cell)
        const uint32_t gz = c / (kx * ky), gy = (c - gz * kx * ky) / kx, gx = c - (gz * ky + gy) * kx;
        const uint32_t x1 = sp.res[0] - 1, y1 = sp.res[1] - 1, z1 = sp.res[2] - 1;
        const uint32_t x = min(gx, x1), y = min(gy, y1), z = min(gz, z1);
        const uint32_t row = lin3(0, y, z, sp);
        auto held = [&](uint32_t a, uint32_t b) { return __ldg(first + b + 1) - __ldg(first + a); };
        uint32_t sum = held(row + (x ? x - 1 : 0u), row + min(x + 1, x1));  // x-neighbours are one run
        auto one = [&](uint32_t yy, uint32_t zz) { const uint32_t k = lin3(x, yy, zz, sp); return held(k, k); };
        sum += one(y ? y - 1 : 0u, z) + one(min(y + 1, y1), z) + one(y, z ? z - 1 : 0u) + one(y, min(z + 1, z1));
        gflag[c] = (sum >= kDenseParticles ? kDenseGroup : 0u) | (sum >= kCrowdedParticles ? kCrowdedGroup : 0u);
        if (c >= cells) continue;
        const uint32_t s = __ldg(first + c), e = __ldg(first + c + 1);
        ranges[c] = e > s ? make_uint2(s, e) : make_uint2(kEmpty, kEmpty);
        occ[c] = e > s ? 1 : 0;
        if (cell_rmax) cell_rmax[c] = 0.f;
        if (e - s > kBigCell) big[atomicAdd(&ctr->n_big_cells, 1u)] = c;
    }
}

struct CellSortOut {
    const float* xyz;
    const float* dens;
    float4* sorted;
    uint32_t* skeys;
    uint32_t* perm;
    __device__ __forceinline__ void put(uint32_t at, uint32_t key, uint32_t i) const
    {
        skeys[at] = key;
        perm[at] = i;
        // without densities (computed later by k_density) w is left at 0
        sorted[at] = make_float4(xyz[3ull * i], xyz[3ull * i + 1], xyz[3ull * i + 2], dens ? dens[i] : 0.0f);
    }
};

__global__ void k_cell_rank(const uint32_t* __restrict__ keys, const uint32_t* __restrict__ first,
                            const uint32_t* __restrict__ grouped, uint32_t n, CellSortOut out)
{
    after_launch();
    const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    const uint32_t i = grouped[k];
    const uint32_t key = __ldg(keys + i);
    const uint32_t s = __ldg(first + key), e = __ldg(first + key + 1);
    if (e - s > kBigCell) return;  // k_big_cells
    uint32_t r = 0;
    uint32_t j = s;
    for (; j + 4 <= e; j += 4) {
        const uint32_t a = __ldg(grouped + j), b = __ldg(grouped + j + 1), c = __ldg(grouped + j + 2),
                       d = __ldg(grouped + j + 3);
        r += (a < i ? 1u : 0u) + (b < i ? 1u : 0u) + (c < i ? 1u : 0u) + (d < i ? 1u : 0u);
    }
    for (; j < e; ++j) r += __ldg(grouped + j) < i ? 1u : 0u;
    out.put(s + r, key, i);
}

// One block per big cell: its particle numbers sorted by 8-bit digits in
// global memory between `grouped` and out.perm (stable passes: ranks inside a
// warp by matching, across warps by a scan), then put in place.
constexpr uint32_t kBigThreads = 1024, kBigWarps = kBigThreads / 32;
__global__ void __launch_bounds__(kBigThreads) k_big_cells(const uint32_t* __restrict__ first, uint32_t* grouped,
                                                           uint32_t digits, CellSortOut out,
                                                           const uint32_t* __restrict__ big, const Counters* ctr)
{
    after_launch();
    __shared__ uint32_t whist[kBigWarps][256];
    __shared__ uint32_t base[256];
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    for (uint32_t c = blockIdx.x; c < ctr->n_big_cells; c += gridDim.x) {
        const uint32_t key = big[c], s = first[key], m = first[key + 1] - s;
        uint32_t* from = grouped + s;
        uint32_t* to = out.perm + s;
        for (uint32_t d = 0; d < digits; ++d) {
            const uint32_t shift = 8u * d;
            // digit counts, then their exclusive scan
            if (tid < 256u) base[tid] = 0u;
            __syncthreads();
            for (uint64_t j = tid; j < m; j += kBigThreads) atomicAdd(&base[(from[j] >> shift) & 255u], 1u);
            __syncthreads();
            if (warp == 0) {
                uint32_t run = 0;
                for (uint32_t b = 0; b < 256u; b += 32) {
                    const uint32_t v = base[b + lane];
                    uint32_t x = v;
#pragma unroll
                    for (int o = 1; o < 32; o <<= 1) {
                        const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
                        if (lane >= (uint32_t)o) x += y;
                    }
                    base[b + lane] = run + x - v;
                    run += __shfl_sync(0xffffffffu, x, 31);
                }
            }
            for (uint64_t b = 0; b < m; b += kBigThreads) {
                for (uint32_t k = tid; k < kBigWarps * 256u; k += kBigThreads) whist[k >> 8][k & 255u] = 0u;
                __syncthreads();
                const uint64_t j = b + tid;
                const bool ok = j < m;
                const uint32_t v = ok ? from[j] : 0u;
                const uint32_t digit = (v >> shift) & 255u;
                const uint32_t peers = __match_any_sync(0xffffffffu, ok ? digit : 256u);
                const uint32_t before = (uint32_t)__popc(peers & ((1u << lane) - 1u));
                if (ok && before == 0u) whist[warp][digit] = (uint32_t)__popc(peers);
                __syncthreads();
                if (tid < 256u) {
                    uint32_t run = base[tid];
                    for (uint32_t w = 0; w < kBigWarps; ++w) {
                        const uint32_t x = whist[w][tid];
                        whist[w][tid] = run;
                        run += x;
                    }
                    base[tid] = run;
                }
                __syncthreads();
                if (ok) to[whist[warp][digit] + before] = v;
                __syncthreads();
            }
            uint32_t* t = from;
            from = to;
            to = t;
        }
        // an odd number of passes leaves them in out.perm itself
        for (uint64_t j = tid; j < m; j += kBigThreads) out.put(s + (uint32_t)j, key, from[j]);
        __syncthreads();
    }
}

}  // namespace

// Grids of at most 8 cells per particle (and small ones): the scan of the
// counts (12 bytes a cell) stays below the radix passes (16 bytes a particle
// each); a 12-particle frame on 250k cells sorts its keys instead.
bool cell_sort_wanted(uint64_t cells, uint32_t n) { return n > 0 && cells <= 8ull * n + 16384ull; }

cudaError_t launch_cell_sort(const KernelCtx& c, const CellSort& a, Counters* ctr)
{
    const int threads = 256;
    const unsigned blocks = (unsigned)(((uint64_t)a.n + threads - 1) / threads);
    const uint32_t cells = a.sp.res[0] * a.sp.res[1] * a.sp.res[2];
    const uint32_t groups = (a.sp.res[0] + 1) * (a.sp.res[1] + 1) * (a.sp.res[2] + 1);
    cudaError_t e = cudaSuccess;
    launch_after(k_hash_count, blocks, threads, 0, c.stream, a.xyz, a.n, a.sp, a.keys, a.arrival, a.first, ctr);
    ++g_launches;
    // in place: first[cells] becomes the number of particles
    if ((e = scan_counts(a.first, cells + 1u, a.scan_tmp, c.stream)) != cudaSuccess) return e;
    const unsigned gblocks = (unsigned)std::min<uint64_t>(((uint64_t)std::max(a.n, groups) + threads - 1) / threads,
                                                          (uint64_t)std::max(1, c.num_sms) * 32);
    launch_after(k_group, gblocks, threads, 0, c.stream, a.keys, a.arrival, a.first, a.n, a.sp, cells, groups,
                 a.grouped, a.ranges, a.occ, a.cell_rmax, a.gflag, a.big, ctr);
    const CellSortOut out{a.xyz, a.dens, a.sorted, a.skeys, a.perm};
    launch_after(k_cell_rank, blocks, threads, 0, c.stream, a.keys, a.first, a.grouped, a.n, out);
    g_launches += 2;
    if (a.n > kBigCell) {
        const uint32_t most = a.n / kBigCell;
        launch_after(k_big_cells, std::min<uint32_t>(most, (uint32_t)std::max(1, c.num_sms)), kBigThreads, 0, c.stream,
                     a.first, a.grouped, (bits_for(a.n) + 7u) / 8u, out, a.big, ctr);
        ++g_launches;
    }
    return cudaGetLastError();
}

}  // namespace fsr
