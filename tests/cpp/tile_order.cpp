// The tiles of a pass, laid out by two warps whose lanes reach their atomics in
// opposite orders (the two halves of a split work item of the anisotropic field).
#include "warp_emul.h"

#include "field_aniso.cu"

#include <cstdio>

namespace fsr {
thread_local uint64_t g_launches = 0;
namespace {
unsigned char smem[1];
uint32_t g_loc[256], g_rank[256], g_hist[256];
uint16_t g_order[256];
float4 g_box[16];

__global__ void k_layout(uint32_t nv, Grid sc, bool in_place)
{
    const int lo[3] = {0, 0, 0};
    float4 pl, ph;
    if (in_place) pass_layout<true>(g_loc, g_rank, lo, sc, nullptr, g_hist, g_box, nv, threadIdx.x & 31, pl, ph);
    else pass_layout<false>(g_loc, g_rank, lo, sc, g_order, g_hist, g_box, nv, threadIdx.x & 31, pl, ph);
}
}  // namespace
}  // namespace fsr

int main()
{
    using namespace fsr;
    Grid sc{};
    sc.cs = 0.1f;
    sc.res[0] = sc.res[1] = sc.res[2] = 64;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(1);
    cfg.blockDim = dim3(32);
    uint32_t seed = 1;
    for (int side : {3, 5, 10, 16})
        for (uint32_t nv : {1u, 32u, 33u, 64u, 65u, 200u, 255u, 256u})
            for (int in_place = 0; in_place < 2; ++in_place) {
                uint32_t loc[256], kept[2][256];
                for (uint32_t q = 0; q < nv; ++q) {
                    seed = seed * 1664525u + 1013904223u;
                    const uint32_t r = seed >> 8;
                    loc[q] = vert_loc(r % side, r / side % side, r / side / side % side);
                }
                for (int d = 0; d < 2; ++d) {
                    emu::descending = d != 0;
                    std::copy(loc, loc + nv, g_loc);
                    for (uint32_t q = 0; q < nv; ++q) {
                        g_rank[q] = q;
                        g_order[q] = 0xffff;
                    }
                    emu::launch(&cfg, k_layout, nv, sc, in_place != 0);
                    for (uint32_t q = 0; q < nv; ++q) kept[d][q] = in_place ? g_rank[q] : g_order[q];
                    std::vector<uint32_t> all(kept[d], kept[d] + nv);
                    std::sort(all.begin(), all.end());
                    for (uint32_t q = 0; q < nv; ++q)
                        if (all[q] != q) return std::printf("a vertex is missing: side %d nv %u\n", side, nv), 0;
                }
                // (in place: one warp has the whole pass, any order will do)
                for (uint32_t q = 0; q < nv && !in_place; ++q)
                    if (kept[0][q] != kept[1][q])
                        return std::printf("orders differ: side %d nv %u at %u\n", side, nv, q), 0;
            }
    std::printf("same\n");
    return 0;
}
