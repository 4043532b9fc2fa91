// The smoothing by one lane and by four lanes per particle, over the same
// particles: equal bit for bit for radii below a cell.
#include "warp_emul.h"

#include "kernels.cu"

#include <cstdio>
#include <random>

int main()
{
    using namespace fsr;
    Grid sp{};
    sp.cs = 0.125f;
    sp.res[0] = 12;
    sp.res[1] = sp.res[2] = 6;
    const float R = 0.8f * sp.cs;
    const uint32_t cells = sp.res[0] * sp.res[1] * sp.res[2];
    std::mt19937 rng(15);
    std::vector<std::pair<uint32_t, float4>> all;
    // rows of many particles, so that whole chunks of 32 lie beyond R; near 0 along
    // x, where a mean shows its last bits
    sp.min[0] = -0.75f;
    for (int i = 0; i < 12000; ++i) {
        float4 p;
        p.x = sp.min[0] + 1.5f * (rng() >> 8) * 0x1p-24f;
        p.y = 0.75f * (rng() >> 8) * 0x1p-24f;
        p.z = 0.75f * (rng() >> 8) * 0x1p-24f;
        p.w = 1000.f;
        const uint32_t key = lin3((uint32_t)cell1(p.x, sp.min[0], sp.cs), (uint32_t)cell1(p.y, 0.f, sp.cs),
                                  (uint32_t)cell1(p.z, 0.f, sp.cs), sp);
        all.emplace_back(key, p);
    }
    std::stable_sort(all.begin(), all.end(), [](auto& a, auto& b) { return a.first < b.first; });
    const uint32_t n = (uint32_t)all.size();
    std::vector<float4> sorted(n), mean[2], mean32[2], smoothed[2];
    std::vector<uint2> ranges(cells, make_uint2(kEmpty, kEmpty));
    for (uint32_t i = 0; i < n; ++i) {
        sorted[i] = all[i].second;
        uint2& r = ranges[all[i].first];
        if (r.x == kEmpty) r.x = i;
        r.y = i + 1;
    }
    cudaLaunchConfig_t cfg{};
    for (int quads = 0; quads < 2; ++quads) {
        mean[quads].resize(n);
        mean32[quads].resize(n);
        smoothed[quads].resize(n);
        cfg.blockDim = dim3(quads ? kQuadThreads : kThreads);
        cfg.gridDim = dim3(quads ? (n + 31) / 32 : (n + kThreads - 1) / kThreads);
        const auto kernel = quads ? k_smooth_quads<true> : k_smooth<true, false>;
        emu::launch(&cfg, kernel, sorted.data(), n, ranges.data(), sp, R, 1.0f / R, sqrt_threshold(R, false),
                    tiny_d2(R), 3, 0.1f, 0.9f, 1.0f, mean[quads].data(), mean32[quads].data(), smoothed[quads].data());
    }
    uint32_t off[3] = {0, 0, 0};
    for (uint32_t i = 0; i < n; ++i) {
        off[0] += std::memcmp(&mean[0][i], &mean[1][i], 16) != 0;
        off[1] += std::memcmp(&mean32[0][i], &mean32[1][i], 16) != 0;
        off[2] += std::memcmp(&smoothed[0][i], &smoothed[1][i], 16) != 0;
    }
    std::printf("differing means %u, FP32 means %u, smoothed positions %u\n", off[0], off[1], off[2]);
    return 0;
}
