// Kernels at counts above 2^31, in arrays of which only the touched pages exist.
//   stamp:    a surface particle above 2^31 stamps its band
//   group:    the grouping loop ends at 2^32 - 2 particles
//   blocks:   the counting sort's launches cover 2^32 - 2 particles
//   classify: the classification's loop ends at 2^32 - 2 band vertices
#include "warp_emul.h"

#include "kernels.cu"
#define kThreads kGroupThreads
#include "cell_sort.cu"

#include <sys/mman.h>

#include <cstdio>

template <class T>
static T* sparse(uint64_t n)
{
    void* p = mmap(nullptr, n * sizeof(T), PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS | MAP_NORESERVE, -1, 0);
    if (p == MAP_FAILED) {
        std::printf("no address space\n");
        std::exit(0);
    }
    return (T*)p;
}

namespace fsr {
cudaError_t scan_counts(uint32_t*, uint32_t, uint32_t*, cudaStream_t) { return cudaSuccess; }
uint32_t bits_for(uint64_t) { return 32; }

static uint32_t stamped(uint32_t n, uint32_t at, std::vector<uint32_t>& bits)
{
    Grid sp{}, sc{};
    sp.cs = 0.25f;
    sc.cs = 0.125f;
    for (int a = 0; a < 3; ++a) {
        sp.res[a] = 8;
        sc.res[a] = 16;
    }
    float4* sorted = sparse<float4>(n);
    uint32_t* keys = sparse<uint32_t>(n);
    uint8_t* flags = sparse<uint8_t>(n);
    sorted[at] = make_float4(1.03f, 0.97f, 1.11f, 1.f);
    flags[at] = 1;
    bits.assign(16 * 16 * 16 / 32 + 1, 0);
    Counters ctr{};
    KernelCtx c{};
    c.num_sms = 1;
    const unsigned last = (unsigned)((2ull * n + 255) / 256);
    emu::wanted_block = [=](unsigned b) { return b + 8 > last; };
    launch_band_stamp(c, sorted, keys, nullptr, flags, n, sp, sc, 0.3f, bits.data(), &ctr);
    return ctr.n_surface;
}
}  // namespace fsr

int main(int, char** argv)
{
    using namespace fsr;
    const std::string what = argv[1];
    cudaLaunchConfig_t cfg{};
    cfg.blockDim = dim3(256);
    if (what == "stamp") {
        std::vector<uint32_t> want, got;
        const uint32_t a = stamped(100000u, 100000u - 3u, want);
        const uint32_t b = stamped(0x80000000u + 301u, 0x80000000u + 5u, got);
        const bool some = std::any_of(want.begin(), want.end(), [](uint32_t w) { return w != 0; });
        std::printf(some && a == 1 && b == 1 && want == got ? "ok\n" : "not stamped\n");
    } else if (what == "group") {
        const uint32_t n = 0xFFFFFFFEu;
        Grid sp{};
        sp.cs = 1.f;
        sp.res[0] = sp.res[1] = sp.res[2] = 1;
        uint32_t *keys = sparse<uint32_t>(n), *arrival = sparse<uint32_t>(n), *grouped = sparse<uint32_t>(n);
        uint32_t first[2] = {0, 0};
        arrival[n - 1] = 1;
        Counters ctr{};
        cfg.gridDim = dim3(1u << 23);
        emu::wanted_block = [](unsigned b) { return b == (1u << 23) - 1; };
        emu::launch(&cfg, k_group, keys, arrival, first, n, sp, 1u, 8u, grouped, nullptr, nullptr, nullptr, nullptr,
                    nullptr, &ctr);
        std::printf(grouped[1] == n - 1 ? "ok\n" : "last particle not grouped\n");
    } else if (what == "blocks") {
        CellSort a{};
        a.n = 0xFFFFFFFEu;
        a.sp.cs = 1.f;
        a.sp.res[0] = a.sp.res[1] = a.sp.res[2] = 1;
        KernelCtx c{};
        c.num_sms = 1;
        std::vector<uint64_t> grids;  // of the launches, in blocks
        emu::wanted_block = [&](unsigned b) {
            if (b == 0) grids.push_back(0);
            ++grids.back();
            return false;
        };
        launch_cell_sort(c, a, nullptr);
        const bool whole = grids.size() == 4 && grids[0] == 1u << 24 && grids[2] == 1u << 24;
        std::printf(whole ? "ok\n" : "too few blocks\n");
    } else {
        const uint32_t n = 0xFFFFFFFEu;
        McArgs a{};
        for (int k = 0; k < 3; ++k) a.sc.res[k] = 4;
        const std::vector<uint32_t> none(8, 0);
        a.band.bits = a.band.prefix = none.data();
        a.sv = sparse<uint32_t>(n);
        a.mc = sparse<uint32_t>(n);
        a.cap_band = n;
        uint32_t* sums = sparse<uint32_t>(1u << 20);
        Counters ctr{};
        ctr.n_band = n;
        a.mc[n - 1] = 7;
        cfg.gridDim = dim3(1u << 21);
        emu::wanted_block = [](unsigned b) { return b == (1u << 21) - 1; };
        emu::launch(&cfg, k_mc_classify, a, &ctr, sums);
        std::printf(a.mc[n - 1] == 0 ? "ok\n" : "last vertex not classified\n");
    }
    return 0;
}
