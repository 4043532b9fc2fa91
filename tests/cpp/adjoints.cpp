// The field adjoints of a few particles against sums over all vertex pairs in
// 64 bits:
//   nan:    one vertex's dL/dphi is not finite: the particles within reach of it
//           get a gradient that is not finite, the others theirs without it
//   cancel: dL/dphi whose first sums vanish for a particle, but not its dL/dG
//   shared: groups whose candidates several warps share, every second one listed as
//           crowded
#include "warp_emul.h"

#include "field_aniso.cu"

#include <cstdio>
#include <random>

namespace fsr {
thread_local uint64_t g_launches = 0;
namespace {
alignas(16) unsigned char smem[256 << 10];
}

constexpr int kCells = 5, kRatio = 4, kRes = kCells * kRatio + 1;
constexpr float kH = 0.5f;
struct Scene {
    Grid sp{}, sc{};
    std::vector<float4> sorted, grec, qrec, smoothed, gsmooth, gG, gx, mv;
    std::vector<uint2> ranges;
    std::vector<uint8_t> invol;
    std::vector<float> rmax, phi, gphi;
    std::vector<uint32_t> bits, prefix, glist;
    Counters ctr{};
    KernelCtx c{};
    uint32_t n = 0, nv = kRes * kRes * kRes;

    Scene(const std::vector<float4>& pos, const std::vector<float>& G)  // G: 9 per particle
    {
        sp.cs = 0.5f;
        sc.cs = sp.cs / kRatio;
        for (int a = 0; a < 3; ++a) {
            sp.res[a] = kCells;
            sc.res[a] = kRes;
        }
        n = (uint32_t)pos.size();
        std::vector<uint32_t> order(n);
        auto key = [&](uint32_t i) {
            return lin3((uint32_t)(pos[i].x / sp.cs), (uint32_t)(pos[i].y / sp.cs), (uint32_t)(pos[i].z / sp.cs), sp);
        };
        for (uint32_t i = 0; i < n; ++i) order[i] = i;
        std::stable_sort(order.begin(), order.end(), [&](uint32_t a, uint32_t b) { return key(a) < key(b); });
        const uint32_t cells = kCells * kCells * kCells, keys = (kCells + 1) * (kCells + 1) * (kCells + 1);
        ranges.assign(cells, make_uint2(kEmpty, kEmpty));
        invol.assign(cells, 1);
        rmax.assign(cells, 0.9f);
        for (uint32_t s = 0; s < n; ++s) {
            const uint32_t i = order[s];
            uint2& r = ranges[key(i)];
            if (r.x == kEmpty) r.x = s;
            r.y = s + 1;
            sorted.push_back(pos[i]);
            smoothed.push_back(make_float4(pos[i].x, pos[i].y, pos[i].z, 1e-3f));
            const float* g = &G[9 * i];
            auto dot = [&](int a, int b) { return g[a] * g[b] + g[3 + a] * g[3 + b] + g[6 + a] * g[6 + b]; };
            const float r2 = 0.75f, coef = pos[i].w;
            grec.push_back(make_float4(pos[i].x, pos[i].y, pos[i].z, r2));
            grec.push_back(make_float4(g[0], g[1], g[2], coef));
            grec.push_back(make_float4(g[3], g[4], g[5], 0.f));
            grec.push_back(make_float4(g[6], g[7], g[8], 0.f));
            qrec.push_back(make_float4(pos[i].x, pos[i].y, pos[i].z, r2));
            qrec.push_back(make_float4(dot(0, 0), 2 * dot(0, 1), 2 * dot(0, 2), coef));
            qrec.push_back(make_float4(dot(1, 1), 2 * dot(1, 2), dot(2, 2), 0.f));
        }
        const uint32_t words = (nv + 31) / 32;
        bits.assign(words + 1, 0);
        prefix.assign(words + 1, 0);
        for (uint32_t v = 0; v < nv; ++v) bits[v >> 5] |= 1u << (v & 31u);
        for (uint32_t w = 0; w < words; ++w) prefix[w] = 32u * w;
        gphi.assign(nv, 0.f);
        phi.assign(nv, 0.f);
        mv.assign(nv, make_float4(0.f, 0.f, 0.f, 0.f));
        ctr.n_band = nv;
        c.num_sms = 1;
        glist = {keys, 0, 0, 0};
        for (uint32_t k = 0; k < keys; ++k) glist.push_back(k);
        gsmooth.assign(n, make_float4(0.f, 0.f, 0.f, 0.f));
        gx = gsmooth;
        gG.assign(3 * n, make_float4(0.f, 0.f, 0.f, 0.f));
    }
    void vertex(uint32_t v, double p[3]) const
    {
        p[0] = (v % kRes) * (double)sc.cs;
        p[1] = v / kRes % kRes * (double)sc.cs;
        p[2] = v / kRes / kRes * (double)sc.cs;
    }
    void aniso()
    {
        AnisoBwdArgs a{};
        a.sp = sp;
        a.sc = sc;
        a.band = BandView{bits.data(), prefix.data(), phi.data()};
        a.smoothed = smoothed.data();
        a.grec = grec.data();
        a.qrec = qrec.data();
        a.ranges = ranges.data();
        a.invol = invol.data();
        a.cell_rmax = rmax.data();
        a.gphi = gphi.data();
        a.glist = glist.data();
        a.gsmooth = gsmooth.data();
        a.gG = gG.data();
        a.sigma = 1.5f;
        a.cap = nv;
        launch_field_aniso_backward(c, a, kRatio, &ctr);
    }
    void iso(bool tc01)
    {
        BwdArgs a{};
        a.sp = sp;
        a.sc = sc;
        a.ratio = kRatio;
        a.n = n;
        a.band = BandView{bits.data(), prefix.data(), phi.data()};
        a.gphi = gphi.data();
        a.glist = glist.data();
        a.sorted = sorted.data();
        a.ranges = ranges.data();
        a.mv = mv.data();
        a.gx = gx.data();
        a.h = kH;
        a.cap_band = nv;
        launch_field_iso_backward(c, a, tc01, &ctr);
    }
};

// the particle's part in 64 bits: 3 of its position, 9 of G; near: a vertex with a
// dL/dphi that is not finite lies in its support
static void exact(const Scene& s, int kind, uint32_t i, double out[12], bool& near, bool& clear)
{
    std::fill(out, out + 12, 0.0);
    near = false;
    clear = true;
    const double x[3] = {s.sorted[i].x, s.sorted[i].y, s.sorted[i].z}, h2 = (double)kH * kH;
    for (uint32_t v = 0; v < s.nv; ++v) {
        if (s.gphi[v] == 0.f) continue;
        double p[3], d[3], t[3], q = 0.0;
        s.vertex(v, p);
        for (int a = 0; a < 3; ++a) d[a] = x[a] - p[a];
        const float4* g = &s.grec[4 * i + 1];
        const bool wide = kind == 2 && !s.invol[0];  // G = I
        for (int a = 0; a < 3; ++a) {
            t[a] = kind < 2 || wide ? d[a] : g[a].x * d[0] + g[a].y * d[1] + g[a].z * d[2];
            q += t[a] * t[a];
        }
        if (kind < 2) q /= h2;
        if (!std::isfinite(s.gphi[v])) {
            clear = clear && std::fabs(q - 1.0) > 1e-3;
            near = near || q < 1.0;
            continue;
        }
        if (!(q < 1.0)) continue;
        const double u = 1.0 - q, gp = s.gphi[v];
        if (kind == 1) {
            for (int a = 0; a < 3; ++a) out[a] += gp * (q - 1.0) / h2 * d[a];
        } else if (kind == 0) {
            const float4 m = s.mv[v];
            const double mm[3] = {m.x, m.y, m.z}, ml = std::sqrt(mm[0] * mm[0] + mm[1] * mm[1] + mm[2] * mm[2]);
            double proj = 0.0;
            for (int a = 0; a < 3; ++a) proj += gp * mm[a] / ml * (d[a] - mm[a]);
            for (int a = 0; a < 3; ++a)
                out[a] += (u * u * u * gp * mm[a] / ml + proj * -6.0 * u * u / h2 * d[a]) / m.w;
        } else {
            const double c = wide ? 1.5 * s.smoothed[i].w : g[0].w, A = -6.0 * gp * c * u * u;
            for (int a = 0; a < 3; ++a) {
                out[a] += wide ? A * d[a]
                               : A * ((&g[0].x)[a] * t[0] + (&g[1].x)[a] * t[1] + (&g[2].x)[a] * t[2]);
                for (int b = 0; b < 3 && !wide; ++b) out[3 + 3 * a + b] += A * t[a] * d[b];
            }
        }
    }
}

static bool check(const Scene& s, int kind, const char* what)
{
    double scale = 0.0;
    std::vector<double> want(12 * s.n);
    std::vector<uint8_t> near(s.n), clear(s.n);
    for (uint32_t i = 0; i < s.n; ++i) {
        bool nr, cl;
        exact(s, kind, i, &want[12 * i], nr, cl);
        near[i] = nr;
        clear[i] = cl;
        for (int k = 0; k < 12; ++k) scale = std::max(scale, std::fabs(want[12 * i + k]));
    }
    uint32_t some = 0;
    for (uint32_t i = 0; i < s.n; ++i) {
        const float4 g = kind == 2 ? s.gsmooth[i] : s.gx[i];
        float got[12] = {g.x, g.y, g.z};
        for (int k = 0; k < 9; ++k) got[3 + k] = (&s.gG[3 * i + k / 3].x)[k % 3];
        bool finite = true;
        for (float v : got) finite = finite && std::isfinite(v);
        if (!clear[i]) continue;
        some += near[i];
        if (finite == (near[i] != 0)) {
            std::printf("%s, kind %d: particle %u %s\n", what, kind, i,
                        finite ? "misses the vertex" : "out of reach is not finite");
            return false;
        }
        for (int k = 0; k < 12 && !near[i]; ++k)
            if (!(std::fabs(got[k] - want[12 * i + k]) <= 1e-5 * scale)) {
                std::printf("%s, kind %d: particle %u term %d is %g, not %g\n", what, kind, i, k, got[k], want[12 * i + k]);
                return false;
            }
    }
    if (!(scale > 0.0) || (std::string(what) == "nan" && some == 0)) {
        std::printf("%s, kind %d: nothing to see\n", what, kind);
        return false;
    }
    return true;
}
}  // namespace fsr

int main(int, char** argv)
{
    using namespace fsr;
    const std::string what = argv[1];
    std::mt19937 rng(7);
    auto uniform = [&] { return (rng() >> 8) * 0x1p-24f; };
    if (what == "nan") {
        for (int kind = 0; kind < 4; ++kind)  // ZB05, TC01, anisotropic, its particles of non-involved cells
            for (float odd : {INFINITY, -INFINITY, NAN}) {
                std::vector<float4> pos;
                std::vector<float> G;
                for (int i = 0; i < 60; ++i) {
                    pos.push_back(make_float4(0.75f + uniform(), 0.75f + uniform(), 0.75f + uniform(), 0.5f + uniform()));
                    float m[9];
                    for (int a = 0; a < 3; ++a)
                        for (int b = a; b < 3; ++b) m[3 * a + b] = m[3 * b + a] = (a == b ? 2.f : 0.f) + 0.8f * (uniform() - 0.5f);
                    G.insert(G.end(), m, m + 9);
                }
                Scene s(pos, G);
                for (uint32_t v = 0; v < s.nv; ++v) {
                    if (uniform() < 0.5f) s.gphi[v] = uniform() - 0.5f;
                    s.mv[v] = make_float4(uniform() - 0.5f, uniform() - 0.5f, uniform() - 0.5f, 1.f + uniform());
                }
                s.gphi[8 + kRes * (9 + kRes * 10)] = odd;
                if (kind == 3) std::fill(s.invol.begin(), s.invol.end(), 0);
                if (kind >= 2) s.aniso();
                else s.iso(kind == 1);
                if (!check(s, std::min(kind, 2), "nan")) return 0;
            }
    } else if (what == "shared") {
        for (int kind = 0; kind < 3; ++kind) {
            std::vector<float4> pos;
            std::vector<float> G;
            for (int i = 0; i < 900; ++i) {
                pos.push_back(make_float4(0.75f + uniform(), 0.75f + uniform(), 0.75f + uniform(), 0.5f + uniform()));
                for (int a = 0; a < 9; ++a) G.push_back(a % 4 == 0 ? 1.75f + 0.5f * uniform() : 0.f);
            }
            Scene s(pos, G);
            for (uint32_t v = 0; v < s.nv; ++v) {
                if (uniform() < 0.5f) s.gphi[v] = uniform() - 0.5f;
                s.mv[v] = make_float4(uniform() - 0.5f, uniform() - 0.5f, uniform() - 0.5f, 1.f + uniform());
            }
            const uint32_t keys = s.glist[0];
            s.glist[0] = 0;
            BwdGroupList list(s.glist.data(), s.sp);
            for (uint32_t k = 0; k < keys; ++k) list.add(k, k % 2 == 0);
            if (kind == 2) s.aniso();
            else s.iso(kind == 1);
            if (!check(s, kind, "shared")) return 0;
        }
    } else {
        // at a vertex, G = 1.75 I: +1 a step away along x, -1 along y
        const uint32_t at[3] = {10, 10, 10};
        const float x = 10 * 0.125f;
        Scene s({make_float4(x, x, x, 1.f)}, {1.75f, 0.f, 0.f, 0.f, 1.75f, 0.f, 0.f, 0.f, 1.75f});
        auto set = [&](int dx, int dy, float g) { s.gphi[at[0] + dx + kRes * (at[1] + dy + kRes * at[2])] = g; };
        set(1, 0, 1.f);
        set(-1, 0, 1.f);
        set(0, 1, -1.f);
        set(0, -1, -1.f);
        s.aniso();
        if (!check(s, 2, "cancel")) return 0;
    }
    std::printf("ok\n");
    return 0;
}
