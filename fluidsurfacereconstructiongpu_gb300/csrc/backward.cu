// Adjoint (backward) kernels: gradient of a scalar loss through the last
// frame's triangle soup back to the particle positions, with the discrete
// structure of the frame held fixed (sorted order, band, valid cubes and MC
// cases, neighbourhoods, isolated-particle decisions, FP64 re-solves).
//
//   mesh vertex p = p_a + f (p_b - p_a), f = (iso - phi_a) / (phi_b - phi_a)
//     -> dL/dphi at the two corners of each edge (k_mc_backward)
//   ZB05:  phi = |xbar - v| - r_p, xbar = sum w x / sum w, w = (1 - d^2/h^2)^3
//   TC01:  phi = sum t^2 - t + 1/4, t = d^2 / 2h^2
//   Yu13:  phi = sum c_j (1 - |G_j (x~_j - v)|^2)^3 - 1/2, c_j = sigma det(G_j) m/rho_j
//          (unscaled kernel with G = I, c = sigma m/rho for non-involved particles)
//     -> dL/dx (ZB05, TC01) or dL/dx~ and dL/dG (Yu13), gathered per particle
//        over the band vertices of its support and window (k_field_iso_backward,
//        k_field_aniso_backward: by window group)
//   G = (1/h) cbrt(s1 s2 s3) V diag(1/s) V^T, s = eigenvalues of C clamped
//       from below at max/4, C = (h^2 I + sum w v v^T) / sum w, v = x_j - mean
//     -> dL/dC by the derivative of a spectral function (Daleckii-Krein form
//        with the cross terms of the clamp and of the volume factor), then
//        dL/dx_j and dL/dmean over the neighbours, recomputed (k_cov_backward)
//   x~ = (1 - lambda) x + lambda mean, mean = sum w x / sum w, w = 1 - (d/R)^3
//     -> dL/dx over the neighbours, recomputed (k_smooth_backward)
// Neighbour gradients are added with atomics (their order is not fixed; the
// results agree with finite differences within FP32 rounding).
#include "backward.h"

#include "cov_solver.cuh"

#include <algorithm>

namespace fsr {
namespace {

constexpr int kT = 256;

// ---------------------------------------------------------------- MC
// One cube per thread.  The mesh vertices' terms are summed per corner in
// shared memory first, one atomic per touched corner, and the corners are looked
// up as four rows of two x-neighbours (as in k_mc_classify).  The cube also
// marks the window centres (keys) its corners fall in; the first mark of a key
// appends it to the list the grouped adjoints take their groups from (a key
// without a gradient vertex is found empty there).  Bound by the latency of its
// scattered reads and atomics (ncu, 256k ZB05: 53 % of the issue slots, 29 % of
// the DRAM peak).  With the marking and the radius's sum as passes over the band
// of their own a 500k ZB05 frame took 151 us, now about 125.
__global__ void __launch_bounds__(kT) k_mc_backward(BwdArgs a, const Counters* ctr)
{
    after_launch();
    __shared__ float s_val[8 * kT], s_g[8 * kT];  // [corner][thread]
    float* val = s_val + threadIdx.x;
    float* g = s_g + threadIdx.x;
    const uint32_t nq = min(ctr->n_valid, a.cap_valid);
    const uint32_t rx = a.sc.res[0], rxy = a.sc.res[0] * a.sc.res[1];
    const uint32_t kx = a.sp.res[0] + 1, ky = a.sp.res[1] + 1;
    BwdGroupList groups(a.glist, a.sp);
    for (uint32_t q = blockIdx.x * blockDim.x + threadIdx.x; q < nq; q += gridDim.x * blockDim.x) {
        const uint32_t t = a.valid[q];
        const uint32_t info = a.mc[t];
        const uint32_t cs = info >> 8, nv = info & 0xFFu, base = a.vofs[t];
        const uint32_t v = a.sv[t];
        uint32_t r0[4];  // rank of each row's x corner; its x + 1 corner follows
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const int dy = r & 1, dz = r >> 1;
            const int i0 = dy ? (dz ? 2 : 3) : (dz ? 1 : 0);  // corner (0, dy, dz); (1, dy, dz) is i0 + 4
            r0[r] = r == 0 ? t : band_rank(a.band, v + (uint32_t)dy * rx + (uint32_t)dz * rxy);
            val[i0 * kT] = __ldg(a.band.phi + r0[r]);
            val[(i0 + 4) * kT] = __ldg(a.band.phi + r0[r] + 1);
            g[i0 * kT] = g[(i0 + 4) * kT] = 0.f;
        }
        const uint64_t tri = a.tri[cs];
        for (uint32_t k = 0; k < nv; ++k) {
            const int e = (int)((tri >> (4u * k)) & 0xFu);
            const int ia = mc::edgeA(e), ib = mc::edgeB(e);
            const float fa = val[ia * kT], fb = val[ib * kT];
            const float d = fb - fa;
            if (d > -1.0e-7f && d < 1.0e-7f) continue;  // f = 0.5 is constant there
            // p_b - p_a is one grid spacing along the edge's axis
            const int ax = mc::cornerDx(ib) != mc::cornerDx(ia) ? 0 : (mc::cornerDy(ib) != mc::cornerDy(ia) ? 1 : 2);
            const int sgn = (ax == 0 ? mc::cornerDx(ib) - mc::cornerDx(ia)
                                     : ax == 1 ? mc::cornerDy(ib) - mc::cornerDy(ia) : mc::cornerDz(ib) - mc::cornerDz(ia));
            const float gp = __ldg(a.gmesh + 3ull * (base + k) + ax);
            const float gf = gp * (float)sgn * a.sc.cs;
            const float inv = 1.0f / (d * d);
            const float ga = gf * (a.iso - fb) * inv, gb = -gf * (a.iso - fa) * inv;
            g[ia * kT] += ga;
            g[ib * kT] += gb;
        }
        bool any = false;
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const int dy = r & 1, dz = r >> 1;
            const int i0 = dy ? (dz ? 2 : 3) : (dz ? 1 : 0);
            const float g0 = g[i0 * kT], g1 = g[(i0 + 4) * kT];
            if (g0 != 0.f) atomicAdd(a.gphi + r0[r], g0);
            if (g1 != 0.f) atomicAdd(a.gphi + r0[r] + 1, g1);
            any = any || g0 != 0.f || g1 != 0.f;
        }
        if (!any) continue;
        // the keys of the corners: the cell of each end per axis
        uint32_t x, y, z;
        unlin3(v, a.sc, x, y, z);
        const uint32_t p[3] = {x, y, z};
        uint32_t lo[3], hi[3];
#pragma unroll
        for (int ax = 0; ax < 3; ++ax) {
            lo[ax] = (uint32_t)cell1(vpos1(p[ax], a.sc.min[ax], a.sc.cs), a.sp.min[ax], a.sp.cs);
            hi[ax] = (uint32_t)cell1(vpos1(p[ax] + 1, a.sc.min[ax], a.sc.cs), a.sp.min[ax], a.sp.cs);
        }
        for (uint32_t cz = lo[2]; cz <= hi[2]; ++cz)
            for (uint32_t cy = lo[1]; cy <= hi[1]; ++cy)
                for (uint32_t cx = lo[0]; cx <= hi[0]; ++cx) {
                    const uint32_t key = (cz * ky + cy) * kx + cx;
                    if (a.gkey[key] != 0u) continue;
                    const uint32_t flag = __ldg(a.gflag + key);  // (in flight with the mark)
                    if (atomicExch(&a.gkey[key], 1u) == 0u) groups.add(key, (flag & kCrowdedGroup) != 0u);
                }
    }
}

// dL/d(particle radius) of ZB05: -sum of dL/dphi over vertices with weight.  The
// weight sums are read only where dL/dphi is not zero (500k-particle frame: 50 ->
// 35 us).  In FP32, joined per warp: an FP64 sum repeats from run to run, but the
// field's own roundings put it 0.02 to 3.5e-6 of the result off the FP64 gradient,
// as far as this one (0 to 8e-6).
__global__ void __launch_bounds__(kT) k_radius_grad(BwdArgs a, const Counters* ctr, float* out)
{
    after_launch();
    const uint32_t nb = min(ctr->n_band, a.cap_band);
    float s = 0.f;
    for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < nb; t += gridDim.x * blockDim.x) {
        const float g = a.gphi[t];
        if (g != 0.f && a.mv[t].w > 0.f) s -= g;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if ((threadIdx.x & 31) == 0 && s != 0.f) atomicAdd(out, s);
}

// c = sigma det(G) m / rho: adds (sum dL/dphi (1 - q2)^3) dc/dG = that sum
// times c G^-T (G is symmetric) to dL/dG of each involved particle, after
// the grouped adjoint has accumulated the sum in gsmooth.w.
__global__ void k_det_term(BwdArgs a)
{
    after_launch();
    const uint32_t j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= a.n || !a.invol[a.skeys[j]]) return;
    const float sc = a.gsmooth[j].w;
    if (sc == 0.f) return;
    const float4 g0 = a.grec[4ull * j + 1], g1 = a.grec[4ull * j + 2], g2 = a.grec[4ull * j + 3];
    const float G[9] = {g0.x, g0.y, g0.z, g1.x, g1.y, g1.z, g2.x, g2.y, g2.z};
    const float det = G[0] * (G[4] * G[8] - G[5] * G[7]) - G[1] * (G[3] * G[8] - G[5] * G[6]) +
                      G[2] * (G[3] * G[7] - G[4] * G[6]);
    if (det == 0.f) return;
    const float k = sc * g0.w / det;
    float4* r = a.gG + 3ull * j;
    float4 r0 = r[0], r1 = r[1], r2 = r[2];
    r0.x += k * (G[4] * G[8] - G[5] * G[7]);
    r0.y += k * (G[5] * G[6] - G[3] * G[8]);
    r0.z += k * (G[3] * G[7] - G[4] * G[6]);
    r1.x += k * (G[2] * G[7] - G[1] * G[8]);
    r1.y += k * (G[0] * G[8] - G[2] * G[6]);
    r1.z += k * (G[1] * G[6] - G[0] * G[7]);
    r2.x += k * (G[1] * G[5] - G[2] * G[4]);
    r2.y += k * (G[2] * G[3] - G[0] * G[5]);
    r2.z += k * (G[0] * G[4] - G[1] * G[3]);
    r[0] = r0;
    r[1] = r1;
    r[2] = r2;
}

// ---------------------------------------------------------------- covariance / G
// dL/dC of G = V diag(d) V^T, d_i = cof / s_i, s_i = max(l_i, lmax/4),
// cof = h_inv cbrt(s_1 s_2 s_3).
template <class T>
__device__ void g_to_c(const T V[3][3], const T l[3], float h_inv, const float gG[9], T gC[3][3])
{
    T s[3], Jd[3];  // s and which eigenvalue each clamped s follows
    int imax = 0;
    T lmax = fabs(l[0]);
    for (int i = 1; i < 3; ++i)
        if (fabs(l[i]) > lmax) {
            lmax = fabs(l[i]);
            imax = i;
        }
    const T lo = lmax / T(4);
    bool clamped[3];
    for (int i = 0; i < 3; ++i) {
        const T li = fabs(l[i]);
        clamped[i] = li < lo;
        s[i] = clamped[i] ? lo : li;
        Jd[i] = l[i] < T(0) ? T(-1) : T(1);  // d|l|/dl
    }
    const T cof = T(h_inv) * cbrt(s[0] * s[1] * s[2]);
    T d[3];
    for (int i = 0; i < 3; ++i) d[i] = cof / s[i];
    // P = V^T sym(gG) V
    T gs[3][3];
    for (int i = 0; i < 3; ++i)
        for (int k = 0; k < 3; ++k) gs[i][k] = T(0.5) * (T(gG[3 * i + k]) + T(gG[3 * k + i]));
    T P[3][3];
    for (int i = 0; i < 3; ++i)
        for (int k = 0; k < 3; ++k) {
            T acc = T(0);
            for (int m = 0; m < 3; ++m)
                for (int n = 0; n < 3; ++n) acc += V[m][i] * gs[m][n] * V[n][k];
            P[i][k] = acc;
        }
    // ds_i/dl_k (J) and dd_i/dl_k = d_i ((1/3) sum_m J_mk / s_m - J_ik / s_i)
    T J[3][3];
    for (int i = 0; i < 3; ++i)
        for (int k = 0; k < 3; ++k) J[i][k] = T(0);
    for (int i = 0; i < 3; ++i) {
        if (clamped[i]) J[i][imax] = Jd[imax] / T(4);
        else J[i][i] = Jd[i];
    }
    T gl[3] = {T(0), T(0), T(0)};
    for (int k = 0; k < 3; ++k) {
        T third = T(0);
        for (int m = 0; m < 3; ++m) third += J[m][k] / s[m];
        third /= T(3);
        for (int i = 0; i < 3; ++i) gl[k] += P[i][i] * d[i] * (third - J[i][k] / s[i]);
    }
    // M = diag(gl) + K o P_offdiag, K_ik = (d_i - d_k) / (l_i - l_k)
    T M[3][3];
    for (int i = 0; i < 3; ++i)
        for (int k = 0; k < 3; ++k) {
            if (i == k) {
                M[i][k] = gl[i];
                continue;
            }
            // divided difference (d_i - d_k) / (l_i - l_k) with d = cof / s:
            // unclamped pairs (s = l > 0) reduce to -cof / (l_i l_k) exactly,
            // which avoids the cancellation of near-degenerate eigenvalues
            T K;
            if (!clamped[i] && !clamped[k]) {
                K = -cof / (s[i] * s[k]);
            } else if (clamped[i] && clamped[k]) {
                K = T(0);
            } else {
                const T dl = l[i] - l[k];
                K = dl != T(0) ? cof * (s[k] - s[i]) / (s[i] * s[k] * dl) : T(0);
            }
            M[i][k] = K * P[i][k];
        }
    for (int i = 0; i < 3; ++i)
        for (int k = 0; k < 3; ++k) {
            T acc = T(0);
            for (int m = 0; m < 3; ++m)
                for (int n = 0; n < 3; ++n) acc += V[i][m] * M[m][n] * V[k][n];
            gC[i][k] = acc;
        }
}

// Calls fn(i, q) for the sorted particles of each particle's cell window (rows
// of x-adjacent cells merged), P lanes per particle taking every P-th of them.
// Every lane of the warp calls it; lanes with active = false take none.
// Lanes whose windows span few cells per axis walk their union together, 32
// particles staged in sq at a time (one load per particle for the whole warp).
// Staged particles beyond r of the box of the active lanes' centres (cx, cy, cz)
// are dropped (they fail every lane's range test); their index rides in the
// staged w.
// kSets = false: the whole warp is one set, or each lane walks on its own; coop
// says that every particle the union adds fails each lane's own range test.
// kSets = true (wide windows, which may cut the range): sets of lanes
// (window_mates), and a lane takes only its own window's particles, a run of the
// sorted ones in each row.
template <int P, bool kSets, class Fn>
__device__ __forceinline__ void walk_windows(const Window& w, bool active, bool coop, const Grid& sp,
                                             const uint2* __restrict__ ranges, const float4* __restrict__ sorted,
                                             float4* sq, float cx, float cy, float cz, float r, Fn fn)
{
    const int lane = threadIdx.x & 31;
    const uint32_t sub = threadIdx.x % P;
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
    auto walk = [&](bool in_set) {
        int ulo[3], uhi[3];
        bool compact = coop;
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            ulo[a] = (int)__reduce_min_sync(0xffffffffu, in_set ? (unsigned)w.lo[a] : 0x7fffffffu);
            uhi[a] = (int)__reduce_max_sync(0xffffffffu, in_set ? (unsigned)(w.hi[a] + 1) : 0u) - 1;
            compact = compact && uhi[a] - ulo[a] <= 3;
        }
        if (!kSets && !compact) return false;
        const WarpBox box = warp_box(in_set, cx, cy, cz, r);
        for (int zz = ulo[2]; zz <= uhi[2]; ++zz)
            for (int yy = ulo[1]; yy <= uhi[1]; ++yy) {
                uint32_t beg, end, own = 0, len = 0;
                row_range(ulo[0], uhi[0], yy, zz, beg, end);
                if (kSets && in_set && zz >= w.lo[2] && zz <= w.hi[2] && yy >= w.lo[1] && yy <= w.hi[1]) {
                    row_range(w.lo[0], w.hi[0], yy, zz, own, len);
                    len = len > own ? len - own : 0u;
                }
                for (uint32_t b = beg; b < end; b += 32) {
                    float4 q = make_float4(0.f, 0.f, 0.f, 0.f);
                    bool keep = false;
                    if (b + lane < end) {
                        q = __ldg(&sorted[b + lane]);
                        keep = box.keeps(q);
                    }
                    const uint32_t m = __ballot_sync(0xffffffffu, keep);
                    if (keep) sq[__popc(m & ((1u << lane) - 1u))] = make_float4(q.x, q.y, q.z, __uint_as_float(b + lane));
                    __syncwarp();
                    const uint32_t cnt = __popc(m);
                    if (in_set)
                        for (uint32_t k = sub; k < cnt; k += P) {
                            const float4 e = sq[k];
                            const uint32_t i = __float_as_uint(e.w);
                            if (!kSets || i - own < len) fn(i, e);
                        }
                    __syncwarp();
                }
            }
        return true;
    };
    uint32_t left = __ballot_sync(0xffffffffu, active);
    if (kSets) {
        for (int sets = 0; left != 0u && sets < kMaxSets; ++sets) {
            const uint32_t set = window_mates(left, w, 5, lane);
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
                for (uint32_t i = beg + sub; i < end; i += P) fn(i, __ldg(&sorted[i]));
            }
    }
    __syncwarp();
}

// The sum of v over a particle's P lanes.
template <int P>
__device__ __forceinline__ float lanes_sum(float v)
{
#pragma unroll
    for (int o = 1; o < P; o <<= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Blocks of two warps (at the registers of 3 blocks of 256 threads per SM):
// a warp without work exits at once, and a small block gives its registers
// back as soon as its two warps are done.
constexpr int kCovBT = 64;

// P lanes per particle (neither kernel has an order to keep), kSets for radii of
// a cell and more, as in the forward walks.  The whole backward pass, P = 1 / 4 /
// 8 (ms): R = 0.8 cells: 3k particles 0.40 / 0.26 / 0.23, 60k 0.49 / 0.34 / 0.35,
// 150k 0.61 / 0.50 / 0.54, 4M 3.60 / 3.86 / 4.68; R = 1.54 cells, P = 1 / 4 / 8 with
// sets and P = 1 without: 20k 1.85 / 0.68 / 0.59, 2.11; 60k 2.29 / 1.18 / 1.07, 2.82.
template <int P, bool kSets>
__global__ void __launch_bounds__(kCovBT, 12) k_cov_backward(BwdArgs a, CovArgs f)
{
    after_launch();
    __shared__ float4 s_q[kCovBT];  // 32 staged particles per warp
    const uint32_t t = (blockIdx.x * blockDim.x + threadIdx.x) / P;
    const bool first = threadIdx.x % P == 0;
    const bool valid = t < f.n;
    float4 gmo = make_float4(0.f, 0.f, 0.f, 0.f);
    float gG[9] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    bool act = false;
    float4 c0 = make_float4(0.f, 0.f, 0.f, 0.f), c1 = c0;
    if (valid) {
        const float4 gr0 = a.gG[3ull * t], gr1 = a.gG[3ull * t + 1], gr2 = a.gG[3ull * t + 2];
        const float g9[9] = {gr0.x, gr0.y, gr0.z, gr1.x, gr1.y, gr1.z, gr2.x, gr2.y, gr2.z};
        bool any = false;
        for (int k = 0; k < 9; ++k) {
            gG[k] = g9[k];
            any = any || g9[k] != 0.f;
        }
        // only involved particles with a non-zero dL/dG whose G used their
        // covariance have work; the forward kept the normalised covariance and
        // its weight sum (k_cov; flag 0: too few neighbours)
        if (any && f.invol[f.skeys[t]] != 0) {
            c0 = f.crec[2ull * t];
            c1 = f.crec[2ull * t + 1];
            act = c1.w != 0.f;
        }
    }
    if (__all_sync(0xffffffffu, !act)) {
        if (valid && first) a.gmean[t] = gmo;
        return;
    }
    const float4 p = act ? f.sorted[t] : make_float4(0.f, 0.f, 0.f, 1.f);
    const float4 m = act ? f.mean[t] : p;
    const Window w = narrow(window(cell1(p.x, f.sp.min[0], f.sp.cs), cell1(p.y, f.sp.min[1], f.sp.cs),
                                   cell1(p.z, f.sp.min[2], f.sp.cs), 2, f.sp),
                            m.x, m.y, m.z, cull_radius(f.R, f.sp.cs), f.sp);
    float gA[3][3] = {{0.f, 0.f, 0.f}, {0.f, 0.f, 0.f}, {0.f, 0.f, 0.f}};
    float gW = 0.f;
    if (act) {
        const float W = c1.z, iw = 1.0f / W;
        float C[3][3] = {{c0.x, c0.y, c0.z}, {c0.y, c0.w, c1.x}, {c0.z, c1.x, c1.y}};
        float C0[3][3];
        for (int i = 0; i < 3; ++i)
            for (int k = 0; k < 3; ++k) C0[i][k] = C[i][k];
        float lv[3], V[3][3], gC[3][3];
        sym_eig3<float>(C, lv, V);
        const float smax = fmaxf(fabsf(lv[0]), fmaxf(fabsf(lv[1]), fabsf(lv[2])));
        const float smin = fminf(fabsf(lv[0]), fminf(fabsf(lv[1]), fabsf(lv[2])));
        if (!(smin > 0.f) || smax > 1e4f * smin) {
            double Cd[3][3], ld[3], Vd[3][3], gCd[3][3];
            for (int i = 0; i < 3; ++i)
                for (int k = 0; k < 3; ++k) Cd[i][k] = C0[i][k];
            sym_eig3<double>(Cd, ld, Vd);
            g_to_c<double>(Vd, ld, f.h_inv, gG, gCd);
            for (int i = 0; i < 3; ++i)
                for (int k = 0; k < 3; ++k) gC[i][k] = (float)gCd[i][k];
        } else {
            g_to_c<float>(V, lv, f.h_inv, gG, gC);
        }
        // C = A / W: dL/dA = gC / W, dL/dW = -<gC, C> / W
        for (int i = 0; i < 3; ++i)
            for (int k = 0; k < 3; ++k) gW -= gC[i][k] * C0[i][k];
        gW *= iw;
        for (int i = 0; i < 3; ++i)
            for (int k = 0; k < 3; ++k) gA[i][k] = gC[i][k] * iw;
    }
    const float R = f.R, invR = 1.0f / R, invR3 = invR * invR * invR;
    float gmx = 0.f, gmy = 0.f, gmz = 0.f;
    walk_windows<P, kSets>(w, act, f.coop_ok != 0, f.sp, f.ranges, f.sorted, s_q + (threadIdx.x & ~31u), m.x, m.y, m.z,
                           cull_radius(R, f.sp.cs), [&](uint32_t i, const float4& q) {
        const float vx = __fsub_rn(q.x, m.x), vy = __fsub_rn(q.y, m.y), vz = __fsub_rn(q.z, m.z);
        const float d2 = dot3_rn(vx, vy, vz);
        if (!(d2 < f.R_lt2)) return;  // the forward's weight test (d < R), exactly
        const float d = d2 > 0.f ? d2 * rsqrtf(d2) : 0.f;  // the gradient needs no correctly rounded root
        const float s = d * invR;
        const float wt = 1.0f - s * s * s;
        const float Avx = gA[0][0] * vx + gA[0][1] * vy + gA[0][2] * vz;
        const float Avy = gA[1][0] * vx + gA[1][1] * vy + gA[1][2] * vz;
        const float Avz = gA[2][0] * vx + gA[2][1] * vy + gA[2][2] * vz;
        const float vAv = vx * Avx + vy * Avy + vz * Avz;
        // d w / d v = -3 d v / R^3
        const float kw = (vAv + gW) * (-3.0f * d * invR3);
        const float gx = 2.f * wt * Avx + kw * vx, gy = 2.f * wt * Avy + kw * vy, gz = 2.f * wt * Avz + kw * vz;
        atomicAdd(a.gx + i, make_float4(gx, gy, gz, 0.f));
        gmx -= gx;
        gmy -= gy;
        gmz -= gz;
    });
    gmo = make_float4(lanes_sum<P>(gmx), lanes_sum<P>(gmy), lanes_sum<P>(gmz), 0.f);  // (0 when not active)
    if (valid && first) a.gmean[t] = gmo;
}

// ---------------------------------------------------------------- smoothing
template <int P, bool kSets>
__global__ void __launch_bounds__(kT) k_smooth_backward(BwdArgs a, const float4* sorted, const float4* mean,
                                                        const uint2* ranges, Grid sp, uint32_t n, float R, float R_lt2,
                                                        int coop_ok, float lambda)
{
    after_launch();
    __shared__ float4 s_q[kT];  // 32 staged particles per warp
    const uint32_t t = (blockIdx.x * blockDim.x + threadIdx.x) / P;
    const bool first = threadIdx.x % P == 0;
    const bool valid = t < n;
    float4 gs = make_float4(0.f, 0.f, 0.f, 0.f), gmc = gs;
    if (valid) {
        gs = a.gsmooth[t];
        gmc = a.gmean[t];
    }
    const float gmx = lambda * gs.x + gmc.x, gmy = lambda * gs.y + gmc.y, gmz = lambda * gs.z + gmc.z;
    float gix = 0.f, giy = 0.f, giz = 0.f;
    const bool act = valid && (gmx != 0.f || gmy != 0.f || gmz != 0.f);
    if (__any_sync(0xffffffffu, act)) {
        const float4 p = act ? sorted[t] : make_float4(0.f, 0.f, 0.f, 1.f);
        const float4 m = act ? mean[t] : make_float4(0.f, 0.f, 0.f, 1.f);  // m.w: the forward's weight sum W
        const Window w = narrow(window(cell1(p.x, sp.min[0], sp.cs), cell1(p.y, sp.min[1], sp.cs),
                                       cell1(p.z, sp.min[2], sp.cs), 2, sp),
                                p.x, p.y, p.z, cull_radius(R, sp.cs), sp);
        const float iw = 1.0f / m.w;
        const float gnx = gmx * iw, gny = gmy * iw, gnz = gmz * iw;
        const float invR = 1.0f / R, invR3 = invR * invR * invR;
        walk_windows<P, kSets>(w, act, coop_ok != 0, sp, ranges, sorted, s_q + (threadIdx.x & ~31u), p.x, p.y, p.z,
                               cull_radius(R, sp.cs), [&](uint32_t i, const float4& q) {
            // the forward's neighbour decision, exactly
            const float d2 = dot3_rn(__fsub_rn(p.x, q.x), __fsub_rn(p.y, q.y), __fsub_rn(p.z, q.z));
            if (!(d2 < R_lt2)) return;
            const float dx = p.x - q.x, dy = p.y - q.y, dz = p.z - q.z;
            const float d = d2 > 0.f ? d2 * rsqrtf(d2) : 0.f;
            const float s = d * invR;
            const float wt = 1.0f - s * s * s;
            // mean = sum w x / W: dL/dx_j += w gN, dL/dw = <gN, x_j - mean>
            const float gw = gnx * (q.x - m.x) + gny * (q.y - m.y) + gnz * (q.z - m.z);
            // dw/dd (x_i - x_j) / d = -3 d / R^3 (x_i - x_j)
            const float k = gw * (-3.0f * d * invR3);
            const float ex = k * dx, ey = k * dy, ez = k * dz;
            gix += ex;
            giy += ey;
            giz += ez;
            atomicAdd(a.gx + i, make_float4(wt * gnx - ex, wt * gny - ey, wt * gnz - ez, 0.f));
        });
    }
    gix = lanes_sum<P>(gix) + (1.0f - lambda) * gs.x;
    giy = lanes_sum<P>(giy) + (1.0f - lambda) * gs.y;
    giz = lanes_sum<P>(giz) + (1.0f - lambda) * gs.z;
    if (valid && first) atomicAdd(a.gx + t, make_float4(gix, giy, giz, 0.f));
}

__global__ void k_unsort(const float4* gx, const uint32_t* perm, uint32_t n, float* out)
{
    after_launch();
    const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    const float4 g = gx[k];
    const uint32_t s = perm[k];
    out[3ull * s] = g.x;
    out[3ull * s + 1] = g.y;
    out[3ull * s + 2] = g.z;
}

inline unsigned nblk(uint64_t n) { return (unsigned)std::max<uint64_t>(1, (n + kT - 1) / kT); }

}  // namespace

void launch_backward(const KernelCtx& c, const BwdArgs& a, const CovArgs* cov, const Counters* ctr, int method,
                     float lambda, float R, float* radius_grad_dev, float* out_grad_xyz)
{
    const unsigned pb = (unsigned)std::max<uint64_t>(1, std::min<uint64_t>((a.cap_valid + kT - 1) / kT,
                                                                          (uint64_t)c.num_sms * 16));
    launch_after(k_mc_backward, pb, kT, 0, c.stream, a, ctr);
    ++g_launches;
    if (radius_grad_dev) {
        const unsigned bb = (unsigned)std::max<uint64_t>(1, std::min<uint64_t>((a.cap_band + kT - 1) / kT,
                                                                              (uint64_t)c.num_sms * 16));
        launch_after(k_radius_grad, bb, kT, 0, c.stream, a, ctr, radius_grad_dev);
        ++g_launches;
    }
    if (method == FSR_METHOD_YU13) {
        AnisoBwdArgs fb{};
        fb.sp = a.sp;
        fb.sc = a.sc;
        fb.band = a.band;
        fb.smoothed = a.smoothed;
        fb.grec = a.grec;
        fb.qrec = a.qrec;
        fb.ranges = a.ranges;
        fb.invol = a.invol;
        fb.cell_rmax = a.cell_rmax;
        fb.gphi = a.gphi;
        fb.glist = a.glist;
        fb.gsmooth = a.gsmooth;
        fb.gG = a.gG;
        fb.sigma = a.sigma;
        fb.cap = a.cap_band;
        launch_field_aniso_backward(c, fb, a.ratio, ctr);
        launch_after(k_det_term, nblk(a.n), kT, 0, c.stream, a);
        // warps may walk the union of their windows when the cull radius stays below 2 cells
        const int smooth_coop = (R * 1.0001f + 1e-4f * cov->sp.cs) < 2.0f * cov->sp.cs * 0.9999f ? 1 : 0;
        auto launch = [&](auto cov_kernel, auto smooth_kernel, uint64_t lanes) {
            launch_after(cov_kernel, (unsigned)((a.n * lanes + kCovBT - 1) / kCovBT), kCovBT, 0, c.stream, a, *cov);
            launch_after(smooth_kernel, nblk(a.n * lanes), kT, 0, c.stream, a, cov->sorted, cov->mean, cov->ranges,
                         cov->sp, a.n, R, cov->R_lt2, smooth_coop, lambda);
        };
        const bool sets = cov->coop_ok == 0;  // R near or above a cell
        if (a.n < (sets ? 131072u : 40960u)) {
            if (sets) launch(k_cov_backward<8, true>, k_smooth_backward<8, true>, 8);
            else launch(k_cov_backward<8, false>, k_smooth_backward<8, false>, 8);
        } else if (a.n < (1u << 21)) {
            if (sets) launch(k_cov_backward<4, true>, k_smooth_backward<4, true>, 4);
            else launch(k_cov_backward<4, false>, k_smooth_backward<4, false>, 4);
        } else {
            if (sets) launch(k_cov_backward<1, true>, k_smooth_backward<1, true>, 1);
            else launch(k_cov_backward<1, false>, k_smooth_backward<1, false>, 1);
        }
        g_launches += 3;
    } else {
        launch_field_iso_backward(c, a, method == FSR_METHOD_TC01, ctr);
    }
    launch_after(k_unsort, nblk(a.n), kT, 0, c.stream, a.gx, a.perm, a.n, out_grad_xyz);
    ++g_launches;
}

}  // namespace fsr
