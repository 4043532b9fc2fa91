// Anisotropic field, grouped by window (computationOfScalarFieldGrid,
// ReconstructionCUDA.cu:830-906).
//
// A band vertex's candidate particles are the particles of the +-2 cells
// around the spatial cell its FP32 position falls in; every vertex that
// falls in the same cell has the same window.  Along each axis that cell
// index is a non-decreasing function of the vertex index, so the vertices
// of one cell form an index box, found exactly without sorting.  One warp
// handles one such group (or one z slab of it, for frames with few groups),
// taken from a work counter:
//   1. it lists the group's band vertices row by row from the bitset, with
//      their rank in the band, in passes of up to 256 vertices ordered into
//      eight brick tiles of 32;
//   2. it lists the window's candidate cells, dropping involved cells that
//      lie beyond the reach (largest support radius + smoothing shift) of all
//      their particles from the group's vertex box;
//   3. it streams the involved candidates 32 at a time (one record per lane,
//      kept in shared memory when its support reaches the pass's box); per
//      tile, the candidates that reach the tile are listed two to a pair
//      block and each lane evaluates one block per step for its vertex with
//      packed FP32x2 operations.
// Particles of non-involved cells use the unscaled kernel (cuh:312-322),
// G = I with support 1: their part of each vertex's sum is the group's
// moment polynomial where it applies, else they are streamed as well.  Only
// terms that are exactly zero are skipped; the summation order is the
// candidate order, the same for every vertex, so results are deterministic.
#include "kernels.h"
#include "backward.h"

#include <algorithm>
#include <type_traits>

namespace fsr {
namespace {

constexpr int kMaxCells = 125;      // 5 x 5 x 5 window

struct GroupArgs {
    Grid sp, sc;
    BandView band;
    const float4* grec;
    const float4* qrec;  // per involved particle: (x~, r2max) (M00, 2M01, 2M02, coef) (M11, 2M12, M22, 0)
    const float4* smoothed;
    const uint32_t* glist;  // groups holding band vertices
    const uint2* ranges;
    const uint8_t* invol;
    const float* reach;
    float* phi;
    float sigma;
    uint32_t cap;
};

// Shared-memory tables of one group's candidate cells.
struct CandTables {
    uint32_t* cstart;  // first sorted particle of each window cell (kMaxCells)
    uint32_t* cpre;    // exclusive prefix of the kept cells' particle counts (kMaxCells + 1)
    uint32_t* cinv;    // the cell is involved (its particles carry a G record)
};

// Group g (a key of the (res + 1)^3 window-centre grid): its cell and its
// vertex index box [x0, x1) x [y0, y1) x [z0, z1).  Every lane of the warp calls it.
__device__ __forceinline__ bool group_box(uint32_t g, const Grid& sp, const Grid& sc, uint32_t ratio, int c[3],
                                          int lo[3], int hi[3])
{
    const uint32_t kx = sp.res[0] + 1, ky = sp.res[1] + 1;
    c[0] = (int)(g % kx);
    c[1] = (int)((g / kx) % ky);
    c[2] = (int)(g / (kx * ky));
    // the six ends, one per lane (lane 2 a: lo of axis a, 2 a + 1: hi)
    const int lane = threadIdx.x & 31, axis = min(lane >> 1, 2);
    const int ca = (axis == 0 ? c[0] : axis == 1 ? c[1] : c[2]) + (lane & 1);
    const int nres = (int)(axis == 0 ? sc.res[0] : axis == 1 ? sc.res[1] : sc.res[2]);
    const float vmin = axis == 0 ? sc.min[0] : axis == 1 ? sc.min[1] : sc.min[2];
    const float cmin = axis == 0 ? sp.min[0] : axis == 1 ? sp.min[1] : sp.min[2];
    const int end = first_vertex(ca, ratio, nres, vmin, sc.cs, cmin, sp.cs);
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        lo[a] = __shfl_sync(0xffffffffu, end, 2 * a);
        hi[a] = __shfl_sync(0xffffffffu, end, 2 * a + 1);
    }
    return hi[0] > lo[0] && hi[1] > lo[1] && hi[2] > lo[2];
}

// Work items of the forward field kernels: a frame with few window groups
// (a small frame) would leave most SMs idle with one warp per group, so each
// group's vertex box is then cut into S slabs along z, each a work item of
// its own (a vertex lies in one slab; a slab is listed, culled and summed
// like a group).  S depends only on the number of groups, so a frame's
// results do not depend on the launch shape.
constexpr uint32_t kSlabTarget = 8192;  // work items wanted (measured: 4096 and 8 slabs at most, 12-16 % slower on 32k frames)
constexpr uint32_t kSlabMax = 16;
__device__ __forceinline__ uint32_t field_slabs(uint32_t ngroups)
{
    return ngroups >= kSlabTarget ? 1u : min(kSlabMax, (kSlabTarget + ngroups - 1) / max(ngroups, 1u));
}
// The anisotropic field's items run 0.1 to 0.3 ms each, two to twelve per
// resident warp, so their order and size decide how long the last ones keep a
// few SMs busy (ncu, 150k particles: the busiest scheduler issued 1.6 times the
// average).  The dense groups come first (GroupList); the last kSplitItems of
// them, about one per resident warp, are split in two, each half taking every
// second tile of the passes; the sparse groups fill the end.  A vertex's sum does
// not depend on the split.  Measured (ms, all / last 7296 / last 3648 split, none
// before): 256k particles 1.00 / 0.98 / 0.99, 1.38 before; 1M 2.34 / 2.27 / 2.19,
// 2.53; 8M 9.73 / 9.37 / 9.33, 9.67; in four parts 1M 2.29.
constexpr uint32_t kSplitItems = 4096;
// Restricts the box [lo, hi) to slab `part` of S along z; false when empty.
__device__ __forceinline__ bool slab_box(uint32_t part, uint32_t S, int lo[3], int hi[3])
{
    if (S == 1) return true;
    const uint32_t nz = (uint32_t)(hi[2] - lo[2]);
    const int z0 = lo[2] + (int)(nz * part / S), z1 = lo[2] + (int)(nz * (part + 1) / S);
    if (z0 >= z1) return false;
    lo[2] = z0;
    hi[2] = z1;
    return true;
}

// Candidate j of the group: its sorted particle index and window cell.
__device__ __forceinline__ uint32_t candidate(uint32_t j, const CandTables& t, int* cell, int ncells = kMaxCells)
{
    int lo = 0, hi = ncells;  // find k with cpre[k] <= j < cpre[k+1]
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (t.cpre[mid] <= j) lo = mid;
        else hi = mid;
    }
    *cell = lo;
    return t.cstart[lo] + (j - t.cpre[lo]);
}

// ---------------------------------------------------------------- forward
constexpr int kFT = 128;                 // threads per block of the forward kernel
#ifndef FSR_FIELD_MIN_BLOCKS
#define FSR_FIELD_MIN_BLOCKS 6               // blocks per SM of the anisotropic field (80 registers)
#endif
constexpr int kFWarps = kFT / 32;
constexpr int kPassTiles = 8;            // 32-vertex tiles per pass (sums kept per lane in the warp's slice)
constexpr int kPassVerts = 32 * kPassTiles;
constexpr int kMoments = 35;             // moments of the unscaled kernel's polynomial (unscaled_sum)
constexpr int kPairF4 = 5;               // float4 per pair block of listed candidates (list_pair_record)

// Per-warp shared memory of the forward kernel.
struct WarpSlice {
    float4 rec[80];              // the current chunk's candidates: 5 float2 per lane (involved, stage_record),
                                 // a float4 per lane (the others)
    float4 lst[16 * kPairF4];    // one tile's involved candidates in lane order, two to a pair block
    uint32_t vloc[kPassVerts];   // the pass's band vertices: index in the group's box (vert_loc)
    uint32_t vrank[kPassVerts];  // and band rank
    float4 box[2 * kPassTiles];  // per tile: lo, hi
    float psum[kPassTiles][32];  // per tile and lane: sum over the involved candidates
    float usum[kPassTiles][32];  // and over the non-involved ones
    uint16_t order[kPassVerts];  // the pass's vertices in brick order (tile t: entries 32t .. 32t+31)
    float mom[kMoments];         // moments of the group's non-involved candidates (unscaled_moments)
    uint32_t use_mom;            // the moment form applies to this group
    uint32_t cstart[128];
    uint32_t cpre[kMaxCells + 1];
    uint32_t cinv[128];
    uint32_t ncells;             // entries of the candidate tables
    uint32_t total_inv;          // candidates of involved cells (they come first)
    uint32_t ninv_cells;         // and the number of those cells
};

// The window cells of candidates cb .. cb + 31 of a sweep through the
// tables, one per lane, from the table boundaries that fall inside the
// chunk (one shared load and a warp OR instead of a binary search per
// lane).  k0 is a cell with cpre[k0] <= cb < cpre[k0 + 1] on entry (the
// sweep's first cell, or the value the previous chunk left) and is advanced
// to the cell of cb + 31.  Every lane calls it; the cell of a lane whose
// candidate lies at or beyond the sweep's end is not used.
__device__ __forceinline__ int chunk_cell(uint32_t cb, int lane, const uint32_t* cpre, uint32_t ncells, uint32_t& k0)
{
    const uint32_t k = k0 + 1u + (uint32_t)lane;
    uint32_t bit = 0;
    if (k <= ncells) {
        const uint32_t d = cpre[k] - cb;  // cpre[k] >= cpre[k0 + 1] > cb
        if (d < 32u) bit = 1u << d;
    }
    const uint32_t bm = __reduce_or_sync(0xffffffffu, bit);
    const int cell = (int)(k0 + (uint32_t)__popc(bm & (0xffffffffu >> (31 - lane))));
    k0 += (uint32_t)__popc(bm);
    return cell;
}

// Lists the candidate cells of the window around cell c (clamped as in the
// reference, cu:856-864), dropping involved cells whose reach cannot touch
// the box [b0, b1]; by the warp: listed with the
// involved cells first and the other non-empty cells after them (each part
// in window order); only non-empty kept cells get an entry.
template <class Slice>
__device__ uint32_t warp_candidates(const Grid& sp, const uint2* __restrict__ ranges,
                                    const uint8_t* __restrict__ invol, const float* __restrict__ reach,
                                    const int c[3], const float b0[3], const float b1[3], Slice& w)
{
    const int lane = threadIdx.x & 31;
    const int lx = clampi(c[0] - 2, 0, (int)sp.res[0] - 1), hx = clampi(c[0] + 2, 0, (int)sp.res[0] - 1);
    const int ly = clampi(c[1] - 2, 0, (int)sp.res[1] - 1), hy = clampi(c[1] + 2, 0, (int)sp.res[1] - 1);
    const int lz = clampi(c[2] - 2, 0, (int)sp.res[2] - 1), hz = clampi(c[2] + 2, 0, (int)sp.res[2] - 1);
    uint32_t st4[4], cnt4[4], inv4[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        const int k = 32 * r + lane;
        uint32_t cnt = 0, st = 0, inv = 0;
        if (k < kMaxCells) {
            const int xx = lx + k % 5, yy = ly + (k / 5) % 5, zz = lz + k / 25;
            if (xx <= hx && yy <= hy && zz <= hz) {
                const uint32_t cell = lin3(xx, yy, zz, sp);
                const uint2 rg = __ldg(&ranges[cell]);
                if (rg.x != kEmpty) {
                    inv = __ldg(&invol[cell]);
                    bool keep = true;
                    if (inv) {
                        const float cs = sp.cs;
                        const float cx0 = sp.min[0] + xx * cs, cy0 = sp.min[1] + yy * cs, cz0 = sp.min[2] + zz * cs;
                        const float gx = fmaxf(0.f, fmaxf(cx0 - b1[0], b0[0] - (cx0 + cs)));
                        const float gy = fmaxf(0.f, fmaxf(cy0 - b1[1], b0[1] - (cy0 + cs)));
                        const float gz = fmaxf(0.f, fmaxf(cz0 - b1[2], b0[2] - (cz0 + cs)));
                        const float cr = cull_radius(__ldg(&reach[cell]), cs);
                        keep = fmaf(gx, gx, fmaf(gy, gy, gz * gz)) < cr * cr;
                    }
                    if (keep) {
                        st = rg.x;
                        cnt = rg.y - rg.x;
                    }
                }
            }
        }
        st4[r] = st;
        cnt4[r] = cnt;
        inv4[r] = inv;
    }
    // two sweeps: involved cells, then the others; entries and prefix sums
    // are appended in window order within each sweep
    uint32_t running = 0, slot = 0;
#pragma unroll
    for (int part = 0; part < 2; ++part) {
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const bool take = cnt4[r] > 0 && (inv4[r] != 0) == (part == 0);
            const uint32_t m = __ballot_sync(0xffffffffu, take);
            const uint32_t c = take ? cnt4[r] : 0u;
            uint32_t x = c;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
                if (lane >= o) x += y;
            }
            if (take) {
                const uint32_t e = slot + __popc(m & ((1u << lane) - 1u));
                w.cstart[e] = st4[r];
                w.cinv[e] = inv4[r];
                w.cpre[e] = running + x - c;
            }
            slot += __popc(m);
            running += __shfl_sync(0xffffffffu, x, 31);
        }
        if (part == 0 && lane == 0) {
            w.total_inv = running;
            w.ninv_cells = slot;
        }
    }
    if (lane == 0) {
        w.cpre[slot] = running;
        w.ncells = slot;
    }
    __syncwarp();
    return running;
}

// A staged involved candidate: 10 floats per lane, as 5 float2
//   (x~, y~) (z~, M00) (2M01, 2M02) (M11, 2M12) (M22, coef)
// (M = G^T G; coef = sigma det(G) m / rho).
__device__ __forceinline__ void stage_record(float2* rec, int lane, float4 r0, float4 m0, float4 m1)
{
    float2* d = rec + 5 * lane;
    d[0] = make_float2(r0.x, r0.y);
    d[1] = make_float2(r0.z, m0.x);
    d[2] = make_float2(m0.y, m0.z);
    d[3] = make_float2(m1.x, m1.y);
    d[4] = make_float2(m1.z, m0.w);
}

// A tile's candidates are listed two to a pair block of 5 float4: entry pos
// of the list in the x (and z) components, entry pos + 1 in y (and w), so
// that each float2 of the block holds one quantity of both candidates and
// feeds one packed FP32x2 operation:
//   (x~, x~') (y~, y~') | (z~, z~') (M00, M00') | (2M01, 2M01') (2M02, 2M02') |
//   (M11, M11') (2M12, 2M12') | (M22, M22') (coef, coef')
__device__ __forceinline__ void list_pair_record(const float2* rec, int lane, float* lst, uint32_t pos)
{
    const float2* src = rec + 5 * lane;
    float* d = lst + (pos >> 1) * (4 * kPairF4) + (pos & 1u);
#pragma unroll
    for (int c = 0; c < 5; ++c) {
        const float2 v = src[c];
        d[4 * c] = v.x;
        d[4 * c + 2] = v.y;
    }
}

// The (1 - q2)^3 terms of both candidates of a pair block for vertex v
// (nv = (-v, -v) per axis): q2 = d^T M d for d = x~ - v, each component
// rounded as the scalar form
//   t1 = fma(M00, dx, fma(2M01, dy, 2M02 dz)),  t2 = fma(M11, dy, 2M12 dz),
//   q2 = fma(dx, t1, fma(dy, t2, dz (M22 dz))),  (1 - q2)^3 = ((1 - q2)^2)(1 - q2)
// (no product feeds a separate sum, so no contraction can change a rounding).
__device__ __forceinline__ void pair_terms(const float4* P, float2 nvx, float2 nvy, float2 nvz, float2& q2,
                                           float2& u3, float2& coef)
{
    const float4 A = P[0], B = P[1], C = P[2], D = P[3], E = P[4];
    const float2 dx = __fadd2_rn(make_float2(A.x, A.y), nvx);
    const float2 dy = __fadd2_rn(make_float2(A.z, A.w), nvy);
    const float2 dz = __fadd2_rn(make_float2(B.x, B.y), nvz);
    float2 t1 = __fmul2_rn(make_float2(C.z, C.w), dz);
    t1 = __ffma2_rn(make_float2(C.x, C.y), dy, t1);
    t1 = __ffma2_rn(make_float2(B.z, B.w), dx, t1);
    float2 t2 = __fmul2_rn(make_float2(D.z, D.w), dz);
    t2 = __ffma2_rn(make_float2(D.x, D.y), dy, t2);
    float2 q = __fmul2_rn(make_float2(E.x, E.y), dz);
    q = __fmul2_rn(dz, q);
    q = __ffma2_rn(dy, t2, q);
    q = __ffma2_rn(dx, t1, q);
    // 1 - q2 as fma(q2, -1, 1): the product is exact, so one rounding, as in
    // the subtraction
    const float2 u = __ffma2_rn(q, make_float2(-1.0f, -1.0f), make_float2(1.0f, 1.0f));
    u3 = __fmul2_rn(__fmul2_rn(u, u), u);
    q2 = q;
    coef = make_float2(E.z, E.w);
}

__device__ __forceinline__ bool reaches(float4 r0, float4 lo, float4 hi)
{
    const float gx = fmaxf(0.f, fmaxf(lo.x - r0.x, r0.x - hi.x));
    const float gy = fmaxf(0.f, fmaxf(lo.y - r0.y, r0.y - hi.y));
    const float gz = fmaxf(0.f, fmaxf(lo.z - r0.z, r0.z - hi.z));
    return fmaf(gx, gx, fmaf(gy, gy, gz * gz)) < r0.w;
}

// A listed vertex is kept as its index in the group's box, 10 bits per axis
// (the box spans at most ratio + 1 <= 1001 vertices per axis); its position
// is the scalar grid's vertex position (getVertexPos, FP32).
__device__ __forceinline__ uint32_t vert_loc(int lx, int ly, int lz)
{
    return (uint32_t)lx | ((uint32_t)ly << 10) | ((uint32_t)lz << 20);
}

__device__ __forceinline__ float4 vert_pos(uint32_t loc, const int lo[3], const Grid& sc)
{
    return make_float4(vpos1(lo[0] + (int)(loc & 1023u), sc.min[0], sc.cs),
                       vpos1(lo[1] + (int)((loc >> 10) & 1023u), sc.min[1], sc.cs),
                       vpos1(lo[2] + (int)(loc >> 20), sc.min[2], sc.cs), 0.f);
}

// The layout of a pass of nv <= kPassVerts listed vertices: the pass's box
// (pl, ph, on every lane), their order in 4 x 4 x 2-vertex bricks (tiles of
// compact bricks instead of runs of rows: a smaller box per tile, fewer
// candidates reaching it; a counting sort by brick), and the box of each
// 32-vertex tile (kVerts: the most vertices of a pass).  Boxes are formed from
// the vertices' indices by warp reductions (positions do not decrease with the
// index); frames of many small groups spent a fifth of their field time on the
// float boxes this replaces.  hist: kVerts words of scratch.
struct IndexBox {
    uint32_t lo[3], hi[3];
    __device__ __forceinline__ void clear()
    {
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            lo[a] = 1023u;
            hi[a] = 0u;
        }
    }
    __device__ __forceinline__ void add(uint32_t loc)
    {
        const uint32_t i[3] = {loc & 1023u, (loc >> 10) & 1023u, loc >> 20};
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            lo[a] = min(lo[a], i[a]);
            hi[a] = max(hi[a], i[a]);
        }
    }
    // the box of all lanes' boxes
    __device__ __forceinline__ void join()
    {
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            lo[a] = __reduce_min_sync(0xffffffffu, lo[a]);
            hi[a] = __reduce_max_sync(0xffffffffu, hi[a]);
        }
    }
    __device__ __forceinline__ float4 low(const int o[3], const Grid& sc) const
    {
        return make_float4(vpos1(o[0] + (int)lo[0], sc.min[0], sc.cs), vpos1(o[1] + (int)lo[1], sc.min[1], sc.cs),
                           vpos1(o[2] + (int)lo[2], sc.min[2], sc.cs), 0.f);
    }
    __device__ __forceinline__ float4 high(const int o[3], const Grid& sc) const
    {
        return make_float4(vpos1(o[0] + (int)hi[0], sc.min[0], sc.cs), vpos1(o[1] + (int)hi[1], sc.min[1], sc.cs),
                           vpos1(o[2] + (int)hi[2], sc.min[2], sc.cs), 0.f);
    }
};

// kInPlace: vloc and vrank are reordered (order is not used), the order inside a
// brick that of the atomics: it changes no result, since a vertex's sum does not
// depend on its tile.  Else order[v] is the place of the v-th vertex, a function
// of the listed vertices alone (a stable sort): the two warps of a split work item
// lay out the pass each for itself and write every second tile.  (Atomics there,
// which left the order to the hardware: 1M particles 4.162 -> 4.170 ms.)
template <bool kInPlace, int kVerts = kPassVerts>
__device__ __forceinline__ void pass_layout(uint32_t* vloc, uint32_t* vrank, const int lo[3], const Grid& sc,
                                            uint16_t* order, uint32_t* hist, float4* box, uint32_t nv, int lane,
                                            float4& pl, float4& ph)
{
    const uint32_t ntiles = (nv + 31) / 32;
    IndexBox pass;
    pass.clear();
    for (uint32_t q = lane; q < nv; q += 32) pass.add(vloc[q]);
    pass.join();
    pl = pass.low(lo, sc);
    ph = pass.high(lo, sc);
    if (ntiles == 1u) {  // one tile: any order, the pass's box
        if (!kInPlace && (uint32_t)lane < nv) order[lane] = (uint16_t)lane;
        if (lane == 0) {
            box[0] = pl;
            box[1] = ph;
        }
        __syncwarp();
        return;
    }
    const uint32_t gx = ((pass.hi[0] - pass.lo[0]) >> 2) + 1u;
    const uint32_t gy = ((pass.hi[1] - pass.lo[1]) >> 2) + 1u;
    const uint32_t gz = ((pass.hi[2] - pass.lo[2]) >> 1) + 1u;
    const uint32_t nbins = gx * gy * gz;
    if (nbins <= (uint32_t)kVerts) {
        for (uint32_t b = lane; b < nbins; b += 32) hist[b] = 0u;
        __syncwarp();
        uint32_t at[kVerts / 32];  // brick | place in it << 16
        uint32_t loc[kVerts / 32], rank[kVerts / 32];
#pragma unroll
        for (int k = 0; k < kVerts / 32; ++k) {
            at[k] = 0;
            if (32u * k >= nv) continue;
            const uint32_t q = lane + 32 * k;
            uint32_t key = kEmpty, place = 0;
            if (q < nv) {
                const uint32_t l = vloc[q];
                loc[k] = l;
                if (kInPlace) rank[k] = vrank[q];
                const uint32_t ix = ((l & 1023u) - pass.lo[0]) >> 2, iy = (((l >> 10) & 1023u) - pass.lo[1]) >> 2;
                const uint32_t iz = ((l >> 20) - pass.lo[2]) >> 1;
                key = ix + gx * (iy + gy * iz);
            }
            if (kInPlace) {
                if (q < nv) place = atomicAdd(hist + key, 1u);
            } else {
                // the lanes of a brick are counted at once, by its first lane
                const uint32_t mates = __match_any_sync(0xffffffffu, key);
                const int first = __ffs((int)mates) - 1;
                if (q < nv && lane == first) {
                    place = hist[key];
                    hist[key] = place + __popc(mates);
                }
                place = __shfl_sync(0xffffffffu, place, first) + __popc(mates & ((1u << lane) - 1u));
                __syncwarp();
            }
            at[k] = key | (place << 16);
        }
        __syncwarp();
        // exclusive scan of the bins, lane by lane in blocks of nbins / 32
        const uint32_t per = (nbins + 31u) / 32u, b0 = lane * per, b1 = min(nbins, b0 + per);
        uint32_t tot = 0;
        for (uint32_t b = b0; b < b1; ++b) tot += hist[b];
        uint32_t x = tot;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        uint32_t run = x - tot;
        for (uint32_t b = b0; b < b1; ++b) {
            const uint32_t hcount = hist[b];
            hist[b] = run;
            run += hcount;
        }
        __syncwarp();
#pragma unroll
        for (int k = 0; k < kVerts / 32; ++k) {
            const uint32_t q = lane + 32 * k;
            if (q < nv) {
                const uint32_t to = hist[at[k] & 0xffffu] + (at[k] >> 16);
                if (kInPlace) {
                    vloc[to] = loc[k];
                    vrank[to] = rank[k];
                } else {
                    order[to] = (uint16_t)q;
                }
            }
        }
    } else if (!kInPlace) {
        for (uint32_t q = lane; q < nv; q += 32) order[q] = (uint16_t)q;
    }
    __syncwarp();
#pragma unroll 1
    for (uint32_t t = 0; t < ntiles; ++t) {
        IndexBox tile;
        tile.clear();
        const uint32_t q = 32u * t + (uint32_t)lane;
        if (q < nv) tile.add(vloc[kInPlace ? q : (uint32_t)order[q]]);
        tile.join();
        if (lane == 0) box[2 * t] = tile.low(lo, sc);
        if (lane == 1) box[2 * t + 1] = tile.high(lo, sc);
    }
    __syncwarp();
}

// The band vertices of a group's index box [lo, hi), listed into (vloc,
// vrank) by row segments of at most 32 vertices (two bitset
// words), `per` segments per step so that one step adds at most kVerts
// vertices; pass(count) runs whenever the next step would not fit, and at
// the end.  keep(bits, r0): which of a segment's vertices (the first set bit
// of rank r0) are wanted.
template <int kVerts, class KeepFn, class PassFn>
__device__ __forceinline__ void list_band_vertices(const Grid& sc, const BandView& band, const int lo[3],
                                                   const int hi[3], uint32_t* vloc, uint32_t* vrank, int lane,
                                                   KeepFn&& keep, PassFn&& pass)
{
    const int nx = hi[0] - lo[0], ny = hi[1] - lo[1], nz = hi[2] - lo[2];
    const int nseg = (nx + 31) / 32;
    const int units = ny * nz * nseg;
    const int per = max(1, min(32, kVerts / min(nx, 32)));
    int ub = 0;
    while (ub < units) {
        uint32_t count = 0;
        for (; ub < units; ub += per) {
            const int u = ub + lane;
            uint32_t rm = 0, v0 = 0, r0 = 0;
            int x0 = 0, ry = 0, rz = 0;
            if (lane < per && u < units) {
                const int seg = u % nseg, row = u / nseg;
                x0 = lo[0] + 32 * seg;
                const int wd = min(32, hi[0] - x0);
                ry = lo[1] + row % ny;
                rz = lo[2] + row / ny;
                v0 = lin3(x0, ry, rz, sc);
                const uint32_t w0 = v0 >> 5, sh = v0 & 31u;
                uint64_t bits = __ldg(band.bits + w0);
                if (sh + (uint32_t)wd > 32u) bits |= (uint64_t)__ldg(band.bits + w0 + 1) << 32;
                rm = (uint32_t)(bits >> sh) & (wd >= 32 ? 0xffffffffu : ((1u << wd) - 1u));
                // band rank of v0 (whether or not v0 is in the band); bit b of
                // rm is vertex v0 + b, so its rank adds the set bits below b
                r0 = __ldg(band.prefix + w0) + __popc((uint32_t)bits & ((1u << sh) - 1u));
            }
            const uint32_t all = rm;
            rm = keep(rm, r0);
            const uint32_t n = __popc(rm);
            uint32_t x = n;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
                if (lane >= o) x += y;
            }
            const uint32_t tot = __shfl_sync(0xffffffffu, x, 31);
            // (tot <= kVerts by the choice of `per`: an empty pass always takes the step)
            if (count > 0 && count + tot > (uint32_t)kVerts) break;  // run the pass, then this step again
            uint32_t slot = count + x - n;
            for (uint32_t m = rm; m; m &= m - 1u) {
                const int bx = __ffs(m) - 1;
                vloc[slot] = vert_loc(x0 + bx - lo[0], ry - lo[1], rz - lo[2]);
                vrank[slot++] = r0 + __popc(all & ((1u << bx) - 1u));
            }
            count += tot;
        }
        __syncwarp();
        if (count > 0) pass(count);
    }
}

__device__ __forceinline__ uint32_t keep_all(uint32_t bits, uint32_t) { return bits; }

// The unscaled kernel's part of the field at vertex v, sum_j c_j (1 - |x_j -
// v|^2)^3 over the group's non-involved candidates j, is one polynomial in
// v for the whole group when every candidate is inside the support of every
// vertex (then no term is cut at q2 = 1).  With y_j = x_j - o, z = v - o
// (o: the centre of the group's vertex box), a_j = 1 - |y_j|^2, w = |z|^2:
//   1 - |x_j - v|^2 = (a_j - w) + 2 y_j.z, and the cube of that sums to
//   sum c (a-w)^3 + 6 sum c (a-w)^2 (y.z) + 12 sum c (a-w) (y.z)^2 + 8 sum c (y.z)^3,
// which needs 35 moments of (c, a, y): A_k = sum c a^k (k = 0..3),
// B_k = sum c a^k y (k = 0..2), C_k = sum c a^k y y^T (k = 0, 1) and
// D = sum c y y y.  The expansion holds exactly; it is used when
// max |y| + max |z| < 0.5 (all pairs well inside the unit support, every
// term of order 1, no cancellation), else the candidates are streamed.

struct MomAcc {
    float m[kMoments];
    __device__ __forceinline__ void zero()
    {
#pragma unroll
        for (int k = 0; k < kMoments; ++k) m[k] = 0.f;
    }
    __device__ __forceinline__ void add(float c, float yx, float yy, float yz)
    {
        const float a = 1.0f - fmaf(yx, yx, fmaf(yy, yy, yz * yz));
        const float ca = c * a, ca2 = ca * a;
        m[0] += c;
        m[1] += ca;
        m[2] += ca2;
        m[3] += ca2 * a;
        m[4] = fmaf(c, yx, m[4]);   m[5] = fmaf(c, yy, m[5]);   m[6] = fmaf(c, yz, m[6]);
        m[7] = fmaf(ca, yx, m[7]);  m[8] = fmaf(ca, yy, m[8]);  m[9] = fmaf(ca, yz, m[9]);
        m[10] = fmaf(ca2, yx, m[10]); m[11] = fmaf(ca2, yy, m[11]); m[12] = fmaf(ca2, yz, m[12]);
        const float cx = c * yx, cy = c * yy, cz = c * yz;
        m[13] = fmaf(cx, yx, m[13]); m[14] = fmaf(cy, yy, m[14]); m[15] = fmaf(cz, yz, m[15]);
        m[16] = fmaf(cx, yy, m[16]); m[17] = fmaf(cx, yz, m[17]); m[18] = fmaf(cy, yz, m[18]);
        m[19] = fmaf(cx * a, yx, m[19]); m[20] = fmaf(cy * a, yy, m[20]); m[21] = fmaf(cz * a, yz, m[21]);
        m[22] = fmaf(cx * a, yy, m[22]); m[23] = fmaf(cx * a, yz, m[23]); m[24] = fmaf(cy * a, yz, m[24]);
        const float cxx = cx * yx, cyy = cy * yy, czz = cz * yz;
        m[25] = fmaf(cxx, yx, m[25]);  // xxx
        m[26] = fmaf(cyy, yy, m[26]);  // yyy
        m[27] = fmaf(czz, yz, m[27]);  // zzz
        m[28] = fmaf(cxx, yy, m[28]);  // xxy
        m[29] = fmaf(cxx, yz, m[29]);  // xxz
        m[30] = fmaf(cyy, yx, m[30]);  // xyy
        m[31] = fmaf(cyy, yz, m[31]);  // yyz
        m[32] = fmaf(czz, yx, m[32]);  // xzz
        m[33] = fmaf(czz, yy, m[33]);  // yzz
        m[34] = fmaf(cx * yy, yz, m[34]);  // xyz
    }
    // The warp's sums to out.  32 of the moments are halved from lane to lane: a
    // lane hands over half of what it holds and keeps the sums of the other
    // half, so that 31 shuffles leave one moment per lane (in the order of the
    // pairwise sums of an all-lanes reduction, which takes 160).
    __device__ __forceinline__ void store(float* out, int lane)
    {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const bool up = (lane & o) != 0;
#pragma unroll
            for (int k = 0; k < o; ++k) {
                const float give = up ? m[k] : m[k + o], keep = up ? m[k + o] : m[k];
                m[k] = keep + __shfl_xor_sync(0xffffffffu, give, o);
            }
        }
        out[lane] = m[0];
#pragma unroll
        for (int k = 32; k < kMoments; ++k) {
            float v = m[k];
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
            if (lane == 0) out[k] = v;
        }
    }
};

// The polynomial at z = v - o.
__device__ __forceinline__ float unscaled_sum(const float* m, float zx, float zy, float zz)
{
    const float w = fmaf(zx, zx, fmaf(zy, zy, zz * zz));
    const float t1 = fmaf(w, fmaf(w, fmaf(-w, m[0], 3.0f * m[1]), -3.0f * m[2]), m[3]);
    const float b0 = fmaf(m[4], zx, fmaf(m[5], zy, m[6] * zz));
    const float b1 = fmaf(m[7], zx, fmaf(m[8], zy, m[9] * zz));
    const float b2 = fmaf(m[10], zx, fmaf(m[11], zy, m[12] * zz));
    const float t2 = 6.0f * fmaf(w, fmaf(w, b0, -2.0f * b1), b2);
    const float xx = zx * zx, yy = zy * zy, zz2 = zz * zz, xy = zx * zy, xz = zx * zz, yz = zy * zz;
    const float q0 = fmaf(m[13], xx, fmaf(m[14], yy, fmaf(m[15], zz2, 2.0f * fmaf(m[16], xy, fmaf(m[17], xz, m[18] * yz)))));
    const float q1 = fmaf(m[19], xx, fmaf(m[20], yy, fmaf(m[21], zz2, 2.0f * fmaf(m[22], xy, fmaf(m[23], xz, m[24] * yz)))));
    const float t3 = 12.0f * fmaf(-w, q0, q1);
    const float d3 = fmaf(m[25], xx * zx, fmaf(m[26], yy * zy, m[27] * zz2 * zz));
    const float d21 = fmaf(m[28], xx * zy, fmaf(m[29], xx * zz, fmaf(m[30], yy * zx,
                      fmaf(m[31], yy * zz, fmaf(m[32], zz2 * zx, m[33] * zz2 * zy)))));
    const float t4 = 8.0f * fmaf(6.0f, m[34] * xy * zz, fmaf(3.0f, d21, d3));
    return (t1 + t2) + (t3 + t4);
}

// One warp per window group, groups handed out dynamically; no block-wide
// barriers.  The warp walks the group's index box 32 vertices at a time and
// collects up to 256 band vertices per pass (8 tiles of 32).  Per pass it
// streams the window's candidates 32 at a time: each lane loads one
// candidate's record into the warp's shared-memory slice once (candidates
// that reach none of the pass's tiles are dropped first), then for every
// tile the warp keeps the candidates whose support sphere reaches the
// tile's box and each lane adds their terms for its vertex of that tile.
// A vertex's sum takes the candidates in window order.
__global__ void __launch_bounds__(kFT, FSR_FIELD_MIN_BLOCKS) k_field_aniso_grouped(GroupArgs a, uint32_t ratio, Counters* ctr)
{
    after_launch();
    __shared__ WarpSlice slices[kFWarps];
    const int lane = threadIdx.x & 31;
    WarpSlice& w = slices[threadIdx.x >> 5];
    const uint32_t nb = min(ctr->n_band, a.cap);
    const GroupList groups(a.glist, a.sp, ctr);
    const uint32_t ngroups = groups.size();
    const uint32_t nslab = field_slabs(ngroups);
    const uint32_t dense = groups.dense * nslab, sparse = groups.sparse * nslab;
    const uint32_t split = min(dense, kSplitItems), whole = dense - split;

    for (;;) {
        uint32_t k = 0;
        if (lane == 0) k = atomicAdd(&ctr->work_field, 1u);
        k = __shfl_sync(0xffffffffu, k, 0);
        if (k >= whole + 2u * split + sparse) break;
        // a work item takes every nsub-th tile of its slab's passes
        uint32_t nsub = 1u, sub = 0u, slab = k;
        if (k >= whole + 2u * split) {
            slab = k - split;
        } else if (k >= whole) {
            nsub = 2u;
            sub = (k - whole) & 1u;
            slab = whole + ((k - whole) >> 1);
        }
        const uint32_t g = groups[slab / nslab];
        int c[3], lo[3], hi[3];
        if (!group_box(g, a.sp, a.sc, ratio, c, lo, hi) || !slab_box(slab % nslab, nslab, lo, hi)) continue;
        bool tables = false;
        uint32_t total = 0;

        auto pass = [&](uint32_t nv) {
            const uint32_t ntiles = (nv + 31) / 32;
            if (sub >= ntiles) return;
            if (!tables) {
                const float b0[3] = {vpos1(lo[0], a.sc.min[0], a.sc.cs), vpos1(lo[1], a.sc.min[1], a.sc.cs),
                                     vpos1(lo[2], a.sc.min[2], a.sc.cs)};
                const float b1[3] = {vpos1(hi[0] - 1, a.sc.min[0], a.sc.cs), vpos1(hi[1] - 1, a.sc.min[1], a.sc.cs),
                                     vpos1(hi[2] - 1, a.sc.min[2], a.sc.cs)};
                total = warp_candidates(a.sp, a.ranges, a.invol, a.reach, c, b0, b1, w);
                tables = true;
                // moments of the non-involved candidates about the box centre
                const float ox = 0.5f * (b0[0] + b1[0]), oy = 0.5f * (b0[1] + b1[1]), oz = 0.5f * (b0[2] + b1[2]);
                const float hx = 0.5f * (b1[0] - b0[0]), hy = 0.5f * (b1[1] - b0[1]), hz = 0.5f * (b1[2] - b0[2]);
                // (a group without such candidates has no unscaled part)
                if (total > w.total_inv) {
                    MomAcc acc;
                    acc.zero();
                    float y2max = 0.f;
                    const CandTables tabs{w.cstart, w.cpre, w.cinv};
                    for (uint32_t j = w.total_inv + lane; j < total; j += 32) {
                        int cell;
                        const uint32_t i = candidate(j, tabs, &cell, (int)w.ncells);
                        const float4 sm = __ldg(&a.smoothed[i]);
                        const float yx = sm.x - ox, yy = sm.y - oy, yz = sm.z - oz;
                        y2max = fmaxf(y2max, fmaf(yx, yx, fmaf(yy, yy, yz * yz)));
                        acc.add(a.sigma * sm.w, yx, yy, yz);
                    }
                    acc.store(w.mom, lane);
#pragma unroll
                    for (int o = 16; o > 0; o >>= 1) y2max = fmaxf(y2max, __shfl_xor_sync(0xffffffffu, y2max, o));
                    const float zmax = sqrtf(fmaf(hx, hx, fmaf(hy, hy, hz * hz)));
                    if (lane == 0) w.use_mom = (sqrtf(y2max) + zmax) * 1.001f < 0.5f ? 1u : 0u;
                }
                __syncwarp();
            }
            // the pass's box, brick order and tile boxes
            float4 pl, ph;
            pass_layout<false>(w.vloc, w.vrank, lo, a.sc, w.order, reinterpret_cast<uint32_t*>(&w.psum[0][0]), w.box, nv, lane, pl, ph);  // psum is zeroed below
            // two sums per vertex: the involved particles' terms, then the
            // non-involved particles' (the unscaled kernel: about 1e-7 each,
            // thousands of them) and the rounding errors of the first sum,
            // added among themselves and joined at the end, so that FP32
            // rounding does not drop or inflate them against a sum of order 1
            // the sums live in the warp's shared slice, so that the tile loops
            // need not be unrolled (the kernel's code stays small enough for
            // the instruction cache)
            for (uint32_t t = sub; t < ntiles; t += nsub) w.psum[t][lane] = w.usum[t][lane] = 0.f;
            const uint32_t total_inv = w.total_inv;
            // involved candidates: staged with their G, culled per tile by
            // their support sphere, evaluated two at a time
            uint32_t k0 = 0;
            for (uint32_t cb = 0; cb < total_inv; cb += 32) {
                const uint32_t j = cb + lane;
                bool keep = false;
                float4 r0 = make_float4(0.f, 0.f, 0.f, -1.f);
                const int cell = chunk_cell(cb, lane, w.cpre, w.ncells, k0);
                if (j < total_inv) {
                    const uint32_t i = w.cstart[cell] + (j - w.cpre[cell]);
                    // the three loads in flight together (most candidates are kept)
                    const float4* qsrc = a.qrec + 3ull * i;
                    r0 = __ldg(qsrc);
                    const float4 r1 = __ldg(qsrc + 1), r2 = __ldg(qsrc + 2);
                    keep = reaches(r0, pl, ph);
                    if (keep) stage_record(reinterpret_cast<float2*>(w.rec), lane, r0, r1, r2);
                }
                const uint32_t any = __ballot_sync(0xffffffffu, keep);
                __syncwarp();
                if (any) {
#pragma unroll 1
                    for (uint32_t t = sub; t < ntiles; t += nsub) {
                        const uint32_t m = __ballot_sync(0xffffffffu, keep && reaches(r0, w.box[2 * t], w.box[2 * t + 1]));
                        if (m) {
                            // the candidates that reach the tile, listed in
                            // lane order two to a pair block
                            if ((m >> lane) & 1u)
                                list_pair_record(reinterpret_cast<const float2*>(w.rec), lane,
                                                 reinterpret_cast<float*>(w.lst), __popc(m & ((1u << lane) - 1u)));
                            // the other half of a last single: zeros, which add 0
                            if ((__popc(m) & 1) && lane < 10)
                                reinterpret_cast<float*>(w.lst)[(__popc(m) >> 1) * (4 * kPairF4) + 1 + 2 * lane] = 0.f;
                            __syncwarp();
                            const uint32_t v = 32 * t + lane;
                            if (v < nv) {
                                const float4 vp = vert_pos(w.vloc[w.order[v]], lo, a.sc);
                                // the chunk's terms are summed on their own and
                                // then added to the vertex's sum with the
                                // rounding error of that addition (two-sum)
                                // kept in the second sum: with tens of
                                // thousands of neighbours one running FP32 sum
                                // drifts by more than 1e-5 of the field
                                float s = 0.f;
                                // one pair block per step, both candidates
                                // evaluated at once by packed operations; the
                                // terms of vertices inside the support enter
                                // the sum in list (lane) order
                                const float2 nvx = make_float2(-vp.x, -vp.x), nvy = make_float2(-vp.y, -vp.y),
                                             nvz = make_float2(-vp.z, -vp.z);
                                const uint32_t cnt = __popc(m);
                                // (two copies: 8M particles 9.36 -> 9.21 ms; three
                                // crowd the instruction cache: 9.62)
#pragma unroll 2
                                for (uint32_t j = 0; j < cnt; j += 2) {
                                    float2 q2, u3, c;
                                    pair_terms(w.lst + (j >> 1) * kPairF4, nvx, nvy, nvz, q2, u3, c);
                                    if (q2.x < 1.0f) s = fmaf(c.x, u3.x, s);
                                    if (q2.y < 1.0f) s = fmaf(c.y, u3.y, s);
                                }
                                const float a0 = w.psum[t][lane];
                                const float t0 = a0 + s;
                                const float bp = t0 - a0;
                                w.psum[t][lane] = t0;
                                w.usum[t][lane] += (a0 - (t0 - bp)) + (s - bp);
                            }
                            __syncwarp();
                        }
                    }
                }
                __syncwarp();
            }
            // non-involved candidates: G = I and support 1 (world units), which
            // reaches every vertex of the window.  Their sum is the group's
            // moment polynomial when it applies; else they are streamed: only
            // the position and the coefficient sigma m / rho are staged, and
            // q2 is |x~ - v|^2
            const bool use_mom = total > total_inv && w.use_mom != 0u;
            if (use_mom) {
                const float ox = 0.5f * (vpos1(lo[0], a.sc.min[0], a.sc.cs) + vpos1(hi[0] - 1, a.sc.min[0], a.sc.cs));
                const float oy = 0.5f * (vpos1(lo[1], a.sc.min[1], a.sc.cs) + vpos1(hi[1] - 1, a.sc.min[1], a.sc.cs));
                const float oz = 0.5f * (vpos1(lo[2], a.sc.min[2], a.sc.cs) + vpos1(hi[2] - 1, a.sc.min[2], a.sc.cs));
#pragma unroll 1
                for (uint32_t t = sub; t < ntiles; t += nsub) {
                    const uint32_t v = 32 * t + lane;
                    if (v < nv) {
                        const float4 vp = vert_pos(w.vloc[w.order[v]], lo, a.sc);
                        w.usum[t][lane] += unscaled_sum(w.mom, vp.x - ox, vp.y - oy, vp.z - oz);
                    }
                }
            }
            k0 = w.ninv_cells;
            for (uint32_t cb = use_mom ? total : total_inv; cb < total; cb += 32) {
                const uint32_t j = cb + lane;
                const int cell = chunk_cell(cb, lane, w.cpre, w.ncells, k0);
                if (j < total) {
                    const uint32_t i = w.cstart[cell] + (j - w.cpre[cell]);
                    const float4 sm = __ldg(&a.smoothed[i]);
                    w.rec[lane] = make_float4(sm.x, sm.y, sm.z, a.sigma * sm.w);
                }
                const uint32_t cnt = min(32u, total - cb);
                __syncwarp();
#pragma unroll 1
                for (uint32_t t = sub; t < ntiles; t += nsub) {
                    const uint32_t v = 32 * t + lane;
                    if (v < nv) {
                        const float4 vp = vert_pos(w.vloc[w.order[v]], lo, a.sc);
                        float su = 0.f;  // the chunk's terms, as for the involved candidates
                        uint32_t k = 0;
                        for (; k + 2 <= cnt; k += 2) {
                            const float4 qa = w.rec[k], qb = w.rec[k + 1];
                            const float ax = qa.x - vp.x, ay = qa.y - vp.y, az = qa.z - vp.z;
                            const float bx = qb.x - vp.x, by = qb.y - vp.y, bz = qb.z - vp.z;
                            const float q2a = fmaf(ax, ax, fmaf(ay, ay, az * az));
                            const float q2b = fmaf(bx, bx, fmaf(by, by, bz * bz));
                            const float ua = 1.0f - q2a, ub = 1.0f - q2b;
                            if (q2a < 1.0f) su = fmaf(qa.w, ua * ua * ua, su);
                            if (q2b < 1.0f) su = fmaf(qb.w, ub * ub * ub, su);
                        }
                        if (k < cnt) {
                            const float4 qa = w.rec[k];
                            const float ax = qa.x - vp.x, ay = qa.y - vp.y, az = qa.z - vp.z;
                            const float q2a = fmaf(ax, ax, fmaf(ay, ay, az * az));
                            const float ua = 1.0f - q2a;
                            if (q2a < 1.0f) su = fmaf(qa.w, ua * ua * ua, su);
                        }
                        w.usum[t][lane] += su;
                    }
                }
                __syncwarp();
            }
            for (uint32_t t = sub; t < ntiles; t += nsub) {
                const uint32_t v = 32 * t + lane;
                if (v < nv) {
                    const uint32_t rank = w.vrank[w.order[v]];
                    if (rank < nb) a.phi[rank] = (w.psum[t][lane] + w.usum[t][lane]) - 0.5f;
                }
            }
            __syncwarp();
        };

        list_band_vertices<kPassVerts>(a.sc, a.band, lo, hi, w.vloc, w.vrank, lane, keep_all, pass);
        __syncwarp();
    }
}

// ---------------------------------------------------------------- ZB05 / TC01
// updateScalarFieldValueZB05 (cu:230-289) and updateScalarFieldValueTC01
// (cu:178-227) grouped like the anisotropic field: a band vertex's
// candidates are the particles of the +-1 cells around its cell, the same for
// every vertex of the cell.  One warp streams them once per pass of up to 256
// vertices, stages up to kIsoSeg of those within h of the pass's box and then
// goes through the brick tiles: the ones within h of the tile are listed two to
// a pair and every lane evaluates one pair per step.  (Issue-bound: 29.8 of 32
// threads per instruction, 70 % of the issue slots.  Tiles inside the chunk of
// 32 candidates, as before, cost each tile its vertices' positions and sums, a
// list and a half-empty pair per chunk: 910 -> 637 M instructions and 1.07 ->
// 0.81 ms on the 256k Akinci12 frame; 1.10 -> 0.85 ms on the 1M ZB05 frame.)  Each vertex sums its terms in window order (cells z, y, x,
// particles in sorted order); candidates of the window cells the per-vertex
// walk narrows away lie beyond h and add nothing.
// Candidates staged at a time: with 120 six blocks fit an SM (64: 1.07 -> 0.88
// ms instead of 0.81 on the 256k Akinci12 frame; 128, five blocks: 0.81, but
// 0.88 instead of 0.85 on the 1M ZB05 frame, of small groups).
constexpr uint32_t kIsoSeg = 120;
struct IsoSlice {
    float4 lxy[kIsoSeg / 2];       // one tile's candidates in order, two to a pair: (x, x', y, y')
    float2 lz[kIsoSeg / 2];        // and (z, z')
    float cx[kIsoSeg], cy[kIsoSeg], cz[kIsoSeg];  // the staged candidates
    uint32_t vloc[kPassVerts];     // the pass's band vertices in brick order: index in the group's box (vert_loc)
    uint32_t vrank[kPassVerts];    // and band rank
    float4 box[2 * kPassTiles];    // per tile: lo, hi
    float sum[4][kPassTiles][32];  // per vertex: weight sum, then (ZB05) sum w (x - v)
    uint32_t rb[9], rp[10];        // the window's rows: first particle, prefix of lengths
};

// The rows of the +-1 window around cell c (clamped as window() clamps), z then
// y: first particles rb[9] and the prefix of their lengths rp[10]; returns the
// number of particles.  Every lane of the warp calls it.
__device__ __forceinline__ uint32_t window_rows(const Grid& sp, const uint2* __restrict__ ranges, const int c[3],
                                                uint32_t* rb, uint32_t* rp, int lane)
{
    uint32_t beg = kEmpty, end = 0;
    if (lane < 9) {
        const int x0 = clampi(c[0] - 1, 0, (int)sp.res[0] - 1), x1 = clampi(c[0] + 1, 0, (int)sp.res[0] - 1);
        const int y0 = clampi(c[1] - 1, 0, (int)sp.res[1] - 1), y1 = clampi(c[1] + 1, 0, (int)sp.res[1] - 1);
        const int z0 = clampi(c[2] - 1, 0, (int)sp.res[2] - 1), z1 = clampi(c[2] + 1, 0, (int)sp.res[2] - 1);
        const int yy = y0 + lane % 3, zz = z0 + lane / 3;
        if (yy <= y1 && zz <= z1) {
            const uint32_t c0 = lin3(x0, yy, zz, sp);
            for (int xx = 0; xx <= x1 - x0; ++xx) {
                const uint2 r = __ldg(&ranges[c0 + xx]);
                if (r.x != kEmpty) {
                    beg = min(beg, r.x);
                    end = max(end, r.y);
                }
            }
        }
    }
    const uint32_t len = end > beg ? end - beg : 0u;
    uint32_t x = len;
#pragma unroll
    for (int o = 1; o < 16; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane < 9) {
        rb[lane] = beg;
        rp[lane] = x - len;
    }
    if (lane == 8) rp[9] = x;
    __syncwarp();
    return __shfl_sync(0xffffffffu, x, 8);
}

__device__ __forceinline__ bool within(float4 q, float4 lo, float4 hi, float r2)
{
    const float gx = fmaxf(0.f, fmaxf(lo.x - q.x, q.x - hi.x));
    const float gy = fmaxf(0.f, fmaxf(lo.y - q.y, q.y - hi.y));
    const float gz = fmaxf(0.f, fmaxf(lo.z - q.z, q.z - hi.z));
    return fmaf(gx, gx, fmaf(gy, gy, gz * gz)) < r2;
}

template <bool TC01>
__global__ void __launch_bounds__(kFT, 6) k_field_iso_grouped(IsoFieldArgs a, BandView band, uint32_t ratio, Counters* ctr)
{
    after_launch();
    __shared__ IsoSlice slices[kFWarps];
    const int lane = threadIdx.x & 31;
    IsoSlice& w = slices[threadIdx.x >> 5];
    const uint32_t nb = min(ctr->n_band, a.cap);
    const GroupList groups(a.glist, a.sp, ctr);
    const uint32_t ngroups = groups.size();
    const uint32_t nslab = field_slabs(ngroups);
    const float cr = cull_radius(a.h, a.sp.cs), cr2 = cr * cr;
    constexpr int kSums = TC01 ? 1 : 4;

    for (;;) {
        uint32_t k = 0;
        if (lane == 0) k = atomicAdd(&ctr->work_field, 1u);
        k = __shfl_sync(0xffffffffu, k, 0);
        if (k >= ngroups * nslab) break;
        const uint32_t g = groups[k / nslab];
        int c[3], lo[3], hi[3];
        if (!group_box(g, a.sp, a.sc, ratio, c, lo, hi) || !slab_box(k % nslab, nslab, lo, hi)) continue;
        const uint32_t total = window_rows(a.sp, a.ranges, c, w.rb, w.rp, lane);

        auto pass = [&](uint32_t nv) {
            float4 pl, ph;
            pass_layout<true>(w.vloc, w.vrank, lo, a.sc, nullptr, reinterpret_cast<uint32_t*>(&w.sum[0][0][0]), w.box, nv, lane, pl, ph);  // the sums are zeroed next
            const uint32_t ntiles = (nv + 31) / 32;
            for (int k = 0; k < kSums; ++k)
                for (uint32_t t = 0; t < ntiles; ++t) w.sum[k][t][lane] = 0.f;
            __syncwarp();
            // a candidate's place in the list: two to a pair
            auto list = [&](const float4& q, uint32_t pos) {
                float* d = reinterpret_cast<float*>(w.lxy + (pos >> 1)) + (pos & 1u);
                d[0] = q.x;
                d[2] = q.y;
                reinterpret_cast<float*>(w.lz)[pos] = q.z;
            };
            // the listed candidates [0, cnt) for tile t: each lane takes one pair
            // per step for its vertex, in order
            auto evaluate = [&](uint32_t t, uint32_t cnt) {
                if ((cnt & 1u) && lane == 0) {  // the last pair's other half: beyond h of everything
                    float* d = reinterpret_cast<float*>(w.lxy + (cnt >> 1)) + 1;
                    d[0] = d[2] = reinterpret_cast<float*>(w.lz)[cnt] = 1.0e18f;
                }
                __syncwarp();
                const uint32_t v = 32 * t + lane;
                if (v < nv) {
                    const float4 vp = vert_pos(w.vloc[v], lo, a.sc);
                    float ws = w.sum[0][t][lane];
                    float ax = 0.f, ay = 0.f, az = 0.f;
                    if (!TC01) {
                        ax = w.sum[1][t][lane];
                        ay = w.sum[2][t][lane];
                        az = w.sum[3][t][lane];
                    }
                    const float2 nvx = make_float2(-vp.x, -vp.x), nvy = make_float2(-vp.y, -vp.y),
                                 nvz = make_float2(-vp.z, -vp.z);
                    const float2 ninv = make_float2(-a.inv_h2, -a.inv_h2), one = make_float2(1.0f, 1.0f);
                    const uint32_t pairs = (cnt + 1) >> 1;
                    // (two copies: 0.90 -> 0.82 ms on the 256k Akinci12 frame;
                    // four crowd the instruction cache: 0.90)
#pragma unroll 2
                    for (uint32_t j = 0; j < pairs; ++j) {
                        const float4 A = w.lxy[j];
                        const float2 dx = __fadd2_rn(make_float2(A.x, A.y), nvx);
                        const float2 dy = __fadd2_rn(make_float2(A.z, A.w), nvy);
                        const float2 dz = __fadd2_rn(w.lz[j], nvz);
                        const float2 d2 = __ffma2_rn(dx, dx, __ffma2_rn(dy, dy, __fmul2_rn(dz, dz)));
                        if (TC01) {
                            const float ua = d2.x * a.inv_h2 * 0.5f, ub = d2.y * a.inv_h2 * 0.5f;
                            const float ta = ua * ua - ua + 0.25f, tb = ub * ub - ub + 0.25f;
                            if (d2.x <= a.h2) ws += ta;
                            if (d2.y <= a.h2) ws += tb;
                        } else {
                            const float2 u = __ffma2_rn(d2, ninv, one);
                            const float2 u2 = __fmul2_rn(u, u);
                            const float2 wt = __fmul2_rn(u2, u);
                            if (d2.x < a.h2) {
                                ws = ws + wt.x;
                                ax = fmaf(dx.x, wt.x, ax);
                                ay = fmaf(dy.x, wt.x, ay);
                                az = fmaf(dz.x, wt.x, az);
                            }
                            if (d2.y < a.h2) {
                                ws = ws + wt.y;
                                ax = fmaf(dx.y, wt.y, ax);
                                ay = fmaf(dy.y, wt.y, ay);
                                az = fmaf(dz.y, wt.y, az);
                            }
                        }
                    }
                    w.sum[0][t][lane] = ws;
                    if (!TC01) {
                        w.sum[1][t][lane] = ax;
                        w.sum[2][t][lane] = ay;
                        w.sum[3][t][lane] = az;
                    }
                }
                __syncwarp();  // the list is rewritten next
            };
            // the staged candidates [0, fill) against every tile: the ones within
            // h of the tile are listed and evaluated; with one tile, whose box is
            // the pass's, the candidates are listed as they are staged
            uint32_t fill = 0;
            const bool one_tile = ntiles == 1u;
            auto tiles = [&]() {
                if (one_tile) {
                    evaluate(0, fill);
                    fill = 0;
                    return;
                }
                __syncwarp();
#pragma unroll 1
                for (uint32_t t = 0; t < ntiles; ++t) {
                    const float4 tl = w.box[2 * t], th = w.box[2 * t + 1];
                    uint32_t cnt = 0;
                    for (uint32_t b = 0; b < fill; b += 32) {
                        const uint32_t i = b + (uint32_t)lane;
                        float4 q = make_float4(0.f, 0.f, 0.f, 0.f);
                        if (i < fill) {
                            q.x = w.cx[i];
                            q.y = w.cy[i];
                            q.z = w.cz[i];
                        }
                        const bool in = i < fill && within(q, tl, th, cr2);
                        const uint32_t m = __ballot_sync(0xffffffffu, in);
                        if (in) list(q, cnt + __popc(m & ((1u << lane) - 1u)));
                        cnt += __popc(m);
                    }
                    if (cnt != 0u) evaluate(t, cnt);
                }
                fill = 0;
            };
            int row = 0;
            for (uint32_t cb = 0; cb < total; cb += 32) {
                const uint32_t j = cb + lane;
                bool keep = false;
                float4 q = make_float4(0.f, 0.f, 0.f, 0.f);
                if (j < total) {
                    while (row < 8 && w.rp[row + 1] <= j) ++row;
                    q = __ldg(&a.sorted[w.rb[row] + (j - w.rp[row])]);
                    keep = within(q, pl, ph, cr2);
                }
                const uint32_t m = __ballot_sync(0xffffffffu, keep);
                if (keep) {
                    const uint32_t pos = fill + __popc(m & ((1u << lane) - 1u));
                    if (one_tile) {
                        list(q, pos);
                    } else {
                        w.cx[pos] = q.x;
                        w.cy[pos] = q.y;
                        w.cz[pos] = q.z;
                    }
                }
                fill += __popc(m);
                if (fill > kIsoSeg - 32) tiles();
            }
            if (fill) tiles();
            __syncwarp();
            for (int t = 0; t < (int)ntiles; ++t) {
                const uint32_t v = 32 * t + lane;
                if (v < nv) {
                    const uint32_t rank = w.vrank[v];
                    if (rank < nb) {
                        const float ws = w.sum[0][t][lane];
                        if (TC01) {
                            a.phi[rank] = ws;
                        } else {
                            const float ax = w.sum[1][t][lane], ay = w.sum[2][t][lane], az = w.sum[3][t][lane];
                            // |v - sum w p / sum w| = |sum w (p - v)| / sum w; a vertex with no
                            // weight keeps 0, the reference's memset value (cu:284)
                            a.phi[rank] = ws > 0.f ? sqrtf(fmaf(ax, ax, fmaf(ay, ay, az * az))) / ws - a.rp : 0.f;
                            if (a.mv) {
                                const float inv = ws > 0.f ? 1.0f / ws : 0.f;
                                a.mv[rank] = make_float4(ax * inv, ay * inv, az * inv, ws);
                            }
                        }
                    }
                }
            }
            __syncwarp();
        };
        list_band_vertices<kPassVerts>(a.sc, band, lo, hi, w.vloc, w.vrank, lane, keep_all, pass);
        __syncwarp();
    }
}

// ---------------------------------------------------------------- adjoint
struct BwdGroupArgs {
    Grid sp, sc;
    BandView band;
    const float4* grec;
    const float4* qrec;
    const float4* smoothed;
    const uint2* ranges;
    const uint8_t* invol;
    const float* reach;
    const float* gphi;
    uint32_t* glist;
    float4* gsmooth;
    float4* gG;
    float sigma;
    uint32_t cap;
};

// Adjoint of the ZB05 / TC01 fields (updateScalarFieldValueZB05 cu:230-289,
// TC01 cu:178-227), grouped like the forward field with the roles swapped: a
// warp takes a group (or a z slab of it), lists the vertices with dL/dphi != 0 in
// brick tiles, stages the window's particles within h of their box, and per tile
// gives the particles within h of the tile one lane each; a lane walks the
// tile's vertices two at a time with packed FP32x2 operations (the clamp of 1 -
// d^2/h^2 at 0 drops the ones beyond h) and adds its sums to the particle's in
// shared memory; one float4 atomic per particle and segment ends it.
//   ZB05: phi = |xbar - v| - r_p; with e = (xbar - v) dL/dphi / (|xbar - v| W) per
//   vertex, dL/dx_j += w e + (e.d - e.(xbar - v)) (-6 u^2 / h^2) d, d = x_j - v,
//   u = 1 - d^2/h^2, w = u^3
//   TC01: phi = sum t^2 - t + 1/4, t = d^2 / 2h^2: dL/dx_j += dL/dphi (2t - 1) / h^2 d
// (A block per group, whose eight warps met at five barriers per group, spent
// most of its time waiting there; 500k-particle ZB05 frame: 0.67 -> 0.17 ms.)
constexpr int kBwdVerts = 128;        // vertices of a pass
constexpr float kFinite = 3.0e38f;    // larger factors are taken as not finite
constexpr uint32_t kBwdSeg = 96;      // particles staged at a time
// Its work items.  Few groups are cut into more of them: on fine grids by slabs of
// vertices, on coarse ones (up to 4 vertices per cell: two to five slabs at most) by
// runs of candidates; crowded groups (kCrowdedGroup) are shared in runs of candidates
// on all grids, however many groups there are.  Backward, us, block per group / a warp
// per group or slab / now: default grid, ZB05: 20k-particle block 50 / 66 / 46, 30k at 140
// a cell 57 / 97 / 47, 1M at 200 a cell 122 / 160 / 118; TC01, 300k at 1000 a cell 82 /
// 166 / 55; 90k ZB05 particles of which 85k lie in a few cells, default grid 419 / 2380 /
// 371, fine 2330 / 5990 / 541.  Frames without such groups: 500k fine 907 / 396 / 398.
constexpr uint32_t kCrowdParts = 64, kPartCandidates = 128;
__device__ __forceinline__ uint32_t crowd_parts(uint32_t ncrowd)
{
    return min(kCrowdParts, (kSlabTarget + ncrowd) / max(ncrowd, 1u));
}

template <bool TC01>
struct IsoBwdSlice {
    float4 vxy[kBwdVerts / 2];                // the pass's vertices two to a pair: (x, x', y, y')
    float2 vz[kBwdVerts / 2];                 // (z, z')
    float4 exy[TC01 ? 1 : kBwdVerts / 2];     // ZB05: e of the two, (ex, ex', ey, ey')
    float4 ezw[TC01 ? 1 : kBwdVerts / 2];     // (ez, ez', e.(xbar - v), ...')
    float2 g[TC01 ? kBwdVerts / 2 : 1];       // TC01: dL/dphi of the two
    uint32_t vloc[kBwdVerts], vrank[kBwdVerts];
    uint32_t hist[kBwdVerts];
    float4 box[2 * (kBwdVerts / 32)];
    float cx[kBwdSeg], cy[kBwdSeg], cz[kBwdSeg];  // the staged particles
    float gx[kBwdSeg], gy[kBwdSeg], gz[kBwdSeg];  // their dL/dx
    uint32_t cj[kBwdSeg];                         // their sorted index
    uint32_t list[kBwdSeg];                       // those within h of the tile
    uint32_t nodd;                                // vertices that are not finite, listed in hist
    uint32_t rb[9], rp[10];
};

template <bool TC01>
__global__ void __launch_bounds__(kFT, 6) k_field_iso_backward(BwdArgs a, const Counters* ctr)
{
    after_launch();
    __shared__ IsoBwdSlice<TC01> slices[kFWarps];
    const int lane = threadIdx.x & 31;
    IsoBwdSlice<TC01>& w = slices[threadIdx.x >> 5];
    const uint32_t nb = min(ctr->n_band, a.cap_band);
    const BwdGroupList groups(a.glist, a.sp);
    const uint32_t ncrowd = groups.crowded(), cparts = crowd_parts(ncrowd);
    const uint32_t nusual = groups.usual(), nsub = field_slabs(nusual);
    const float h2 = a.h * a.h, inv_h2 = 1.0f / h2;
    const float cr = cull_radius(a.h, a.sp.cs), cr2 = cr * cr;
    const float2 inv2 = make_float2(inv_h2, inv_h2), ninv2 = make_float2(-inv_h2, -inv_h2);
    const float2 one2 = make_float2(1.0f, 1.0f), mone2 = make_float2(-1.0f, -1.0f);

    for (;;) {
        uint32_t k = 0;
        if (lane == 0) k = atomicAdd(&a.glist[2], 1u);
        k = __shfl_sync(0xffffffffu, k, 0);
        if (k >= ncrowd * cparts + nusual * nsub) break;
        const bool crowd = k < ncrowd * cparts;
        const uint32_t item = crowd ? k : k - ncrowd * cparts, cut = crowd ? cparts : nsub;
        const bool by_slab = !crowd && a.ratio > 4;
        int c[3], lo[3], hi[3];
        if (!group_box(groups.at((crowd ? 0u : ncrowd) + item / cut, ncrowd), a.sp, a.sc, a.ratio, c, lo, hi) ||
            (by_slab && !slab_box(item % cut, cut, lo, hi)))
            continue;
        uint32_t begin = 0, total = window_rows(a.sp, a.ranges, c, w.rb, w.rp, lane);  // the item's candidates
        if (!by_slab && cut > 1u) {
            const uint32_t step = max(kPartCandidates, (total / cut + 32u) & ~31u);
            begin = (item % cut) * step;
            if (begin >= total) continue;
            total = min(total, begin + step);
        }

        auto pass = [&](uint32_t nv) {
            float4 pl, ph;
            pass_layout<true, kBwdVerts>(w.vloc, w.vrank, lo, a.sc, nullptr, w.hist, w.box, nv, lane, pl, ph);
            const uint32_t ntiles = (nv + 31) / 32;
            // the vertices' positions and factors; the places up to the last
            // tile's end lie beyond h of everything.  Vertices whose factors are not
            // finite are set apart (odd_vertices)
            uint32_t nodd = 0;
            for (uint32_t q = lane; q < 32u * ntiles; q += 32) {
                float4 vp = make_float4(1.0e18f, 1.0e18f, 1.0e18f, 0.f);
                float4 e = make_float4(0.f, 0.f, 0.f, 0.f);
                float gv = 0.f;
                if (q < nv) {
                    vp = vert_pos(w.vloc[q], lo, a.sc);
                    const uint32_t rank = w.vrank[q];
                    gv = __ldg(a.gphi + rank);
                    if (!TC01) {
                        const float4 m = __ldg(a.mv + rank);  // mean - v, weight sum
                        const float ml = sqrtf(fmaf(m.x, m.x, fmaf(m.y, m.y, m.z * m.z)));
                        if (m.w > 0.f && ml > 0.f) {
                            const float f = gv / ml / m.w;
                            e = make_float4(m.x * f, m.y * f, m.z * f, 0.f);
                            e.w = fmaf(e.x, m.x, fmaf(e.y, m.y, e.z * m.z));
                        }
                    }
                }
                const bool odd = !(fabsf(TC01 ? gv : (e.x + e.y) + (e.z + e.w)) <= kFinite);
                const uint32_t om = __ballot_sync(0xffffffffu, odd);
                if (odd) {
                    w.hist[nodd + __popc(om & ((1u << lane) - 1u))] = q;
                    gv = 0.f;
                    e = make_float4(0.f, 0.f, 0.f, 0.f);
                }
                nodd += __popc(om);
                const uint32_t p = q >> 1, s = q & 1u;
                float* d = reinterpret_cast<float*>(w.vxy + p) + s;
                d[0] = vp.x;
                d[2] = vp.y;
                reinterpret_cast<float*>(w.vz)[q] = vp.z;
                if (TC01) {
                    reinterpret_cast<float*>(w.g)[q] = gv;
                } else {
                    d = reinterpret_cast<float*>(w.exy + p) + s;
                    d[0] = e.x;
                    d[2] = e.y;
                    d = reinterpret_cast<float*>(w.ezw + p) + s;
                    d[0] = e.z;
                    d[2] = e.w;
                }
            }
            if (lane == 0) w.nodd = nodd;
            __syncwarp();
            uint32_t fill = 0;
            // The clamp in the pair loop would let a vertex that is not finite reach
            // every particle of its tile (0 x inf): these take the range test, and reach
            // the staged particles within h of them only.  (The test in the pair loop
            // of passes that need it, a second copy of the loop: 500k ZB05 frame's
            // backward 397 -> 409 us without such a vertex; this way 401 -> 404.)
            auto odd_vertices = [&]() {
#pragma unroll 1
                for (uint32_t o = 0; o < w.nodd; ++o) {
                    const uint32_t q = w.hist[o], rank = w.vrank[q];
                    const float4 vp = vert_pos(w.vloc[q], lo, a.sc);
                    const float gv = __ldg(a.gphi + rank);
#pragma unroll 1
                    for (uint32_t i = lane; i < fill; i += 32) {
                        const float dx = w.cx[i] - vp.x, dy = w.cy[i] - vp.y, dz = w.cz[i] - vp.z;
                        const float d2 = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
                        if (!(d2 < h2)) continue;
                        float sx = 0.f, sy = 0.f, sz = 0.f, k = gv * (d2 * inv_h2 - 1.0f) * inv_h2;
                        if (!TC01) {
                            const float4 m = __ldg(a.mv + rank);
                            const float f = gv / sqrtf(fmaf(m.x, m.x, fmaf(m.y, m.y, m.z * m.z))) / m.w;
                            const float u = 1.0f - d2 * inv_h2, wt = u * u * u;
                            sx = wt * (f * m.x);
                            sy = wt * (f * m.y);
                            sz = wt * (f * m.z);
                            k = f * (m.x * (dx - m.x) + m.y * (dy - m.y) + m.z * (dz - m.z)) * (-6.0f * u * u * inv_h2);
                        }
                        w.gx[i] += fmaf(k, dx, sx);
                        w.gy[i] += fmaf(k, dy, sy);
                        w.gz[i] += fmaf(k, dz, sz);
                    }
                }
                __syncwarp();
            };
            auto tiles = [&]() {
                for (uint32_t i = lane; i < fill; i += 32) w.gx[i] = w.gy[i] = w.gz[i] = 0.f;
                __syncwarp();
#pragma unroll 1
                for (uint32_t t = 0; t < ntiles; ++t) {
                    const float4 tl = w.box[2 * t], th = w.box[2 * t + 1];
                    uint32_t cnt = 0;
                    for (uint32_t b = 0; b < fill; b += 32) {
                        const uint32_t i = b + (uint32_t)lane;
                        bool in = false;
                        if (i < fill) in = within(make_float4(w.cx[i], w.cy[i], w.cz[i], 0.f), tl, th, cr2);
                        const uint32_t m = __ballot_sync(0xffffffffu, in);
                        if (in) w.list[cnt + __popc(m & ((1u << lane) - 1u))] = i;
                        cnt += __popc(m);
                    }
                    __syncwarp();
                    const uint32_t pairs = (min(32u, nv - 32u * t) + 1u) >> 1;
                    for (uint32_t b = lane; b < cnt; b += 32) {
                        const uint32_t i = w.list[b];
                        const float2 qx = make_float2(w.cx[i], w.cx[i]), qy = make_float2(w.cy[i], w.cy[i]),
                                     qz = make_float2(w.cz[i], w.cz[i]);
                        // (ZB05) sum w e; sum k d with the factors common to all pairs left out
                        float2 sx = make_float2(0.f, 0.f), sy = sx, sz = sx, tx = sx, ty = sx, tz = sx;
#pragma unroll 2
                        for (uint32_t j = 0; j < pairs; ++j) {
                            const float4 A = w.vxy[16u * t + j];
                            const float2 dx = __ffma2_rn(make_float2(A.x, A.y), mone2, qx);
                            const float2 dy = __ffma2_rn(make_float2(A.z, A.w), mone2, qy);
                            const float2 dz = __ffma2_rn(w.vz[16u * t + j], mone2, qz);
                            const float2 d2 = __ffma2_rn(dx, dx, __ffma2_rn(dy, dy, __fmul2_rn(dz, dz)));
                            float2 kk;
                            if (TC01) {
                                kk = __ffma2_rn(d2, inv2, mone2);
                                kk.x = fminf(kk.x, 0.f);
                                kk.y = fminf(kk.y, 0.f);
                                kk = __fmul2_rn(kk, w.g[16u * t + j]);
                            } else {
                                float2 u = __ffma2_rn(d2, ninv2, one2);
                                u.x = fmaxf(u.x, 0.f);
                                u.y = fmaxf(u.y, 0.f);
                                const float2 u2 = __fmul2_rn(u, u), wt = __fmul2_rn(u2, u);
                                const float4 E = w.exy[16u * t + j], Z = w.ezw[16u * t + j];
                                const float2 ex = make_float2(E.x, E.y), ey = make_float2(E.z, E.w),
                                             ez = make_float2(Z.x, Z.y), ew = make_float2(Z.z, Z.w);
                                kk = __ffma2_rn(ex, dx, __ffma2_rn(ey, dy, __ffma2_rn(ez, dz, __fmul2_rn(ew, mone2))));
                                kk = __fmul2_rn(kk, u2);
                                sx = __ffma2_rn(wt, ex, sx);
                                sy = __ffma2_rn(wt, ey, sy);
                                sz = __ffma2_rn(wt, ez, sz);
                            }
                            tx = __ffma2_rn(kk, dx, tx);
                            ty = __ffma2_rn(kk, dy, ty);
                            tz = __ffma2_rn(kk, dz, tz);
                        }
                        const float f = TC01 ? inv_h2 : -6.0f * inv_h2;
                        w.gx[i] += fmaf(f, tx.x + tx.y, sx.x + sx.y);
                        w.gy[i] += fmaf(f, ty.x + ty.y, sy.x + sy.y);
                        w.gz[i] += fmaf(f, tz.x + tz.y, sz.x + sz.y);
                    }
                    __syncwarp();
                }
                if (w.nodd != 0u) odd_vertices();
                for (uint32_t i = lane; i < fill; i += 32) {
                    const float4 g = make_float4(w.gx[i], w.gy[i], w.gz[i], 0.f);
                    if (g.x != 0.f || g.y != 0.f || g.z != 0.f) atomicAdd(a.gx + w.cj[i], g);
                }
                __syncwarp();
                fill = 0;
            };
            int row = 0;
            for (uint32_t cb = begin; cb < total; cb += 32) {
                const uint32_t j = cb + lane;
                bool keep = false;
                float4 q = make_float4(0.f, 0.f, 0.f, 0.f);
                uint32_t idx = 0;
                if (j < total) {
                    while (row < 8 && w.rp[row + 1] <= j) ++row;
                    idx = w.rb[row] + (j - w.rp[row]);
                    q = __ldg(&a.sorted[idx]);
                    keep = within(q, pl, ph, cr2);
                }
                const uint32_t m = __ballot_sync(0xffffffffu, keep);
                if (keep) {
                    const uint32_t pos = fill + __popc(m & ((1u << lane) - 1u));
                    w.cx[pos] = q.x;
                    w.cy[pos] = q.y;
                    w.cz[pos] = q.z;
                    w.cj[pos] = idx;
                }
                fill += __popc(m);
                if (fill > kBwdSeg - 32) tiles();
            }
            if (fill) tiles();
        };
        // the vertices of a row segment with dL/dphi != 0
        auto with_gradient = [&](uint32_t bits, uint32_t r0) {
            uint32_t kept = 0;
            for (uint32_t m = bits, r = r0; m; m &= m - 1u, ++r)
                if (r < nb && __ldg(a.gphi + r) != 0.f) kept |= m & (0u - m);
            return kept;
        };
        list_band_vertices<kBwdVerts>(a.sc, a.band, lo, hi, w.vloc, w.vrank, lane, with_gradient, pass);
        __syncwarp();
    }
}

// dL/d(smoothed position), dL/dG (without the determinant's term) and the sums
// that term takes, for the particles of each group holding gradient vertices
// (cu:938-1031 differentiated).  As the isotropic adjoint above: a warp per group,
// passes of up to 128 vertices with dL/dphi != 0 in tiles of 32, the candidates
// staged, those whose support sphere reaches a tile listed, a lane per listed
// candidate, two vertices per packed operation.  Per pair, with M = G^T G (the
// forward's quadratic form), q2 = d^T M d, u = 1 - q2 and b = g u^2:
//   sum b d, sum b d d^T, sum g u^3,
// from which dL/dx~ = -6 c M (sum b d) and dL/dG = -6 c G (sum b d d^T) follow
// once per candidate.  Bound by the FP32 pipe.  A block per group with a candidate
// per thread and the vertices one by one ran 13 of 32 lanes (whole backward: 20k
// particles 0.25 -> 0.215 ms, 150k 0.49 -> 0.45, 1M 1.44 -> 1.36).  Staged 64 / 96 / 128
// at a time: 150k 0.47 / 0.45 / 0.46 ms; vertex pairs one, two or four to a step: 20k
// 0.233 / 0.233 / 0.211.
constexpr uint32_t kAnisoBwdSeg = 96;  // candidates staged at a time
constexpr int kBwdSums = 10;
struct AnisoBwdSlice {
    float4 vxy[kBwdVerts / 2];  // the pass's vertices two to a pair: (x, x', y, y')
    float4 vzg[kBwdVerts / 2];  // (z, z', dL/dphi, dL/dphi')
    uint32_t vloc[kBwdVerts], vrank[kBwdVerts];
    uint32_t hist[kBwdVerts];
    float4 box[2 * (kBwdVerts / 32)];
    float4 c[kAnisoBwdSeg];                // the staged candidates: x, y, z, squared support radius
    float m[6][kAnisoBwdSeg];              // their quadratic forms: m00, 2 m01, 2 m02, m11, 2 m12, m22
    float s[kBwdSums][kAnisoBwdSeg];       // their sums: b d, g u^3, b d d^T
    float coef[kAnisoBwdSeg];              // sigma det(G) m / rho
    uint32_t cj[kAnisoBwdSeg];             // their sorted index
    uint32_t list[kAnisoBwdSeg];           // those that reach the tile
    uint32_t cstart[128], cpre[kMaxCells + 1], cinv[128];
    uint32_t ncells, total_inv, ninv_cells;
};

__global__ void __launch_bounds__(kFT, 4) k_field_aniso_backward(BwdGroupArgs a, uint32_t ratio, const Counters* ctr)
{
    after_launch();
    extern __shared__ __align__(16) unsigned char smem[];
    const int lane = threadIdx.x & 31;
    AnisoBwdSlice& w = reinterpret_cast<AnisoBwdSlice*>(smem)[threadIdx.x >> 5];
    const uint32_t nb = min(ctr->n_band, a.cap);
    const BwdGroupList groups(a.glist, a.sp);
    const uint32_t ncrowd = groups.crowded(), nlist = groups.usual() + ncrowd;  // groups holding gradient vertices
    // Few groups are cut into more work items: fine grids by slabs of vertices,
    // coarse ones, whose groups hold few vertices, by runs of candidates (backward
    // by slabs / runs, ms: 10 vertices per cell, 20k particles 0.21 / 0.25, 150k 0.44 / 0.53;
    // 3 per cell, 20k 0.62 / 0.585).
    const uint32_t nsub = field_slabs(nlist), nslab = ratio > 4 ? nsub : 1u, nparts = ratio > 4 ? 1u : nsub;
    const float2 one2 = make_float2(1.0f, 1.0f), mone2 = make_float2(-1.0f, -1.0f);

    for (;;) {
        uint32_t k = 0;
        if (lane == 0) k = atomicAdd(&a.glist[1], 1u);
        k = __shfl_sync(0xffffffffu, k, 0);
        if (k >= nlist * nsub) break;
        const uint32_t part = k % nparts;
        int c[3], lo[3], hi[3];
        if (!group_box(groups.at(k / nsub, ncrowd), a.sp, a.sc, ratio, c, lo, hi) || !slab_box(k % nslab, nslab, lo, hi))
            continue;
        bool tables = false;
        uint32_t total = 0;

        auto pass = [&](uint32_t nv) {
            if (!tables) {
                const float b0[3] = {vpos1(lo[0], a.sc.min[0], a.sc.cs), vpos1(lo[1], a.sc.min[1], a.sc.cs),
                                     vpos1(lo[2], a.sc.min[2], a.sc.cs)};
                const float b1[3] = {vpos1(hi[0] - 1, a.sc.min[0], a.sc.cs), vpos1(hi[1] - 1, a.sc.min[1], a.sc.cs),
                                     vpos1(hi[2] - 1, a.sc.min[2], a.sc.cs)};
                total = warp_candidates(a.sp, a.ranges, a.invol, a.reach, c, b0, b1, w);
                tables = true;
            }
            float4 pl, ph;
            pass_layout<true, kBwdVerts>(w.vloc, w.vrank, lo, a.sc, nullptr, w.hist, w.box, nv, lane, pl, ph);
            const uint32_t ntiles = (nv + 31) / 32;
            // the places up to the last tile's end lie far away and have dL/dphi = 0
            float all = 0.f;
            for (uint32_t q = lane; q < 32u * ntiles; q += 32) {
                float4 vp = make_float4(1.0e18f, 1.0e18f, 1.0e18f, 0.f);
                if (q < nv) {
                    vp = vert_pos(w.vloc[q], lo, a.sc);
                    vp.w = __ldg(a.gphi + w.vrank[q]);
                    all += vp.w;
                }
                float* d = reinterpret_cast<float*>(w.vxy + (q >> 1)) + (q & 1u);
                d[0] = vp.x;
                d[2] = vp.y;
                d = reinterpret_cast<float*>(w.vzg + (q >> 1)) + (q & 1u);
                d[0] = vp.z;
                d[2] = vp.w;
            }
            // A vertex whose dL/dphi is not finite is not dropped by the clamp of 1 - q2 at
            // 0 (0 x inf): passes that hold one (or whose lanes' sums overflow) test the
            // range of each pair, so that it reaches the particles of its support only
            const bool odd = __any_sync(0xffffffffu, !(fabsf(all) <= kFinite));
            __syncwarp();
            const uint32_t total_inv = w.total_inv;
            uint32_t fill = 0;
            auto tiles = [&]() {
                for (uint32_t i = lane; i < fill; i += 32)
#pragma unroll
                    for (int r = 0; r < kBwdSums; ++r) w.s[r][i] = 0.f;
                __syncwarp();
#pragma unroll 1
                for (uint32_t t = 0; t < ntiles; ++t) {
                    const float4 tl = w.box[2 * t], th = w.box[2 * t + 1];
                    uint32_t cnt = 0;
                    for (uint32_t b = 0; b < fill; b += 32) {
                        const uint32_t i = b + (uint32_t)lane;
                        const bool in = i < fill && reaches(w.c[i], tl, th);
                        const uint32_t m = __ballot_sync(0xffffffffu, in);
                        if (in) w.list[cnt + __popc(m & ((1u << lane) - 1u))] = i;
                        cnt += __popc(m);
                    }
                    __syncwarp();
                    const uint32_t pairs = (min(32u, nv - 32u * t) + 1u) >> 1;
                    for (uint32_t b = lane; b < cnt; b += 32) {
                        const uint32_t i = w.list[b];
                        const float4 q = w.c[i];
                        const float2 qx = make_float2(q.x, q.x), qy = make_float2(q.y, q.y), qz = make_float2(q.z, q.z);
                        const float2 m0 = make_float2(w.m[0][i], w.m[0][i]), m1 = make_float2(w.m[1][i], w.m[1][i]),
                                     m2 = make_float2(w.m[2][i], w.m[2][i]), m3 = make_float2(w.m[3][i], w.m[3][i]),
                                     m4 = make_float2(w.m[4][i], w.m[4][i]), m5 = make_float2(w.m[5][i], w.m[5][i]);
                        float2 s[kBwdSums];
#pragma unroll
                        for (int r = 0; r < kBwdSums; ++r) s[r] = make_float2(0.f, 0.f);
                        auto walk = [&](auto odd_pass) {
                            constexpr bool kOdd = decltype(odd_pass)::value;
#pragma unroll 4
                            for (uint32_t j = 0; j < pairs; ++j) {
                                const float4 A = w.vxy[16u * t + j], Z = w.vzg[16u * t + j];
                                const float2 dx = __ffma2_rn(make_float2(A.x, A.y), mone2, qx);
                                const float2 dy = __ffma2_rn(make_float2(A.z, A.w), mone2, qy);
                                const float2 dz = __ffma2_rn(make_float2(Z.x, Z.y), mone2, qz);
                                const float2 t0 = __ffma2_rn(m0, dx, __ffma2_rn(m1, dy, __fmul2_rn(m2, dz)));
                                const float2 t1 = __ffma2_rn(m3, dy, __fmul2_rn(m4, dz));
                                const float2 q2 =
                                    __ffma2_rn(dx, t0, __ffma2_rn(dy, t1, __fmul2_rn(__fmul2_rn(m5, dz), dz)));
                                float2 u = __ffma2_rn(q2, mone2, one2);
                                u.x = fmaxf(u.x, 0.f);
                                u.y = fmaxf(u.y, 0.f);
                                float2 bb = __fmul2_rn(make_float2(Z.z, Z.w), __fmul2_rn(u, u));
                                if (kOdd) {
                                    if (!(u.x > 0.f)) bb.x = 0.f;
                                    if (!(u.y > 0.f)) bb.y = 0.f;
                                }
                                const float2 bx = __fmul2_rn(bb, dx), by = __fmul2_rn(bb, dy), bz = __fmul2_rn(bb, dz);
                                s[0] = __fadd2_rn(s[0], bx);
                                s[1] = __fadd2_rn(s[1], by);
                                s[2] = __fadd2_rn(s[2], bz);
                                s[3] = __ffma2_rn(bb, u, s[3]);
                                s[4] = __ffma2_rn(bx, dx, s[4]);
                                s[5] = __ffma2_rn(bx, dy, s[5]);
                                s[6] = __ffma2_rn(bx, dz, s[6]);
                                s[7] = __ffma2_rn(by, dy, s[7]);
                                s[8] = __ffma2_rn(by, dz, s[8]);
                                s[9] = __ffma2_rn(bz, dz, s[9]);
                            }
                        };
                        if (odd) walk(std::true_type());
                        else walk(std::false_type());
#pragma unroll
                        for (int r = 0; r < kBwdSums; ++r) w.s[r][i] += s[r].x + s[r].y;
                    }
                    __syncwarp();
                }
                for (uint32_t i = lane; i < fill; i += 32) {
                    const float gx = w.s[0][i], gy = w.s[1][i], gz = w.s[2][i], sc = w.s[3][i];
                    // (the first moments can cancel where the second ones do not)
                    bool some = gx != 0.f || gy != 0.f || gz != 0.f || sc != 0.f;
#pragma unroll
                    for (int r = 4; r < kBwdSums; ++r) some = some || w.s[r][i] != 0.f;
                    if (!some) continue;
                    const uint32_t id = w.cj[i];
                    const float f = -6.0f * w.coef[i];
                    const float m01 = 0.5f * w.m[1][i], m02 = 0.5f * w.m[2][i], m12 = 0.5f * w.m[4][i];
                    atomicAdd(a.gsmooth + id,
                              make_float4(f * (w.m[0][i] * gx + m01 * gy + m02 * gz),
                                          f * (m01 * gx + w.m[3][i] * gy + m12 * gz),
                                          f * (m02 * gx + m12 * gy + w.m[5][i] * gz), sc));
                    const float s00 = f * w.s[4][i], s01 = f * w.s[5][i], s02 = f * w.s[6][i];
                    const float s11 = f * w.s[7][i], s12 = f * w.s[8][i], s22 = f * w.s[9][i];
#pragma unroll
                    for (int r = 0; r < 3; ++r) {
                        const float4 g = __ldg(a.grec + 4ull * id + 1 + r);
                        atomicAdd(a.gG + 3ull * id + r, make_float4(g.x * s00 + g.y * s01 + g.z * s02,
                                                                    g.x * s01 + g.y * s11 + g.z * s12,
                                                                    g.x * s02 + g.y * s12 + g.z * s22, 0.f));
                    }
                }
                __syncwarp();
                fill = 0;
            };
            const CandTables tabs{w.cstart, w.cpre, w.cinv};
            // the part's candidates: a run of the involved ones, whole 32s
            const uint32_t n32 = (total_inv + 31) / 32;
            for (uint32_t cb = 32 * (n32 * part / nparts); cb < 32 * (n32 * (part + 1) / nparts); cb += 32) {
                const uint32_t j = cb + lane;
                bool keep = false;
                uint32_t id = 0;
                float4 r0 = make_float4(0.f, 0.f, 0.f, 0.f), r1 = r0, r2 = r0;
                if (j < total_inv) {
                    int cell;
                    id = candidate(j, tabs, &cell, (int)w.ncells);
                    const float4* src = a.qrec + 3ull * id;
                    r0 = __ldg(src);
                    r1 = __ldg(src + 1);
                    r2 = __ldg(src + 2);
                    keep = reaches(r0, pl, ph);
                }
                const uint32_t m = __ballot_sync(0xffffffffu, keep);
                if (keep) {
                    const uint32_t i = fill + __popc(m & ((1u << lane) - 1u));
                    w.c[i] = r0;
                    w.m[0][i] = r1.x;
                    w.m[1][i] = r1.y;
                    w.m[2][i] = r1.z;
                    w.m[3][i] = r2.x;
                    w.m[4][i] = r2.y;
                    w.m[5][i] = r2.z;
                    w.coef[i] = r1.w;
                    w.cj[i] = id;
                }
                fill += __popc(m);
                if (fill > kAnisoBwdSeg - 32) tiles();
            }
            if (fill) tiles();
            // the others: G = I and support 1, which reaches every vertex; no dL/dG
            for (uint32_t j = total_inv + 32 * part + lane; j < total; j += 32 * nparts) {
                int cell;
                const uint32_t id = candidate(j, tabs, &cell, (int)w.ncells);
                const float4 q = __ldg(&a.smoothed[id]);
                const float2 qx = make_float2(q.x, q.x), qy = make_float2(q.y, q.y), qz = make_float2(q.z, q.z);
                float2 sx = make_float2(0.f, 0.f), sy = sx, sz = sx;
#pragma unroll 1
                for (uint32_t v = 0; v < (nv + 1u) >> 1; ++v) {
                    const float4 A = w.vxy[v], Z = w.vzg[v];
                    const float2 dx = __ffma2_rn(make_float2(A.x, A.y), mone2, qx);
                    const float2 dy = __ffma2_rn(make_float2(A.z, A.w), mone2, qy);
                    const float2 dz = __ffma2_rn(make_float2(Z.x, Z.y), mone2, qz);
                    const float2 q2 = __ffma2_rn(dx, dx, __ffma2_rn(dy, dy, __fmul2_rn(dz, dz)));
                    float2 u = __ffma2_rn(q2, mone2, one2);
                    u.x = fmaxf(u.x, 0.f);
                    u.y = fmaxf(u.y, 0.f);
                    float2 bb = __fmul2_rn(make_float2(Z.z, Z.w), __fmul2_rn(u, u));
                    if (odd) {
                        if (!(u.x > 0.f)) bb.x = 0.f;
                        if (!(u.y > 0.f)) bb.y = 0.f;
                    }
                    sx = __ffma2_rn(bb, dx, sx);
                    sy = __ffma2_rn(bb, dy, sy);
                    sz = __ffma2_rn(bb, dz, sz);
                }
                const float f = -6.0f * (a.sigma * q.w);
                const float4 g = make_float4(f * (sx.x + sx.y), f * (sy.x + sy.y), f * (sz.x + sz.y), 0.f);
                if (g.x != 0.f || g.y != 0.f || g.z != 0.f) atomicAdd(a.gsmooth + id, g);
            }
            __syncwarp();
        };
        // the vertices of a row segment with dL/dphi != 0
        auto with_gradient = [&](uint32_t bits, uint32_t r0) {
            uint32_t kept = 0;
            for (uint32_t m = bits, r = r0; m; m &= m - 1u, ++r)
                if (r < nb && __ldg(a.gphi + r) != 0.f) kept |= m & (0u - m);
            return kept;
        };
        list_band_vertices<kBwdVerts>(a.sc, a.band, lo, hi, w.vloc, w.vrank, lane, with_gradient, pass);
        __syncwarp();
    }
}

}  // namespace

void launch_field_aniso_backward(const KernelCtx& c, const AnisoBwdArgs& f, uint32_t ratio, const Counters* ctr)
{
    BwdGroupArgs a;
    a.sp = f.sp;
    a.sc = f.sc;
    a.band = f.band;
    a.grec = f.grec;
    a.qrec = f.qrec;
    a.smoothed = f.smoothed;
    a.ranges = f.ranges;
    a.invol = f.invol;
    a.reach = f.cell_rmax;
    a.gphi = f.gphi;
    a.glist = f.glist;
    a.gsmooth = f.gsmooth;
    a.gG = f.gG;
    a.sigma = f.sigma;
    a.cap = f.cap;
    const size_t smem = sizeof(AnisoBwdSlice) * kFWarps;
    cudaFuncSetAttribute(k_field_aniso_backward, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    const unsigned grid = (unsigned)std::max(1, c.num_sms * 4 / std::max(1, c.grid_div));
    launch_after(k_field_aniso_backward, grid, kFT, smem, c.stream, a, ratio, ctr);
    ++g_launches;
}

void launch_field_aniso_grouped(const KernelCtx& c, const AnisoFieldArgs& f, const BandView& band, uint32_t ratio,
                                Counters* ctr)
{
    GroupArgs a;
    a.sp = f.sp;
    a.sc = f.sc;
    a.band = band;
    a.grec = f.grec;
    a.qrec = f.qrec;
    a.smoothed = f.smoothed;
    a.glist = f.glist;
    a.ranges = f.ranges;
    a.invol = f.invol;
    a.reach = f.cell_rmax;
    a.phi = f.phi;
    a.sigma = f.sigma;
    a.cap = f.cap;
    const uint64_t groups = (uint64_t)(f.sp.res[0] + 1) * (f.sp.res[1] + 1) * (f.sp.res[2] + 1);
    const unsigned grid = (unsigned)std::min<uint64_t>(
        (groups + kFWarps - 1) / kFWarps, std::max<uint64_t>(1, (uint64_t)c.num_sms * 16 / std::max(1, c.grid_div)));
    launch_after(k_field_aniso_grouped, grid, kFT, 0, c.stream, a, ratio, ctr);
    ++g_launches;
}

void launch_field_iso_backward(const KernelCtx& c, const BwdArgs& a, bool tc01, const Counters* ctr)
{
    const uint64_t groups = (uint64_t)(a.sp.res[0] + 1) * (a.sp.res[1] + 1) * (a.sp.res[2] + 1);
    const unsigned grid = (unsigned)std::min<uint64_t>(
        (groups * kSlabMax + kFWarps - 1) / kFWarps, std::max<uint64_t>(1, (uint64_t)c.num_sms * 12 / std::max(1, c.grid_div)));
    if (tc01) launch_after(k_field_iso_backward<true>, grid, kFT, 0, c.stream, a, ctr);
    else launch_after(k_field_iso_backward<false>, grid, kFT, 0, c.stream, a, ctr);
    ++g_launches;
}

void launch_field_iso_grouped(const KernelCtx& c, bool tc01, const IsoFieldArgs& f, const BandView& band, uint32_t ratio,
                              Counters* ctr)
{
    const uint64_t groups = (uint64_t)(f.sp.res[0] + 1) * (f.sp.res[1] + 1) * (f.sp.res[2] + 1);
    const unsigned grid = (unsigned)std::min<uint64_t>(
        (groups + kFWarps - 1) / kFWarps, std::max<uint64_t>(1, (uint64_t)c.num_sms * 16 / std::max(1, c.grid_div)));
    if (tc01) launch_after(k_field_iso_grouped<true>, grid, kFT, 0, c.stream, f, band, ratio, ctr);
    else launch_after(k_field_iso_grouped<false>, grid, kFT, 0, c.stream, f, band, ratio, ctr);
    ++g_launches;
}

}  // namespace fsr
