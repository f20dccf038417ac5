// stencil.cu -- the per-triangle guide stencil search of build_asset on sm_100a.
//
// For every triangle the reference (src/asset.cpp:252-269) scores each guide
// by |centroid - root|^2, plus 1e20 when the face normal and the guide's root
// normal disagree (dot < -0.25), and keeps the 8 smallest (score, guide)
// pairs in ascending order.  That is triangles x guides candidates (8.2e8 for
// a 200,000-triangle mesh with 4,096 guides), the only super-linear step of
// the asset build.
//
// Two searches, the same rows:
//
// All pairs (search_all): one thread per triangle, 128-thread CTAs; the guide
// roots (one plane per axis) and normals stream through shared memory in tiles
// of kStencilTile guides, read by every lane at the same address (broadcast).
// The eight best candidates live in registers.  Scores use the exact helpers
// of strand_math.cuh (__f*_rn, never contracted), so they equal the host
// build's bit for bit, and the insertion replays the host's procedure
// (host.cpp build_stencils), so the rows are identical even for ties and
// non-finite scores.  A candidate whose |centroid - root|^2 alone is above the
// current eighth score cannot enter (the penalty only adds); four guides at a
// time are tested with packed f32x2 arithmetic and the rare group that passes
// is scored exactly.  Bound by FP32 issue: 502 us for 200,000 triangles x
// 4,096 guides.
//
// Clusters (search_clusters), for enough of both: the guides are sorted along
// a Morton curve into clusters of 32 with bounding boxes, and a warp looks
// only into clusters that some lane's eighth score does not rule out --
// a handful of 128, since a mesh's neighbouring triangles share their guides.
// For finite positions the (score, guide) order is a total one, so the eight
// smallest do not depend on the order of search; a CTA that meets a wild
// position (not finite, or beyond kWild) takes all pairs.  So does one whose
// warps' triangles lie scattered over too many clusters, and the whole call
// where the sort finds a sample of the warps scattered over the mesh: a visit
// to a cluster costs a warp as much as all pairs cost it over six to eight
// clusters' guides (200,000 x 4,096 in random triangle order 3,609 us by
// clusters, 1,200 by all pairs).  149 us at the size
// above (sorting 23, search 90, the last rows' search mostly beside it): bound
// by the latency of a warp's chain of clusters.  The sorted guides need memory this entry point has no argument
// for: they are put into the last rows of the output, whose triangles a second
// kernel searches from its own shared-memory copy and writes last.
//
// guide_nearest_kernel, one warp per guide, finds each guide's nearest
// other root for the automatic support radius (guide_count^2 distances).
#include "generator_core.cuh"
#include "nxg_internal.h"
#include "strand_math.cuh"

#include <cuda_runtime.h>

#include <cfloat>
#include <cmath>
#include <cstdint>

namespace nxg {
namespace dev {
namespace {

constexpr uint32_t kStencilThreads = 128u;
constexpr uint32_t kStencilTile = 512u;  // guides per shared-memory tile (14 KB)

struct Candidate {
    float key;
    uint32_t guide;
};

// std::pair<float, uint32_t>::operator<, as host.cpp candidate_less.
__device__ __forceinline__ bool candidate_less(float ak, uint32_t ag, float bk, uint32_t bg) {
    return ak < bk || (!(bk < ak) && ag < bg);
}

// The host's insertion step: the hole is at `hole`; entries move up while the
// new candidate orders before them, and it lands where that first fails.
// Unrolled over fixed indices so the list stays in registers.
__device__ __forceinline__ void insert_candidate(Candidate (&best)[kSlots], Candidate c, uint32_t hole) {
    bool moving = true;
#pragma unroll
    for (int k = static_cast<int>(kSlots) - 1; k >= 1; --k) {
        if (static_cast<uint32_t>(k) <= hole && moving) {
            if (candidate_less(c.key, c.guide, best[k - 1].key, best[k - 1].guide)) {
                best[k] = best[k - 1];
            } else {
                best[k] = c;
                moving = false;
            }
        }
    }
    if (moving) { best[0] = c; }
}

// Packed pairs of floats (sm_100a f32x2 arithmetic), half the issued
// instructions of the scalar form.  On the GPU their |d|^2 did not equal the
// scalar __f*_rn result bit for bit (tied guides came out in the wrong
// order), so they only filter: a group of guides is skipped when its
// smallest packed |d|^2, shrunk by kFilterMargin, still exceeds the eighth
// score, and every guide of a group that passes is scored again with the
// exact scalar helpers.  Both are sums of the same three squares of the
// same differences, so they can differ by rounding only (a few ulps, about
// 2^-21 relative); the margin is 2^-16, so no guide the host keeps is ever
// skipped, and a packed value that is too small only lets a group through.
constexpr float kFilterMargin = 0.9999847412109375f;  // 1 - 2^-16

struct GuideTile {
    float x[kStencilTile], y[kStencilTile], z[kStencilTile];  // roots, one plane per axis
    float4 normal[kStencilTile];
};

// One candidate, exactly as the host: skip when |d|^2 alone already loses
// (the score is |d|^2 + 0 or 1e20 >= |d|^2), else score with the penalty and
// insert.  `hole` is the fill position while the list is not yet full.
__device__ __forceinline__ void consider(Candidate (&best)[kSlots], float l2, uint32_t gi, uint32_t count,
                                         F3 face, float4 m) {
    if (gi >= count && best[kSlots - 1].key < l2) { return; }
    const float penalty = xdot(face, F3{m.x, m.y, m.z}) < -0.25f ? 1.0e20f : 0.0f;
    const Candidate c{__fadd_rn(l2, penalty), gi};
    uint32_t hole = gi;
    if (gi >= count) {
        if (!candidate_less(c.key, c.guide, best[kSlots - 1].key, best[kSlots - 1].guide)) { return; }
        hole = kSlots - 1;
    }
    insert_candidate(best, c, hole);
}

__device__ __forceinline__ float root_distance2(F3 centroid, const GuideTile &t, uint32_t j) {
    const F3 d = xsub(centroid, F3{t.x[j], t.y[j], t.z[j]});
    return xdot(d, d);
}

// One triangle's search state, all in registers.
struct TriangleSearch {
    F3 centroid, face;
    f32x2 cx, cy, cz;  // the centroid's coordinates, each in both halves
    bool live, invalid;  // invalid: out of range, keeps an all-invalid row
    Candidate best[kSlots];
};

__device__ __forceinline__ void begin_triangle(TriangleSearch &t, uint32_t ti, const nxg_vec3 *__restrict__ positions,
                                               uint32_t vertex_count, const nxg_uint3 *__restrict__ triangles,
                                               uint32_t triangle_count) {
    t.live = ti < triangle_count;
    t.invalid = false;
    t.centroid = F3{0.0f, 0.0f, 0.0f};
    t.face = F3{0.0f, 1.0f, 0.0f};
    if (t.live) {
        const nxg_uint3 tri = triangles[ti];
        if (tri.x < vertex_count && tri.y < vertex_count && tri.z < vertex_count) {
            const nxg_vec3 a = positions[tri.x], b = positions[tri.y], c = positions[tri.z];
            const F3 p0{a.x, a.y, a.z}, p1{b.x, b.y, b.z}, p2{c.x, c.y, c.z};
            t.centroid = xdiv(xadd(xadd(p0, p1), p2), 3.0f);
            t.face = xnormalize(xcross(xsub(p1, p0), xsub(p2, p0)));
        } else {
            t.live = false;
            t.invalid = true;
        }
    }
    t.cx = pair2(t.centroid.x, t.centroid.x);
    t.cy = pair2(t.centroid.y, t.centroid.y);
    t.cz = pair2(t.centroid.z, t.centroid.z);
#pragma unroll
    for (uint32_t k = 0; k < kSlots; ++k) { t.best[k] = {0.0f, kInvalid}; }
}

// Guides j..j+3 of the tile for one triangle: packed |d|^2 of all four, and
// the group skipped when even its smallest one (less the margin) loses.  A
// NaN |d|^2 past the fill can never enter (its guide index is larger than
// every listed one), so fminf dropping it is exact.
__device__ __forceinline__ void consider_group(TriangleSearch &t, const GuideTile &tile, uint32_t j, uint32_t gi,
                                               uint32_t count, ulonglong2 gx, ulonglong2 gy, ulonglong2 gz) {
    const f32x2 dx0 = sub2(t.cx, gx.x), dx1 = sub2(t.cx, gx.y);
    const f32x2 dy0 = sub2(t.cy, gy.x), dy1 = sub2(t.cy, gy.y);
    const f32x2 dz0 = sub2(t.cz, gz.x), dz1 = sub2(t.cz, gz.y);
    const float2 a = unpair2(add2(add2(mul2(dx0, dx0), mul2(dy0, dy0)), mul2(dz0, dz0)));
    const float2 b = unpair2(add2(add2(mul2(dx1, dx1), mul2(dy1, dy1)), mul2(dz1, dz1)));
    const float low = fminf(fminf(a.x, a.y), fminf(b.x, b.y));
    if (t.best[kSlots - 1].key < low * kFilterMargin) { return; }
    // The group passed: each guide is checked on its own packed value before
    // its exact score (a warp runs a guide's exact path only when one of its
    // lanes needs it).
    const float packed[4] = {a.x, a.y, b.x, b.y};
#pragma unroll
    for (uint32_t k = 0; k < 4u; ++k) {
        if (t.best[kSlots - 1].key < packed[k] * kFilterMargin) { continue; }
        consider(t.best, root_distance2(t.centroid, tile, j + k), gi + k, count, t.face, tile.normal[j + k]);
    }
}

__device__ __forceinline__ void end_triangle(const TriangleSearch &t, uint32_t ti, uint32_t keep,
                                             uint32_t *__restrict__ stencil) {
    if (!t.live && !t.invalid) { return; }
    uint32_t out[kSlots];
#pragma unroll
    for (uint32_t k = 0; k < kSlots; ++k) { out[k] = t.live && k < keep ? t.best[k].guide : kInvalid; }
    uint4 *row = reinterpret_cast<uint4 *>(stencil + static_cast<size_t>(ti) * kSlots);
    row[0] = make_uint4(out[0], out[1], out[2], out[3]);
    row[1] = make_uint4(out[4], out[5], out[6], out[7]);
}

// The all-pairs search of a CTA's triangles (every thread calls it).
__device__ __forceinline__ void search_all(TriangleSearch &t, GuideTile &tile, const nxg_vec3 *__restrict__ guide_roots,
                                           const nxg_vec3 *__restrict__ guide_normals, uint32_t guide_count) {
    const uint32_t count = guide_count < kSlots ? guide_count : kSlots;
    for (uint32_t base = 0; base < guide_count; base += kStencilTile) {
        const uint32_t n = guide_count - base < kStencilTile ? guide_count - base : kStencilTile;
        __syncthreads();
        for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) {
            const nxg_vec3 r = guide_roots[base + i], m = guide_normals[base + i];
            tile.x[i] = r.x;
            tile.y[i] = r.y;
            tile.z[i] = r.z;
            tile.normal[i] = make_float4(m.x, m.y, m.z, 0.0f);
        }
        __syncthreads();
        if (!t.live) { continue; }
        // The first `count` guides fill the lists (tile 0 only; count <= 8).
        uint32_t j = base == 0u ? count : 0u;
        for (uint32_t f = 0; f < j; ++f) {
            consider(t.best, root_distance2(t.centroid, tile, f), f, count, t.face, tile.normal[f]);
        }
        for (; j + 4u <= n; j += 4u) {
            const ulonglong2 gx = *reinterpret_cast<const ulonglong2 *>(&tile.x[j]);
            const ulonglong2 gy = *reinterpret_cast<const ulonglong2 *>(&tile.y[j]);
            const ulonglong2 gz = *reinterpret_cast<const ulonglong2 *>(&tile.z[j]);
            consider_group(t, tile, j, base + j, count, gx, gy, gz);
        }
        for (; j < n; ++j) {
            consider(t.best, root_distance2(t.centroid, tile, j), base + j, count, t.face, tile.normal[j]);
        }
    }
}

// One triangle per thread, 128-thread CTAs (56 registers, 9 CTAs per SM).
// Measured slower: two triangles per thread sharing each guide load (fewer
// warps per SM to hide the dependency chains), and a 40-register cap that
// fits a 200,000-triangle mesh in one wave (spills).
__global__ void __launch_bounds__(kStencilThreads, 9)
stencil_kernel(const nxg_vec3 *__restrict__ positions, uint32_t vertex_count, const nxg_uint3 *__restrict__ triangles,
               uint32_t triangle_count, const nxg_vec3 *__restrict__ guide_roots,
               const nxg_vec3 *__restrict__ guide_normals, uint32_t guide_count, uint32_t keep,
               uint32_t *__restrict__ stencil) {
    __shared__ __align__(16) GuideTile tile;
    const uint32_t ti = blockIdx.x * kStencilThreads + threadIdx.x;
    TriangleSearch t;
    begin_triangle(t, ti, positions, vertex_count, triangles, triangle_count);
    search_all(t, tile, guide_roots, guide_normals, guide_count);
    end_triangle(t, ti, keep, stencil);
}

// ---------------------------------------------------------------------------
// The cluster search.
// ---------------------------------------------------------------------------
constexpr uint32_t kClusterGuides = 32u;
constexpr uint32_t kClusterWords = 4u * kClusterGuides / 4u;  // float4 per cluster: planes x, y, z, guide index
constexpr uint32_t kMaxClusters = 160u;    // 92 KB of shared memory in the second kernel
constexpr uint32_t kTailCtas = 8u;         // CTAs of the second kernel, one thread-block cluster
constexpr uint32_t kTailMaxThreads = 384u;
constexpr uint32_t kClusterMinGuides = 640u;
constexpr float kWild = 1.0e15f;           // |coordinate| past it: |d|^2 could overflow

constexpr uint32_t kClusterBoxes = 4u;     // float4 per cluster: roots' box low (and guide count), high, normals' box

// Scratch: kClusterWords float4 per cluster | kClusterBoxes float4 per cluster
// | one float4, in the last row of all: its first word nonzero where every
// triangle takes all pairs, its second where that is because a guide is wild.
__host__ __device__ constexpr uint32_t cluster_scratch_words(uint32_t clusters) {
    return clusters * (kClusterWords + kClusterBoxes) + 1u;
}
// Output rows (two float4 each) the scratch takes.
__host__ __device__ constexpr uint32_t cluster_scratch_rows(uint32_t clusters) {
    return (cluster_scratch_words(clusters) + 1u) / 2u;
}

__device__ __forceinline__ uint32_t spread3(uint32_t v) {  // bits of v three apart
    uint32_t r = 0u;
#pragma unroll
    for (uint32_t k = 0; k < 4u; ++k) { r |= ((v >> k) & 1u) << (3u * k); }
    return r;
}

// A warp of the sample is scattered where its triangles reach further than 1.7
// clusters would if they shared out the mesh as squares: neighbours reach
// 0.07 to 0.15 of a mesh of 50,000 to 200,000 triangles (0.8 to 1.3 of 32 to
// 128 clusters), a quarter of a ring of 64 quads 0.34 (1.9 of 32, where all
// pairs are level), two patches of sixteen triangles 0.56 (2.5 of 20).
constexpr float kScattered = 1.7f * 1.7f;

// The box of the warp's triangles.
struct WarpBox {
    F3 lo, hi;
};
__device__ __forceinline__ WarpBox warp_box(const TriangleSearch &t) {
    WarpBox b;
    b.lo = t.live ? t.centroid : F3{FLT_MAX, FLT_MAX, FLT_MAX};
    b.hi = t.live ? t.centroid : F3{-FLT_MAX, -FLT_MAX, -FLT_MAX};
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        b.lo = F3{fminf(b.lo.x, __shfl_xor_sync(kFull, b.lo.x, o)), fminf(b.lo.y, __shfl_xor_sync(kFull, b.lo.y, o)),
                  fminf(b.lo.z, __shfl_xor_sync(kFull, b.lo.z, o))};
        b.hi = F3{fmaxf(b.hi.x, __shfl_xor_sync(kFull, b.hi.x, o)), fmaxf(b.hi.y, __shfl_xor_sync(kFull, b.hi.y, o)),
                  fmaxf(b.hi.z, __shfl_xor_sync(kFull, b.hi.z, o))};
    }
    return b;
}

// Sorts the guides by the Morton code of their cell (16 cells per axis of
// the roots' box) and writes the scratch; one CTA.  The order within a cell is
// arbitrary.  Each warp also looks at the triangles of one warp of the search.
__global__ void __launch_bounds__(1024) cluster_kernel(const nxg_vec3 *__restrict__ positions, uint32_t vertex_count,
                                                       const nxg_uint3 *__restrict__ triangles,
                                                       uint32_t triangle_count, const nxg_vec3 *__restrict__ guide_roots,
                                                       const nxg_vec3 *__restrict__ guide_normals, uint32_t guide_count,
                                                       uint32_t clusters, float4 *scratch) {
    constexpr uint32_t kBits = 4u;  // 4,096 cells, of which a surface meets about a fifth
    constexpr uint32_t bin_count = 1u << (3u * kBits);
    __shared__ uint32_t bins[bin_count];
    __shared__ float bounds[6][32], mesh[6][32];
    __shared__ uint32_t warp_sums[32];
    chain_start();
    chain_wait();
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    for (uint32_t i = tid; i < bin_count; i += 1024u) { bins[i] = 0u; }
    constexpr uint32_t kOwn = (kMaxClusters * kClusterGuides + 1023u) / 1024u;  // guides of a thread
    nxg_vec3 root[kOwn];
    float lo[3] = {FLT_MAX, FLT_MAX, FLT_MAX}, hi[3] = {-FLT_MAX, -FLT_MAX, -FLT_MAX};
    bool wild = false;
    TriangleSearch sample;
    begin_triangle(sample, warp * (triangle_count / 1024u) * 32u + lane, positions, vertex_count, triangles,
                   triangle_count);
#pragma unroll
    for (uint32_t q = 0; q < kOwn; ++q) {
        const uint32_t i = q * 1024u + tid;
        root[q] = i < guide_count ? guide_roots[i] : nxg_vec3{0.0f, 0.0f, 0.0f};
    }
#pragma unroll
    for (uint32_t q = 0; q < kOwn; ++q) {
        if (q * 1024u + tid >= guide_count) { continue; }
        const float v[3] = {root[q].x, root[q].y, root[q].z};
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            wild = wild || !(fabsf(v[k]) <= kWild);
            lo[k] = fminf(lo[k], v[k]);
            hi[k] = fmaxf(hi[k], v[k]);
        }
    }
#pragma unroll
    for (int k = 0; k < 3; ++k) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            lo[k] = fminf(lo[k], __shfl_xor_sync(kFull, lo[k], o));
            hi[k] = fmaxf(hi[k], __shfl_xor_sync(kFull, hi[k], o));
        }
        if (lane == 0u) {
            bounds[k][warp] = lo[k];
            bounds[3 + k][warp] = hi[k];
        }
    }
    const WarpBox box = warp_box(sample);
    if (lane == 0u) {
        mesh[0][warp] = box.lo.x;
        mesh[1][warp] = box.lo.y;
        mesh[2][warp] = box.lo.z;
        mesh[3][warp] = box.hi.x;
        mesh[4][warp] = box.hi.y;
        mesh[5][warp] = box.hi.z;
    }
    wild = __syncthreads_or(wild);
    // Most of the sample scattered: all pairs (every warp counts alike).
    float across = 0.0f, own = 0.0f;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        float low = mesh[k][lane], high = mesh[3 + k][lane];
        own = fmaxf(own, high - low);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            low = fminf(low, __shfl_xor_sync(kFull, low, o));
            high = fmaxf(high, __shfl_xor_sync(kFull, high, o));
        }
        across = fmaxf(across, high - low);
    }
    const bool all = wild ||
        __popc(__ballot_sync(kFull, own * own * static_cast<float>(clusters) > kScattered * across * across)) > 16;
    if (tid == 0u) {
        scratch[clusters * (kClusterWords + kClusterBoxes)] = make_float4(all ? 1.0f : 0.0f, wild ? 1.0f : 0.0f, 0.0f, 0.0f);
    }
    if (all) { return; }
    float extent = 0.0f;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        lo[k] = bounds[k][lane];
        hi[k] = bounds[3 + k][lane];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            lo[k] = fminf(lo[k], __shfl_xor_sync(kFull, lo[k], o));
            hi[k] = fmaxf(hi[k], __shfl_xor_sync(kFull, hi[k], o));
        }
        extent = fmaxf(extent, hi[k] - lo[k]);
    }
    const float cells = static_cast<float>(1u << kBits);
    const float scale = extent > 0.0f ? cells / extent : 0.0f;
    const auto cell = [&](nxg_vec3 r) {
        const float v[3] = {r.x, r.y, r.z};
        uint32_t code = 0u;
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const float q = fminf(fmaxf((v[k] - lo[k]) * scale, 0.0f), cells - 1.0f);
            code |= spread3(static_cast<uint32_t>(q)) << k;
        }
        return min(code, bin_count - 1u);
    };
#pragma unroll
    for (uint32_t q = 0; q < kOwn; ++q) {
        if (q * 1024u + tid < guide_count) { atomicAdd(&bins[cell(root[q])], 1u); }
    }
    __syncthreads();
    const uint32_t per = (bin_count + 1023u) / 1024u, begin = min(bin_count, tid * per),
                   end = min(bin_count, begin + per);
    uint32_t sum = 0u;
    for (uint32_t i = begin; i < end; ++i) { sum += bins[i]; }
    uint32_t incl = sum;
#pragma unroll
    for (uint32_t o = 1u; o < 32u; o <<= 1) {
        const uint32_t u = __shfl_up_sync(kFull, incl, o);
        if (lane >= o) { incl += u; }
    }
    if (lane == 31u) { warp_sums[warp] = incl; }
    __syncthreads();
    uint32_t running = incl - sum + __reduce_add_sync(kFull, lane < warp ? warp_sums[lane] : 0u);
    for (uint32_t i = begin; i < end; ++i) {
        const uint32_t n = bins[i];
        bins[i] = running;
        running += n;
    }
    __syncthreads();
    float *planes = reinterpret_cast<float *>(scratch);
    const auto put = [planes](uint32_t at, nxg_vec3 r, uint32_t guide) {
        float *plane = planes + (at / kClusterGuides) * (4u * kClusterWords) + at % kClusterGuides;
        plane[0] = r.x;
        plane[kClusterGuides] = r.y;
        plane[2u * kClusterGuides] = r.z;
        plane[3u * kClusterGuides] = __uint_as_float(guide);
    };
#pragma unroll
    for (uint32_t q = 0; q < kOwn; ++q) {
        const uint32_t i = q * 1024u + tid;
        if (i < guide_count) { put(atomicAdd(&bins[cell(root[q])], 1u), root[q], i); }
    }
    // The last cluster's free entries: no guide, further than any.
    for (uint32_t i = guide_count + tid; i < clusters * kClusterGuides; i += 1024u) {
        put(i, nxg_vec3{1.0e18f, 1.0e18f, 1.0e18f}, kInvalid);
    }
    __syncthreads();
#pragma unroll 2
    for (uint32_t c = warp; c < clusters; c += 32u) {
        const float *plane = planes + c * (4u * kClusterWords) + lane;
        const bool guide = c * kClusterGuides + lane < guide_count;
        const uint32_t gi = __float_as_uint(plane[3u * kClusterGuides]);
        const nxg_vec3 m = guide ? guide_normals[gi] : nxg_vec3{0.0f, 0.0f, 0.0f};
        const float v[6] = {plane[0], plane[kClusterGuides], plane[2u * kClusterGuides], m.x, m.y, m.z};
        // A normal that is not finite agrees with every face: a box of all.
        const bool all = __any_sync(kFull, guide && !(fabsf(m.x) <= kWild && fabsf(m.y) <= kWild && fabsf(m.z) <= kWild));
        float low[6], high[6];
#pragma unroll
        for (int k = 0; k < 6; ++k) {
            low[k] = guide ? v[k] : FLT_MAX;
            high[k] = guide ? v[k] : -FLT_MAX;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                low[k] = fminf(low[k], __shfl_xor_sync(kFull, low[k], o));
                high[k] = fmaxf(high[k], __shfl_xor_sync(kFull, high[k], o));
            }
        }
        if (lane == 0u) {
            float4 *box = scratch + clusters * kClusterWords + kClusterBoxes * c;
            box[0] = make_float4(low[0], low[1], low[2],
                                 static_cast<float>(min(kClusterGuides, guide_count - c * kClusterGuides)));
            box[1] = make_float4(high[0], high[1], high[2], 0.0f);
            box[2] = all ? make_float4(-kWild, -kWild, -kWild, 0.0f) : make_float4(low[3], low[4], low[5], 0.0f);
            box[3] = all ? make_float4(kWild, kWild, kWild, 0.0f) : make_float4(high[3], high[4], high[5], 0.0f);
        }
    }
}

// Squared distance between the boxes [alo, ahi] and [blo, bhi].
__device__ __forceinline__ float box_distance2(F3 alo, F3 ahi, float4 blo, float4 bhi) {
    const float x = fmaxf(fmaxf(blo.x - ahi.x, alo.x - bhi.x), 0.0f);
    const float y = fmaxf(fmaxf(blo.y - ahi.y, alo.y - bhi.y), 0.0f);
    const float z = fmaxf(fmaxf(blo.z - ahi.z, alo.z - bhi.z), 0.0f);
    return x * x + y * y + z * z;
}

// The warp's triangles as one: the middle of their centroids' box and the
// largest distance of a centroid from it.
struct WarpBall {
    F3 middle;
    float radius;
};

// A triangle whose nearest guide is penalised (a degenerate one, whose face
// normal is (0, 1, 0) wherever it lies) has to reach guides that are not, past
// all the near ones.  For those of a warp that share one face normal, where at
// least eight guides agree with it, those eight come before every penalised
// one, so to the end of the search only guides that agree matter to them, and
// within `reach2` squared distance there are eight.
constexpr float kPenalty = 1.0e20f;
struct WarpAim {
    bool active;   // some triangle of the warp is aimed
    bool aimed;    // this lane's is
    F3 face;
    float reach2;
};

// What a guide has to be near enough for: the largest eighth score of the
// other triangles (any guide), and of the aimed ones (one that agrees), there at
// most their reach; -1 or 0 where there is no such triangle.
struct WarpWorst {
    float own, aimed;
};
__device__ __forceinline__ WarpWorst worst_scores(const TriangleSearch &t, const WarpAim &aim) {
    // Non-negative floats order as their bits.
    const uint32_t key = __float_as_uint(t.best[kSlots - 1].key);
    WarpWorst w;
    w.own = __uint_as_float(__reduce_max_sync(kFull, t.live && !aim.aimed ? key : 0u));
    w.aimed = -1.0f;
    if (aim.active) {
        w.aimed = fminf(__uint_as_float(__reduce_max_sync(kFull, aim.aimed ? key : 0u)), aim.reach2);
    }
    return w;
}

// The guides of one cluster for this warp's triangles.  A lane takes one guide;
// the lanes are sorted by their guides' distance from the warp's middle and
// hand round, nearest first, those near enough for some triangle: in that
// order few guides enter any list (a warp pays for an insertion of any of its
// lanes), and the loop reads no memory.
__device__ __forceinline__ void consider_cluster(TriangleSearch &t, const WarpBall &ball, const WarpAim &aim,
                                                 const float4 *cluster, const nxg_vec3 *__restrict__ guide_normals) {
    const uint32_t lane = threadIdx.x & 31u;
    const float *plane = reinterpret_cast<const float *>(cluster) + lane;
    const F3 own = {plane[0], plane[kClusterGuides], plane[2u * kClusterGuides]};
    const uint32_t own_guide = __float_as_uint(plane[3u * kClusterGuides]);
    const bool guide = own_guide != kInvalid;
    const nxg_vec3 own_normal = guide ? guide_normals[own_guide] : nxg_vec3{0.0f, 0.0f, 0.0f};
    const F3 off = own - ball.middle;
    const float distance = guide ? sqrtf(dot(off, off)) : FLT_MAX;
    // Bitonic sort of (distance, lane): the low five bits of the distance give
    // way to the lane, which only blurs the order.
    uint32_t key = (__float_as_uint(distance) & ~31u) | lane;
#pragma unroll
    for (uint32_t k = 2u; k <= 32u; k <<= 1) {
#pragma unroll
        for (uint32_t j = k >> 1; j > 0u; j >>= 1) {
            const uint32_t other = __shfl_xor_sync(kFull, key, j);
            const bool up = (lane & k) == 0u, low = (lane & j) == 0u;
            key = up == low ? min(key, other) : max(key, other);
        }
    }
    const int from = static_cast<int>(key & 31u);
    const F3 root = {__shfl_sync(kFull, own.x, from), __shfl_sync(kFull, own.y, from), __shfl_sync(kFull, own.z, from)};
    const F3 normal = {__shfl_sync(kFull, own_normal.x, from), __shfl_sync(kFull, own_normal.y, from),
                       __shfl_sync(kFull, own_normal.z, from)};
    const uint32_t gi = __shfl_sync(kFull, own_guide, from);
    // The least |d|^2 of this lane's guide from any of the triangles.
    const float reach = fmaxf(__shfl_sync(kFull, distance, from) - ball.radius, 0.0f);
    const float bound = gi != kInvalid ? reach * reach * kFilterMargin : FLT_MAX;
    const bool agrees = aim.active && !(xdot(aim.face, normal) < -0.25f);
    const auto near = [&]() {
        const WarpWorst w = worst_scores(t, aim);
        return __ballot_sync(kFull, gi != kInvalid && (bound <= w.own || (agrees && bound <= w.aimed)));
    };
    for (unsigned mask = near(); mask != 0u; mask &= mask - 1u) {
        const int i = __ffs(mask) - 1;
        const F3 d = xsub(t.centroid, F3{__shfl_sync(kFull, root.x, i), __shfl_sync(kFull, root.y, i),
                                         __shfl_sync(kFull, root.z, i)});
        const float l2 = xdot(d, d);
        if (!__any_sync(kFull, t.live && !(t.best[kSlots - 1].key < l2))) { continue; }  // the penalty only adds
        const F3 m = {__shfl_sync(kFull, normal.x, i), __shfl_sync(kFull, normal.y, i),
                      __shfl_sync(kFull, normal.z, i)};
        const Candidate c{__fadd_rn(l2, xdot(t.face, m) < -0.25f ? kPenalty : 0.0f), __shfl_sync(kFull, gi, i)};
        const bool enters = t.live && candidate_less(c.key, c.guide, t.best[kSlots - 1].key, t.best[kSlots - 1].guide);
        if (!__any_sync(kFull, enters)) { continue; }
        if (enters) { insert_candidate(t.best, c, kSlots - 1u); }
        mask &= near() | (1u << i);
    }
}

// The range of dot(face, normal) over a box of normals, widened by more than
// the rounding of both.
__device__ __forceinline__ float2 dot_range(F3 face, float4 lo, float4 hi) {
    const float x0 = face.x * lo.x, x1 = face.x * hi.x, y0 = face.y * lo.y, y1 = face.y * hi.y;
    const float z0 = face.z * lo.z, z1 = face.z * hi.z;
    const float slack = 1.0e-5f * (fmaxf(fabsf(x0), fabsf(x1)) + fmaxf(fabsf(y0), fabsf(y1)) + fmaxf(fabsf(z0), fabsf(z1)));
    return make_float2(fminf(x0, x1) + fminf(y0, y1) + fminf(z0, z1) - slack,
                       fmaxf(x0, x1) + fmaxf(y0, y1) + fmaxf(z0, z1) + slack);
}

// Finds the warp's aim for the triangles that the guide of `normal`, the
// nearest to the warp's middle, is penalised for: the nearest (by its furthest
// corner) cluster of at least eight guides that all agree with the face of the
// first of them.  Every lane of the warp calls it.
__device__ __forceinline__ WarpAim find_aim(const TriangleSearch &t, const WarpBall &ball, F3 normal,
                                            const float4 *boxes, uint32_t clusters) {
    WarpAim aim{false, false, F3{0.0f, 0.0f, 0.0f}, 0.0f};
    const bool open = t.live && xdot(t.face, normal) < -0.25f;
    const unsigned any = __ballot_sync(kFull, open);
    if (any == 0u) { return aim; }
    const int leader = __ffs(any) - 1;
    aim.face = F3{__shfl_sync(kFull, t.face.x, leader), __shfl_sync(kFull, t.face.y, leader),
                  __shfl_sync(kFull, t.face.z, leader)};
    float nearest = FLT_MAX;
    for (uint32_t c = threadIdx.x & 31u; c < clusters; c += 32u) {
        const float4 *box = boxes + kClusterBoxes * c;
        if (box[0].w < static_cast<float>(kSlots) || dot_range(aim.face, box[2], box[3]).x < -0.25f) { continue; }
        const F3 far = {fmaxf(fabsf(box[0].x - ball.middle.x), fabsf(box[1].x - ball.middle.x)),
                        fmaxf(fabsf(box[0].y - ball.middle.y), fabsf(box[1].y - ball.middle.y)),
                        fmaxf(fabsf(box[0].z - ball.middle.z), fabsf(box[1].z - ball.middle.z))};
        nearest = fminf(nearest, sqrtf(dot(far, far)));
    }
    nearest = __uint_as_float(__reduce_min_sync(kFull, __float_as_uint(nearest)));
    if (nearest == FLT_MAX) { return aim; }
    const float reach = nearest + ball.radius;
    aim.reach2 = reach * reach * 1.00002f;
    aim.active = aim.reach2 < 0.5f * kPenalty;
    aim.aimed = aim.active && open && t.face.x == aim.face.x && t.face.y == aim.face.y && t.face.z == aim.face.z;
    return aim;
}

// The search of this warp's triangles over the scratch's clusters; every lane
// of the warp calls it.  The nearest cluster first (its guides give bounds
// near the final ones), then, 32 clusters at a time and nearest first, those
// whose box is near enough to the box of the warp's centroids.  A box or ball
// distance is at most the computed |d|^2 of any pair it covers but for
// rounding, which kFilterMargin covers.
__device__ __forceinline__ void search_clusters(TriangleSearch &t, const WarpBox &bounds, const float4 *scratch,
                                                uint32_t clusters, const nxg_vec3 *__restrict__ guide_normals) {
    const uint32_t lane = threadIdx.x & 31u;
    const float4 *boxes = scratch + clusters * kClusterWords;
#pragma unroll
    for (uint32_t k = 0; k < kSlots; ++k) { t.best[k] = {INFINITY, kInvalid}; }
    if (__ballot_sync(kFull, t.live) == 0u) { return; }
    const F3 lo = bounds.lo, hi = bounds.hi;
    WarpBall ball;
    ball.middle = (lo + hi) * 0.5f;
    const F3 out = t.centroid - ball.middle;
    // (Rounded up: the radius is subtracted from distances to the middle, whose
    // own rounding is relative to the coordinates.)
    const F3 size = {fmaxf(fabsf(lo.x), fabsf(hi.x)), fmaxf(fabsf(lo.y), fabsf(hi.y)),
                     fmaxf(fabsf(lo.z), fabsf(hi.z))};
    const float slack = 1.0e-6f * (size.x + size.y + size.z);
    ball.radius = __uint_as_float(__reduce_max_sync(
                      kFull, t.live ? __float_as_uint(sqrtf(dot(out, out)) * 1.000001f) : 0u)) + slack;
    float nearest = FLT_MAX;
    uint32_t first = 0u;
    for (uint32_t c = lane; c < clusters; c += 32u) {
        const float d = box_distance2(ball.middle, ball.middle, boxes[kClusterBoxes * c], boxes[kClusterBoxes * c + 1u]);
        if (d < nearest) {
            nearest = d;
            first = c;
        }
    }
    const uint32_t least = __reduce_min_sync(kFull, __float_as_uint(nearest));
    first = __shfl_sync(kFull, first, __ffs(__ballot_sync(kFull, __float_as_uint(nearest) == least)) - 1);
    F3 normal;
    {
        const float *plane = reinterpret_cast<const float *>(scratch + first * kClusterWords) + lane;
        const F3 off = F3{plane[0], plane[kClusterGuides], plane[2u * kClusterGuides]} - ball.middle;
        const uint32_t gi = __float_as_uint(plane[3u * kClusterGuides]);
        const uint32_t bits = __float_as_uint(gi == kInvalid ? FLT_MAX : dot(off, off));
        const int lead = __ffs(__ballot_sync(kFull, bits == __reduce_min_sync(kFull, bits))) - 1;
        const nxg_vec3 m = guide_normals[__shfl_sync(kFull, gi, lead)];
        normal = F3{m.x, m.y, m.z};
    }
    const WarpAim aim = find_aim(t, ball, normal, boxes, clusters);
    consider_cluster(t, ball, aim, scratch + first * kClusterWords, guide_normals);
    for (uint32_t base = 0; base < clusters; base += 32u) {
        const float4 *mine = boxes + kClusterBoxes * (base + lane);
        float box = FLT_MAX;
        bool agrees = false;
        if (base + lane < clusters && base + lane != first) {
            box = box_distance2(lo, hi, mine[0], mine[1]) * kFilterMargin;
            agrees = aim.active && !(dot_range(aim.face, mine[2], mine[3]).y < -0.25f);
        }
        for (uint32_t guard = 0; guard < 32u; ++guard) {
            const WarpWorst worst = worst_scores(t, aim);
            const bool near = box <= worst.own || (agrees && box <= worst.aimed);
            const uint32_t next = __reduce_min_sync(kFull, __float_as_uint(near ? box : FLT_MAX));
            if (next == __float_as_uint(FLT_MAX)) { break; }
            const uint32_t c = static_cast<uint32_t>(__ffs(__ballot_sync(kFull, near && __float_as_uint(box) == next))) - 1u;
            if (lane == c) { box = FLT_MAX; }
            consider_cluster(t, ball, aim, scratch + (base + c) * kClusterWords, guide_normals);
        }
    }
}

__device__ __forceinline__ bool wild_triangle(const TriangleSearch &t) {
    return t.live && !(fabsf(t.centroid.x) <= kWild && fabsf(t.centroid.y) <= kWild && fabsf(t.centroid.z) <= kWild);
}

// Whether the CTA's triangles lie scattered over too many clusters: whether its
// warps' boxes touch more than a quarter of the clusters and three on average
// (neighbours touch 2 to 5; all pairs cost as much as visits to a seventh of
// them, but a CTA alone takes as long for them as the whole search does).  Every
// thread of the CTA calls it.
__device__ __forceinline__ bool scattered_triangles(const WarpBox &bounds, const float4 *scratch, uint32_t clusters) {
    const float4 *boxes = scratch + clusters * kClusterWords;
    uint32_t touched = 0u;
    for (uint32_t c = threadIdx.x & 31u; c < clusters; c += 32u) {
        touched += box_distance2(bounds.lo, bounds.hi, boxes[kClusterBoxes * c], boxes[kClusterBoxes * c + 1u]) == 0.0f;
    }
    __shared__ uint32_t sum;
    if (threadIdx.x == 0u) { sum = 0u; }
    __syncthreads();
    touched = __reduce_add_sync(kFull, touched);
    if ((threadIdx.x & 31u) == 0u) { atomicAdd(&sum, touched); }
    __syncthreads();
    return sum * 4u > (blockDim.x >> 5) * (clusters + 12u);
}

// The all-pairs search of one triangle, which every thread of the CTA holds, for
// finite positions: each takes every blockDim-th guide, and the CTA picks the
// least (score, guide) eight times.  (By one thread, a triangle that every
// guide is penalised for takes 70 us of 1,024 guides.)
__device__ __forceinline__ void share_triangle(TriangleSearch &t, const nxg_vec3 *__restrict__ guide_roots,
                                               const nxg_vec3 *__restrict__ guide_normals, uint32_t guide_count) {
    constexpr unsigned long long kNone = ~0ull;
    __shared__ unsigned long long least[2], row[kSlots];
    unsigned long long last = 0ull;
    if (threadIdx.x < 2u) { least[threadIdx.x] = kNone; }
    __syncthreads();
#pragma unroll 1
    for (uint32_t k = 0; k < kSlots; ++k) {
        unsigned long long mine = kNone;
        for (uint32_t gi = threadIdx.x; gi < guide_count; gi += blockDim.x) {
            const nxg_vec3 r = guide_roots[gi], m = guide_normals[gi];
            const F3 d = xsub(t.centroid, F3{r.x, r.y, r.z});
            const float key = __fadd_rn(xdot(d, d), xdot(t.face, F3{m.x, m.y, m.z}) < -0.25f ? kPenalty : 0.0f);
            const unsigned long long c = static_cast<unsigned long long>(__float_as_uint(key)) << 32 | gi;
            if ((k == 0u || c > last) && c < mine) { mine = c; }
        }
        if (mine != kNone) { atomicMin(&least[k & 1u], mine); }
        __syncthreads();
        last = least[k & 1u];
        if (threadIdx.x == 0u) {
            least[(k + 1u) & 1u] = kNone;
            row[k] = last;
        }
        __syncthreads();
    }
#pragma unroll
    for (uint32_t k = 0; k < kSlots; ++k) {
        t.best[k] = {__uint_as_float(static_cast<uint32_t>(row[k] >> 32)), static_cast<uint32_t>(row[k])};
    }
}

// Triangles [0, first) from the scratch in global memory (the rows from `first`
// on); where every triangle takes all pairs, those of the scratch's rows too but
// for the last row, which says so.
__global__ void __launch_bounds__(kStencilThreads, 8)
stencil_cluster_kernel(const nxg_vec3 *__restrict__ positions, uint32_t vertex_count,
                       const nxg_uint3 *__restrict__ triangles, uint32_t first, uint32_t triangle_count,
                       const nxg_vec3 *__restrict__ guide_roots, const nxg_vec3 *__restrict__ guide_normals,
                       uint32_t guide_count, uint32_t clusters, uint32_t keep, uint32_t *stencil) {
    __shared__ __align__(16) GuideTile tile;
    chain_wait();
    chain_start();  // from here on the scratch is complete, which the next kernel relies on
    const float4 *scratch = reinterpret_cast<const float4 *>(stencil + static_cast<size_t>(first) * kSlots);
    const bool all = __ldcg(&scratch[clusters * (kClusterWords + kClusterBoxes)].x) != 0.0f;
    const uint32_t end = all ? triangle_count - 1u : first;
    if (blockIdx.x * kStencilThreads >= end) { return; }
    const uint32_t ti = blockIdx.x * kStencilThreads + threadIdx.x;
    TriangleSearch t;
    begin_triangle(t, ti, positions, vertex_count, triangles, end);
    const WarpBox bounds = warp_box(t);
    if (__syncthreads_or(all || wild_triangle(t)) || scattered_triangles(bounds, scratch, clusters)) {
        search_all(t, tile, guide_roots, guide_normals, guide_count);
    } else {
        search_clusters(t, bounds, scratch, clusters, guide_normals);
    }
    end_triangle(t, ti, keep, stencil);
}

// The rows the scratch is in: one thread-block cluster, whose CTAs copy the
// scratch to shared memory before any of them writes a row.  It starts once
// every CTA of stencil_cluster_kernel has seen the scratch complete, searches
// beside that kernel's end and writes after it.  Where every triangle takes all
// pairs (the last row, which nobody else writes, says so) it has that row
// alone, and one CTA shares its guides out to its threads unless one is wild.
__global__ void __launch_bounds__(kTailMaxThreads)
stencil_tail_kernel(const nxg_vec3 *__restrict__ positions, uint32_t vertex_count,
                    const nxg_uint3 *__restrict__ triangles, uint32_t first, uint32_t triangle_count,
                    const nxg_vec3 *__restrict__ guide_roots, const nxg_vec3 *__restrict__ guide_normals,
                    uint32_t guide_count, uint32_t clusters, uint32_t keep, uint32_t *stencil) {
    extern __shared__ float4 copy[];
    __shared__ __align__(16) GuideTile tile;
    const float4 *scratch = reinterpret_cast<const float4 *>(stencil + static_cast<size_t>(first) * kSlots);
    for (uint32_t i = threadIdx.x; i < cluster_scratch_words(clusters); i += blockDim.x) {
        copy[i] = __ldcg(scratch + i);
    }
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    const float4 flags = copy[clusters * (kClusterWords + kClusterBoxes)];
    const bool all = flags.x != 0.0f;
    TriangleSearch t;
    if (all && flags.y == 0.0f) {
        begin_triangle(t, triangle_count - 1u, positions, vertex_count, triangles, triangle_count);
        if (!wild_triangle(t)) {  // the same triangle in every thread
            if (blockIdx.x != 0u) { return; }
            if (t.live) { share_triangle(t, guide_roots, guide_normals, guide_count); }
            chain_wait();
            if (threadIdx.x == 0u) { end_triangle(t, triangle_count - 1u, keep, stencil); }
            return;
        }
    }
    const uint32_t ti = first + blockIdx.x * blockDim.x + threadIdx.x;
    begin_triangle(t, ti, positions, vertex_count, triangles, triangle_count);
    if (all && ti != triangle_count - 1u) { t.live = t.invalid = false; }
    const WarpBox bounds = warp_box(t);
    if (__syncthreads_or(all || wild_triangle(t))) {
        if (!__syncthreads_or(t.live || t.invalid)) { return; }
        search_all(t, tile, guide_roots, guide_normals, guide_count);
    } else {
        search_clusters(t, bounds, copy, clusters, guide_normals);
    }
    chain_wait();
    end_triangle(t, ti, keep, stencil);
}

// Distance from every guide root to its nearest other root (the automatic
// support radius, src/asset.cpp automatic_support_radius): |root_i - root_j|
// with IEEE sqrt, minimum over j != i with a CV count > 0.  One warp per
// guide, lanes striding over j, then a warp minimum: every distance is >= +0,
// a NaN one never replaces a lane's running value (which starts at FLT_MAX,
// as the host's), so the minimum is the host's whatever the order.
__global__ void __launch_bounds__(kStencilThreads)
guide_nearest_kernel(const nxg_vec3 *__restrict__ roots, const uint32_t *__restrict__ cv_counts, uint32_t guide_count,
                     float *__restrict__ nearest) {
    const uint32_t gi = (blockIdx.x * kStencilThreads + threadIdx.x) >> 5, lane = threadIdx.x & 31u;
    if (gi >= guide_count) { return; }  // whole warps
    const nxg_vec3 r = roots[gi];
    const F3 root{r.x, r.y, r.z};
    float best = 3.402823466e38f;  // FLT_MAX
    for (uint32_t j = lane; j < guide_count; j += 32u) {
        if (j == gi || cv_counts[j] == 0u) { continue; }
        const nxg_vec3 o = roots[j];
        const F3 d = xsub(root, F3{o.x, o.y, o.z});
        const float dist = __fsqrt_rn(xdot(d, d));
        best = dist < best ? dist : best;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) { best = fminf(best, __shfl_xor_sync(kFull, best, o)); }
    if (lane == 0u) { nearest[gi] = best; }
}

uint32_t slots_kept(uint32_t guide_count, uint32_t stencil_slots) {
    const uint32_t count = guide_count < kSlots ? guide_count : kSlots;
    return stencil_slots == 0u || stencil_slots > count ? count : stencil_slots;
}

static_assert((cluster_scratch_rows(kMaxClusters) + kTailCtas - 1u) / kTailCtas <= kTailMaxThreads, "one CTA cluster");

cudaError_t launch_stencils(const nxg_vec3 *positions, uint32_t vertex_count, const nxg_uint3 *triangles,
                         uint32_t triangle_count, const nxg_vec3 *guide_roots, const nxg_vec3 *guide_normals,
                         uint32_t guide_count, uint32_t stencil_slots, uint32_t *stencil, cudaStream_t stream) {
    const uint32_t keep = slots_kept(guide_count, stencil_slots);
    const uint32_t clusters = (guide_count + kClusterGuides - 1u) / kClusterGuides;
    const uint32_t rows = cluster_scratch_rows(clusters);
    // The cluster search where it is faster: enough pairs to pay for the sort
    // (all pairs against clusters: 20,000 x 1,000 96 / 80 us, 20,000 x 640 72 /
    // 105, 200,000 x 640 123 / 81), triangles close enough together that a warp
    // shares its guides (50,000 x 4,096 320 / 190 us, 10,000 x 4,096 297 / 429),
    // and up to kMaxClusters.
    if (guide_count < kClusterMinGuides || clusters > kMaxClusters || triangle_count / 12u < guide_count ||
        uint64_t{triangle_count} * guide_count < 20000000u) {
        const uint32_t blocks = (triangle_count + kStencilThreads - 1u) / kStencilThreads;
        stencil_kernel<<<blocks, kStencilThreads, 0, stream>>>(positions, vertex_count, triangles, triangle_count,
                                                               guide_roots, guide_normals, guide_count, keep, stencil);
        return cudaGetLastError();
    }
    const uint32_t first = triangle_count - rows;  // row of the scratch
    const size_t copy = sizeof(float4) * cluster_scratch_words(clusters);
    const uint32_t tail_threads = ((rows + kTailCtas - 1u) / kTailCtas + 31u) / 32u * 32u;
    // The largest copy, whatever this call's: the limit is the process's.
    cudaError_t e = cudaFuncSetAttribute(stencil_tail_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         static_cast<int>(sizeof(float4) * cluster_scratch_words(kMaxClusters)));
    // The same share of the SM's memory for both kernels: with the shares of
    // their own occupancies the second did not start beside the first until its
    // SMs were empty (39,600 x 1,000 62 -> 53 us, 200,000 x 4,096 130 -> 118).
    for (const void *fn : {reinterpret_cast<const void *>(stencil_cluster_kernel),
                           reinterpret_cast<const void *>(stencil_tail_kernel)}) {
        if (e == cudaSuccess) { e = cudaFuncSetAttribute(fn, cudaFuncAttributePreferredSharedMemoryCarveout, 58); }
    }
    if (e != cudaSuccess) { return e; }
    cudaLaunchConfig_t config{};
    cudaLaunchAttribute attributes[2];
    attributes[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attributes[0].val.programmaticStreamSerializationAllowed = 1;
    attributes[1].id = cudaLaunchAttributeClusterDimension;
    attributes[1].val.clusterDim.x = kTailCtas;
    attributes[1].val.clusterDim.y = attributes[1].val.clusterDim.z = 1u;
    config.stream = stream;
    config.attrs = attributes;
    config.gridDim = dim3(1);
    config.blockDim = dim3(1024);
    config.dynamicSmemBytes = 0u;
    e = cudaLaunchKernelEx(&config, cluster_kernel, positions, vertex_count, triangles, triangle_count, guide_roots,
                           guide_normals, guide_count, clusters,
                           reinterpret_cast<float4 *>(stencil + static_cast<size_t>(first) * kSlots));
    if (e != cudaSuccess) { return e; }
    config.numAttrs = 1u;
    config.gridDim = dim3((triangle_count + kStencilThreads - 1u) / kStencilThreads);
    config.blockDim = dim3(kStencilThreads);
    config.dynamicSmemBytes = 0u;
    e = cudaLaunchKernelEx(&config, stencil_cluster_kernel, positions, vertex_count, triangles, first, triangle_count,
                           guide_roots, guide_normals, guide_count, clusters, keep, stencil);
    if (e != cudaSuccess) { return e; }
    config.numAttrs = 2u;
    config.gridDim = dim3(kTailCtas);
    config.blockDim = dim3(tail_threads);
    config.dynamicSmemBytes = copy;
    return cudaLaunchKernelEx(&config, stencil_tail_kernel, positions, vertex_count, triangles, first, triangle_count,
                              guide_roots, guide_normals, guide_count, clusters, keep, stencil);
}

size_t align256(size_t n) { return (n + 255u) & ~size_t{255u}; }

} // namespace
} // namespace dev

int device_guide_search(const nxg_vec3 *positions, uint32_t vertex_count, const nxg_uint3 *triangles,
                        uint32_t triangle_count, const nxg_vec3 *guide_roots, const nxg_vec3 *guide_normals,
                        const uint32_t *guide_cv_counts, uint32_t guide_count, uint32_t stencil_slots,
                        uint32_t *stencil, float *nearest, void *stream, const char **what) noexcept {
    using dev::align256;
    const cudaStream_t s = static_cast<cudaStream_t>(stream);
    const size_t vb = size_t{vertex_count} * sizeof(nxg_vec3), tb = size_t{triangle_count} * sizeof(nxg_uint3);
    const size_t gb = size_t{guide_count} * sizeof(nxg_vec3), sb = size_t{triangle_count} * NXG_GUIDE_STENCIL_SIZE * 4u;
    const size_t o_tri = align256(vb), o_root = o_tri + align256(tb), o_normal = o_root + align256(gb);
    const size_t cb = size_t{guide_count} * 4u, o_counts = o_normal + align256(gb);
    const size_t o_nearest = o_counts + align256(cb), o_stencil = o_nearest + align256(cb);
    const size_t total = o_stencil + align256(sb);
    char *base = nullptr;
    cudaError_t e = cudaMallocAsync(reinterpret_cast<void **>(&base), total, s);
    if (e != cudaSuccess) {
        *what = cudaGetErrorString(e);
        set_last_cuda_error(static_cast<int32_t>(e));
        return static_cast<int>(e);
    }
    auto *d_pos = reinterpret_cast<nxg_vec3 *>(base);
    auto *d_tri = reinterpret_cast<nxg_uint3 *>(base + o_tri);
    auto *d_root = reinterpret_cast<nxg_vec3 *>(base + o_root);
    auto *d_normal = reinterpret_cast<nxg_vec3 *>(base + o_normal);
    auto *d_counts = reinterpret_cast<uint32_t *>(base + o_counts);
    auto *d_nearest = reinterpret_cast<float *>(base + o_nearest);
    auto *d_stencil = reinterpret_cast<uint32_t *>(base + o_stencil);
    if ((e = cudaMemcpyAsync(d_pos, positions, vb, cudaMemcpyHostToDevice, s)) == cudaSuccess &&
        (e = cudaMemcpyAsync(d_tri, triangles, tb, cudaMemcpyHostToDevice, s)) == cudaSuccess &&
        (e = cudaMemcpyAsync(d_root, guide_roots, gb, cudaMemcpyHostToDevice, s)) == cudaSuccess &&
        (e = cudaMemcpyAsync(d_normal, guide_normals, gb, cudaMemcpyHostToDevice, s)) == cudaSuccess &&
        (e = cudaMemcpyAsync(d_counts, guide_cv_counts, cb, cudaMemcpyHostToDevice, s)) == cudaSuccess) {
        const uint64_t threads = uint64_t{guide_count} * 32u;
        const uint32_t blocks = static_cast<uint32_t>((threads + dev::kStencilThreads - 1u) / dev::kStencilThreads);
        dev::guide_nearest_kernel<<<blocks, dev::kStencilThreads, 0, s>>>(d_root, d_counts, guide_count, d_nearest);
        if ((e = cudaGetLastError()) == cudaSuccess &&
            (e = dev::launch_stencils(d_pos, vertex_count, d_tri, triangle_count, d_root, d_normal, guide_count,
                                      stencil_slots, d_stencil, s)) == cudaSuccess &&
            (e = cudaMemcpyAsync(nearest, d_nearest, cb, cudaMemcpyDeviceToHost, s)) == cudaSuccess) {
            e = cudaMemcpyAsync(stencil, d_stencil, sb, cudaMemcpyDeviceToHost, s);
        }
    }
    const cudaError_t freed = cudaFreeAsync(base, s);
    const cudaError_t synced = cudaStreamSynchronize(s);
    if (e == cudaSuccess) { e = freed != cudaSuccess ? freed : synced; }
    if (e != cudaSuccess) {
        *what = cudaGetErrorString(e);
        set_last_cuda_error(static_cast<int32_t>(e));
        return static_cast<int>(e);
    }
    return 0;
}

} // namespace nxg

extern "C" uint32_t nxg_build_stencils_device(const nxg_vec3 *positions, uint32_t vertex_count,
                                              const nxg_uint3 *triangles, uint32_t triangle_count,
                                              const nxg_vec3 *guide_roots, const nxg_vec3 *guide_normals,
                                              uint32_t guide_count, uint32_t stencil_slots, uint32_t *stencil,
                                              void *stream) {
    if (!positions || !triangles || !guide_roots || !guide_normals || !stencil || vertex_count == 0u ||
        triangle_count == 0u || guide_count == 0u || stencil_slots > NXG_GUIDE_STENCIL_SIZE) {
        return NXG_ERROR_INVALID_ARGUMENT;
    }
    if (reinterpret_cast<uintptr_t>(stencil) % 16u != 0u) { return NXG_ERROR_MISALIGNED_OUTPUT; }
    nxg::set_last_cuda_error(0);
    return nxg::record_cuda(nxg::dev::launch_stencils(positions, vertex_count, triangles, triangle_count, guide_roots,
                                                      guide_normals, guide_count, stencil_slots, stencil,
                                                      static_cast<cudaStream_t>(stream)));
}
