// generate.cu -- the packed strand generator for sm_100a and its C-ABI entry
// points (nxg_generate_packed, nxg_generate_packed_range,
// nxg_packed_workspace_size, nxg_query_strand_states).
//
// Pipeline per call, all enqueued on the caller's stream as chained launches
// (chain_wait); 2 to 4 only where the strand order pays (wants_order):
//   1. guide_offsets   : the frame's guide-offset table and guide frame
//                        records;
//   2. strand_keys     : alias-sample every strand's root triangle and bin the
//                        strand by its triangle's nearest stencil guide
//                        (a counting sort's histogram pass);
//   3. exclusive_scan  : bin offsets;
//   4. scatter_order   : the permutation that groups strands sharing guides,
//                        so one CTA's strands read the same guide CVs from L1
//                        (ranks in shared memory per block, one global atomic
//                        per block and bin);
//   5. generate        : persistent CTAs walk contiguous ranges of the strands
//                        (in that order) with the lane-walk generator
//                        (walk.cuh).  Where a lane-group tile is registered
//                        (nxg_set_tile, up to 128 CVs): a group of L lanes
//                        owns one strand, the transported frame as prefix
//                        scans over shuffles (generator_core.cuh), with a
//                        separate roots kernel.
// Strands whose guide-offset table does not fit (the table's cap, more than
// 1,024 CVs, or past 128 CVs a workspace without room for it) take a serial
// per-thread kernel that walks the reference's cursor directly.
#include "generator_core.cuh"
#include "walk.cuh"
#include "nxg_internal.h"
#include "strand_math.cuh"

#include <cuda_runtime.h>

#include <cfloat>
#include <cmath>
#include <cstdint>
#include <algorithm>
#include <atomic>
#include <mutex>
#include <cstring>

namespace nxg {
namespace dev {

// Persistent CTAs over contiguous ranges of the strand order.  Each warp
// takes 32 strands at a time: phase A sets them up one lane per strand,
// phase B emits them one L-lane group per strand.
template <int L, int PPT, bool NOISE, bool CLASSIC>
__global__ void generate_kernel(LaunchArgs g, const float4 *offsets) {
    extern __shared__ float4 smem[];
    constexpr int kGroups = 32 / L;
    constexpr int kLatticePerWarp = 384;                 // float2 columns per warp (3 axes)
    constexpr int kLatticeMax = kLatticePerWarp / 3 / kGroups;
    const int P = static_cast<int>(g.p.cvs_per_strand);
    const int warps = blockDim.x >> 5;
    // Layout: gradient table | t values | per warp: records, stage, lattice.
    float4 *table = smem;
    float *tvals = reinterpret_cast<float *>(smem + kTableFloat4);
    unsigned char *warp_base = reinterpret_cast<unsigned char *>(tvals + ((P + 3) & ~3));
    const size_t rec_bytes = sizeof(uint32_t) * kRecFields * 32;
    const size_t stage_bytes = sizeof(float4) * kGroups * L * PPT;
    const size_t lattice_bytes = NOISE ? sizeof(float2) * kLatticePerWarp : 0;
    const size_t per_warp = rec_bytes + stage_bytes + lattice_bytes;
    if constexpr (NOISE) {
        for (int i = threadIdx.x; i < kTableFloat4; i += blockDim.x) {
            table[i] = make_float4(__ldg(g.a.gradients + 3 * i), __ldg(g.a.gradients + 3 * i + 1),
                                   __ldg(g.a.gradients + 3 * i + 2), 0.0f);
        }
    }
    for (int i = threadIdx.x; i < P; i += blockDim.x) {  // t = cv / (P - 1) (generate.h:295-298)
        tvals[i] = __fdiv_rn(static_cast<float>(i), static_cast<float>(P - 1));
    }
    __syncthreads();
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    const int group = lane / L;
    const int gl = lane % L;
    unsigned char *mine = warp_base + per_warp * warp;
    const Records rec{reinterpret_cast<uint32_t *>(mine)};
    float4 *stage = reinterpret_cast<float4 *>(mine + rec_bytes) + group * (L * PPT);
    float2 *lattice = reinterpret_cast<float2 *>(mine + rec_bytes + stage_bytes) + group * (kLatticePerWarp / kGroups);
    const uint32_t begin = static_cast<uint32_t>(static_cast<uint64_t>(blockIdx.x) * g.count / gridDim.x);
    const uint32_t end = static_cast<uint32_t>(static_cast<uint64_t>(blockIdx.x + 1u) * g.count / gridDim.x);
    for (uint32_t batch = begin + static_cast<uint32_t>(warp) * 32u; batch < end;
         batch += static_cast<uint32_t>(warps) * 32u) {
        const uint32_t item = batch + static_cast<uint32_t>(lane);
        const bool valid = item < end;
        setup_strand<NOISE>(g, rec, lane, valid ? item : batch, valid);
        __syncwarp();
        const uint32_t in_batch = min(32u, end - batch);
#pragma unroll 1
        for (uint32_t r = 0; r < in_batch; r += kGroups) {
            emit_strand<L, PPT, NOISE, CLASSIC>(g, rec, static_cast<int>(r) + group, gl, table, offsets, tvals, stage,
                                       lattice, kLatticeMax);
        }
        __syncwarp();
    }
}

// The lane-walk generator (walk.cuh).  Persistent CTAs over contiguous ranges
// of the strand order; each warp takes g.batch strands at a time.  Register
// budgets: the noise variant runs one CTA of up to twelve warps per SM (at
// most 168 registers), the plain one three CTAs of eight warps (at most 80
// registers; with Classic scalars on 4,000,000 strands x 24, 902 us, two CTAs
// 1,037, four 1,135).  The arguments stay in the constant
// bank (__grid_constant__): an out-of-line call taking them by reference
// otherwise copies them to every thread's stack first.
template <bool NOISE, bool CLASSIC, int CHUNK = kWalkChunk>
__global__ void __launch_bounds__(NOISE ? 32 * walk_noise_warps(CHUNK) : 256, NOISE ? 1 : 3)
    generate_walk_kernel(const __grid_constant__ LaunchArgs g, const float4 *offsets) {
    extern __shared__ float4 smem[];
    const uint32_t P = g.p.cvs_per_strand;
    const uint32_t padded = walk_padded(P);
    float *tvals = reinterpret_cast<float *>(smem + (NOISE ? kTableFloat4 << walk_table_copies(blockDim.x >> 5, CHUNK) : 0));
    float *rvals = tvals + padded;
    walk_fill_head<NOISE, CHUNK>(g, smem, tvals, rvals);  // of the asset and the arguments alone
    __syncthreads();
    chain_start();
    chain_wait();
    const int lane = threadIdx.x & 31;
    const uint32_t warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
    unsigned char *mine = reinterpret_cast<unsigned char *>(rvals + padded) + walk_warp_bytes(NOISE, CLASSIC, CHUNK) * warp;
    const uint32_t begin = static_cast<uint32_t>(static_cast<uint64_t>(blockIdx.x) * g.count / gridDim.x);
    const uint32_t end = static_cast<uint32_t>(static_cast<uint64_t>(blockIdx.x + 1u) * g.count / gridDim.x);
    for (uint32_t batch = begin + warp * g.batch; batch < end; batch += warps * g.batch) {
        const int in_batch = static_cast<int>(min(g.batch, end - batch));
        if constexpr (NOISE) {
            walk_noise_batch<CLASSIC, CHUNK>(g, offsets, mine, smem, tvals, rvals, lane, batch, in_batch);
        } else {
            walk_plain_batch<CLASSIC>(g, offsets, mine, tvals, rvals, lane, batch, in_batch);
        }
    }
}

// The Classic application for the serial generator: one thread
// per strand re-reads its written points (xgen_classic_runtime.cpp:1650-1678,
// :1827-1858), measuring cLength for every strand.
__global__ void classic_serial_apply_kernel(LaunchArgs g) {
    const int P = static_cast<int>(g.p.cvs_per_strand);
    const float rs = g.p.radius_scale;
    for (uint32_t local = blockIdx.x * blockDim.x + threadIdx.x; local < g.count; local += gridDim.x * blockDim.x) {
        float4 *pts = g.points + static_cast<uint64_t>(local) * static_cast<uint32_t>(P);
        const float2 sc = g.scalars[local];
        const float s = g.classic_length ? sc.x : 1.0f;
        const float raw_width = g.classic_width ? sc.y : (rs > 0.0f ? __fdiv_rn(__fmul_rn(2.0f, pts[0].w), rs) : 0.0f);
        bool keep = !(raw_width < 1.0e-4f);
        if (keep) { keep = !(__fmul_rn(classic_spline_length(pts, P), s) < 1.0e-4f); }
        const F3 front = xyz(pts[0]);
        const float radius = __fmul_rn(__fmul_rn(0.5f, raw_width < 0.0f ? 0.0f : raw_width), rs);
        for (int cv = 0; cv < P; ++cv) {
            float4 q = pts[cv];
            if (g.classic_length) {
                const F3 v = xadd(front, xmul(xsub(xyz(q), front), s));
                q.x = v.x;
                q.y = v.y;
                q.z = v.z;
            }
            if (g.classic_width) { q.w = radius; }
            pts[cv] = q;
        }
        if (!keep && g.point_counts != nullptr) { g.point_counts[local] = 0u; }
    }
}

// RootSample, root UV and point count of every strand of the range, in
// output order (coalesced), for the frame (generate.h:101-135, :621-623).
__global__ void strand_roots_kernel(LaunchArgs g) {
    __shared__ uint32_t staged[8][32 * 12];
    chain_start();
    chain_wait();
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    const uint32_t P = g.p.cvs_per_strand;
    for (uint32_t base = (blockIdx.x * (blockDim.x >> 5) + warp) * 32u; base < g.count;
         base += gridDim.x * (blockDim.x >> 5) * 32u) {
        const uint32_t i = base + lane;
        const bool valid = i < g.count;
        const Root r = sample_root(g.a, g.f, g.p.seed, g.first_strand + (valid ? i : base));
        uint32_t *rec = staged[warp] + lane * 12;
        rec[0] = __float_as_uint(r.position.x);
        rec[1] = __float_as_uint(r.position.y);
        rec[2] = __float_as_uint(r.position.z);
        rec[3] = __float_as_uint(r.normal.x);
        rec[4] = __float_as_uint(r.normal.y);
        rec[5] = __float_as_uint(r.normal.z);
        rec[6] = __float_as_uint(r.u);
        rec[7] = __float_as_uint(r.v);
        rec[8] = r.triangle;
        rec[9] = __float_as_uint(r.b1);
        rec[10] = __float_as_uint(r.b2);
        rec[11] = r.triangle;  // surface_face_id == triangle_index (generate.h:134)
        __syncwarp();
        const uint32_t n = min(32u, g.count - base);
        if (g.roots) {
            uint32_t *dst = g.roots + static_cast<uint64_t>(base) * 12u;
            for (uint32_t w = lane; w < n * 12u; w += 32u) { dst[w] = staged[warp][w]; }
        }
        if (valid) {
            if (g.root_uvs) { g.root_uvs[i] = make_float2(r.u, r.v); }
            if (g.point_counts) { g.point_counts[i] = P; }
        }
        __syncwarp();
    }
}

// The frame's guide-offset table (G x P float4) and, after it, the guide
// frame records (2 float4 per guide) the lane-walk generator reads; also
// clears the `bins` words of a strand order that follows.
__global__ void guide_offsets_kernel(AssetArgs a, FrameArgs f, uint32_t P, float support_scale, float4 *offsets,
                                     uint32_t *hist, uint32_t bins) {
    chain_start();
    chain_wait();
    const uint64_t n = static_cast<uint64_t>(a.guide_count) * P;
    const uint64_t stride = static_cast<uint64_t>(gridDim.x) * blockDim.x;
    const uint64_t first = blockIdx.x * static_cast<uint64_t>(blockDim.x) + threadIdx.x;
    for (uint64_t k = first; k < bins; k += stride) { hist[k] = 0u; }
    for (uint64_t idx = first; idx < n; idx += stride) {
        offsets[idx] = guide_offset_entry(a, f, P, static_cast<uint32_t>(idx / P), static_cast<uint32_t>(idx % P));
    }
    for (uint64_t gi = first; gi < a.guide_count; gi += stride) {
        guide_frame_entry(a, f, support_scale, static_cast<uint32_t>(gi),
                          guide_offset_entry(a, f, P, static_cast<uint32_t>(gi), 0u), offsets + n + 2u * gi);
    }
}

// Strands whose offset table does not fit: one thread walks the reference's cursor
// (generate.h:445-642) directly.  Slot records live in registers.
__device__ F3 serial_base_cv(const LaunchArgs &g, const Root &root, const Slot *slots, float wsum,
                             int nearest, uint32_t cv) {
    const float t = __fdiv_rn(static_cast<float>(cv), static_cast<float>(g.p.cvs_per_strand - 1u));
    F3 off = {0.0f, 0.0f, 0.0f};
    if (wsum > 1.0e-12f) {
        for (uint32_t j = 0; j < kSlots; ++j) {
            if (slots[j].flags & kSlotBlended) { off = off + guide_offset(g.f.guide_cvs, slots[j], t) * slots[j].w; }
        }
        off = off * (1.0f / wsum);
    } else if (nearest >= 0) {
        off = guide_offset(g.f.guide_cvs, slots[nearest], t);
    } else {
        off = root.normal * t;
    }
    return root.position + off * g.p.length_scale;
}

struct SerialCursor {
    uint32_t cv;
    F3 previous_base, current_base, next_base, tangent, transported_normal;
    float arc_length;
};

__device__ F3 serial_advance(const LaunchArgs &g, const Root &root, const Slot *slots, float wsum, int nearest,
                             const F3 &domain, float f_eff, const float4 *table, SerialCursor &cur) {
    const ParamArgs &p = g.p;
    if (cur.cv > 0u) {
        const F3 d = cur.current_base - cur.previous_base;
        cur.arc_length += sqrtf(dot(d, d));
    }
    F3 next_tangent = cur.tangent;
    if (cur.cv + 1u < p.cvs_per_strand) {
        const F3 seg = xsub(cur.next_base, cur.current_base);
        if (xdot(seg, seg) > 0.0f) { next_tangent = xnormalize(seg); }
    }
    const F3 axis = xcross(cur.tangent, next_tangent);
    if (xdot(axis, axis) > 0.0f) {
        const float angle = acosf(fminf(fmaxf(dot(cur.tangent, next_tangent), -1.0f), 1.0f));
        cur.transported_normal = normalize(apply3(rotation3(axis, angle), cur.transported_normal));
    }
    const F3 n = cur.transported_normal;
    const F3 b = cross(n, next_tangent);
    const F3 t = cross(b, n);
    F3 point = cur.current_base;
    if (cur.cv > 0u) {
        const float distance = cur.arc_length * f_eff;
        const float magnitude = p.noise_mask * p.noise_amplitude *
                                __fdiv_rn(static_cast<float>(cur.cv), static_cast<float>(p.cvs_per_strand - 1u));
        const float lx = (gradient_noise(table, domain.x + distance, domain.y, domain.z) - 0.5f) * magnitude;
        const float ly = (gradient_noise(table, domain.x, domain.y + distance, domain.z) - 0.5f) * magnitude;
        const float lz = (gradient_noise(table, domain.x, domain.y, domain.z + distance) - 0.5f) * magnitude;
        point = point + n * lx + b * ly + t * lz;
    }
    cur.tangent = next_tangent;
    cur.previous_base = cur.current_base;
    if (cur.cv + 1u < p.cvs_per_strand) {
        cur.current_base = cur.next_base;
        if (cur.cv + 2u < p.cvs_per_strand) {
            cur.next_base = serial_base_cv(g, root, slots, wsum, nearest, cur.cv + 2u);
        }
    }
    ++cur.cv;
    return point;
}

__device__ __forceinline__ void serial_store(const LaunchArgs &g, uint32_t local, uint32_t cv, F3 q, float radius) {
    const uint64_t index = static_cast<uint64_t>(local) * g.p.cvs_per_strand + cv;
    if (g.vec3_points) {
        g.vec3_points[3u * index] = q.x;
        g.vec3_points[3u * index + 1u] = q.y;
        g.vec3_points[3u * index + 2u] = q.z;
    } else {
        g.points[index] = make_float4(q.x, q.y, q.z, radius);
    }
}

__global__ void generate_serial_kernel(LaunchArgs g) {
    __shared__ float4 table[kTableFloat4];
    for (int i = threadIdx.x; i < kTableFloat4; i += blockDim.x) {
        table[i] = make_float4(__ldg(g.a.gradients + 3 * i), __ldg(g.a.gradients + 3 * i + 1),
                               __ldg(g.a.gradients + 3 * i + 2), 0.0f);
    }
    __syncthreads();
    const ParamArgs &p = g.p;
    const uint32_t P = p.cvs_per_strand;
    for (uint32_t item = blockIdx.x * blockDim.x + threadIdx.x; item < g.count; item += gridDim.x * blockDim.x) {
        const uint32_t local = g.order ? min(__ldg(g.order + item), g.count - 1u) : item;
        const Root root = sample_root(g.a, g.f, p.seed, g.first_strand + local);
        Slot slots[kSlots];
        float wsum = 0.0f, nd2 = FLT_MAX;
        int nearest = -1;
        for (uint32_t j = 0; j < kSlots; ++j) {
            slots[j] = eval_slot(g.a, g.f, p, root, j);
            if ((slots[j].flags & kSlotEligible) && slots[j].d2 < nd2) {
                nd2 = slots[j].d2;
                nearest = static_cast<int>(j);
            }
            if (slots[j].flags & kSlotBlended) { wsum = __fadd_rn(wsum, slots[j].w); }
        }
        float scale = 1.0f;
        F3 domain = {0.0f, 0.0f, 0.0f};
        float f_eff = 0.0f;
        F3 surface_u = {0.0f, 0.0f, 0.0f};
        if (p.noise) {
            surface_u = root_surface_u(g.a, g.f, root);
            F3 prev = serial_base_cv(g, root, slots, wsum, nearest, 0u);
            float length = 0.0f;
            for (uint32_t cv = 1u; cv < P; ++cv) {
                const F3 cur = serial_base_cv(g, root, slots, wsum, nearest, cv);
                const F3 d = cur - prev;
                length += sqrtf(dot(d, d));
                prev = cur;
            }
            f_eff = length > 0.0f ? fmaxf(0.5f / length, p.noise_frequency) : p.noise_frequency;
            const float dec = 1.0f - p.noise_correlation;
            domain = (rest_root_position(g.a, root) + F3{0.419276f, 0.184247f, 0.805721f}) * (100.0f * dec * dec);
            if (p.noise_preserve_length > 0.001f) {
                SerialCursor c{0u, {}, {}, {}, root.normal, surface_u, 0.0f};
                c.current_base = serial_base_cv(g, root, slots, wsum, nearest, 0u);
                c.previous_base = c.current_base;
                c.next_base = serial_base_cv(g, root, slots, wsum, nearest, 1u);
                F3 pv = serial_advance(g, root, slots, wsum, nearest, domain, f_eff, table, c);
                float noisy = 0.0f;
                for (uint32_t cv = 1u; cv < P; ++cv) {
                    const F3 cur = serial_advance(g, root, slots, wsum, nearest, domain, f_eff, table, c);
                    const F3 d = cur - pv;
                    noisy += sqrtf(dot(d, d));
                    pv = cur;
                }
                if (noisy > 0.0f) {
                    const float target = length * p.noise_preserve_length + noisy * (1.0f - p.noise_preserve_length);
                    if (fabsf(noisy - target) >= 0.0001f) { scale = target / noisy; }
                }
            }
            SerialCursor c{0u, {}, {}, {}, root.normal, surface_u, 0.0f};
            c.current_base = serial_base_cv(g, root, slots, wsum, nearest, 0u);
            c.previous_base = c.current_base;
            c.next_base = serial_base_cv(g, root, slots, wsum, nearest, 1u);
            for (uint32_t cv = 0u; cv < P; ++cv) {
                F3 q = serial_advance(g, root, slots, wsum, nearest, domain, f_eff, table, c);
                if (scale != 1.0f) { q = root.position + (q - root.position) * scale; }
                const float t = __fdiv_rn(static_cast<float>(cv), static_cast<float>(P - 1u));
                serial_store(g, local, cv, q, strand_radius(p, t));
            }
        } else {
            for (uint32_t cv = 0u; cv < P; ++cv) {
                const F3 q = serial_base_cv(g, root, slots, wsum, nearest, cv);
                const float t = __fdiv_rn(static_cast<float>(cv), static_cast<float>(P - 1u));
                serial_store(g, local, cv, q, strand_radius(p, t));
            }
        }
        if (g.roots) {
            for (int w = 0; w < 12; ++w) { g.roots[static_cast<uint64_t>(local) * 12u + w] = root_word(root, w); }
        }
        if (g.root_uvs) { g.root_uvs[local] = make_float2(root.u, root.v); }
        if (g.point_counts) { g.point_counts[local] = P; }
    }
}

// ---------------------------------------------------------------------------
// Strand-locality counting sort.
// ---------------------------------------------------------------------------
constexpr uint32_t kPrivateBins = 8192u;

__global__ void strand_keys_kernel(AssetArgs a, uint32_t seed, uint32_t first, uint32_t count, uint32_t *keys,
                                   uint32_t *hist, uint32_t bins) {
    extern __shared__ uint32_t local_hist[];
    const bool priv = bins <= kPrivateBins;
    chain_start();
    chain_wait();
    if (priv) {
        for (uint32_t b = threadIdx.x; b < bins; b += blockDim.x) { local_hist[b] = 0u; }
        __syncthreads();
    }
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < count; i += gridDim.x * blockDim.x) {
        const uint32_t tri = sample_triangle(a, seed, first + i);
        const uint32_t gi = __ldg(a.stencil + static_cast<uint64_t>(tri) * kSlots);
        const uint32_t key = gi < a.guide_count ? gi : a.guide_count;
        keys[i] = key;
        if (priv) {
            atomicAdd(&local_hist[key], 1u);
        } else {
            atomicAdd(&hist[key], 1u);
        }
    }
    if (priv) {
        __syncthreads();
        for (uint32_t b = threadIdx.x; b < bins; b += blockDim.x) {
            const uint32_t v = local_hist[b];
            if (v) { atomicAdd(&hist[b], v); }
        }
    }
}

// Exclusive scan of n words in place, one CTA of 1024 threads.
__global__ void __launch_bounds__(1024) exclusive_scan_kernel(uint32_t *data, uint32_t n) {
    __shared__ uint32_t warp_sums[32];
    chain_start();
    chain_wait();
    const uint32_t tid = threadIdx.x;
    const uint32_t per = (n + blockDim.x - 1u) / blockDim.x;
    const uint32_t lo = min(n, tid * per), hi = min(n, lo + per);
    uint32_t sum = 0u;
    for (uint32_t i = lo; i < hi; ++i) { sum += data[i]; }
    uint32_t incl = sum;
    const int lane = tid & 31;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const uint32_t u = __shfl_up_sync(kFull, incl, d);
        if (lane >= d) { incl += u; }
    }
    if (lane == 31) { warp_sums[tid >> 5] = incl; }
    __syncthreads();
    if (tid < 32) {
        uint32_t w = tid < (blockDim.x >> 5) ? warp_sums[tid] : 0u;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const uint32_t u = __shfl_up_sync(kFull, w, d);
            if (lane >= d) { w += u; }
        }
        warp_sums[tid] = w;
    }
    __syncthreads();
    uint32_t running = incl - sum + ((tid >> 5) ? warp_sums[(tid >> 5) - 1u] : 0u);
    for (uint32_t i = lo; i < hi; ++i) {
        const uint32_t v = data[i];
        data[i] = running;
        running += v;
    }
}

__global__ void scatter_order_kernel(const uint32_t *keys, uint32_t *offsets, uint32_t count, uint32_t bins,
                                     uint32_t *order) {
    chain_start();
    chain_wait();
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < count; i += gridDim.x * blockDim.x) {
        const uint32_t key = min(keys[i], bins - 1u);
        const uint32_t pos = atomicAdd(&offsets[key], 1u);
        if (pos < count) { order[pos] = i; }
    }
}

// The same scatter with one global atomic per (block, non-empty bin): block
// b owns strands [b * chunk, (b + 1) * chunk); it counts its keys in shared
// memory, reserves each bin's range of the order with one atomicAdd on the
// bin offset, then places each strand at that range plus its shared-memory
// rank.  For up to kPrivateBins bins (the count array is in shared memory).
__global__ void __launch_bounds__(1024) scatter_order_blocked_kernel(const uint32_t *keys, uint32_t *offsets,
                                                                     uint32_t count, uint32_t bins, uint32_t chunk,
                                                                     uint32_t *order) {
    extern __shared__ uint32_t slots[];  // per bin: count, then the next free position
    const uint32_t begin = blockIdx.x * chunk;
    const uint32_t end = min(count, begin + chunk);
    for (uint32_t b = threadIdx.x; b < bins; b += blockDim.x) { slots[b] = 0u; }
    chain_start();
    chain_wait();
    __syncthreads();
    for (uint32_t i = begin + threadIdx.x; i < end; i += blockDim.x) { atomicAdd(&slots[min(keys[i], bins - 1u)], 1u); }
    __syncthreads();
    for (uint32_t b = threadIdx.x; b < bins; b += blockDim.x) {
        const uint32_t n = slots[b];
        slots[b] = n ? atomicAdd(&offsets[b], n) : 0u;
    }
    __syncthreads();
    for (uint32_t i = begin + threadIdx.x; i < end; i += blockDim.x) {
        const uint32_t pos = atomicAdd(&slots[min(keys[i], bins - 1u)], 1u);
        if (pos < count) { order[pos] = i; }
    }
}

// Per-strand state for stencil/root parity checks (generate.h:568-575).
struct StrandStateOut {
    uint32_t root[12];
    uint32_t indices[8];
    float weights[8];
    float weight_sum;
    uint32_t nearest;
    float surface_u[3];
    float noise_domain[3];
};

__global__ void query_states_kernel(AssetArgs a, FrameArgs f, ParamArgs p, const uint32_t *strands,
                                    uint32_t count, StrandStateOut *out) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= count) { return; }
    const Root root = sample_root(a, f, p.seed, strands[i]);
    StrandStateOut s;
    for (int w = 0; w < 12; ++w) { s.root[w] = root_word(root, w); }
    s.weight_sum = 0.0f;
    s.nearest = kInvalid;
    float nd2 = FLT_MAX;
    for (uint32_t j = 0; j < kSlots; ++j) {
        const Slot slot = eval_slot(a, f, p, root, j);
        s.indices[j] = (slot.flags & kSlotBlended) ? slot.guide : kInvalid;
        s.weights[j] = (slot.flags & kSlotBlended) ? slot.w : 0.0f;
        if ((slot.flags & kSlotEligible) && slot.d2 < nd2) {
            nd2 = slot.d2;
            s.nearest = slot.guide;
        }
        if (slot.flags & kSlotBlended) { s.weight_sum = __fadd_rn(s.weight_sum, slot.w); }
    }
    F3 su = {0.0f, 0.0f, 0.0f}, dom = {0.0f, 0.0f, 0.0f};
    if (p.noise) {
        su = root_surface_u(a, f, root);
        const float dec = 1.0f - p.noise_correlation;
        dom = (rest_root_position(a, root) + F3{0.419276f, 0.184247f, 0.805721f}) * (100.0f * dec * dec);
    }
    s.surface_u[0] = su.x;
    s.surface_u[1] = su.y;
    s.surface_u[2] = su.z;
    s.noise_domain[0] = dom.x;
    s.noise_domain[1] = dom.y;
    s.noise_domain[2] = dom.z;
    out[i] = s;
}

// The lane walk's own setup decisions for listed strands (one warp per CTA,
// g.order = the strand ids, first_strand 0): walk_setup itself, with the
// frame's guide records already in g.guide_frames, outputs off.
__global__ void __launch_bounds__(32) walk_states_kernel(LaunchArgs g, uint32_t count, WalkDecision *out) {
    __shared__ float4 records[kWalkRecords * 32];
    __shared__ uint32_t locals[32];
    const int lane = threadIdx.x & 31;
    const uint32_t i = blockIdx.x * 32u + static_cast<uint32_t>(lane);
    const bool valid = i < count;
    WalkDecision d;
    walk_setup<false>(g, records, locals, lane, valid ? i : 0u, valid, g.p.cvs_per_strand, false, &d);
    if (valid) { out[i] = d; }
}

} // namespace dev

using dev::LaunchArgs;

namespace {

constexpr uint64_t kWorkspaceAlign = 256u;
inline uint64_t align_up(uint64_t v, uint64_t a) { return (v + a - 1u) / a * a; }

struct WorkspaceLayout {
    uint64_t keys, order, hist, offsets, total, walked;
};

// Largest guide-offset table the warp-parallel generator stages; beyond it
// strands take the serial per-thread kernel.
constexpr uint64_t kMaxOffsetTableBytes = uint64_t{1} << 30;
constexpr uint32_t kMaxParallelCvs = 128u;  // of the lane groups, and of what a workspace must hold a table for

bool parallel_path(uint32_t guide_count, uint32_t P) {
    return P <= kMaxParallelCvs && uint64_t{guide_count} * P * 16u <= kMaxOffsetTableBytes;
}

// Strands of more than kMaxParallelCvs CVs take the lane walk too where the
// workspace holds their offset table (20,011 strands x 160 CVs with noise, 512
// guides: 1,214 us on the serial kernel).  The workspace need not: a caller's
// that holds the order alone stays valid and takes the serial kernel.  The
// queried size asks for the table while it is no larger than the description's
// own points, so it never dominates a caller's memory: by the strands of the
// whole description, whose ranges are then generated alike.
bool long_walk_path(uint32_t guide_count, uint32_t strands, uint32_t P) {
    return P > kMaxParallelCvs && P <= dev::kWalkMaxCvs && guide_count <= strands &&
           uint64_t{guide_count} * P * 16u <= kMaxOffsetTableBytes;
}

// keys[count] | order[count] | bins[guides + 1] | offsets[guides * P] (float4)
// followed by the guide frame records [guides * 2] (float4).  `total` is what
// a caller has to provide, `walked` what the lane walk needs.
// `strands`: the description's, where the launch is a range of them.
WorkspaceLayout workspace_layout(uint32_t guide_count, uint32_t count, uint32_t P, uint32_t strands = 0u) {
    WorkspaceLayout w{};
    w.keys = 0u;
    w.order = align_up(uint64_t{count} * 4u, kWorkspaceAlign);
    w.hist = w.order + align_up(uint64_t{count} * 4u, kWorkspaceAlign);
    w.offsets = w.hist + align_up((uint64_t{guide_count} + 1u) * 4u, kWorkspaceAlign);
    const uint64_t table = align_up(uint64_t{guide_count} * (P + 2u) * 16u, kWorkspaceAlign);
    w.total = w.offsets + (parallel_path(guide_count, P) ? table : 0u);
    const bool walked = parallel_path(guide_count, P) || long_walk_path(guide_count, std::max(count, strands), P);
    w.walked = w.offsets + (walked ? table : 0u);
    return w;
}

} // namespace

int device_sm_count() {
    int device = 0;
    if (cudaGetDevice(&device) != cudaSuccess) { return 148; }
    int sms = 0;
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess || sms <= 0) {
        return 148;
    }
    return sms;
}

dev::AssetArgs resolve_asset(const nxg_device_asset_desc &desc) {
    const auto *base = static_cast<const unsigned char *>(desc.asset);
    const nxg_asset_header &h = desc.header;
    dev::AssetArgs a{};
    a.positions = reinterpret_cast<const float *>(base + h.positions_offset);
    a.normals = reinterpret_cast<const float *>(base + h.normals_offset);
    a.texcoords = (h.flags & NXG_ASSET_HAS_TEXCOORDS) && h.texcoords_offset
        ? reinterpret_cast<const float *>(base + h.texcoords_offset) : nullptr;
    a.triangles = reinterpret_cast<const uint32_t *>(base + h.triangles_offset);
    a.alias = reinterpret_cast<const uint2 *>(base + h.alias_table_offset);
    a.guides = reinterpret_cast<const uint32_t *>(base + h.guides_offset);
    a.guide_cvs = reinterpret_cast<const float *>(base + h.guide_cvs_offset);
    a.stencil = reinterpret_cast<const uint32_t *>(base + h.triangle_guides_offset);
    a.gradients = reinterpret_cast<const float *>(base + h.noise_gradients_offset);
    a.vertex_count = h.vertex_count;
    a.triangle_count = h.triangle_count;
    a.guide_count = h.guide_count;
    a.guide_cv_count = h.guide_cv_count;
    a.flags = h.flags;
    return a;
}

dev::FrameArgs resolve_frame(const dev::AssetArgs &a, const nxg_deformed_desc &d) {
    dev::FrameArgs f{};
    f.positions = d.positions ? reinterpret_cast<const float *>(d.positions) : a.positions;
    f.normals = d.normals ? reinterpret_cast<const float *>(d.normals) : a.normals;
    f.guide_cvs = d.guide_cvs ? reinterpret_cast<const float *>(d.guide_cvs) : a.guide_cvs;
    f.deformed_positions = d.positions != nullptr;
    f.deformed_normals = d.normals != nullptr;
    f.deformed_guide_cvs = d.guide_cvs != nullptr;
    return f;
}

dev::ParamArgs resolve_params(const nxg_generation_params &p, float radius_scale) {
    dev::ParamArgs r{};
    r.strand_count = p.strand_count;
    r.cvs_per_strand = p.cvs_per_strand;
    r.seed = p.seed;
    r.support_scale = p.guide_support_scale;
    r.weight_power = p.guide_weight_power > 0.0f ? p.guide_weight_power : 0.0f;
    r.rejection_cos = p.normal_rejection_cos;
    r.length_scale = p.length_scale;
    r.root_width = p.root_width;
    r.tip_width = p.tip_width;
    r.noise_amplitude = p.noise_amplitude;
    r.noise_frequency = p.noise_frequency;
    r.noise_mask = p.noise_mask;
    r.noise_correlation = p.noise_correlation;
    r.noise_preserve_length = p.noise_preserve_length;
    r.radius_scale = radius_scale;
    r.noise = (p.noise_amplitude != 0.0f && p.noise_mask != 0.0f) ? 1u : 0u;
    return r;
}

namespace {

using KernelFn = void (*)(LaunchArgs, const float4 *);

// Classic variants (scalars applied in the kernel) are separate
// instantiations, so the plain generator keeps its register budget.
template <int L, int PPT>
KernelFn pick_noise(bool noise, bool classic) {
    if (classic) {
        return noise ? dev::generate_kernel<L, PPT, true, true> : dev::generate_kernel<L, PPT, false, true>;
    }
    return noise ? dev::generate_kernel<L, PPT, true, false> : dev::generate_kernel<L, PPT, false, false>;
}

template <int PPT>
KernelFn pick_lanes(int lanes, bool noise, bool classic) {
    switch (lanes) {
        case 2: return pick_noise<2, PPT>(noise, classic);
        case 4: return pick_noise<4, PPT>(noise, classic);
        case 8: return pick_noise<8, PPT>(noise, classic);
        case 16: return pick_noise<16, PPT>(noise, classic);
        default: return pick_noise<32, PPT>(noise, classic);
    }
}

// Tile registry: the (lanes per strand, CVs per lane, CTA size) used for
// strands of P CVs with noise off/on, set by nxg_set_tile or the autotuner.
// Packed as lanes | ppt << 8 | (block / 32) << 16; 0 means "not set".
std::atomic<uint32_t> g_tiles[kMaxParallelCvs + 1][2];

uint32_t packed_tile(const nxg_tile &t) {
    return t.lanes_per_strand | (t.cvs_per_lane << 8) | ((t.block_size + 31u) / 32u << 16);
}

uint32_t registered_tile(uint32_t P, bool noise) {
    return P <= kMaxParallelCvs ? g_tiles[P][noise ? 1 : 0].load(std::memory_order_relaxed) : 0u;
}

bool lane_groups(uint32_t packed) { return packed != 0u && (packed & 0xffu) != 1u; }

// The lane walk's tile has one lane per strand.  Its CVs per lane read 1 up to
// 32 CVs, and the strand's CV count past them.
uint32_t lane_walk_ppt(uint32_t P) { return P <= 32u ? 1u : P; }

bool valid_tile(uint32_t P, uint32_t lanes, uint32_t ppt) {
    if (lanes == 1u) { return ppt == lane_walk_ppt(P) && P >= 2u && P <= kMaxParallelCvs; }
    const bool lanes_ok = lanes == 2u || lanes == 4u || lanes == 8u || lanes == 16u || lanes == 32u;
    const bool ppt_ok = ppt == 1u || ppt == 2u || ppt == 4u;
    return lanes_ok && ppt_ok && lanes * ppt >= P && P >= 2u && P <= kMaxParallelCvs;
}

// The tile of strands without a registered one: the lane walk.  Registering it
// registers none.  (Up to 32 CVs with noise the launch is free to take CTAs of
// up to kWalkNoiseWarps, more than the 352 threads its callers have been told.)
nxg_tile builtin_tile(uint32_t P, bool noise) {
    return {1u, lane_walk_ppt(P), !noise ? 256u : (P <= 32u ? 352u : 32u * static_cast<uint32_t>(dev::kWalkNoiseWarps))};
}

KernelFn pick_kernel(int lanes, int ppt, bool noise, bool classic) {
    switch (ppt) {
        case 1: return pick_lanes<1>(lanes, noise, classic);
        case 2: return pick_lanes<2>(lanes, noise, classic);
        default: return pick_lanes<4>(lanes, noise, classic);
    }
}

// Dynamic shared memory of the lane-group kernels.
size_t generate_smem_bytes(uint32_t P, int lanes, int ppt, bool noise, uint32_t warps) {
    const size_t per_warp = sizeof(uint32_t) * dev::kRecFields * 32u + sizeof(float4) * 32u / lanes * lanes * ppt +
                            (noise ? sizeof(float2) * 384u : 0u);
    return sizeof(float4) * dev::kTableFloat4 + sizeof(float) * ((P + 3u) & ~3u) + per_warp * warps;
}

} // namespace

uint32_t record_cuda(cudaError_t e) {
    if (e == cudaSuccess) { return NXG_ERROR_NONE; }
    set_last_cuda_error(static_cast<int32_t>(e));
    return NXG_ERROR_CUDA;
}


uint32_t check_launch_inputs(const nxg_device_asset_desc &asset, const nxg_packed_output_desc *output) {
    if (!sections_in_bounds(asset.header)) { return NXG_ERROR_INVALID_ASSET_METADATA; }
    if (output && (reinterpret_cast<std::uintptr_t>(output->points) % 16u != 0u ||
                   reinterpret_cast<std::uintptr_t>(output->roots) % 4u != 0u ||
                   reinterpret_cast<std::uintptr_t>(output->root_uvs) % 8u != 0u ||
                   reinterpret_cast<std::uintptr_t>(output->point_counts) % 4u != 0u)) {
        return NXG_ERROR_MISALIGNED_OUTPUT;
    }
    return NXG_ERROR_NONE;
}

uint32_t check_workspace(const nxg_device_asset_desc &asset, uint32_t count, uint32_t P, const void *workspace,
                         uint64_t workspace_bytes) {
    const WorkspaceLayout ws = workspace_layout(asset.header.guide_count, count, P);
    if (!workspace || workspace_bytes < ws.total) { return NXG_ERROR_WORKSPACE_TOO_SMALL; }
    if (reinterpret_cast<std::uintptr_t>(workspace) % kWorkspaceAlign != 0u) { return NXG_ERROR_MISALIGNED_OUTPUT; }
    return NXG_ERROR_NONE;
}

// Counting sort of strands [first, first + count) by their triangle's first
// stencil guide; leaves the permutation in the workspace's order section.
// `cleared`: the launch before on the stream has cleared the bins.
uint32_t launch_order(const nxg_device_asset_desc &asset, uint32_t seed, uint32_t first, uint32_t count,
                      uint32_t P, void *workspace, cudaStream_t stream, bool cleared) {
    const WorkspaceLayout ws = workspace_layout(asset.header.guide_count, count, P);
    auto *wbase = static_cast<unsigned char *>(workspace);
    auto *keys = reinterpret_cast<uint32_t *>(wbase + ws.keys);
    auto *order = reinterpret_cast<uint32_t *>(wbase + ws.order);
    auto *hist = reinterpret_cast<uint32_t *>(wbase + ws.hist);
    const uint32_t bins = asset.header.guide_count + 1u;
    const int sms = device_sm_count();
    const dev::AssetArgs a = resolve_asset(asset);
    uint32_t status = cleared ? uint32_t{NXG_ERROR_NONE}
                              : record_cuda(cudaMemsetAsync(hist, 0, uint64_t{bins} * 4u, stream));
    if (status) { return status; }
    const uint32_t threads = 256u;
    const uint32_t blocks = static_cast<uint32_t>(std::min<uint64_t>((count + threads - 1u) / threads,
                                                                      static_cast<uint64_t>(sms) * 4u));
    const size_t shm = bins <= dev::kPrivateBins ? bins * 4u : 0u;
    // An ordinary launch: chained to the guide offsets before it, both kernels
    // share the SMs to neither's gain (whole calls of 1,000,000 x 32 without noise
    // 238 us chained, 231 not; with noise 577, 569).
    if ((status = launch_chained(false, dev::strand_keys_kernel, blocks, threads, shm, stream, a, seed, first,
                                 count, keys, hist, bins)) ||
        (status = launch_chained(true, dev::exclusive_scan_kernel, 1u, 1024u, 0u, stream, hist, bins))) {
        return status;
    }
    if (bins > dev::kPrivateBins) {
        return launch_chained(true, dev::scatter_order_kernel, blocks, threads, 0u, stream, keys, hist, count, bins,
                              order);
    }
    // One block per SM, shared-memory ranks.
    const uint32_t scatter_blocks = static_cast<uint32_t>(std::max(1, sms));
    const uint32_t chunk = (count + scatter_blocks - 1u) / scatter_blocks;
    const uint32_t used = (count + chunk - 1u) / chunk;
    return launch_chained(true, dev::scatter_order_blocked_kernel, used, 1024u, bins * 4u, stream, keys, hist, count,
                          bins, chunk, order);
}

namespace {

// Whether the lane walk takes its strands in the order of their guides.  The
// order makes the warps of an SM read the same guide rows from L1, and costs
// three launches, two passes over a key per strand, and scattered instead of
// sequential outputs.  It pays where that locality is missing (a table beyond
// L1) over enough points.  Whole calls, ordered against not, 4,096 guides unless
// said otherwise: with noise 100,000 x 32 85.5 / 78.1 us, 200,000 x 32 142.1 /
// 143.2, 300,000 x 32 196.2 / 207.1 (of 700 guides 196.9 / 201.1).  Without noise more warps
// hide the rows' latency and the scattered root outputs weigh more (60 bytes per
// strand), so only long strands gain: 300,000 x 100 197.3 / 200.8, but 1,000,000 x
// 32 241.1 / 238.9, 800,000 x 31 230.6 / 219.1, 2,000,000 x 32 498 / 462.
// A motion call orders its strands once for all samples (each then as below).  An order that the
// caller has prepared costs nothing more and is always taken: with noise
// 100,000 x 32 71.5 us against 78.5 without it, 1,000,000 x 24 and 200 guides
// 492 / 513; without noise 100,000 x 32 31.8 / 36.8, 500,000 x 12 87.5 / 110.5,
// 2,000,000 x 24 378 / 414.
// Whole stages leave the rows little of L1, so there it pays earlier: 170,000 x 24
// 103.4 / 110.7 us (of 700 guides 102.2 / 104.4), 130,000 x 24 95.4 / 96.2 (of 700
// guides 93.9 / 90.2), 1,000,000 x 24 of 700 guides 490 / 533, 4,000,000 x 24 1,947 /
// 2,218; with Classic scalars 170,000 x 24 109.5 / 117.5.
bool wants_order(uint32_t guide_count, uint32_t count, uint32_t P, bool noise, bool whole, uint32_t samples) {
    const uint64_t points = uint64_t{count} * P * samples;
    if (uint64_t{guide_count} * P * 16u <= (uint64_t{128} << 10)) { return false; }
    if (noise) { return points >= (whole ? 4000000u : 7000000u); }
    return points >= 24000000u && count <= (samples > 1u ? 1700000u : 500000u);
}

// CVs of a strand that the noisy walk stages at a time (walk.cuh).  Up to 24 the
// whole strand, where two chunks leave the second half empty (1,000,000 x 24 488
// us, in chunks 522; x 17 468 / 506).  Up to 32 only where its points are
// rewritten: otherwise two full chunks are the faster (1,000,000 x 32 570, whole
// 604), except below the frequency floor, where a chunked strand is staged twice
// (703, whole 582).  A range of strands takes the whole call's path, so the
// number of strands has no part in it.
int noise_chunk(uint32_t P, bool classic, const nxg_generation_params &params) {
    if (P <= static_cast<uint32_t>(dev::kWalkChunk) || P > static_cast<uint32_t>(dev::kWalkWholeCvs)) {
        return dev::kWalkChunk;
    }
    if (P <= 24u) { return 24; }
    return classic || params.noise_preserve_length > 0.001f ? 32 : dev::kWalkChunk;
}

} // namespace

LaunchForm launch_form(uint32_t guide_count, const nxg_generation_params &params, uint32_t count, uint32_t samples,
                       bool prepared, bool classic) {
    const uint32_t P = params.cvs_per_strand;
    const bool noise = resolve_params(params, 1.0f).noise != 0u;
    LaunchForm form;
    form.tile = registered_tile(P, noise);
    form.ordered = prepared || lane_groups(form.tile) ||
                   wants_order(guide_count, count, P, noise, noise_chunk(P, classic, params) != dev::kWalkChunk, samples);
    return form;
}

// The guide-offset table for this frame, the strand order where one is wanted
// and not ready, then the persistent generate kernel.
uint32_t launch_generate(const nxg_device_asset_desc &asset, const nxg_deformed_desc &deformed,
                         const nxg_generation_params &params, const nxg_packed_output_desc &output,
                         const nxg_launch_config &config, uint32_t first, uint32_t count, void *workspace,
                         uint64_t workspace_bytes, cudaStream_t stream, float *vec3_points,
                         const nxg_classic_apply_desc *classic, LaunchForm form, bool order_ready) {
    set_last_cuda_error(0);
    const uint32_t P = params.cvs_per_strand;
    const WorkspaceLayout ws = workspace_layout(asset.header.guide_count, count, P, params.strand_count);
    auto *wbase = static_cast<unsigned char *>(workspace);
    LaunchArgs g{};
    g.a = resolve_asset(asset);
    g.f = resolve_frame(g.a, deformed);
    g.p = resolve_params(params, output.radius_scale);
    g.first_strand = first;
    g.count = count;
    g.points = reinterpret_cast<float4 *>(output.points);
    g.vec3_points = vec3_points;
    g.roots = reinterpret_cast<uint32_t *>(output.roots);
    g.root_uvs = reinterpret_cast<float2 *>(output.root_uvs);
    g.point_counts = output.point_counts;
    g.order = reinterpret_cast<const uint32_t *>(wbase + ws.order);
    if (classic != nullptr) {
        g.scalars = reinterpret_cast<const float2 *>(classic->root_scalars);
        g.classic_length = classic->apply_length != 0u;
        g.classic_width = classic->apply_width != 0u;
    }
    const int sms = device_sm_count();
    uint32_t status = NXG_ERROR_NONE;
    const bool parallel = parallel_path(asset.header.guide_count, P);
    if (!parallel && (ws.walked == ws.total || workspace_bytes < ws.walked)) {  // without the table
        if (!order_ready &&
            (status = launch_order(asset, params.seed, first, count, P, workspace, stream, false))) {
            return status;
        }
        const uint32_t threads = 128u;
        const uint32_t blocks = static_cast<uint32_t>(std::min<uint64_t>((count + threads - 1u) / threads,
                                                                          static_cast<uint64_t>(sms) * 8u));
        dev::generate_serial_kernel<<<blocks, threads, 0, stream>>>(g);
        if ((status = record_cuda(cudaGetLastError())) || g.scalars == nullptr) { return status; }
        dev::classic_serial_apply_kernel<<<blocks, threads, 0, stream>>>(g);
        return record_cuda(cudaGetLastError());
    }
    auto *offsets = reinterpret_cast<float4 *>(wbase + ws.offsets);
    g.guide_frames = offsets + uint64_t{asset.header.guide_count} * P;
    const bool noise = g.p.noise != 0u;
    // The lane walk, unless a lane-group tile is registered for these strands.
    const uint32_t packed = form.tile;
    const bool walk = !lane_groups(packed);
    {
        const uint64_t n = uint64_t{asset.header.guide_count} * P;
        const uint32_t threads = 256u;
        const uint32_t blocks = static_cast<uint32_t>(std::min<uint64_t>((n + threads - 1u) / threads,
                                                                          static_cast<uint64_t>(sms) * 16u));
        const bool sort = form.ordered && !order_ready;
        // The first launch is an ordinary one.  (Chained to the walk of the
        // motion sample before, its CTAs and the next walk's took the SMs that
        // walk still needed: five samples of 250,000 x 24, 791 against 735 us.)
        if ((status = launch_chained(false, dev::guide_offsets_kernel, blocks, threads, 0u, stream, g.a, g.f, P,
                                     g.p.support_scale, offsets, reinterpret_cast<uint32_t *>(wbase + ws.hist),
                                     sort ? asset.header.guide_count + 1u : 0u)) ||
            (sort && (status = launch_order(asset, params.seed, first, count, P, workspace, stream, true)))) {
            return status;
        }
    }
    if (!form.ordered) { g.order = nullptr; }
    const bool classic_scalars = g.scalars != nullptr;
    int device = 0, smem_optin = 48 * 1024;
    if (cudaGetDevice(&device) == cudaSuccess) {
        cudaDeviceGetAttribute(&smem_optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, device);
    }
    // Launches `fn` persistently over the strand order, `per_warp` strands per
    // warp at a time.  `requested` threads are rounded up to whole warps, then
    // capped at what the kernel's registers and shared memory (smem(warps)
    // bytes) can launch.
    auto launch = [&](auto fn, uint32_t requested, uint32_t per_warp, auto smem) -> uint32_t {
        cudaFuncAttributes attr{};
        uint32_t st = record_cuda(cudaFuncGetAttributes(&attr, reinterpret_cast<const void *>(fn)));
        if (st) { return st; }
        const uint32_t launchable =
            std::max<uint32_t>(32u, static_cast<uint32_t>(attr.maxThreadsPerBlock) / 32u * 32u);
        uint32_t block = std::min(launchable, std::max<uint32_t>(32u, (requested + 31u) / 32u * 32u));
        while (block > 32u && smem(block / 32u) > static_cast<size_t>(smem_optin)) { block -= 32u; }
        const uint32_t warps = block / 32u;
        const size_t shm = smem(warps);
        if (shm > 48u * 1024u) {
            st = allow_shared(reinterpret_cast<const void *>(fn), attr.sharedSizeBytes, smem_optin);
            if (st) { return st; }
        }
        int per_sm = 0;
        st = record_cuda(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, reinterpret_cast<const void *>(fn),
                                                                       static_cast<int>(block), shm));
        if (st) { return st; }
        per_sm = std::max(per_sm, 1);
        const uint64_t needed = (uint64_t{count} + per_warp * warps - 1u) / (uint64_t{per_warp} * warps);
        const uint32_t grid = static_cast<uint32_t>(std::min<uint64_t>(needed, static_cast<uint64_t>(sms) * per_sm));
        return grid ? launch_chained(walk, fn, grid, block, shm, stream, g, static_cast<const float4 *>(offsets))
                    : uint32_t{NXG_ERROR_NONE};
    };
    if (walk) {
        const int chunk = noise_chunk(P, classic_scalars, params);
        const uint32_t full = noise ? dev::walk_noise_warps(chunk) : 8u;
        uint32_t warps = full;
        if (packed) {  // a registered CTA size is a bound
            const uint32_t tile_warps = (packed >> 16) & 0xffu;
            warps = std::min(warps, tile_warps ? tile_warps : (config.block_size + 31u) / 32u);
        }
        {
            // Every warp the GPU holds takes the same number of batches, of
            // equal size: a multiple of four strands, what a base and a store
            // pass take.  A warp's time is the walk along one strand, whatever
            // their number, plus what it does strand by strand, so a call that
            // leaves warps idle with full batches runs faster with smaller ones
            // (20,000 strands x 160 CVs with noise 159 -> 113 us, x 100 CVs
            // without 72 -> 31 us), and the last batches of a larger one are
            // not nearly empty.  Below a warp per SM the CTAs shrink too.
            const uint64_t slots = static_cast<uint64_t>(sms) * (noise ? full : 24u);
            const uint64_t rounds = (count + slots * 32u - 1u) / (slots * 32u);
            const uint64_t share = (count + slots * rounds - 1u) / (slots * rounds);
            g.batch = static_cast<uint32_t>(std::clamp<uint64_t>((share + 3u) / 4u * 4u, noise ? 8u : 4u, 32u));
            const uint64_t needed = (uint64_t{count} + g.batch - 1u) / g.batch;
            warps = static_cast<uint32_t>(std::min<uint64_t>(warps, (needed + sms - 1u) / sms));
        }
        const auto pick = [&](auto plain, auto classic) { return classic_scalars ? classic : plain; };
        const auto fn = !noise ? pick(dev::generate_walk_kernel<false, false>, dev::generate_walk_kernel<false, true>)
            : chunk == 32 ? pick(dev::generate_walk_kernel<true, false, 32>, dev::generate_walk_kernel<true, true, 32>)
            : chunk == 24 ? pick(dev::generate_walk_kernel<true, false, 24>, dev::generate_walk_kernel<true, true, 24>)
                          : pick(dev::generate_walk_kernel<true, false>, dev::generate_walk_kernel<true, true>);
        return launch(fn, warps * 32u, g.batch, [&](uint32_t w) {
            return dev::walk_head_bytes(noise, P, w, chunk) + dev::walk_warp_bytes(noise, classic_scalars, chunk) * w;
        });
    }
    const int lanes = static_cast<int>(packed & 0xffu), ppt = static_cast<int>((packed >> 8) & 0xffu);
    const uint32_t tile_block = ((packed >> 16) & 0xffu) * 32u;
    if (g.roots || g.root_uvs || g.point_counts) {  // the lane-walk kernel writes its own
        const uint32_t threads = 256u;
        const uint32_t per_block = threads;  // one strand per thread
        const uint32_t blocks = static_cast<uint32_t>(std::min<uint64_t>((count + per_block - 1u) / per_block,
                                                                          static_cast<uint64_t>(sms) * 8u));
        dev::strand_roots_kernel<<<blocks, threads, 0, stream>>>(g);
        if ((status = record_cuda(cudaGetLastError()))) { return status; }
    }
    return launch(pick_kernel(lanes, ppt, noise, classic_scalars), tile_block ? tile_block : config.block_size, 32u,
                  [&](uint32_t w) { return generate_smem_bytes(P, lanes, ppt, noise, w); });
}

uint32_t validate_range_request(const nxg_device_asset_desc *asset, const nxg_deformed_desc *deformed,
                                const nxg_generation_params *params, const nxg_packed_output_desc *output,
                                const nxg_launch_config *config, uint32_t first, uint32_t count) {
    if (!asset || !params || !output) { return NXG_ERROR_INVALID_ARGUMENT; }
    const nxg_deformed_desc none{};
    const nxg_launch_config default_config{128u};
    const uint32_t error = validate_common(*asset, deformed ? *deformed : none, *params,
                                           config ? *config : default_config);
    if (error != NXG_ERROR_NONE) { return error; }
    if (first > params->strand_count || count > params->strand_count - first) {
        return NXG_ERROR_INVALID_STRAND_RANGE;
    }
    if (!output->points) { return NXG_ERROR_MISSING_OUTPUT; }
    if (!std::isfinite(output->radius_scale) || output->radius_scale < 0.0f) {
        return NXG_ERROR_INVALID_RADIUS_SCALE;
    }
    const uint64_t point_count = uint64_t{count} * params->cvs_per_strand;
    if (output->point_capacity < point_count) { return NXG_ERROR_POINT_CAPACITY_TOO_SMALL; }
    auto optional_ok = [](const void *ptr, uint64_t cap, uint64_t need) { return ptr ? cap >= need : cap == 0u; };
    if (!optional_ok(output->roots, output->root_capacity, count)) { return NXG_ERROR_ROOT_CAPACITY_TOO_SMALL; }
    if (!optional_ok(output->root_uvs, output->root_uv_capacity, count)) {
        return NXG_ERROR_ROOT_UV_CAPACITY_TOO_SMALL;
    }
    if (!optional_ok(output->point_counts, output->point_count_capacity, count)) {
        return NXG_ERROR_POINT_COUNT_CAPACITY_TOO_SMALL;
    }
    return NXG_ERROR_NONE;
}

} // namespace nxg

extern "C" {

uint64_t nxg_packed_workspace_size(const nxg_device_asset_desc *asset, const nxg_generation_params *params,
                                   uint32_t strand_count) {
    if (!asset || !params || strand_count == 0u) { return 0u; }
    return nxg::workspace_layout(asset->header.guide_count, strand_count, params->cvs_per_strand, params->strand_count)
        .walked;
}

uint32_t nxg_generate_packed(const nxg_device_asset_desc *asset, const nxg_deformed_desc *deformed,
                             const nxg_generation_params *params, const nxg_packed_output_desc *output,
                             const nxg_launch_config *config, void *workspace, uint64_t workspace_bytes,
                             void *stream) {
    const uint32_t error = nxg_validate_packed_request(asset, deformed, params, output, config);
    if (error != NXG_ERROR_NONE) { return error; }
    return nxg_generate_packed_range(asset, deformed, params, output, config, 0u, params->strand_count,
                                     workspace, workspace_bytes, stream);
}

uint32_t nxg_generate_packed_range(const nxg_device_asset_desc *asset, const nxg_deformed_desc *deformed,
                                   const nxg_generation_params *params, const nxg_packed_output_desc *output,
                                   const nxg_launch_config *config, uint32_t first_strand, uint32_t strand_count,
                                   void *workspace, uint64_t workspace_bytes, void *stream) {
    uint32_t error =
        nxg::validate_range_request(asset, deformed, params, output, config, first_strand, strand_count);
    if (error != NXG_ERROR_NONE) { return error; }
    if ((error = nxg::check_launch_inputs(*asset, output)) != NXG_ERROR_NONE) { return error; }
    if (strand_count == 0u) { return NXG_ERROR_NONE; }
    if ((error = nxg::check_workspace(*asset, strand_count, params->cvs_per_strand, workspace, workspace_bytes)) !=
        NXG_ERROR_NONE) {
        return error;
    }
    const auto s = static_cast<cudaStream_t>(stream);
    nxg::set_last_cuda_error(0);
    const nxg_deformed_desc none{};
    const nxg_launch_config default_config{128u};
    return nxg::launch_generate(*asset, deformed ? *deformed : none, *params, *output,
                                config ? *config : default_config, first_strand, strand_count, workspace,
                                workspace_bytes, s, nullptr, nullptr,
                                nxg::launch_form(asset->header.guide_count, *params, strand_count, 1u, false, false), false);
}

uint32_t nxg_prepare_strand_order(const nxg_device_asset_desc *asset, const nxg_generation_params *params,
                                  uint32_t first_strand, uint32_t strand_count, void *workspace,
                                  uint64_t workspace_bytes, void *stream) {
    if (!asset || !params) { return NXG_ERROR_INVALID_ARGUMENT; }
    const nxg_deformed_desc none{};
    const nxg_launch_config default_config{128u};
    uint32_t error = nxg::validate_common(*asset, none, *params, default_config);
    if (error != NXG_ERROR_NONE) { return error; }
    if (first_strand > params->strand_count || strand_count > params->strand_count - first_strand) {
        return NXG_ERROR_INVALID_STRAND_RANGE;
    }
    if ((error = nxg::check_launch_inputs(*asset, nullptr)) != NXG_ERROR_NONE) { return error; }
    if (strand_count == 0u) { return NXG_ERROR_NONE; }
    if ((error = nxg::check_workspace(*asset, strand_count, params->cvs_per_strand, workspace, workspace_bytes)) !=
        NXG_ERROR_NONE) {
        return error;
    }
    nxg::set_last_cuda_error(0);
    return nxg::launch_order(*asset, params->seed, first_strand, strand_count, params->cvs_per_strand, workspace,
                             static_cast<cudaStream_t>(stream), false);
}

uint32_t nxg_generate_packed_ordered(const nxg_device_asset_desc *asset, const nxg_deformed_desc *deformed,
                                     const nxg_generation_params *params, const nxg_packed_output_desc *output,
                                     const nxg_launch_config *config, uint32_t first_strand,
                                     uint32_t strand_count, void *workspace, uint64_t workspace_bytes,
                                     void *stream) {
    uint32_t error =
        nxg::validate_range_request(asset, deformed, params, output, config, first_strand, strand_count);
    if (error != NXG_ERROR_NONE) { return error; }
    if ((error = nxg::check_launch_inputs(*asset, output)) != NXG_ERROR_NONE) { return error; }
    if (strand_count == 0u) { return NXG_ERROR_NONE; }
    if ((error = nxg::check_workspace(*asset, strand_count, params->cvs_per_strand, workspace, workspace_bytes)) !=
        NXG_ERROR_NONE) {
        return error;
    }
    const nxg_deformed_desc none{};
    const nxg_launch_config default_config{128u};
    return nxg::launch_generate(*asset, deformed ? *deformed : none, *params, *output,
                                config ? *config : default_config, first_strand, strand_count, workspace,
                                workspace_bytes, static_cast<cudaStream_t>(stream), nullptr, nullptr,
                                nxg::launch_form(asset->header.guide_count, *params, strand_count, 1u, true, false), true);
}

uint32_t nxg_query_strand_states(const nxg_device_asset_desc *asset, const nxg_deformed_desc *deformed,
                                 const nxg_generation_params *params, const uint32_t *strands, uint32_t count,
                                 nxg_strand_state *out, void *stream) {
    if (!asset || !params || (count && (!strands || !out))) { return NXG_ERROR_INVALID_ARGUMENT; }
    const nxg_deformed_desc none{};
    const nxg_launch_config default_config{128u};
    const uint32_t error = nxg::validate_common(*asset, deformed ? *deformed : none, *params, default_config);
    if (error != NXG_ERROR_NONE) { return error; }
    if (!nxg::sections_in_bounds(asset->header)) { return NXG_ERROR_INVALID_ASSET_METADATA; }
    if (count == 0u) { return NXG_ERROR_NONE; }
    const nxg::dev::AssetArgs a = nxg::resolve_asset(*asset);
    const nxg::dev::FrameArgs f = nxg::resolve_frame(a, deformed ? *deformed : none);
    const nxg::dev::ParamArgs p = nxg::resolve_params(*params, 1.0f);
    nxg::set_last_cuda_error(0);
    const uint32_t threads = 128u;
    nxg::dev::query_states_kernel<<<(count + threads - 1u) / threads, threads, 0,
                                    static_cast<cudaStream_t>(stream)>>>(
        a, f, p, strands, count, reinterpret_cast<nxg::dev::StrandStateOut *>(out));
    return nxg::record_cuda(cudaGetLastError());
}

uint32_t nxg_query_walk_states(const nxg_device_asset_desc *asset, const nxg_deformed_desc *deformed,
                               const nxg_generation_params *params, const uint32_t *strands, uint32_t count,
                               nxg_walk_state *out, void *workspace, uint64_t workspace_bytes, void *stream) {
    static_assert(sizeof(nxg_walk_state) == sizeof(nxg::dev::WalkDecision), "nxg_walk_state layout");
    if (!asset || !params || (count && (!strands || !out))) { return NXG_ERROR_INVALID_ARGUMENT; }
    const nxg_deformed_desc none{};
    const nxg_launch_config default_config{128u};
    const nxg_deformed_desc &frame = deformed ? *deformed : none;
    uint32_t error = nxg::validate_common(*asset, frame, *params, default_config);
    if (error != NXG_ERROR_NONE) { return error; }
    if ((error = nxg::check_launch_inputs(*asset, nullptr)) != NXG_ERROR_NONE) { return error; }
    if (count == 0u) { return NXG_ERROR_NONE; }
    const uint32_t P = params->cvs_per_strand;
    if (!nxg::parallel_path(asset->header.guide_count, P)) { return NXG_ERROR_INVALID_ARGUMENT; }
    if ((error = nxg::check_workspace(*asset, count, P, workspace, workspace_bytes)) != NXG_ERROR_NONE) {
        return error;
    }
    const auto s = static_cast<cudaStream_t>(stream);
    const nxg::WorkspaceLayout ws = nxg::workspace_layout(asset->header.guide_count, count, P);
    auto *offsets = reinterpret_cast<float4 *>(static_cast<unsigned char *>(workspace) + ws.offsets);
    nxg::LaunchArgs g{};
    g.a = nxg::resolve_asset(*asset);
    g.f = nxg::resolve_frame(g.a, frame);
    g.p = nxg::resolve_params(*params, 1.0f);
    g.first_strand = 0u;
    g.count = 0xffffffffu;  // strand ids are global: every id is a valid order entry
    g.order = strands;
    g.guide_frames = offsets + uint64_t{asset->header.guide_count} * P;
    nxg::set_last_cuda_error(0);
    const uint64_t n = uint64_t{asset->header.guide_count} * P;
    const uint32_t threads = 256u;
    const uint32_t blocks = static_cast<uint32_t>(std::max<uint64_t>(1u, std::min<uint64_t>(
        (n + threads - 1u) / threads, static_cast<uint64_t>(nxg::device_sm_count()) * 16u)));
    nxg::dev::guide_offsets_kernel<<<blocks, threads, 0, s>>>(g.a, g.f, P, g.p.support_scale, offsets, nullptr, 0u);
    if ((error = nxg::record_cuda(cudaGetLastError()))) { return error; }
    nxg::dev::walk_states_kernel<<<(count + 31u) / 32u, 32, 0, s>>>(g, count,
                                                                  reinterpret_cast<nxg::dev::WalkDecision *>(out));
    return nxg::record_cuda(cudaGetLastError());
}

uint32_t nxg_set_tile(uint32_t cvs_per_strand, uint32_t noise, const nxg_tile *tile) {
    if (cvs_per_strand < 2u || cvs_per_strand > nxg::kMaxParallelCvs) { return NXG_ERROR_INVALID_ARGUMENT; }
    std::atomic<uint32_t> &slot = nxg::g_tiles[cvs_per_strand][noise ? 1 : 0];
    const uint32_t builtin = nxg::packed_tile(nxg::builtin_tile(cvs_per_strand, noise != 0u));
    if (!tile) {
        slot.store(0u, std::memory_order_relaxed);
        return NXG_ERROR_NONE;
    }
    if (!nxg::valid_tile(cvs_per_strand, tile->lanes_per_strand, tile->cvs_per_lane) || tile->block_size > 1024u) {
        return NXG_ERROR_INVALID_ARGUMENT;
    }
    const uint32_t packed = nxg::packed_tile(*tile);
    slot.store(packed == builtin ? 0u : packed, std::memory_order_relaxed);
    return NXG_ERROR_NONE;
}

uint32_t nxg_get_tile(uint32_t cvs_per_strand, uint32_t noise, nxg_tile *tile) {
    if (!tile || cvs_per_strand < 2u || cvs_per_strand > nxg::kMaxParallelCvs) { return NXG_ERROR_INVALID_ARGUMENT; }
    const uint32_t packed = nxg::registered_tile(cvs_per_strand, noise != 0u);
    *tile = packed ? nxg_tile{packed & 0xffu, (packed >> 8) & 0xffu, (packed >> 16) * 32u}
                   : nxg::builtin_tile(cvs_per_strand, noise != 0u);
    return NXG_ERROR_NONE;
}

uint32_t nxg_autotune_packed(const nxg_device_asset_desc *asset, const nxg_deformed_desc *deformed,
                             const nxg_generation_params *params, const nxg_packed_output_desc *output,
                             uint32_t first_strand, uint32_t strand_count, void *workspace, uint64_t workspace_bytes,
                             uint32_t repeats, void *stream, nxg_tile *best, float *best_ms) {
    const nxg_launch_config config{128u};
    uint32_t error =
        nxg::validate_range_request(asset, deformed, params, output, &config, first_strand, strand_count);
    if (error != NXG_ERROR_NONE) { return error; }
    const uint32_t P = params->cvs_per_strand;
    if (strand_count == 0u || P > nxg::kMaxParallelCvs ||
        !nxg::parallel_path(asset->header.guide_count, P)) {
        return NXG_ERROR_INVALID_ARGUMENT;
    }
    if ((error = nxg_prepare_strand_order(asset, params, first_strand, strand_count, workspace, workspace_bytes,
                                          stream))) {
        return error;
    }
    const bool noise = params->noise_amplitude != 0.0f && params->noise_mask != 0.0f;
    const auto s = static_cast<cudaStream_t>(stream);
    cudaEvent_t start = nullptr, stop = nullptr;
    if ((error = nxg::record_cuda(cudaEventCreate(&start)))) { return error; }
    if ((error = nxg::record_cuda(cudaEventCreate(&stop)))) {
        cudaEventDestroy(start);
        return error;
    }
    const uint32_t saved = nxg::g_tiles[P][noise ? 1 : 0].load(std::memory_order_relaxed);
    nxg_tile winner{0u, 0u, 0u};
    float winner_ms = 0.0f;
    const uint32_t reps = std::max(1u, repeats);
    const auto time = [&](float *ms) -> uint32_t {  // with the tile registered now
        uint32_t e = NXG_ERROR_NONE;
        for (uint32_t r = 0; r <= reps; ++r) {  // one to warm up
            if (r == 1u && (e = nxg::record_cuda(cudaEventRecord(start, s)))) { return e; }
            if ((e = nxg_generate_packed_ordered(asset, deformed, params, output, &config, first_strand, strand_count,
                                                 workspace, workspace_bytes, stream))) {
                return e;
            }
        }
        if ((e = nxg::record_cuda(cudaEventRecord(stop, s))) || (e = nxg::record_cuda(cudaEventSynchronize(stop))) ||
            (e = nxg::record_cuda(cudaEventElapsedTime(ms, start, stop)))) {
            return e;
        }
        *ms /= static_cast<float>(reps);
        return NXG_ERROR_NONE;
    };
    // Nothing registered is the first candidate, and stays unless another is faster.
    winner = nxg::builtin_tile(P, noise);
    nxg_set_tile(P, noise ? 1u : 0u, nullptr);
    error = time(&winner_ms);
    const uint32_t blocks[5] = {64u, 128u, 256u, 384u, 512u};
    for (uint32_t lanes = 1u; lanes <= 32u && !error; lanes *= 2u) {
        for (uint32_t ppt = 1u; ppt <= 4u && !error; ppt *= 2u) {
            // tiles that hold the strand without idling half of their lanes
            if (!nxg::valid_tile(P, lanes, ppt) || (lanes > 2u && lanes * ppt >= 2u * P)) { continue; }
            for (const uint32_t block : blocks) {
                if (lanes == 1u && block >= nxg::builtin_tile(P, noise).block_size) { break; }  // no bound
                const nxg_tile tile{lanes, ppt, block};
                nxg_set_tile(P, noise ? 1u : 0u, &tile);
                float ms = 0.0f;
                if ((error = time(&ms))) { break; }
                if (ms < winner_ms) {
                    winner = tile;
                    winner_ms = ms;
                }
            }
        }
    }
    cudaEventDestroy(start);
    cudaEventDestroy(stop);
    if (error) {
        nxg::g_tiles[P][noise ? 1 : 0].store(saved, std::memory_order_relaxed);
        return error;
    }
    nxg_set_tile(P, noise ? 1u : 0u, &winner);
    if (best) { *best = winner; }
    if (best_ms) { *best_ms = winner_ms; }
    return NXG_ERROR_NONE;
}

} // extern "C"

// ---------------------------------------------------------------------------
// Motion samples (device_contract.h:42-53, :256-288): one description at
// several deformed frames, strand identities shared.  The strand order depends
// only on rest data and the seed, so it is prepared once; each sample then
// rebuilds the offset table for its frame and runs the generator.
// ---------------------------------------------------------------------------
namespace nxg {
namespace {

uint32_t validate_motion_samples(const nxg_device_asset_desc &asset, const nxg_motion_sample_desc *samples,
                                 uint32_t sample_count, const nxg_generation_params &params,
                                 const nxg_launch_config &config) {
    if (!samples || sample_count == 0u) { return NXG_ERROR_MISSING_MOTION_SAMPLES; }
    float previous = -INFINITY;
    for (uint32_t i = 0; i < sample_count; ++i) {
        if (!std::isfinite(samples[i].time) || samples[i].time <= previous) { return NXG_ERROR_INVALID_MOTION_TIMES; }
        previous = samples[i].time;
        const uint32_t error = validate_common(asset, samples[i].deformation, params, config);
        if (error != NXG_ERROR_NONE) { return error; }
    }
    return NXG_ERROR_NONE;
}

} // namespace
} // namespace nxg

extern "C" uint32_t nxg_generate_motion_packed(const nxg_device_asset_desc *asset,
                                               const nxg_motion_sample_desc *samples, uint32_t sample_count,
                                               const nxg_generation_params *params,
                                               const nxg_packed_output_desc *outputs,
                                               const nxg_launch_config *config, void *workspace,
                                               uint64_t workspace_bytes, void *stream) {
    if (!asset || !params || !outputs) { return NXG_ERROR_INVALID_ARGUMENT; }
    const nxg_launch_config cfg = config ? *config : nxg_launch_config{128u};
    uint32_t error = nxg::validate_motion_samples(*asset, samples, sample_count, *params, cfg);
    if (error != NXG_ERROR_NONE) { return error; }
    for (uint32_t i = 0; i < sample_count; ++i) {
        error = nxg::validate_range_request(asset, &samples[i].deformation, params, &outputs[i], &cfg, 0u,
                                            params->strand_count);
        if (error == NXG_ERROR_NONE) { error = nxg::check_launch_inputs(*asset, &outputs[i]); }
        if (error != NXG_ERROR_NONE) { return error; }
    }
    if ((error = nxg::check_workspace(*asset, params->strand_count, params->cvs_per_strand, workspace,
                                      workspace_bytes)) != NXG_ERROR_NONE) {
        return error;
    }
    const auto s = static_cast<cudaStream_t>(stream);
    nxg::set_last_cuda_error(0);
    const nxg::LaunchForm form =
        nxg::launch_form(asset->header.guide_count, *params, params->strand_count, sample_count, false, false);
    for (uint32_t i = 0; i < sample_count && !error; ++i) {
        error = nxg::launch_generate(*asset, samples[i].deformation, *params, outputs[i], cfg, 0u,
                                     params->strand_count, workspace, workspace_bytes, s, nullptr, nullptr, form,
                                     i != 0u);
    }
    return error;
}

extern "C" uint32_t nxg_generate_motion(const nxg_device_asset_desc *asset, const nxg_motion_sample_desc *samples,
                                        uint32_t sample_count, const nxg_generation_params *params,
                                        const nxg_motion_output_desc *output, const nxg_launch_config *config,
                                        void *workspace, uint64_t workspace_bytes, void *stream) {
    uint32_t error = nxg_validate_motion_request(asset, samples, sample_count, params, output, config);
    if (error != NXG_ERROR_NONE) { return error; }
    if ((error = nxg::check_launch_inputs(*asset, nullptr)) != NXG_ERROR_NONE) { return error; }
    if (reinterpret_cast<std::uintptr_t>(output->points) % 4u != 0u) { return NXG_ERROR_MISALIGNED_OUTPUT; }
    if ((error = nxg::check_workspace(*asset, params->strand_count, params->cvs_per_strand, workspace,
                                      workspace_bytes)) != NXG_ERROR_NONE) {
        return error;
    }
    const nxg_launch_config cfg = config ? *config : nxg_launch_config{128u};
    const auto s = static_cast<cudaStream_t>(stream);
    nxg::set_last_cuda_error(0);
    const uint64_t per_sample = uint64_t{params->strand_count} * params->cvs_per_strand * 3u;
    nxg_packed_output_desc none{};
    none.radius_scale = 1.0f;
    const nxg::LaunchForm form =
        nxg::launch_form(asset->header.guide_count, *params, params->strand_count, sample_count, false, false);
    for (uint32_t i = 0; i < sample_count && !error; ++i) {
        float *dst = reinterpret_cast<float *>(output->points) + per_sample * i;
        error = nxg::launch_generate(*asset, samples[i].deformation, *params, none, cfg, 0u, params->strand_count,
                                     workspace, workspace_bytes, s, dst, nullptr, form, i != 0u);
    }
    return error;
}

// ---------------------------------------------------------------------------
// Generation without a caller-provided workspace.
//
// Some callers cannot allocate device memory themselves: a renderer plugin
// whose host application owns every allocation through its own pool and
// memory budget, or a frame loop that must not call cudaMalloc because it
// implicitly synchronises the device and stalls the frame.  For them the
// library keeps its own scratch in a fixed-size array in device memory
// (below), held by every GPU that loads the library until the process exits.
// ---------------------------------------------------------------------------
namespace nxg {
namespace {

__device__ __align__(256) unsigned char g_static_scratch[NXG_STATIC_SCRATCH_BYTES];

constexpr int kMaxScratchDevices = 64;

// Driver entry points for the identity of the current context, so that an
// address looked up before a device reset (which destroys the context and
// unloads this module's device memory) is never handed out after it.
using CtxGetCurrentFn = int (*)(void **context);
using CtxGetIdFn = int (*)(void *context, unsigned long long *id);

struct ScratchSlot {
    unsigned long long context_id;  // 0: not looked up on this device yet
    void *address;
};
ScratchSlot g_static_scratch_slots[kMaxScratchDevices];
std::mutex g_static_scratch_mutex;

// The id of the context current on this thread, or 0 when none is current or
// the driver cannot say.
unsigned long long current_context_id() {
    static CtxGetCurrentFn get_current = nullptr;
    static CtxGetIdFn get_id = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void *fn = nullptr;
        cudaDriverEntryPointQueryResult found{};
        if (cudaGetDriverEntryPoint("cuCtxGetCurrent", &fn, cudaEnableDefault, &found) == cudaSuccess &&
            found == cudaDriverEntryPointSuccess) {
            get_current = reinterpret_cast<CtxGetCurrentFn>(fn);
        }
        fn = nullptr;
        if (cudaGetDriverEntryPoint("cuCtxGetId", &fn, cudaEnableDefault, &found) == cudaSuccess &&
            found == cudaDriverEntryPointSuccess) {
            get_id = reinterpret_cast<CtxGetIdFn>(fn);
        }
    });
    void *context = nullptr;
    unsigned long long id = 0u;
    if (!get_current || !get_id || get_current(&context) != 0 || context == nullptr || get_id(context, &id) != 0) {
        return 0u;
    }
    return id;
}

// The device address of g_static_scratch on the current device (host code
// may not use the array's name as a device pointer).  Looked up with
// cudaGetSymbolAddress once per device and context: again after a device
// reset, or whenever the current context's id cannot be read.
uint32_t static_scratch_address(void **out) {
    int device = 0;
    if (const uint32_t status = record_cuda(cudaGetDevice(&device))) { return status; }
    if (device < 0 || device >= kMaxScratchDevices) { return NXG_ERROR_INVALID_ARGUMENT; }
    std::lock_guard<std::mutex> lock(g_static_scratch_mutex);
    ScratchSlot &slot = g_static_scratch_slots[device];
    const unsigned long long id = current_context_id();
    if (id == 0u || id != slot.context_id || slot.address == nullptr) {
        void *address = nullptr;
        if (const uint32_t status = record_cuda(cudaGetSymbolAddress(&address, g_static_scratch))) {
            return status;
        }
        slot.address = address;
        slot.context_id = current_context_id();  // the lookup makes the device's context current
    }
    *out = slot.address;
    return NXG_ERROR_NONE;
}

} // namespace
} // namespace nxg

extern "C" uint32_t nxg_generate_packed_static_scratch(const nxg_device_asset_desc *asset,
                                                      const nxg_deformed_desc *deformed,
                                                      const nxg_generation_params *params,
                                                      const nxg_packed_output_desc *output,
                                                      const nxg_launch_config *config, void *stream) {
    const uint32_t error = nxg_validate_packed_request(asset, deformed, params, output, config);
    if (error != NXG_ERROR_NONE) { return error; }
    if (nxg::workspace_layout(asset->header.guide_count, params->strand_count, params->cvs_per_strand).total >
        NXG_STATIC_SCRATCH_BYTES) {
        return NXG_ERROR_STATIC_SCRATCH_LIMIT;
    }
    void *scratch = nullptr;
    if (const uint32_t status = nxg::static_scratch_address(&scratch)) { return status; }
    return nxg_generate_packed(asset, deformed, params, output, config, scratch, NXG_STATIC_SCRATCH_BYTES, stream);
}
