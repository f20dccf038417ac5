// batched.cu -- many descriptions in one persistent generate launch.
//
// A frame of several descriptions (each its own .nxg asset, strand count,
// CV count, stencil and noise settings) is generated by:
//   batched_offsets    every description's guide-offset table and guide frame
//                      records; zeroes the bins and the work counters;
//   batched_prepare    one pass over every strand of every description:
//                      root triangle and sort key (first stencil guide)
//                      with its histogram;
//   batched_scan       one CTA per description: bin offsets;
//   batched_scatter    per-description strand-locality orders (ranks in
//                      shared memory, one global atomic per block and bin);
//   batched_generate   one launch per class of work item -- noisy, noise-free
//                      -- each with the CTA shape, shared memory and register
//                      budget of its variant of the lane walk (walk.cuh);
//                      persistent CTAs pull (description, slice of its strand
//                      order) items of their class from an atomic counter --
//                      items of the costliest descriptions first.
// Five or six chained launches per frame whatever the description count, all
// enqueue-only and capturable in one CUDA graph.
#include "generator_core.cuh"
#include "walk.cuh"
#include "nxg_classic.h"
#include "nxg_internal.h"
#include "strand_math.cuh"

#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <numeric>
#include <vector>

namespace nxg {
namespace dev {

constexpr int kMaxBatch = NXG_MAX_BATCH;

struct BatchDesc {
    LaunchArgs g;              // asset, frame, params, count, outputs, order
    const float4 *offsets;     // guide-offset table (G x P)
    uint32_t *keys;            // count
    uint32_t *bins;            // guide_count + 1
    uint32_t strand_begin;     // prefix of strand counts (flat strand index)
    uint32_t item_begin;       // first work item (32 strands each)
    uint64_t offset_begin;     // prefix of guide_count * P (flat table index)
};

struct BatchArgs {
    uint32_t count;
    uint32_t total_strands;
    // Work-item classes, each its own generate launch: 0 = noisy
    // descriptions, 1 = noise-free descriptions.  Descriptions d[k] of class c
    // are k in [desc_first[c], desc_end[c]).
    uint32_t total_items[2];
    uint32_t desc_first[2], desc_end[2];
    uint32_t first_class;      // the class whose launch comes first
    uint32_t *item_counter;    // one counter per class
    uint64_t total_offsets;
    BatchDesc d[kMaxBatch];
};

__device__ __forceinline__ int desc_of_strand(const BatchArgs &b, uint32_t i) {
    int d = 0;
    while (d + 1 < static_cast<int>(b.count) && b.d[d + 1].strand_begin <= i) { ++d; }
    return d;
}

// One CTA (1024 threads) per description: exclusive scan of its bins.
__global__ void __launch_bounds__(1024) batched_scan_kernel(const __grid_constant__ BatchArgs b) {
    __shared__ uint32_t warp_sums[32];
    chain_start();
    chain_wait();
    const BatchDesc &d = b.d[blockIdx.x];
    uint32_t *data = d.bins;
    const uint32_t n = d.g.a.guide_count + 1u;
    const uint32_t tid = threadIdx.x;
    const uint32_t per = (n + blockDim.x - 1u) / blockDim.x;
    const uint32_t lo = min(n, tid * per), hi = min(n, lo + per);
    uint32_t sum = 0u;
    for (uint32_t i = lo; i < hi; ++i) { sum += data[i]; }
    uint32_t incl = sum;
    const int lane = tid & 31;
#pragma unroll
    for (int k = 1; k < 32; k <<= 1) {
        const uint32_t u = __shfl_up_sync(kFull, incl, k);
        if (lane >= k) { incl += u; }
    }
    if (lane == 31) { warp_sums[tid >> 5] = incl; }
    __syncthreads();
    if (tid < 32) {
        uint32_t w = tid < (blockDim.x >> 5) ? warp_sums[tid] : 0u;
#pragma unroll
        for (int k = 1; k < 32; k <<= 1) {
            const uint32_t u = __shfl_up_sync(kFull, w, k);
            if (lane >= k) { w += u; }
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

// Block-aggregated scatter (see scatter_order_blocked_kernel): a block whose
// flat range lies in one description with up to kBatchScatterBins bins
// ranks its strands in shared memory and takes one global atomic per
// non-empty bin; a block straddling descriptions takes one per strand.
constexpr uint32_t kBatchScatterBins = 8192u;

__global__ void __launch_bounds__(1024) batched_scatter_blocked_kernel(const __grid_constant__ BatchArgs b,
                                                                       uint32_t chunk) {
    extern __shared__ uint32_t slots[];
    chain_start();
    chain_wait();
    const uint32_t begin = blockIdx.x * chunk;
    const uint32_t end = min(b.total_strands, begin + chunk);
    if (begin >= end) { return; }
    const int home = desc_of_strand(b, begin);
    const BatchDesc &d = b.d[home];
    const uint32_t bins = d.g.a.guide_count + 1u;
    uint32_t *order = const_cast<uint32_t *>(d.g.order);
    if (desc_of_strand(b, end - 1u) != home || bins > kBatchScatterBins) {
        for (uint32_t i = begin + threadIdx.x; i < end; i += blockDim.x) {
            const BatchDesc &e = b.d[desc_of_strand(b, i)];
            const uint32_t local = i - e.strand_begin;
            const uint32_t pos = atomicAdd(&e.bins[min(e.keys[local], e.g.a.guide_count)], 1u);
            if (pos < e.g.count) { const_cast<uint32_t *>(e.g.order)[pos] = local; }
        }
        return;
    }
    const uint32_t lo = begin - d.strand_begin, hi = end - d.strand_begin;
    for (uint32_t k = threadIdx.x; k < bins; k += blockDim.x) { slots[k] = 0u; }
    __syncthreads();
    for (uint32_t i = lo + threadIdx.x; i < hi; i += blockDim.x) { atomicAdd(&slots[min(d.keys[i], bins - 1u)], 1u); }
    __syncthreads();
    for (uint32_t k = threadIdx.x; k < bins; k += blockDim.x) {
        const uint32_t n = slots[k];
        slots[k] = n ? atomicAdd(&d.bins[k], n) : 0u;
    }
    __syncthreads();
    for (uint32_t i = lo + threadIdx.x; i < hi; i += blockDim.x) {
        const uint32_t pos = atomicAdd(&slots[min(d.keys[i], bins - 1u)], 1u);
        if (pos < d.g.count) { order[pos] = i; }
    }
}

// Also clears the work counters and the descriptions' bins.
__global__ void batched_offsets_kernel(const __grid_constant__ BatchArgs b) {
    chain_start();
    chain_wait();
    if (blockIdx.x == 0 && threadIdx.x < 2) { b.item_counter[threadIdx.x] = 0u; }
    for (uint32_t d = 0; d < b.count; ++d) {
        const uint32_t bins = b.d[d].g.a.guide_count + 1u;
        for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < bins; i += gridDim.x * blockDim.x) {
            b.d[d].bins[i] = 0u;
        }
    }
    for (uint64_t i = blockIdx.x * static_cast<uint64_t>(blockDim.x) + threadIdx.x; i < b.total_offsets;
         i += static_cast<uint64_t>(gridDim.x) * blockDim.x) {
        int di = 0;
        while (di + 1 < static_cast<int>(b.count) && b.d[di + 1].offset_begin <= i) { ++di; }
        const BatchDesc &d = b.d[di];
        const uint64_t local = i - d.offset_begin;
        const uint32_t P = d.g.p.cvs_per_strand;
        const uint64_t table = static_cast<uint64_t>(d.g.a.guide_count) * P;
        if (local < table) {
            const_cast<float4 *>(d.offsets)[local] = guide_offset_entry(d.g.a, d.g.f, P,
                                                                        static_cast<uint32_t>(local / P),
                                                                        static_cast<uint32_t>(local % P));
        } else {
            const uint64_t gi = local - table;
            guide_frame_entry(d.g.a, d.g.f, d.g.p.support_scale, static_cast<uint32_t>(gi),
                              guide_offset_entry(d.g.a, d.g.f, P, static_cast<uint32_t>(gi), 0u),
                              const_cast<float4 *>(d.offsets) + table + 2u * gi);
        }
    }
}

// Per flat strand: the root triangle's sort key (first stencil guide) with
// the description's key histogram.  Block b owns the contiguous flat range
// [b*chunk, (b+1)*chunk), so its strands are mostly one description's and
// that description's histogram is kept in shared memory.
constexpr uint32_t kBatchPrivateBins = 4096u;

__global__ void __launch_bounds__(256) batched_prepare_kernel(const __grid_constant__ BatchArgs b, uint32_t chunk) {
    __shared__ uint32_t hist[kBatchPrivateBins];
    chain_start();
    chain_wait();
    const uint32_t begin = blockIdx.x * chunk;
    const uint32_t end = min(begin + chunk, b.total_strands);
    if (begin >= end) { return; }
    const int home = desc_of_strand(b, begin);
    const uint32_t home_bins = b.d[home].g.a.guide_count + 1u;
    const bool priv = home_bins <= kBatchPrivateBins;
    if (priv) {
        for (uint32_t i = threadIdx.x; i < home_bins; i += blockDim.x) { hist[i] = 0u; }
    }
    __syncthreads();
    for (uint32_t i = begin + threadIdx.x; i < end; i += blockDim.x) {
        const int di = desc_of_strand(b, i);
        const BatchDesc &d = b.d[di];
        const uint32_t local = i - d.strand_begin;
        const uint32_t triangle = sample_triangle(d.g.a, d.g.p.seed, d.g.first_strand + local);
        const uint32_t gi = __ldg(d.g.a.stencil + static_cast<uint64_t>(triangle) * kSlots);
        const uint32_t key = gi < d.g.a.guide_count ? gi : d.g.a.guide_count;
        d.keys[local] = key;
        if (priv && di == home) {
            atomicAdd(&hist[key], 1u);
        } else {
            atomicAdd(&d.bins[key], 1u);
        }
    }
    __syncthreads();
    if (priv) {
        for (uint32_t k = threadIdx.x; k < home_bins; k += blockDim.x) {
            if (hist[k]) { atomicAdd(&b.d[home].bins[k], hist[k]); }
        }
    }
}

// Shared memory of batched_generate: a head per CTA (the current
// description's gradient table with noise, t values and radii for up to
// kBatchMaxCvs CVs -- every warp of a CTA works on the same description), then
// the lane walk's region per warp.
constexpr uint32_t kBatchMaxCvs = 128u;
__host__ __device__ constexpr size_t batch_smem_bytes(int cls, bool classic, uint32_t warps) {
    return walk_head_bytes(cls == 0, kBatchMaxCvs, warps, kWalkChunk) +
           walk_warp_bytes(cls == 0, classic, kWalkChunk) * warps;
}
// 32-strand batches per warp in one work item of each class: four for the
// noisy class (fewer CTA-wide claims between long batches), one for the
// noise-free class (its descriptions are small; finer items balance better).
__host__ __device__ constexpr uint32_t batches_per_warp(int cls) { return cls == 1 ? 1u : 4u; }

// One batch of a description; out of line, one copy per variant.
template <int CLS, bool CLASSIC>
__device__ __noinline__ void batched_walk_item(const BatchDesc &d, uint32_t batch, int in_batch, int lane,
                                               unsigned char *mine, const float4 *table, const float *tvals,
                                               const float *rvals) {
    if constexpr (CLS == 0) {
        walk_noise_batch<CLASSIC>(d.g, d.offsets, mine, table, tvals, rvals, lane, batch, in_batch);
    } else {
        walk_plain_batch<CLASSIC>(d.g, d.offsets, mine, tvals, rvals, lane, batch, in_batch);
    }
}

// CLASSIC: some description applies Classic per-root scalars; descriptions
// without scalars still take the plain item.  CLS: the work-item class this
// launch runs (0: noisy, 1: noise-free), so each launch holds only its
// variants' code and runs at their register and shared-memory footprint.
template <bool CLASSIC, int CLS>
__global__ void __launch_bounds__(CLS == 1 ? 256 : 32 * kWalkNoiseWarps, CLS == 1 ? 3 : 1)
    batched_generate_kernel(const __grid_constant__ BatchArgs b) {
    extern __shared__ float4 smem[];
    __shared__ uint32_t claimed;
    __shared__ uint32_t next_batch;
    const int lane = threadIdx.x & 31;
    const uint32_t warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
    const uint32_t per_item = warps * batches_per_warp(CLS);
    // The strand order and offset tables are complete once this launch may
    // touch memory.  The next class's launch reads nothing this one writes (its
    // own descriptions' outputs), so from then on it may start as soon as this
    // launch's CTAs leave SMs free; it waits at its end only.
    if (b.first_class == static_cast<uint32_t>(CLS)) { chain_wait(); }
    chain_start();
    float *tvals = reinterpret_cast<float *>(smem + (CLS == 0 ? kTableFloat4 << walk_table_copies(warps, kWalkChunk) : 0));
    float *rvals = tvals + walk_padded(kBatchMaxCvs);
    unsigned char *mine = reinterpret_cast<unsigned char *>(rvals + walk_padded(kBatchMaxCvs)) +
                          walk_warp_bytes(CLS == 0, CLASSIC, kWalkChunk) * warp;
    const uint32_t total = b.total_items[CLS];
    const int first = static_cast<int>(b.desc_first[CLS]);
    const int last = static_cast<int>(b.desc_end[CLS]) - 1;
    int current = -1;
    // A work item is a contiguous slice of one description's strand order,
    // batches_per_warp(CLS) 32-strand batches per warp of the CTA, so the CTA's
    // strands share guide-offset rows in L1; its warps take the item's
    // batches from a shared counter, so a slow batch holds up only its own
    // warp until the item ends.  Each pass of the loop consumes one item.
    for (uint32_t guard = 0; guard <= total; ++guard) {
        if (threadIdx.x == 0) {
            claimed = atomicAdd(b.item_counter + CLS, 1u);
            next_batch = 0u;
        }
        __syncthreads();
        const uint32_t item = claimed;
        __syncthreads();
        if (item >= total) { break; }
        int di = first;
        while (di < last && b.d[di + 1].item_begin <= item) { ++di; }
        const BatchDesc &d = b.d[di];
        if (di != current) {  // the whole CTA: every warp works on the item's description
            walk_fill_head<CLS == 0>(d.g, smem, tvals, rvals);
            __syncthreads();
            current = di;
        }
        for (;;) {
            uint32_t k = 0u;
            if (lane == 0) { k = atomicAdd(&next_batch, 1u); }
            k = __shfl_sync(kFull, k, 0);
            if (k >= per_item) { break; }
            const uint32_t batch = ((item - d.item_begin) * per_item + k) * 32u;
            if (batch >= d.g.count) { break; }
            const int in_batch = static_cast<int>(min(32u, d.g.count - batch));
            if (CLASSIC && d.g.scalars != nullptr) {
                batched_walk_item<CLS, CLASSIC>(d, batch, in_batch, lane, mine, smem, tvals, rvals);
            } else {
                batched_walk_item<CLS, false>(d, batch, in_batch, lane, mine, smem, tvals, rvals);
            }
        }
        __syncthreads();  // the item's batches are done before the next claim resets the counter
    }
    // The second launch ends no earlier than the first, so what follows on the
    // stream follows both.
    if (b.first_class != static_cast<uint32_t>(CLS)) { chain_wait(); }
}

} // namespace dev

namespace {

constexpr uint64_t kAlign = 256u;
inline uint64_t up(uint64_t v) { return (v + kAlign - 1u) / kAlign * kAlign; }

struct BatchLayout {
    uint64_t counter;
    std::vector<uint64_t> keys, order, bins, offsets;
    uint64_t total;
};

BatchLayout batch_layout(const nxg_device_asset_desc *assets, const nxg_generation_params *params, uint32_t count) {
    BatchLayout l{};
    l.counter = 0u;
    uint64_t at = kAlign;
    for (uint32_t d = 0; d < count; ++d) {
        const uint64_t S = params[d].strand_count, P = params[d].cvs_per_strand, G = assets[d].header.guide_count;
        l.keys.push_back(at);
        at += up(S * 4u);
        l.order.push_back(at);
        at += up(S * 4u);
        l.bins.push_back(at);
        at += up((G + 1u) * 4u);
        l.offsets.push_back(at);
        at += up(G * (P + 2u) * 16u);  // offset table, 2 guide frame records per guide
    }
    l.total = at;
    return l;
}

int sm_count() {
    int device = 0, sms = 148;
    if (cudaGetDevice(&device) == cudaSuccess) { cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device); }
    return sms > 0 ? sms : 148;
}

} // namespace
} // namespace nxg

extern "C" uint64_t nxg_batched_workspace_size(const nxg_device_asset_desc *assets,
                                               const nxg_generation_params *params, uint32_t count) {
    if (!assets || !params || count == 0u || count > NXG_MAX_BATCH) { return 0u; }
    return nxg::batch_layout(assets, params, count).total;
}

namespace nxg {
namespace {

uint32_t generate_batched(const nxg_device_asset_desc *assets, const nxg_deformed_desc *deformed,
                          const nxg_generation_params *params, const nxg_packed_output_desc *outputs,
                          const nxg_classic_apply_desc *classic, uint32_t count, const nxg_launch_config *config,
                          void *workspace, uint64_t workspace_bytes, void *stream) {
    if (!assets || !params || !outputs || count == 0u || count > NXG_MAX_BATCH) { return NXG_ERROR_INVALID_ARGUMENT; }
    bool any_classic = false;
    if (classic) {
        for (uint32_t d = 0; d < count; ++d) {
            if (classic[d].root_scalars == nullptr) { continue; }
            if (reinterpret_cast<std::uintptr_t>(classic[d].root_scalars) % 8u != 0u) {
                return NXG_ERROR_MISALIGNED_OUTPUT;
            }
            any_classic = true;
        }
    }
    const nxg_launch_config cfg = config ? *config : nxg_launch_config{128u};
    for (uint32_t d = 0; d < count; ++d) {
        const uint32_t error = nxg_validate_packed_request(&assets[d], deformed ? &deformed[d] : nullptr, &params[d],
                                                           &outputs[d], &cfg);
        if (error != NXG_ERROR_NONE) { return error; }
        if (!sections_in_bounds(assets[d].header)) { return NXG_ERROR_INVALID_ASSET_METADATA; }
        if (reinterpret_cast<std::uintptr_t>(outputs[d].points) % 16u != 0u ||
            reinterpret_cast<std::uintptr_t>(outputs[d].roots) % 4u != 0u ||
            reinterpret_cast<std::uintptr_t>(outputs[d].root_uvs) % 8u != 0u ||
            reinterpret_cast<std::uintptr_t>(outputs[d].point_counts) % 4u != 0u) {
            return NXG_ERROR_MISALIGNED_OUTPUT;
        }
        if (params[d].cvs_per_strand > dev::kBatchMaxCvs ||
            uint64_t{assets[d].header.guide_count} * params[d].cvs_per_strand * 16u > (uint64_t{1} << 30)) {
            return NXG_ERROR_INVALID_ARGUMENT;  // more CVs than the CTAs' heads hold (kBatchMaxCvs), or the table's cap
        }
    }
    const BatchLayout layout = batch_layout(assets, params, count);
    if (!workspace || workspace_bytes < layout.total) { return NXG_ERROR_WORKSPACE_TOO_SMALL; }
    if (reinterpret_cast<std::uintptr_t>(workspace) % kAlign != 0u) { return NXG_ERROR_MISALIGNED_OUTPUT; }

    // Work-item class of each description, one generate launch per class at
    // its own occupancy: 0 for noisy descriptions, whose warps need the walk's
    // stage and lattice window; 1 for noise-free descriptions.
    constexpr uint32_t kClasses = 2u;
    std::vector<uint32_t> cls(count);
    for (uint32_t d = 0; d < count; ++d) {
        cls[d] = params[d].noise_amplitude != 0.0f && params[d].noise_mask != 0.0f ? 0u : 1u;
    }
    const auto kernel = [&](uint32_t c) -> const void * {
        if (c == 0u) {
            return any_classic ? reinterpret_cast<const void *>(dev::batched_generate_kernel<true, 0>)
                               : reinterpret_cast<const void *>(dev::batched_generate_kernel<false, 0>);
        }
        return any_classic ? reinterpret_cast<const void *>(dev::batched_generate_kernel<true, 1>)
                           : reinterpret_cast<const void *>(dev::batched_generate_kernel<false, 1>);
    };
    uint32_t status = NXG_ERROR_NONE;
    int device = 0, smem_optin = 48 * 1024;
    if (cudaGetDevice(&device) == cudaSuccess) {
        cudaDeviceGetAttribute(&smem_optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, device);
    }
    // CTA size and static shared memory per class.
    uint32_t class_block[kClasses] = {0u, 0u};
    size_t class_static[kClasses] = {0u, 0u};
    for (uint32_t c = 0; c < kClasses; ++c) {
        cudaFuncAttributes attr{};
        if ((status = record_cuda(cudaFuncGetAttributes(&attr, kernel(c))))) { return status; }
        uint32_t block = std::min(static_cast<uint32_t>(attr.maxThreadsPerBlock) / 32u * 32u,
                                  c == 0u ? 32u * dev::kWalkNoiseWarps
                                          : std::max<uint32_t>(32u, (cfg.block_size + 31u) / 32u * 32u));
        while (block > 32u && dev::batch_smem_bytes(static_cast<int>(c), any_classic, block / 32u) + 64u >
                                  static_cast<size_t>(smem_optin)) {
            block -= 32u;
        }
        class_block[c] = block;
        class_static[c] = attr.sharedSizeBytes;
    }

    auto *w = static_cast<unsigned char *>(workspace);
    dev::BatchArgs b{};
    b.count = count;
    b.item_counter = reinterpret_cast<uint32_t *>(w + layout.counter);
    // Costliest descriptions first (CVs per strand, tripled with noise), so the
    // longest work items start early and the tail is made of cheap ones.
    std::vector<uint32_t> rank(count);
    std::iota(rank.begin(), rank.end(), 0u);
    auto cost = [&](uint32_t d) {
        const bool noise = params[d].noise_amplitude != 0.0f && params[d].noise_mask != 0.0f;
        return uint64_t{params[d].cvs_per_strand} * (noise ? 3u : 1u);
    };
    std::stable_sort(rank.begin(), rank.end(), [&](uint32_t x, uint32_t y) {
        return cls[x] != cls[y] ? cls[x] < cls[y] : cost(x) > cost(y);
    });
    uint32_t strands = 0u, items[kClasses] = {0u, 0u};
    for (uint32_t c = 0; c < kClasses; ++c) { b.desc_first[c] = b.desc_end[c] = count; }
    uint64_t offsets = 0u;
    for (uint32_t k = 0; k < count; ++k) {
        const uint32_t d = rank[k];
        dev::BatchDesc &bd = b.d[k];
        const nxg_deformed_desc none{};
        bd.g.a = resolve_asset(assets[d]);
        bd.g.f = resolve_frame(bd.g.a, deformed ? deformed[d] : none);
        bd.g.p = resolve_params(params[d], outputs[d].radius_scale);
        bd.g.first_strand = 0u;
        bd.g.count = params[d].strand_count;
        bd.g.points = reinterpret_cast<float4 *>(outputs[d].points);
        bd.g.vec3_points = nullptr;
        bd.g.roots = reinterpret_cast<uint32_t *>(outputs[d].roots);
        bd.g.root_uvs = reinterpret_cast<float2 *>(outputs[d].root_uvs);
        bd.g.point_counts = outputs[d].point_counts;
        bd.g.order = reinterpret_cast<const uint32_t *>(w + layout.order[d]);
        if (classic && classic[d].root_scalars) {
            bd.g.scalars = reinterpret_cast<const float2 *>(classic[d].root_scalars);
            bd.g.classic_length = classic[d].apply_length != 0u;
            bd.g.classic_width = classic[d].apply_width != 0u;
        }
        bd.offsets = reinterpret_cast<const float4 *>(w + layout.offsets[d]);
        bd.g.guide_frames = bd.offsets + uint64_t{assets[d].header.guide_count} * params[d].cvs_per_strand;
        bd.keys = reinterpret_cast<uint32_t *>(w + layout.keys[d]);
        bd.bins = reinterpret_cast<uint32_t *>(w + layout.bins[d]);
        bd.strand_begin = strands;
        const uint32_t c = cls[d];
        if (b.desc_first[c] == count) { b.desc_first[c] = k; }
        b.desc_end[c] = k + 1u;
        bd.item_begin = items[c];
        bd.offset_begin = offsets;
        strands += params[d].strand_count;
        const uint32_t per_item = 32u * (class_block[c] / 32u) * dev::batches_per_warp(static_cast<int>(c));
        items[c] += (params[d].strand_count + per_item - 1u) / per_item;
        offsets += uint64_t{assets[d].header.guide_count} * (params[d].cvs_per_strand + 1u);
    }
    b.total_strands = strands;
    for (uint32_t c = 0; c < kClasses; ++c) { b.total_items[c] = items[c]; }
    b.total_offsets = offsets;

    const auto s = static_cast<cudaStream_t>(stream);
    const int sms = sm_count();
    set_last_cuda_error(0);
    b.first_class = items[0] ? 0u : 1u;
    const uint32_t offset_blocks = static_cast<uint32_t>(std::min<uint64_t>((offsets + 255u) / 256u, uint64_t(sms) * 16u));
    const uint32_t prepare_blocks = static_cast<uint32_t>(std::min<uint64_t>((strands + 255u) / 256u,
                                                                             uint64_t(sms) * 8u));
    const uint32_t prepare_chunk = ((strands + prepare_blocks - 1u) / prepare_blocks + 31u) / 32u * 32u;
    const uint32_t scatter_chunk = (strands + static_cast<uint32_t>(std::max(1, sms)) - 1u) /
                                   static_cast<uint32_t>(std::max(1, sms));
    if ((status = launch_chained(false, dev::batched_offsets_kernel, std::max(1u, offset_blocks), 256u, 0u, s, b)) ||
        (status = launch_chained(true, dev::batched_prepare_kernel, std::max(1u, prepare_blocks), 256u, 0u, s, b,
                                 prepare_chunk)) ||
        (status = launch_chained(true, dev::batched_scan_kernel, count, 1024u, 0u, s, b)) ||
        (status = launch_chained(true, dev::batched_scatter_blocked_kernel,
                                 (strands + scatter_chunk - 1u) / scatter_chunk, 1024u,
                                 dev::kBatchScatterBins * sizeof(uint32_t), s, b, scatter_chunk))) {
        return status;
    }

    // One generate launch per class with work, in stream order; each runs
    // persistent CTAs at its own occupancy.
    for (uint32_t c = 0; c < kClasses; ++c) {
        if (items[c] == 0u) { continue; }
        const void *fn = kernel(c);
        const uint32_t block = class_block[c];
        const size_t shm = dev::batch_smem_bytes(static_cast<int>(c), any_classic, block / 32u);
        if ((status = allow_shared(fn, class_static[c], smem_optin))) { return status; }
        int per_sm = 0;
        if ((status = record_cuda(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, static_cast<int>(block),
                                                                                shm)))) {
            return status;
        }
        const uint32_t grid = static_cast<uint32_t>(
            std::min<uint64_t>(items[c], static_cast<uint64_t>(std::max(1, sms * std::max(per_sm, 1)))));
        void *args[] = {&b};
        // The first class's launch is chained to the scatter; the second is a
        // programmatic dependent of the first that does not wait for its end: its
        // CTAs take the SMs that the first class's tail leaves idle.
        cudaLaunchConfig_t lc{};
        lc.gridDim = dim3(grid);
        lc.blockDim = dim3(block);
        lc.dynamicSmemBytes = shm;
        lc.stream = s;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[0].val.programmaticStreamSerializationAllowed = 1;
        lc.attrs = attr;
        lc.numAttrs = 1;
        if ((status = record_cuda(cudaLaunchKernelExC(&lc, fn, args)))) { return status; }
    }
    return record_cuda(cudaGetLastError());
}

} // namespace
} // namespace nxg

extern "C" uint32_t nxg_generate_batched(const nxg_device_asset_desc *assets, const nxg_deformed_desc *deformed,
                                         const nxg_generation_params *params,
                                         const nxg_packed_output_desc *outputs, uint32_t count,
                                         const nxg_launch_config *config, void *workspace,
                                         uint64_t workspace_bytes, void *stream) {
    return nxg::generate_batched(assets, deformed, params, outputs, nullptr, count, config, workspace,
                                 workspace_bytes, stream);
}

extern "C" uint32_t nxg_generate_batched_classic(const nxg_device_asset_desc *assets,
                                                 const nxg_deformed_desc *deformed,
                                                 const nxg_generation_params *params,
                                                 const nxg_packed_output_desc *outputs,
                                                 const nxg_classic_apply_desc *classic, uint32_t count,
                                                 const nxg_launch_config *config, void *workspace,
                                                 uint64_t workspace_bytes, void *stream) {
    if (!classic) { return NXG_ERROR_INVALID_ARGUMENT; }
    return nxg::generate_batched(assets, deformed, params, outputs, classic, count, config, workspace,
                                 workspace_bytes, stream);
}
