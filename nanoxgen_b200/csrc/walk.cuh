// walk.cuh -- the lane-walk generator, for strands of any CV count whose
// guide-offset table fits the workspace.
//
// A warp takes up to 32 strands of the strand order at a time:
//
//   setup  (lane = strand)   root sample, the eight stencil slots and the
//                            blend mode, folded into one weighted-sum record;
//   base   (8 lanes/strand)  the base curve from the guide-offset table, read
//                            as coalesced rows (consecutive lanes on
//                            consecutive CVs of one guide): straight to the
//                            output without noise, else a chunk of 16 CVs per
//                            strand into a stage in shared memory;
//   frame  (lane = strand)   with noise: the reference's cursor walk
//                            (generate.h:445-502) over the staged chunk --
//                            the transported normal is a serial recurrence,
//                            so a lane carries it CV by CV with the
//                            reference's rotation applied as a vector update,
//                            and no matrix products or cross-lane scans are
//                            needed; the noise comes from a window of lattice
//                            columns that moves along the strand;
//   store  (8 lanes/strand)  the chunk's float4s as coalesced streaming
//                            stores; preserveLength and Classic scalars are
//                            applied to the stage before it, or, on strands of
//                            more than 32 CVs (in the batched launch more than
//                            one chunk), to the written points afterwards,
//                            from L2.
//
// What bounds the noisy walk: of 1,000,000 strands x 32 CVs, separately built
// variants put about 120 us each on the walk itself (near the issue rate),
// the lattice (shared-memory wavefronts of random table reads) and the base
// rows (latency of L1 and L2), 60 on the stencil slots and 60 on the stores.
// So a longer strand is not staged whole (kWalkWholeCvs): chunks of 16 CVs
// and a moving window of five lattice columns keep a warp at 13 KB of shared
// memory instead of 20, the L1 at 60 KB instead of 28 for the base rows, and
// any CV count on the same path; the base step requests sixteen rows' entries
// before it uses one; and the gradient table is held eight times, free of
// bank conflicts.
// Twelve warps at 168 registers; sixteen at 128 spilled (729 us).  1,000,000 x
// 32: 601 us staged whole with all columns, 543 us now; 150,000 x 61 with
// preserveLength: 408 us on lane groups with scans, 191 us; 20,000 x 160: 1,241 us
// on one thread per strand, 104 us (121 before the equal batches of small calls).
//
// Stage rows are 49 words apart (73 and 97 where strands are staged whole) and a
// CV takes 3 words; both strides are odd,
// so a warp reading column c of 32 rows (frame step) and a warp reading one
// row are free of shared-memory bank conflicts, and the eight-lane base and
// store steps (four strands of eight CVs per access) meet at most two lanes
// to a bank.
#pragma once

#include "generator_core.cuh"

namespace nxg {
namespace dev {

constexpr int kWalkChunk = 16;                     // CVs staged at a time
// Strands of up to 24 CVs, and rewritten ones of up to 32 (noise_chunk), are staged
// whole instead, CHUNK 24 or 32.  There preserveLength and Classic scalars, which
// rewrite the points once the whole strand is known, do so in the stage: through
// L2 the second pass cost more than the chunks gain.  With noise and Classic
// scalars 500,000 x 24 331 -> 277 us, x 32 370 -> 341; preserveLength 500,000 x 17
// 325 -> 250, x 24 320 -> 268, x 32 357 -> 328.
constexpr int kWalkWholeCvs = 32;
// Words of a stage row: x, y, z per CV, and the strand's radius override (an odd stride).
__host__ __device__ constexpr int walk_row(int chunk) { return 3 * chunk + 1; }
// Noise lattice columns per axis and strand.  Five cover four lattice cells; a
// walk crosses a cell every five or six CVs at the sizes grooms use, so a
// strand refills its window about once (four columns: 533 us against 526 on
// 1,000,000 strands x 32).
constexpr int kWalkWindow = 5;
// Segments of more lattice cells than this leave a window after one pair of CVs,
// whose six values the direct noise gives for less than a window costs (200,000
// strands x 32 at 2 cells a segment 282 us from windows, 252 directly; at 6, where
// no window holds a pair, 406 with the windows tried first, 252).
constexpr float kWalkDirect = 1.5f;
constexpr int kWalkRecords = 6;                    // float4 setup records per strand
constexpr int kWalkClassicRecords = 8;             // with the Classic values of walk_classic_setup
constexpr int kWalkNoiseWarps = 12;                // warps of a full noise CTA

// Copies (log2) of the gradient table in a noise CTA's shared memory, entry e
// of copy k at (e << copies) + k.  With eight, a lane reads copy lane % 8, so
// the eight lanes that a 16-byte shared load serves at a time sit in eight
// different bank groups whatever entries they want (4 wavefronts per warp;
// with one copy, eight random entries in eight bank groups, 11.6): 1,000,000
// strands x 32 CVs 574 -> 551 us.  A CTA of a few warps runs too few strands
// to pay for the copies (2,000 strands x 16: 14.2 us with one, 15.5 with eight).
// A CTA of whole 32-CV stages has room for four.
__host__ __device__ constexpr uint32_t walk_table_copies(uint32_t warps, int chunk) {
    return warps < 8u ? 0u : (chunk > 24 ? 2u : 3u);
}
// Warps of a full CTA: what shared memory holds.
__host__ __device__ constexpr uint32_t walk_noise_warps(int chunk) { return chunk > 24 ? 11u : kWalkNoiseWarps; }

// Shared-memory bytes per warp.  With noise: stage | lattice window | records
// | output words.  Without (the base step writes the output directly):
// records | output words.
__host__ __device__ constexpr size_t walk_stage_bytes(int chunk) {
    return sizeof(float) * 32u * static_cast<size_t>(walk_row(chunk));
}
constexpr size_t kWalkLatticeBytes = sizeof(float2) * 3u * kWalkWindow * 32u;
constexpr size_t kWalkRecordBytes = sizeof(float4) * kWalkRecords * 32u;
constexpr size_t kWalkClassicRecordBytes = sizeof(float4) * kWalkClassicRecords * 32u;
constexpr size_t kWalkLocalBytes = sizeof(uint32_t) * 32u;
__host__ __device__ constexpr size_t walk_warp_bytes(bool noise, bool classic, int chunk) {
    return (noise ? walk_stage_bytes(chunk) + kWalkLatticeBytes + kWalkRecordBytes
                  : (classic ? kWalkClassicRecordBytes : kWalkRecordBytes)) +
           kWalkLocalBytes;
}
// Per CTA, before the warps: gradient table (noise) | t values | radii, each
// of P values and padding to a multiple of four (walk_pair reads t in pairs).
__host__ __device__ constexpr uint32_t walk_padded(uint32_t P) { return (P + 4u) & ~3u; }
__host__ __device__ constexpr size_t walk_head_bytes(bool noise, uint32_t P, uint32_t warps, int chunk) {
    return (noise ? sizeof(float4) * (kTableFloat4 << walk_table_copies(warps, chunk)) : 0u) +
           2u * sizeof(float) * walk_padded(P);
}
// Longest strand the walk takes (its t values and radii are in shared memory).
constexpr uint32_t kWalkMaxCvs = 1024u;

// Record q of strand s lives at records[q * 32 + s]:
//   q = 0..3  (row of slot 2q, weight, row of slot 2q+1, weight) of the
//             strand's weighted slots, zeros past its count; a row is
//             guide * P, the guide's first entry in the offset table
//   q = 4     (root position, 1 / weight sum)
//   q = 5     (root normal in normal mode else 0, slot count as bits)
//   q = 6, 7  Classic scalars without noise (walk_classic_setup): (first
//             point, length scale) and (width radius, width override flag,
//             width below the drop threshold, chord near it)
// Nearest mode becomes one slot of weight 1 and normal mode zero slots, so
// the base step evaluates every strand as
//   base = root + (inv * sum_j w_j offsets[row_j + c] + normal' * t_c) * length_scale.
// Square root by the PTX approximate instruction (one MUFU operation, no
// special-case branch); its relative error (below 2^-22) is far inside the
// position tolerance where it is used (arc lengths, sin(acos x)), and
// arguments below 2^-126 (lengths below 2^-63) read as zero.
__device__ __forceinline__ float sqrt_approx(float x) {
    float r;
    asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
// 1 / sqrt(x) by one MUFU operation, for x that is a normal float: the value
// rsqrtf gives there, without its scaling of subnormal arguments.
__device__ __forceinline__ float rsqrt_normal(float x) {
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

struct WalkRoot {
    F3 position, normal, surface_u, domain;
    bool lead;  // the first base point may not be the root exactly (kGuideLead)
};

// sample_root (generate.h:101-135) plus, with noise, the root's surface_u
// (generate.h:312-341) and rest position (generate.h:343-351), reusing the
// triangle's vertex data instead of loading it again.
template <bool NOISE>
__device__ __forceinline__ Root walk_root(const AssetArgs &a, const FrameArgs &f, uint32_t seed, uint32_t strand,
                                          F3 &surface_u, F3 &rest_position) {
    // The noise walk's instructions, not its lookups, bound it (gather3 there:
    // 706 -> 713 us on 5 samples of 250,000 strands; without noise 1,032 ->
    // 1,021 us on 4,000,000 x 24).
    const auto row = [](const float *p, uint32_t i) { return NOISE ? ld3(p, i) : gather3(p, i); };
    Root r;
    r.triangle = sample_triangle(a, seed, strand);
    const float r1 = random01(seed, strand, 2u);
    const float r2 = random01(seed, strand, 3u);
    const float s = __fsqrt_rn(r1);
    const float b0 = __fsub_rn(1.0f, s);
    r.b1 = __fmul_rn(s, __fsub_rn(1.0f, r2));
    r.b2 = __fmul_rn(s, r2);
    const uint3 t = load_triangle(a, r.triangle);
    const F3 p0 = row(f.positions, t.x), p1 = row(f.positions, t.y), p2 = row(f.positions, t.z);
    // A deformed frame's noise domain needs the rest-pose vertices too:
    // requested with the frame's, before any arithmetic waits on them.
    F3 q0 = p0, q1 = p1, q2 = p2;
    if (NOISE && f.positions != a.positions) {
        q0 = row(a.positions, t.x);
        q1 = row(a.positions, t.y);
        q2 = row(a.positions, t.z);
    }
    r.position = xbary(p0, p1, p2, b0, r.b1, r.b2);
    // The face normal only where the asset has no vertex normals (the
    // reference computes it first and then replaces it).
    if (a.flags & NXG_ASSET_HAS_NORMALS) {
        r.normal = xnormalize(xbary(row(f.normals, t.x), row(f.normals, t.y), row(f.normals, t.z),
                                    b0, r.b1, r.b2));
    } else {
        r.normal = xnormalize(xcross(xsub(p1, p0), xsub(p2, p0)));
    }
    r.u = 0.0f;
    r.v = 0.0f;
    const bool uvs = (a.flags & NXG_ASSET_HAS_TEXCOORDS) && a.texcoords;
    float2 uv0 = make_float2(0.0f, 0.0f), uv1 = uv0, uv2 = uv0;
    if (uvs) {
        uv0 = gather2(a.texcoords, t.x);
        uv1 = gather2(a.texcoords, t.y);
        uv2 = gather2(a.texcoords, t.z);
        r.u = __fadd_rn(__fadd_rn(__fmul_rn(uv0.x, b0), __fmul_rn(uv1.x, r.b1)), __fmul_rn(uv2.x, r.b2));
        r.v = __fadd_rn(__fadd_rn(__fmul_rn(uv0.y, b0), __fmul_rn(uv1.y, r.b1)), __fmul_rn(uv2.y, r.b2));
    }
    if constexpr (NOISE) {
        F3 tangent = {0.0f, 0.0f, 0.0f};
        if (uvs) {
            const F3 e1 = p1 - p0;
            const F3 e2 = p2 - p0;
            const float du1 = uv1.x - uv0.x, dv1 = uv1.y - uv0.y;
            const float du2 = uv2.x - uv0.x, dv2 = uv2.y - uv0.y;
            const float det = du1 * dv2 - dv1 * du2;
            if (fabsf(det) > 1.0e-12f) {
                tangent = (e1 * dv2 - e2 * dv1) * (1.0f / det);
                tangent = tangent - r.normal * dot(tangent, r.normal);
            }
        }
        surface_u = dot(tangent, tangent) > 1.0e-20f ? normalize(tangent) : fallback_surface_u(r.normal);
        const float rb0 = __fsub_rn(__fsub_rn(1.0f, r.b1), r.b2);
        rest_position = xbary(q0, q1, q2, rb0, r.b1, r.b2);
    }
    return r;
}

// The blend weights of generate.h:226-241 in the reference's rounding: every
// value IEEE-rounded and uncontracted.  Rewrites the weights of the strand's
// blended slots (records in slot order, as the setup step staged them) and
// returns their sum in slot order.  For powers other than 2 the setup step
// takes the fast power; it calls this only for strands whose sum may lie on
// the other side of the 1e-12 threshold that chooses between blending and the
// nearest-guide fallback (generate.h:261), so that choice is the reference's
// (to the last-bit agreement of CUDA's powf with the host's).  The hot path
// rarely takes it: the noise walk calls the out-of-line copy below (inlined
// it costs that kernel more registers than the call), the noise-free walk
// this inlined one (the call's saved registers cost it more).
__device__ __forceinline__ float walk_exact_weights_inline(const LaunchArgs &g, uint32_t triangle, F3 position,
                                                          F3 normal, float *slot_words, int lane) {
    const AssetArgs &a = g.a;
    const ParamArgs &p = g.p;
    float wsum = 0.0f;
    uint32_t blended = 0u;
    for (uint32_t j = 0; j < kSlots; ++j) {
        const uint32_t gi = __ldg(a.stencil + static_cast<uint64_t>(triangle) * kSlots + j);
        if (gi == kInvalid || gi >= a.guide_count) { continue; }
        const float4 gr = __ldg(g.guide_frames + 2u * gi);
        const float4 gn = __ldg(g.guide_frames + 2u * gi + 1u);
        if (__float_as_uint(gn.w) == 0u) { continue; }
        const F3 delta = xsub(position, F3{gr.x, gr.y, gr.z});
        const float d2 = xdot(delta, delta);
        if (xdot(normal, F3{gn.x, gn.y, gn.z}) < p.rejection_cos) { continue; }
        const float radius = gr.w;
        if (radius <= 0.0f || d2 >= __fmul_rn(radius, radius)) { continue; }
        const float x = __fsub_rn(1.0f, __fdiv_rn(__fsqrt_rn(d2), radius));
        const float w = p.weight_power == 2.0f ? __fmul_rn(x, x) : powf(x, p.weight_power);
        slot_words[((blended >> 1) * 32u + static_cast<uint32_t>(lane)) * 4u + (blended & 1u) * 2u + 1u] = w;
        ++blended;
        wsum = __fadd_rn(wsum, w);
    }
    return wsum;
}

static __device__ __noinline__ float walk_exact_weights(const LaunchArgs &g, uint32_t triangle, F3 position,
                                                        F3 normal, float *slot_words, int lane) {
    return walk_exact_weights_inline(g, triangle, position, normal, slot_words, lane);
}

// Whether a weight sum from the fast power (__powf, within p * 4e-7 + 1e-5
// relative of powf for exact bases) may lie on the other side of the 1e-12
// blend threshold from the reference's; twice that bound is used.
__device__ __forceinline__ bool walk_blend_uncertain(float wsum, float power) {
    return fabsf(wsum - 1.0e-12f) <= 2.0f * (power * 4.0e-7f + 1.0e-5f) * wsum;
}

// The lane walk's own per-strand decisions, for inspection
// (nxg_query_walk_states): the blend mode (0 blend, 1 nearest guide,
// 2 root normal), the nearest eligible guide, the weight sum the decision
// was taken on, and the weighted slots in the order the base step reads
// them (guide index and weight; one slot of weight 1 in nearest mode).
struct WalkDecision {
    uint32_t mode;
    uint32_t nearest;
    float weight_sum;
    uint32_t slot_count;
    uint32_t guides[kSlots];
    float weights[kSlots];
};

// The strand's RootSample (types.h:126-136) at roots[local]: three 16-byte
// stores when the array is 16-byte aligned, else twelve word stores.
__device__ __forceinline__ void walk_store_root(uint32_t *roots, uint32_t local, const Root &r) {
    uint32_t *dst = roots + static_cast<uint64_t>(local) * 12u;
    if ((reinterpret_cast<std::uintptr_t>(roots) & 15u) == 0u) {
        uint4 *v = reinterpret_cast<uint4 *>(dst);
        v[0] = make_uint4(root_word(r, 0), root_word(r, 1), root_word(r, 2), root_word(r, 3));
        v[1] = make_uint4(root_word(r, 4), root_word(r, 5), root_word(r, 6), root_word(r, 7));
        v[2] = make_uint4(root_word(r, 8), root_word(r, 9), root_word(r, 10), root_word(r, 11));
    } else {
#pragma unroll
        for (int w = 0; w < 12; ++w) { dst[w] = root_word(r, w); }
    }
}

// Setup step for this lane's strand.  The stencil slots follow eval_slot and
// the loop of generate.h:214-244 with the frame's guide roots, normals and
// support radii read from the per-frame guide records.  With `outputs`,
// also writes the strand's RootSample, root UV and point count.  With
// `decision` (inspection only), also reports the choices made.
template <bool NOISE>
__device__ __forceinline__ WalkRoot walk_setup(const LaunchArgs &g, float4 *records, uint32_t *locals, int lane,
                                               uint32_t pick, bool valid, uint32_t P, bool outputs = true,
                                               WalkDecision *decision = nullptr) {
    const AssetArgs &a = g.a;
    const FrameArgs &f = g.f;
    const ParamArgs &p = g.p;
    uint32_t local = g.order != nullptr ? __ldg(g.order + pick) : pick;
    if (local >= g.count) {
        local = 0u;
        valid = false;
    }
    WalkRoot r;
    r.surface_u = F3{0.0f, 0.0f, 0.0f};
    r.lead = false;
    F3 rest_position = {0.0f, 0.0f, 0.0f};
    const Root root = walk_root<NOISE>(a, f, p.seed, g.first_strand + local, r.surface_u, rest_position);
    if (outputs && valid) {  // generate.h:621-623
        if (g.roots) { walk_store_root(g.roots, local, root); }
        if (g.root_uvs) { g.root_uvs[local] = make_float2(root.u, root.v); }
        if (g.point_counts) { g.point_counts[local] = P; }
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) { records[q * 32 + lane] = make_float4(0.0f, 0.0f, 0.0f, 0.0f); }
    uint32_t stencil[kSlots];
    const uint32_t *row = a.stencil + static_cast<uint64_t>(root.triangle) * kSlots;
    if ((reinterpret_cast<std::uintptr_t>(a.stencil) & 15u) == 0u) {
        const uint4 s0 = __ldg(reinterpret_cast<const uint4 *>(row));
        const uint4 s1 = __ldg(reinterpret_cast<const uint4 *>(row) + 1);
        stencil[0] = s0.x; stencil[1] = s0.y; stencil[2] = s0.z; stencil[3] = s0.w;
        stencil[4] = s1.x; stencil[5] = s1.y; stencil[6] = s1.z; stencil[7] = s1.w;
    } else {
#pragma unroll
        for (uint32_t j = 0; j < kSlots; ++j) { stencil[j] = __ldg(row + j); }
    }
    float *slot_words = reinterpret_cast<float *>(records);
    // Guide frame record of slot j (an out-of-range slot reads as a corrupt
    // record: no slot).  With noise (fewer warps per SM to hide latency) four
    // are requested before any is used; without, one at a time, which keeps
    // the register count and the occupancy of the plain kernel.
    constexpr uint32_t kAhead = NOISE ? kSlots : 1u;
    float4 gr[kSlots], gn[kSlots];
    auto load_slot = [&](uint32_t j) {
        const bool in_range = stencil[j] != kInvalid && stencil[j] < a.guide_count;
        const uint32_t gi = in_range ? stencil[j] : 0u;
        gr[j] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        gn[j] = gr[j];
        if (a.guide_count != 0u) {
            gr[j] = __ldg(g.guide_frames + 2u * gi);
            gn[j] = __ldg(g.guide_frames + 2u * gi + 1u);
        }
        if (!in_range) { gn[j].w = 0.0f; }
    };
    // Blend weights (1 - d / r)^power in fast arithmetic (they feed positions
    // only); d^2, the rejection test and the radius test that decide which
    // slots count stay in the reference's exact rounding.
    const bool square = p.weight_power == 2.0f;
    float wsum = 0.0f;
    float nearest_d2 = FLT_MAX;
    uint32_t nearest = kInvalid;
    uint32_t blended = 0u;
#pragma unroll
    for (uint32_t j = 0; j < kSlots; ++j) {
        if (j % kAhead == 0u) {
#pragma unroll
            for (uint32_t k = 0; k < kAhead; ++k) { load_slot(j + k); }
        }
        if (__float_as_uint(gn[j].w) == 0u) { continue; }  // out of range or corrupt record
        r.lead = r.lead || (__float_as_uint(gn[j].w) & kGuideLead) != 0u;
        const F3 delta = xsub(root.position, F3{gr[j].x, gr[j].y, gr[j].z});
        const float d2 = xdot(delta, delta);
        if (xdot(root.normal, F3{gn[j].x, gn[j].y, gn[j].z}) < p.rejection_cos) { continue; }
        if (d2 < nearest_d2) {  // strict first minimum over eligible slots (generate.h:234)
            nearest_d2 = d2;
            nearest = stencil[j];
        }
        const float radius = gr[j].w;
        if (radius <= 0.0f || d2 >= __fmul_rn(radius, radius)) { continue; }
        // The base 1 - sqrt(d2) / r in the reference's rounding: near the
        // edge of the support radius it cancels, and a fast quotient would
        // change the weight there by a large fraction.  The square is then
        // the reference's weight bit for bit; other powers take __powf.
        const float x = __fsub_rn(1.0f, __fdiv_rn(__fsqrt_rn(d2), radius));
        const float w = square ? __fmul_rn(x, x)
                               : (x > 0.0f ? __powf(x, p.weight_power) : (p.weight_power > 0.0f ? 0.0f : 1.0f));
        float *dst = slot_words + ((blended >> 1) * 32u + lane) * 4u + (blended & 1u) * 2u;
        dst[0] = __uint_as_float(stencil[j] * P);
        dst[1] = w;
        ++blended;
        wsum = __fadd_rn(wsum, w);
    }
    if (!square && blended != 0u && walk_blend_uncertain(wsum, p.weight_power)) {
        if constexpr (NOISE) {
            wsum = walk_exact_weights(g, root.triangle, root.position, root.normal, slot_words, lane);
        } else {
            wsum = walk_exact_weights_inline(g, root.triangle, root.position, root.normal, slot_words, lane);
        }
    }
    float inv = 0.0f;
    F3 normal_term = {0.0f, 0.0f, 0.0f};
    uint32_t nb = blended;
    uint32_t mode = 0u;
    if (wsum > 1.0e-12f) {
        inv = 1.0f / wsum;
    } else if (nearest != kInvalid) {
        records[lane] = make_float4(__uint_as_float(nearest * P), 1.0f, 0.0f, 0.0f);
        nb = 1u;
        inv = 1.0f;
        mode = 1u;
    } else {
        nb = 0u;
        normal_term = root.normal;
        mode = 2u;
    }
    if (decision != nullptr) {
        decision->mode = mode;
        decision->nearest = nearest;
        decision->weight_sum = wsum;
        decision->slot_count = nb;
        for (uint32_t j = 0; j < kSlots; ++j) {
            const float *src = slot_words + (((j >> 1) * 32u + lane) * 4u + (j & 1u) * 2u);
            decision->guides[j] = j < nb ? __float_as_uint(src[0]) / P : kInvalid;
            decision->weights[j] = j < nb ? src[1] : 0.0f;
        }
    }
    records[4 * 32 + lane] = make_float4(root.position.x, root.position.y, root.position.z, inv);
    records[5 * 32 + lane] = make_float4(normal_term.x, normal_term.y, normal_term.z, __uint_as_float(nb));
    locals[lane] = local | (valid ? 0u : 0x80000000u);
    r.position = root.position;
    r.normal = root.normal;
    r.domain = F3{0.0f, 0.0f, 0.0f};
    if constexpr (NOISE) {
        const float decorrelation = 1.0f - p.noise_correlation;
        const float domain_scale = 100.0f * decorrelation * decorrelation;
        r.domain = (rest_position + F3{0.419276f, 0.184247f, 0.805721f}) * domain_scale;
    }
    return r;
}

// One output point of the strand whose output word is `word` (skipped when
// the word is marked invalid): float4 (position, radius), or Vec3 positions,
// 3P consecutive floats per strand (device_contract.h:47-52).  `again`: the
// point is read back soon, so it is stored without the streaming hint.
__device__ __forceinline__ void walk_emit(const LaunchArgs &g, uint32_t word, int P, int c, float4 q,
                                          bool again = false) {
    if (word >> 31) { return; }
    const uint64_t index = static_cast<uint64_t>(word) * static_cast<uint32_t>(P) + static_cast<uint32_t>(c);
    if (g.vec3_points) {
        float *out3 = g.vec3_points + 3u * index;
        __stcs(out3, q.x);
        __stcs(out3 + 1, q.y);
        __stcs(out3 + 2, q.z);
    } else if (again) {
        g.points[index] = q;
    } else {
        __stcs(g.points + index, q);
    }
}

// CV c of a staged row.
__device__ __forceinline__ F3 stage_get(const float *row, int c) {
    return F3{row[3 * c], row[3 * c + 1], row[3 * c + 2]};
}
__device__ __forceinline__ void stage_put(float *row, int c, F3 v) {
    row[3 * c] = v.x;
    row[3 * c + 1] = v.y;
    row[3 * c + 2] = v.z;
}

// Base point c of strand s from its records (generate.h:246-267, :300-310).
__device__ __forceinline__ F3 walk_base_point(const float4 *records, int s, int c, float t, float ls,
                                              const float4 *offsets) {
    const float4 head = records[4 * 32 + s];
    const float4 tail = records[5 * 32 + s];
    const uint32_t nb = __float_as_uint(tail.w);
    F3 acc = {0.0f, 0.0f, 0.0f};
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const float4 gw = records[q * 32 + s];
        if (static_cast<uint32_t>(2 * q) < nb) {
            const float4 d = __ldg(offsets + (__float_as_uint(gw.x) + static_cast<uint32_t>(c)));
            acc = acc + F3{d.x, d.y, d.z} * gw.y;
        }
        if (static_cast<uint32_t>(2 * q + 1) < nb) {
            const float4 d = __ldg(offsets + (__float_as_uint(gw.z) + static_cast<uint32_t>(c)));
            acc = acc + F3{d.x, d.y, d.z} * gw.w;
        }
    }
    const F3 off = acc * head.w + F3{tail.x, tail.y, tail.z} * t;
    return F3{head.x, head.y, head.z} + off * ls;
}

// Classic scalars without noise (xgen_classic_runtime.cpp:1650-1678,
// :1827-1858), for this lane's strand before its base step: the first base
// point (the root itself, unless a guide's first offset is not zero), the
// scale and the radius, left in records 6 and 7 for walk_base_direct.
__device__ __forceinline__ void walk_classic_setup(const LaunchArgs &g, float4 *records, int lane, const WalkRoot &root,
                                                   uint32_t local, const float *tvals, const float4 *offsets) {
    const ParamArgs &p = g.p;
    const float2 sc = __ldg(g.scalars + local);
    F3 front = root.position;
    if (root.lead) { front = walk_base_point(records, lane, 0, tvals[0], p.length_scale, offsets); }
    const float scale = g.classic_length ? sc.x : 1.0f;
    const float raw_width = g.classic_width ? sc.y
        : (p.radius_scale > 0.0f ? __fdiv_rn(__fmul_rn(2.0f, strand_radius(p, 0.0f)), p.radius_scale) : 0.0f);
    const float radius = __fmul_rn(__fmul_rn(0.5f, raw_width < 0.0f ? 0.0f : raw_width), p.radius_scale);
    records[6 * 32 + lane] = make_float4(front.x, front.y, front.z, scale);
    records[7 * 32 + lane] = make_float4(radius, g.classic_width ? 1.0f : 0.0f, raw_width < 1.0e-4f ? 1.0f : 0.0f, 0.0f);
}

// The sampled spline's length of this lane's strand.  Out of line: it is rare,
// and inlined its registers leave room for two CTAs per SM instead of three
// (1,022 us on 4,000,000 strands x 24; 935 with three).
static __device__ __noinline__ float walk_spline_length(const float4 *records, int lane, const float *tvals, float ls,
                                                        const float4 *offsets, int P) {
    return classic_spline_length_by(
        [&](int c) { return walk_base_point(records, lane, c, tvals[c], ls, offsets); }, P);
}

// The drop rule after the base step: a strand of too small a width, or one
// whose scaled chord walk_base_direct found near the 1e-4 threshold and whose
// sampled spline is below it, gets point count 0.  (The chord taken in the
// base step instead of from two points gathered before it: 935 -> 902 us on
// 4,000,000 strands x 24.)
__device__ __forceinline__ void walk_classic_drop(const LaunchArgs &g, const float4 *records, int lane, bool valid,
                                                  uint32_t local, const float *tvals, const float4 *offsets, int P) {
    const float4 width = records[7 * 32 + lane];
    bool keep = width.z == 0.0f;
    if (valid && keep && width.w != 0.0f) {
        keep = !(__fmul_rn(walk_spline_length(records, lane, tvals, g.p.length_scale, offsets, P),
                           records[6 * 32 + lane].w) < 1.0e-4f);
    }
    if (!keep && valid && g.point_counts != nullptr) { g.point_counts[local] = 0u; }
}

// An offset-table entry as two pairs, (x, y) and (z, unused).
__device__ __forceinline__ ulonglong2 walk_offset(const float4 *offsets, uint32_t index) {
    return __ldg(reinterpret_cast<const ulonglong2 *>(offsets) + index);
}

// Base step straight to the output (no noise).  Eight lanes per strand and
// four strands per pass: lane (s = pass * 4 + lane / 8, c = lane % 8)
// computes CVs c + 8m of a block of 32 CVs, m < 4.  One address per slot
// serves the lane's loads (the other CVs sit at fixed distances along the
// guide's offset row), every load of a warp instruction stays within one
// 128-byte line per strand, and a lane's t values are fixed for the block.  A
// pass runs as many slot pairs as its strands' largest count; a strand's
// loads past its own count are predicated off (no memory request), and its
// weights there are zero.
// CLASSIC applies records 6 and 7, and marks a strand whose scaled chord is
// near the drop threshold in record 7.  Every lane of the warp calls it.
template <bool CLASSIC>
__device__ __forceinline__ void walk_base_direct(const LaunchArgs &g, float4 *records, const uint32_t *locals,
                                                 const float *tvals, const float *rvals, const float4 *offsets,
                                                 int lane, int in_batch, int P) {
    constexpr int kPerLane = 4;
    const float ls = g.p.length_scale;
    for (int block = 0; block < P; block += 8 * kPerLane) {
        const int c = block + (lane & 7);
        const int cpl = min((P - block + 7) >> 3, kPerLane);
        float tv[kPerLane];
#pragma unroll
        for (int m = 0; m < kPerLane; ++m) { tv[m] = tvals[min(c + 8 * m, P - 1)]; }
        const float4 *column = offsets + c;
        for (int first = 0; first < in_batch; first += 4) {
            const int s = first + (lane >> 3);
            const bool live = s < in_batch;
            const float4 head = records[4 * 32 + s];
            const float4 tail = records[5 * 32 + s];
            const uint32_t nb = live ? __float_as_uint(tail.w) : 0u;
            const uint32_t pairs = __reduce_max_sync(kFull, (nb + 1u) >> 1);
            F3 acc[kPerLane];
            float4 da[kPerLane], db[kPerLane];
#pragma unroll
            for (int m = 0; m < kPerLane; ++m) {
                acc[m] = F3{0.0f, 0.0f, 0.0f};
                da[m] = db[m] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            }
            for (uint32_t q = 0; q < pairs; ++q) {
                // Past a strand's count the registers keep its last entries
                // and the weights are zero.
                const float4 gw = records[q * 32 + s];
                const float4 *ra = column + __float_as_uint(gw.x);
                const float4 *rb = column + __float_as_uint(gw.z);
                const bool la = 2u * q < nb, lb = 2u * q + 1u < nb;
#pragma unroll
                for (int m = 0; m < kPerLane; ++m) {
                    if (m < cpl) {
                        if (la) { da[m] = __ldg(ra + 8 * m); }
                        if (lb) { db[m] = __ldg(rb + 8 * m); }
                    }
                }
#pragma unroll
                for (int m = 0; m < kPerLane; ++m) {
                    if (m < cpl) { acc[m] = acc[m] + xyz(da[m]) * gw.y + xyz(db[m]) * gw.w; }
                }
            }
            const uint32_t word = live ? locals[s] : 0x80000000u;
            float4 front = {0.0f, 0.0f, 0.0f, 1.0f}, width = {0.0f, 0.0f, 0.0f, 0.0f};
            if constexpr (CLASSIC) {
                front = records[6 * 32 + s];
                width = records[7 * 32 + s];
            }
#pragma unroll
            for (int m = 0; m < kPerLane; ++m) {
                const int cm = c + 8 * m;
                if (m < cpl && cm < P) {
                    F3 base = F3{head.x, head.y, head.z} + (acc[m] * head.w + F3{tail.x, tail.y, tail.z} * tv[m]) * ls;
                    float radius = rvals[cm];
                    if constexpr (CLASSIC) {
                        const F3 chord = base - xyz(front);
                        if (live && cm == P - 1 && !(sqrtf(dot(chord, chord)) * front.w > 1.01e-4f)) {
                            records[7 * 32 + s].w = 1.0f;
                        }
                        if (g.classic_length) { base = xadd(xyz(front), xmul(xsub(base, xyz(front)), front.w)); }
                        if (width.y != 0.0f) { radius = width.x; }
                    }
                    walk_emit(g, word, P, cm, make_float4(base.x, base.y, base.z, radius));
                }
            }
        }
    }
}

// Base step of one chunk with noise: base points a + 1 .. a + n of each
// strand (the points after CVs a .. a + n - 1) into stage slots 0 .. n - 1,
// and for an odd n slot n too; past the strand's end they repeat the tip, a
// zero segment to the walk.  Lanes as in walk_base_direct.  Every lane of the
// warp calls it.
template <int CHUNK>
__device__ __forceinline__ void walk_base_chunk(const LaunchArgs &g, const float4 *records, float *stage,
                                                const float *tvals, const float4 *offsets, int lane, int in_batch,
                                                int a, int n, int P) {
    constexpr int kPerLane = CHUNK / 8;
    constexpr int kPasses = CHUNK == kWalkChunk ? 2 : 1;  // at most sixteen loads in flight
    constexpr uint32_t kTrip = 4u;
    const int c = lane & 7;
    const float ls = g.p.length_scale;
    uint32_t cm[kPerLane];
    float tv[kPerLane];
#pragma unroll
    for (int m = 0; m < kPerLane; ++m) {
        cm[m] = static_cast<uint32_t>(min(a + 1 + c + 8 * m, P - 1));
        tv[m] = tvals[cm[m]];
    }
    for (int first = 0; first < in_batch; first += 4 * kPasses) {
        uint32_t nb[kPasses], most = 0u;
        f32x2 xy[kPasses][kPerLane];
        float z[kPasses][kPerLane];
#pragma unroll
        for (int u = 0; u < kPasses; ++u) {
            const int s = first + 4 * u + (lane >> 3);
            nb[u] = s < in_batch ? __float_as_uint(records[5 * 32 + s].w) : 0u;
            most = max(most, nb[u]);
#pragma unroll
            for (int m = 0; m < kPerLane; ++m) {
                xy[u][m] = 0ull;
                z[u][m] = 0.0f;
            }
        }
        const uint32_t trips = __reduce_max_sync(kFull, (most + kTrip - 1u) / kTrip);
        for (uint32_t q = 0; q < trips; ++q) {
            ulonglong2 d[kPasses][kTrip][kPerLane];
            float w[kPasses][kTrip];
#pragma unroll
            for (int u = 0; u < kPasses; ++u) {
                const int s = first + 4 * u + (lane >> 3);
#pragma unroll
                for (uint32_t j = 0; j < kTrip; j += 2u) {
                    const float4 gw = records[(q * kTrip + j) / 2u * 32u + s];
                    const bool la = q * kTrip + j < nb[u], lb = q * kTrip + j + 1u < nb[u];
                    w[u][j] = gw.y;
                    w[u][j + 1u] = gw.w;
#pragma unroll
                    for (int m = 0; m < kPerLane; ++m) {
                        d[u][j][m] = d[u][j + 1u][m] = make_ulonglong2(0ull, 0ull);
                        if (la) { d[u][j][m] = walk_offset(offsets, __float_as_uint(gw.x) + cm[m]); }
                        if (lb) { d[u][j + 1u][m] = walk_offset(offsets, __float_as_uint(gw.z) + cm[m]); }
                    }
                }
            }
#pragma unroll
            for (int u = 0; u < kPasses; ++u) {
#pragma unroll
                for (uint32_t j = 0; j < kTrip; ++j) {
                    const f32x2 ww = both2(w[u][j]);
#pragma unroll
                    for (int m = 0; m < kPerLane; ++m) {
                        xy[u][m] = fma2(d[u][j][m].x, ww, xy[u][m]);
                        z[u][m] = fmaf(low2(d[u][j][m].y), w[u][j], z[u][m]);
                    }
                }
            }
        }
#pragma unroll
        for (int u = 0; u < kPasses; ++u) {
            const int s = first + 4 * u + (lane >> 3);
            if (s >= in_batch) { continue; }
            const float4 head = records[4 * 32 + s];
            const float4 tail = records[5 * 32 + s];
            float *row = stage + s * walk_row(CHUNK);
            const F3 root = {head.x, head.y, head.z}, normal = {tail.x, tail.y, tail.z};
#pragma unroll
            for (int m = 0; m < kPerLane; ++m) {
                stage_put(row, c + 8 * m,
                          root + (F3{low2(xy[u][m]), high2(xy[u][m]), z[u][m]} * head.w + normal * tv[m]) * ls);
            }
        }
    }
}

// Floor by a round-down add: for |x| < 2^22, x + 1.5 * 2^23 lies in
// [2^23, 2^24), where consecutive floats are consecutive integers, so the
// sum rounded toward minus infinity is 1.5 * 2^23 + floor(x) exactly.  Its
// bit pattern minus that of 1.5 * 2^23 is floor(x) as an integer, and the
// sum minus 1.5 * 2^23 is floor(x) as a float (an exact difference).  Two
// adds on the FMA pipe replace the rounding and conversion instructions.
constexpr float kFloorMagic = 12582912.0f;      // 1.5 * 2^23
constexpr uint32_t kFloorMagicBits = 0x4b400000u;
constexpr float kFloorMagicLimit = 4194304.0f;  // 2^22

// A strand's window on its noise lattice: kWalkWindow columns (A, B) per axis
// (see lattice_noise) from the lattice coordinate the walk had reached when
// it was filled.  Column k of axis a is at lat[(a * kWalkWindow + k) * 32] of
// this lane's lattice.  `bias` is per axis the bit pattern of 1.5 * 2^23 plus
// the first column's coordinate minus the axis' first column index.  The
// window holds every distance up to `limit`.
struct WalkWindow {
    uint32_t bias[3];
    float limit;
};

// 2 (noise - 0.5) along one axis at two coordinates from the window's columns
// (the regrouped blend of lattice_noise); the caller folds the 1/2 into the
// magnitude, a product by an exact power of two.  The round-down sum's bits
// minus `bias` index the lattice directly, bounded by the axis' last pair of
// columns whatever the coordinate (lanes with no strand read some column of
// their own lattice).
__device__ __forceinline__ f32x2 walk_lattice_pair(const float2 *lat, uint32_t bias, int axis, float xa, float xb) {
    const uint32_t last = static_cast<uint32_t>(axis * kWalkWindow + kWalkWindow - 2);
    const float ta = __fadd_rd(xa, kFloorMagic), tb = __fadd_rd(xb, kFloorMagic);
    const f32x2 w = sub2(pair2(xa, xb), pair2(ta - kFloorMagic, tb - kFloorMagic));
    const float2 *ca = lat + static_cast<int>(min(__float_as_uint(ta) - bias, last)) * 32;
    const float2 *cb = lat + static_cast<int>(min(__float_as_uint(tb) - bias, last)) * 32;
    const float2 a0 = ca[0], a1 = ca[32], b0 = cb[0], b1 = cb[32];
    const f32x2 w1 = add2(w, both2(-1.0f));
    const f32x2 s = mul2(mul2(mul2(w, w), w), fma2(w, fma2(w, both2(6.0f), both2(-15.0f)), both2(10.0f)));
    const f32x2 v0 = pair2(fmaf(a0.x, low2(w), a0.y), fmaf(b0.x, high2(w), b0.y));
    const f32x2 v1 = pair2(fmaf(a1.x, low2(w1), a1.y), fmaf(b1.x, high2(w1), b1.y));
    return fma2(s, sub2(v1, v0), v0);
}

// The window from `distance` on (bias, limit as a uint4), its columns written
// to `lat`.  Along axis ax the moving coordinate is d_ax + distance, the other
// two stay at the domain; the eight-corner blend of one column folds into
// (A, B), and the corner seeds are linear in the moving lattice coordinate X
// (noise_hash's LCG chain): seed(X + 1) = seed(X) + step.  `limit` keeps every
// coordinate, rounded, below the last column; it is negative (no distance
// fits) beyond the round-down floor's range.  A walk that leaves its window at
// the end starts the next one inside it, so the first two
// columns are moved there from the old window and only the others are
// computed (551 -> 533 us on 1,000,000 strands x 32).  Where one of the lanes says
// `direct`, the old window stays.  Out of line: it is called about twice per strand, and its
// registers inlined spill the walk's loop.  Every one of `lanes` calls it.
static __device__ __noinline__ uint4 walk_fill_window(F3 dom, float distance, WalkWindow old, float2 *lat,
                                                      const float4 *table, uint32_t copies, bool direct,
                                                      unsigned lanes) {
    __builtin_assume(__isShared(lat));
    __builtin_assume(__isShared(table));
    if (__any_sync(lanes, direct)) {
        return make_uint4(old.bias[0], old.bias[1], old.bias[2], __float_as_uint(old.limit));
    }
    uint32_t bias[3], moved[3];
    float lo[3];
    bool near = old.limit >= 0.0f;
#pragma unroll
    for (int ax = 0; ax < 3; ++ax) {
        lo[ax] = floorf(__fadd_rn(component(dom, ax), distance));
        bias[ax] = kFloorMagicBits + static_cast<uint32_t>(static_cast<int>(lo[ax])) -
                   static_cast<uint32_t>(ax * kWalkWindow);
        moved[ax] = bias[ax] - old.bias[ax];
        near = near && moved[ax] <= static_cast<uint32_t>(kWalkWindow) - 2u;
    }
    int first = 0;
    if (__all_sync(lanes, near)) {
        first = 2;
#pragma unroll
        for (int ax = 0; ax < 3; ++ax) {
            const float2 *from = lat + (ax * kWalkWindow + static_cast<int>(moved[ax])) * 32;
            const float2 c0 = from[0], c1 = from[32];
            lat[ax * kWalkWindow * 32] = c0;
            lat[(ax * kWalkWindow + 1) * 32] = c1;
        }
    }
    float limit = FLT_MAX;
#pragma unroll
    for (int ax = 0; ax < 3; ++ax) {
        const int ib = ax == 0 ? 1 : 0;  // the fixed axes, ascending
        const int ic = ax == 2 ? 1 : 2;
        const float d0 = component(dom, ax);
        const int X = static_cast<int>(lo[ax]);
        const float end = lo[ax] + static_cast<float>(kWalkWindow - 1);
        // x = d0 + distance rounds by at most 2^-24 of |x|.
        const float fits = (end - d0) - 4.0e-7f * (fabsf(d0) + fabsf(end));
        limit = fabsf(d0) + fabsf(end) < kFloorMagicLimit ? fminf(limit, fits) : -1.0f;
        const float db = component(dom, ib), dc = component(dom, ic);
        const float fb = floorf(db), fc = floorf(dc);
        const float wb = db - fb, wc = dc - fc;
        const float sb = s_curve(wb), sc = s_curve(wc);
        const int Yb = static_cast<int>(fb), Zc = static_cast<int>(fc);
        const uint32_t step = ax == 0 ? kLcgA2 : (ax == 1 ? kLcgA : 1u);
        uint32_t seed[4];
        float wgt[4], wdb[4], wdc[4];
#pragma unroll
        for (int corner = 0; corner < 4; ++corner) {
            const int ob = corner & 1, oc = corner >> 1;
            const int cx = ax == 0 ? X : Yb + ob;
            const int cy = ax == 1 ? X : (ax == 0 ? Yb + ob : Zc + oc);
            const int cz = ax == 2 ? X : Zc + oc;
            seed[corner] = static_cast<uint32_t>(cx) * kLcgA2 + static_cast<uint32_t>(cy) * kLcgA +
                           static_cast<uint32_t>(cz) + kLcgK;
            wgt[corner] = (ob ? sb : 1.0f - sb) * (oc ? sc : 1.0f - sc);
            wdb[corner] = wgt[corner] * (wb - static_cast<float>(ob));
            wdc[corner] = wgt[corner] * (wc - static_cast<float>(oc));
        }
#pragma unroll 1
        for (int k = first; k < kWalkWindow; ++k) {
            float A = 0.0f, B = 0.0f;
#pragma unroll
            for (int corner = 0; corner < 4; ++corner) {
                const float4 gr = table[temper_index(seed[corner] + static_cast<uint32_t>(k) * step) << copies];
                A += wgt[corner] * component4(gr, ax);
                B += component4(gr, ib) * wdb[corner] + component4(gr, ic) * wdc[corner];
            }
            lat[(ax * kWalkWindow + k) * 32] = make_float2(A, B);
        }
    }
    return make_uint4(bias[0], bias[1], bias[2], __float_as_uint(limit));
}

// 2 (noise - 0.5) at a point, for a segment longer than the window.
static __device__ __noinline__ float walk_direct_noise(const float4 *table, uint32_t copies, float x, float y,
                                                       float z) {
    __builtin_assume(__isShared(table));
    return 2.0f * (gradient_noise(table, x, y, z, copies) - 0.5f);
}

__device__ __forceinline__ float walk_effective_frequency(const ParamArgs &p, float original_length) {
    return original_length > 0.0f ? fmaxf(0.5f / original_length, p.noise_frequency) : p.noise_frequency;
}

// A strand's cursor between two CVs: the tangent after the last CV handled
// and the transported normal there, the base point of the next CV and the
// arc length at it.
struct WalkCursor {
    F3 tan, v, cur;
    float arc;
};

// A vector per half: one of CV c and one of CV c + 1.
struct F3x2 {
    f32x2 x, y, z;
};
__device__ __forceinline__ f32x2 dot2(const F3x2 &a, const F3x2 &b) {
    return fma2(a.z, b.z, fma2(a.y, b.y, mul2(a.x, b.x)));
}
// a x b; the products' sign is folded into `minus_a` = -a.
__device__ __forceinline__ F3x2 cross2(const F3x2 &a, const F3x2 &minus_a, const F3x2 &b) {
    return {fma2(a.y, b.z, mul2(minus_a.z, b.y)), fma2(a.z, b.x, mul2(minus_a.x, b.z)),
            fma2(a.x, b.y, mul2(minus_a.y, b.x))};
}
__device__ __forceinline__ F3x2 scale2(const F3x2 &a, f32x2 s) { return {mul2(a.x, s), mul2(a.y, s), mul2(a.z, s)}; }

// The transported normal over one CV: rotate_by(axis, acos(cos)) applied to v
// (generate.h:404-418, :475-481) as the vector update
//   M v = cos v + (1 - cos)(axis . v) axis + sin (axis x v).
__device__ __forceinline__ F3 walk_turn(F3 v, F3 axis, float cs, float omc, float sn) {
    const float k = omc * dot(axis, v);
    const F3 axv = cross(axis, v);
    return F3{v.x * cs + axis.x * k + axv.x * sn, v.y * cs + axis.y * k + axv.y * sn,
              v.z * cs + axis.z * k + axv.z * sn};
}

// Two steps of the cursor walk (generate.h:465-502): the noisy points qa, qb
// of the CV at the cursor and of the one after it, whose next base points are
// n0 and n1 (a strand's tip repeats the last base point: a zero segment).
// Tangent after a CV: the next segment's direction, carried over zero-length
// segments and at the tip; the transported normal turns by walk_turn with
// cos(acos x) = x and sin(acos x) = sqrt(1 - x^2), and is left unchanged when
// the axis is zero (the axis and that test in ordinary arithmetic: where the
// reference's rounded cross product vanishes for nearly parallel tangents,
// the rotation left here is within rounding of the identity).
//
// What the two CVs do alike runs as packed f32x2 arithmetic, one instruction
// for both (segments, tangents, rotation axes, frame vectors, the noise
// blend): the walk is bound by instruction issue and by its dependency
// chains, and only the turn of v is a chain from CV to CV.  The segment's
// squared length serves both its direction and the arc length.  `turn` is the
// CVs' t and `mscale` half the noise magnitude at t = 1 (the noise comes
// doubled).  The warp refills its windows when a strand that counts has
// reached the end of its own; a segment that no window holds makes the warp
// evaluate gradient noise directly.  Every lane of the warp calls it.
__device__ __forceinline__ void walk_pair(WalkCursor &s, F3 n0, F3 n1, f32x2 t, float mscale, float f_eff, F3 dom,
                                          bool counts, WalkWindow &wl, float2 *lat, const float4 *table,
                                          uint32_t copies, F3 &qa, F3 &qb) {
    const F3 sa = n0 - s.cur, sb = n1 - n0;
    const F3x2 seg = {pair2(sa.x, sb.x), pair2(sa.y, sb.y), pair2(sa.z, sb.z)};
    const f32x2 l2 = dot2(seg, seg);
    const float la = low2(l2), lb = high2(l2);
    F3x2 tn = scale2(seg, pair2(rsqrt_normal(la), rsqrt_normal(lb)));
    if (fminf(la, lb) <= 1.0e-20f) {  // a zero segment keeps the tangent; normalize() of a tiny one is (0, 1, 0)
        F3 ta = la > 1.0e-20f ? F3{low2(tn.x), low2(tn.y), low2(tn.z)} : la > 0.0f ? F3{0.0f, 1.0f, 0.0f} : s.tan;
        F3 tb = lb > 1.0e-20f ? F3{high2(tn.x), high2(tn.y), high2(tn.z)} : lb > 0.0f ? F3{0.0f, 1.0f, 0.0f} : ta;
        tn = F3x2{pair2(ta.x, tb.x), pair2(ta.y, tb.y), pair2(ta.z, tb.z)};
    }
    const float arc_b = __fadd_rn(s.arc, sqrt_approx(la));
    const f32x2 minus = both2(-1.0f);
    const F3x2 tp = {pair2(s.tan.x, low2(tn.x)), pair2(s.tan.y, low2(tn.y)), pair2(s.tan.z, low2(tn.z))};
    const F3x2 axis = cross2(tp, scale2(tp, minus), tn);
    const f32x2 d = dot2(tp, tn);
    const f32x2 a2 = dot2(axis, axis);
    const f32x2 d1 = fma2(d, d, minus);  // cos^2 - 1
    const float ca = low2(a2) > 0.0f ? low2(d) : 1.0f, cb = high2(a2) > 0.0f ? high2(d) : 1.0f;
    const f32x2 omc = sub2(both2(1.0f), pair2(ca, cb));
    const F3 va = walk_turn(s.v, F3{low2(axis.x), low2(axis.y), low2(axis.z)}, ca, low2(omc),
                            sqrt_approx(fmaxf(-low2(d1), 0.0f)));
    const F3 vb = walk_turn(va, F3{high2(axis.x), high2(axis.y), high2(axis.z)}, cb, high2(omc),
                            sqrt_approx(fmaxf(-high2(d1), 0.0f)));
    // The update is linear in v and the reference renormalises after every
    // step, a positive factor each time; here both steps' directions come from
    // one pair of roots, and the second goes on to the next pair.  (Carried
    // unnormalised over a whole strand, v underflows: a turn by theta, axis of
    // length sin theta, shortens it to sqrt(1 - c^2 + c^4) across the axis,
    // 0.866 at 45 degrees, and to |c + (1 - c)(1 - c^2)| along it, c = cos
    // theta, which vanishes near 139 degrees.)  No step lengthens v, so where
    // the second leaves some of it the first did too; where nothing is left
    // (`lost`), the second step is taken again with the reference's
    // normalisation of each, (0, 1, 0) below 1e-20.
    const F3x2 v = {pair2(va.x, vb.x), pair2(va.y, vb.y), pair2(va.z, vb.z)};
    const f32x2 v2 = dot2(v, v);
    F3x2 vu = scale2(v, pair2(rsqrt_normal(low2(v2)), rsqrt_normal(high2(v2))));
    F3x2 mv = scale2(vu, minus);
    F3x2 bn = cross2(vu, mv, tn);
    // The frame's third vector cross(bn, vu) is tn - vu (vu . tn) for a unit
    // vu; its part along vu joins vu's coefficient below.
    f32x2 mvn = dot2(mv, tn);
    const float da = __fmul_rn(s.arc, f_eff), db = __fmul_rn(arc_b, f_eff);
    const bool lost = !(high2(v2) > 1.0e-20f);
    bool lattice = true;
    if (__any_sync(kFull, counts && (lost || !(db <= wl.limit)))) {
        if (lost) {
            const F3 ua = normalize(va);
            const F3 ub = normalize(walk_turn(ua, F3{high2(axis.x), high2(axis.y), high2(axis.z)}, cb, high2(omc),
                                              sqrt_approx(fmaxf(-high2(d1), 0.0f))));
            vu = F3x2{pair2(ua.x, ub.x), pair2(ua.y, ub.y), pair2(ua.z, ub.z)};
            mv = scale2(vu, minus);
            bn = cross2(vu, mv, tn);
            mvn = dot2(mv, tn);
        }
        if (__any_sync(kFull, counts && !(db <= wl.limit))) {
            const uint4 w = walk_fill_window(dom, da, wl, lat, table, copies,
                                             counts && !(db - da <= kWalkDirect), kFull);
            wl = WalkWindow{{w.x, w.y, w.z}, __uint_as_float(w.w)};
            lattice = __all_sync(kFull, db <= wl.limit || !counts);
        }
    }
    f32x2 gx, gy, gz;
    if (lattice) {
        gx = walk_lattice_pair(lat, wl.bias[0], 0, __fadd_rn(dom.x, da), __fadd_rn(dom.x, db));
        gy = walk_lattice_pair(lat, wl.bias[1], 1, __fadd_rn(dom.y, da), __fadd_rn(dom.y, db));
        gz = walk_lattice_pair(lat, wl.bias[2], 2, __fadd_rn(dom.z, da), __fadd_rn(dom.z, db));
    } else {
        gx = pair2(walk_direct_noise(table, copies, __fadd_rn(dom.x, da), dom.y, dom.z),
                   walk_direct_noise(table, copies, __fadd_rn(dom.x, db), dom.y, dom.z));
        gy = pair2(walk_direct_noise(table, copies, dom.x, __fadd_rn(dom.y, da), dom.z),
                   walk_direct_noise(table, copies, dom.x, __fadd_rn(dom.y, db), dom.z));
        gz = pair2(walk_direct_noise(table, copies, dom.x, dom.y, __fadd_rn(dom.z, da)),
                   walk_direct_noise(table, copies, dom.x, dom.y, __fadd_rn(dom.z, db)));
    }
    const f32x2 magnitude = mul2(both2(mscale), t);  // 0 at CV 0
    const f32x2 lx = mul2(gx, magnitude), ly = mul2(gy, magnitude), lz = mul2(gz, magnitude);
    const f32x2 along = fma2(lz, mvn, lx);
    const f32x2 ox = fma2(tn.x, lz, fma2(bn.x, ly, mul2(vu.x, along)));
    const f32x2 oy = fma2(tn.y, lz, fma2(bn.y, ly, mul2(vu.y, along)));
    const f32x2 oz = fma2(tn.z, lz, fma2(bn.z, ly, mul2(vu.z, along)));
    qa = s.cur + F3{low2(ox), low2(oy), low2(oz)};
    qb = n0 + F3{high2(ox), high2(oy), high2(oz)};
    s.tan = F3{high2(tn.x), high2(tn.y), high2(tn.z)};
    s.v = F3{high2(vu.x), high2(vu.y), high2(vu.z)};
    s.cur = n1;
    s.arc = __fadd_rn(arc_b, sqrt_approx(lb));
}

// Fills a CTA's head (every thread calls it; a barrier must follow): the
// gradient table with noise, t = cv / (P - 1) (generate.h:295-298) and the
// radii, the padding after the tip repeating it.
template <bool NOISE, int CHUNK = kWalkChunk>
__device__ __forceinline__ void walk_fill_head(const LaunchArgs &g, float4 *table, float *tvals, float *rvals) {
    if constexpr (NOISE) {
        const uint32_t copies = walk_table_copies(blockDim.x >> 5, CHUNK);
        for (uint32_t i = threadIdx.x; i < static_cast<uint32_t>(kTableFloat4) << copies; i += blockDim.x) {
            const float *gradient = g.a.gradients + 3u * (i >> copies);
            table[i] = make_float4(__ldg(gradient), __ldg(gradient + 1), __ldg(gradient + 2), 0.0f);
        }
    }
    const uint32_t P = g.p.cvs_per_strand;
    for (uint32_t i = threadIdx.x; i < walk_padded(P); i += blockDim.x) {
        const float t = __fdiv_rn(static_cast<float>(min(i, P - 1u)), static_cast<float>(P - 1u));
        tvals[i] = t;
        rvals[i] = strand_radius(g.p, t);
    }
}

// preserveLength scale (generate.h:553-563), or 1.
__device__ __forceinline__ float walk_preserve_scale(const ParamArgs &p, float original_length, float noisy) {
    if (!(p.noise_preserve_length > 0.001f) || !(noisy > 0.0f)) { return 1.0f; }
    const float target = original_length * p.noise_preserve_length + noisy * (1.0f - p.noise_preserve_length);
    return fabsf(noisy - target) >= 0.0001f ? target / noisy : 1.0f;
}

// Store step of one chunk, eight lanes per strand as in walk_base_chunk: each
// store instruction writes four strands' runs of eight consecutive float4s.
// RADII: a strand's last stage word overrides its radius unless it is negative.
// Every lane of the warp calls it.
template <int CHUNK, bool RADII>
__device__ __forceinline__ void walk_store_chunk(const LaunchArgs &g, const float *stage, const uint32_t *locals,
                                                 const float *rvals, int lane, int in_batch, int a, int n, int P,
                                                 bool again) {
    constexpr int kPerLane = CHUNK / 8;
    const int c = lane & 7;
    float rv[kPerLane];
#pragma unroll
    for (int m = 0; m < kPerLane; ++m) { rv[m] = rvals[min(a + c + 8 * m, P - 1)]; }
    for (int first = 0; first < in_batch; first += 4) {
        const int s = first + (lane >> 3);  // at most 31
        const uint32_t word = s < in_batch ? locals[s] : 0x80000000u;
        const float *row = stage + s * walk_row(CHUNK);
        float radius = -1.0f;
        if constexpr (RADII) { radius = row[3 * CHUNK]; }
#pragma unroll
        for (int m = 0; m < kPerLane; ++m) {
            if (c + 8 * m < n) {
                const F3 q = stage_get(row, c + 8 * m);
                walk_emit(g, word, P, a + c + 8 * m, make_float4(q.x, q.y, q.z, RADII && !(radius < 0.0f) ? radius : rv[m]),
                          again);
            }
        }
    }
}

__device__ __forceinline__ F3 walk_scaled(F3 centre, F3 q, float k) { return centre + (q - centre) * k; }

// Rewrites the written points of the warp's strands: each lane holds its own
// strand's preserveLength scale (points to centre + (q - centre) * keep) and,
// CLASSIC, the Classic one (about `front`, in its uncontracted operations) and
// radius override (negative: none).  The points are this warp's own writes of
// a moment ago, so what bounds it is the latency of L2: eight lanes per strand
// and four strands at a time as in the store step, a lane's loads requested
// together, both scales in one pass.  500,000 strands x 24 with noise, one
// strand at a time and now: Classic scalars 424 -> 356 us, preserveLength 398
// -> 340, both 524 -> 361.  (Longer runs in flight, or out of line, the walk's
// own registers spill.)  Every lane of the warp calls it, after a __syncwarp.
template <bool CLASSIC>
__device__ __forceinline__ void walk_rescale(const LaunchArgs &g, const uint32_t *locals, F3 centre, float keep,
                                             F3 front, float scale, float radius, int lane, int in_batch, int P) {
    const bool length = CLASSIC && g.classic_length != 0u;
    constexpr int kPerLane = 4;
#pragma unroll 1
    for (int first = 0; first < in_batch; first += 4) {
        const int s = first + (lane >> 3);  // at most 31
        const uint32_t word = s < in_batch ? locals[s] : 0x80000000u;
        const F3 o = {__shfl_sync(kFull, centre.x, s), __shfl_sync(kFull, centre.y, s),
                      __shfl_sync(kFull, centre.z, s)};
        const float k = __shfl_sync(kFull, keep, s);
        F3 f = {0.0f, 0.0f, 0.0f};
        float by = 1.0f, r = -1.0f;
        if constexpr (CLASSIC) {
            f = F3{__shfl_sync(kFull, front.x, s), __shfl_sync(kFull, front.y, s), __shfl_sync(kFull, front.z, s)};
            by = __shfl_sync(kFull, scale, s);
            r = __shfl_sync(kFull, radius, s);
        }
        if ((word >> 31) || (k == 1.0f && !length && r < 0.0f)) { continue; }
        const uint64_t begin = static_cast<uint64_t>(word) * static_cast<uint32_t>(P);
        if (g.vec3_points) {
            for (int c = lane & 7; c < P; c += 8) {
                float *q = g.vec3_points + 3u * (begin + static_cast<uint32_t>(c));
                const F3 v = walk_scaled(o, F3{q[0], q[1], q[2]}, k);
                q[0] = v.x;
                q[1] = v.y;
                q[2] = v.z;
            }
            continue;
        }
        float4 *points = g.points + begin;
#pragma unroll 1
        for (int c = lane & 7; c < P; c += 8 * kPerLane) {
            float4 q[kPerLane];
#pragma unroll
            for (int m = 0; m < kPerLane; ++m) { q[m] = points[min(c + 8 * m, P - 1)]; }
#pragma unroll
            for (int m = 0; m < kPerLane; ++m) {
                F3 v = xyz(q[m]);
                if (k != 1.0f) { v = walk_scaled(o, v, k); }
                if (length) { v = xadd(f, xmul(xsub(v, f), by)); }
                if (c + 8 * m < P) { points[c + 8 * m] = make_float4(v.x, v.y, v.z, r < 0.0f ? q[m].w : r); }
            }
        }
    }
}

// The Classic application to noisy strands once their points are written
// (the rules of emit_strand: scale about the first point, width override, the
// drop rule with its chord bound and sampled-spline measure), after their
// preserveLength scale `kept` about the root `centre`, which is the first point
// too unless `lead`; `back` is the tip as written.  A dropped strand's point
// count becomes 0.  Every lane of the warp calls it, after a
// __syncwarp.
__device__ __forceinline__ void walk_classic_finish(const LaunchArgs &g, const uint32_t *locals, F3 centre,
                                                    float kept, bool lead, F3 back, int lane, int in_batch, int P) {
    const ParamArgs &p = g.p;
    const uint32_t word = lane < in_batch ? locals[lane] : 0x80000000u;
    F3 front = {0.0f, 0.0f, 0.0f};
    float scale = 1.0f, radius = -1.0f;
    if (!(word >> 31)) {
        const float4 *points = g.points + static_cast<uint64_t>(word) * static_cast<uint32_t>(P);
        const float2 sc = __ldg(g.scalars + word);
        const auto point = [=](int i) {
            const F3 q = xyz(points[i]);
            return kept != 1.0f ? walk_scaled(centre, q, kept) : q;
        };
        front = lead ? point(0) : centre;  // its displacement is 0
        if (kept != 1.0f) { back = walk_scaled(centre, back, kept); }
        scale = g.classic_length ? sc.x : 1.0f;
        const float raw_width = g.classic_width ? sc.y
            : (p.radius_scale > 0.0f ? __fdiv_rn(__fmul_rn(2.0f, strand_radius(p, 0.0f)), p.radius_scale) : 0.0f);
        bool keep = !(raw_width < 1.0e-4f);
        const F3 chord = back - front;
        if (keep && !(sqrtf(dot(chord, chord)) * scale > 1.01e-4f)) {
            keep = !(__fmul_rn(classic_spline_length_by(point, P), scale) <
                     1.0e-4f);
        }
        if (g.classic_width) {
            radius = __fmul_rn(__fmul_rn(0.5f, raw_width < 0.0f ? 0.0f : raw_width), p.radius_scale);
        }
        if (!keep && g.point_counts != nullptr) { g.point_counts[word] = 0u; }
    }
    __syncwarp();
    walk_rescale<true>(g, locals, centre, kept, front, scale, radius, lane, in_batch, P);
}

// The sampled spline's length of a staged strand, out of line: it is rare.
static __device__ __noinline__ float walk_stage_spline_length(const float *row, int P) {
    __builtin_assume(__isShared(row));
    return classic_spline_length_by([row](int c) { return stage_get(row, c); }, P);
}

// This lane's staged strand, all its points there: its preserveLength scale
// `keep` about the root `centre` and, CLASSIC, the rules of emit_strand (scale
// about the first point, width override into the row's last word, the drop
// rule with its chord bound and sampled-spline measure; a dropped strand's
// point count becomes 0).
template <bool CLASSIC, int CHUNK>
__device__ __forceinline__ void walk_finish_stage(const LaunchArgs &g, float *row, uint32_t word, F3 centre, float keep,
                                                  int P) {
    const auto point = [=](int c) {
        const F3 q = stage_get(row, c);
        return keep != 1.0f ? walk_scaled(centre, q, keep) : q;
    };
    F3 front = {0.0f, 0.0f, 0.0f};
    float scale = 1.0f;
    bool length = false;
    if constexpr (CLASSIC) {
        const ParamArgs &p = g.p;
        float radius = -1.0f;
        if (!(word >> 31)) {
            const float2 sc = __ldg(g.scalars + word);
            front = point(0);
            length = g.classic_length != 0u;
            scale = length ? sc.x : 1.0f;
            const float raw_width = g.classic_width ? sc.y
                : (p.radius_scale > 0.0f ? __fdiv_rn(__fmul_rn(2.0f, strand_radius(p, 0.0f)), p.radius_scale) : 0.0f);
            bool stays = !(raw_width < 1.0e-4f);
            const F3 chord = point(P - 1) - front;
            if (stays && !(sqrtf(dot(chord, chord)) * scale > 1.01e-4f)) {
                if (keep != 1.0f) {
                    for (int c = 0; c < P; ++c) { stage_put(row, c, point(c)); }
                    keep = 1.0f;
                }
                stays = !(__fmul_rn(walk_stage_spline_length(row, P), scale) < 1.0e-4f);
            }
            if (g.classic_width) {
                radius = __fmul_rn(__fmul_rn(0.5f, raw_width < 0.0f ? 0.0f : raw_width), p.radius_scale);
            }
            if (!stays && g.point_counts != nullptr) { g.point_counts[word] = 0u; }
        }
        row[3 * CHUNK] = radius;
    }
    if (keep == 1.0f && !length) { return; }
    for (int c = 0; c < P; ++c) {
        F3 v = stage_get(row, c);
        if (keep != 1.0f) { v = walk_scaled(centre, v, keep); }
        if (length) { v = xadd(front, xmul(xsub(v, front), scale)); }
        stage_put(row, c, v);
    }
}

// One batch of a warp with noise: strands [batch, batch + in_batch) of the
// order through setup, base, frame and store.  Every lane of the warp calls
// it; lanes past in_batch set up its first strand again and are ignored.
template <bool CLASSIC, int CHUNK = kWalkChunk>
__device__ __forceinline__ void walk_noise_batch(const LaunchArgs &g, const float4 *offsets, unsigned char *mine,
                                                 const float4 *table, const float *tvals, const float *rvals,
                                                 int lane, uint32_t batch, int in_batch) {
    float *stage = reinterpret_cast<float *>(mine);
    float2 *lattice = reinterpret_cast<float2 *>(mine + walk_stage_bytes(CHUNK)) + lane;
    const uint32_t copies = walk_table_copies(blockDim.x >> 5, CHUNK);
    table += static_cast<uint32_t>(lane) & ((1u << copies) - 1u);
    float4 *records = reinterpret_cast<float4 *>(mine + walk_stage_bytes(CHUNK) + kWalkLatticeBytes);
    uint32_t *locals =
        reinterpret_cast<uint32_t *>(mine + walk_stage_bytes(CHUNK) + kWalkLatticeBytes + kWalkRecordBytes);
    const ParamArgs &p = g.p;
    const int P = static_cast<int>(p.cvs_per_strand);
    const bool counts = lane < in_batch;
    const WalkRoot wr = walk_setup<true>(g, records, locals, lane, batch + (counts ? static_cast<uint32_t>(lane) : 0u),
                                         counts, static_cast<uint32_t>(P));
    __syncwarp();
    WalkCursor s{wr.normal, wr.surface_u, wr.position, 0.0f};
    if (__any_sync(kFull, wr.lead)) { s.cur = walk_base_point(records, lane, 0, tvals[0], p.length_scale, offsets); }
    float f_eff = p.noise_frequency;
    const float mscale = 0.5f * (p.noise_mask * p.noise_amplitude);
    const bool preserve = p.noise_preserve_length > 0.001f;
    const bool one_chunk = CHUNK != kWalkChunk || P <= CHUNK;  // staged whole
    const bool again = (CLASSIC || preserve) && !one_chunk;
    float *row = stage + lane * walk_row(CHUNK);
    WalkWindow window;
    window.limit = -1.0f;
    F3 previous = s.cur;
    float noisy = 0.0f;
    // Below the frequency floor the chunks are staged once to measure the base
    // curve (`measuring`) and once more to be walked: 200,000 strands x 32 225 ->
    // 187 us against a routine of its own that staged them all first; one chunk,
    // staged once, x 16 135 -> 94.
    bool measuring = false;
    float base_length = 0.0f;
    F3 measured = s.cur;
    for (int a = 0; a < P;) {
        const int n = min(CHUNK, P - a);
        walk_base_chunk<CHUNK>(g, records, stage, tvals, offsets, lane, in_batch, a, n, P);
        __syncwarp();
        if (a == 0 && base_length >= 0.0f) {
            // The effective frequency max(0.5 / length, frequency)
            // (generate.h:543) is the frequency itself for a strand of at
            // least 0.5 / frequency, which a chord that long from the root to
            // the chunk's last point or to the tip shows; else the base curve
            // is measured (generate.h:420-433).
            const auto sure = [&](F3 point) {
                const F3 chord = point - s.cur;
                return sqrt_approx(dot(chord, chord)) * p.noise_frequency * 0.9999f >= 0.5f || !counts;
            };
            measuring = !__all_sync(kFull, sure(stage_get(row, min(n, P - 1) - 1))) &&
                        (P <= CHUNK || !__all_sync(kFull, sure(walk_base_point(records, lane, P - 1, tvals[P - 1],
                                                                               p.length_scale, offsets))));
        }
        if (measuring) {
            for (int i = 0; i < min(n, P - 1 - a); ++i) {
                const F3 next = stage_get(row, i);
                const F3 d = next - measured;
                base_length = __fadd_rn(base_length, sqrt_approx(dot(d, d)));
                measured = next;
            }
            if (a + CHUNK >= P - 1) {
                f_eff = walk_effective_frequency(p, base_length);
                base_length = -1.0f;  // measured
                measuring = false;
            }
            if (a + CHUNK < P - 1 || a > 0) {  // the next chunk, or the first again
                a = measuring ? a + CHUNK : 0;
                __syncwarp();
                continue;
            }
        }
        F3 n0 = stage_get(row, 0), n1 = stage_get(row, 1);
#pragma unroll 1
        for (int i = 0; i < n; i += 2) {
            // The next pair is requested before this one is replaced (past
            // the chunk: slots that are not used).
            const int ahead = min(i + 2, CHUNK - 2);
            const F3 ahead0 = stage_get(row, ahead), ahead1 = stage_get(row, ahead + 1);
            F3 qa, qb;
            walk_pair(s, n0, n1, *reinterpret_cast<const f32x2 *>(tvals + a + i), mscale, f_eff, wr.domain, counts,
                      window, lattice, table, copies, qa, qb);
            if (preserve) {
                const F3 e = qa - previous, f = qb - qa;
                noisy += sqrt_approx(dot(e, e));
                if (i + 1 < n) { noisy += sqrt_approx(dot(f, f)); }
                previous = qb;
            }
            stage_put(row, i, qa);
            stage_put(row, i + 1, qb);
            n0 = ahead0;
            n1 = ahead1;
        }
        if (one_chunk && (CLASSIC || preserve)) {
            walk_finish_stage<CLASSIC, CHUNK>(g, row, counts ? locals[lane] : 0x80000000u, wr.position,
                                              preserve ? walk_preserve_scale(p, s.arc, noisy) : 1.0f, P);
        }
        __syncwarp();
        if (CLASSIC && one_chunk) {
            walk_store_chunk<CHUNK, true>(g, stage, locals, rvals, lane, in_batch, a, n, P, false);
        } else {
            walk_store_chunk<CHUNK, false>(g, stage, locals, rvals, lane, in_batch, a, n, P, again);
        }
        __syncwarp();
        a += CHUNK;
    }
    if constexpr (CHUNK == kWalkChunk) {
        const float kept = preserve && !one_chunk && counts ? walk_preserve_scale(p, s.arc, noisy) : 1.0f;
        if constexpr (CLASSIC) {
            if (!one_chunk) {
                walk_classic_finish(g, locals, wr.position, kept, wr.lead, stage_get(row, (P - 1) % kWalkChunk), lane,
                                    in_batch, P);
            }
        } else if (__any_sync(kFull, kept != 1.0f)) {
            walk_rescale<false>(g, locals, wr.position, kept, wr.position, 1.0f, -1.0f, lane, in_batch, P);
        }
        __syncwarp();
    }
}

// One batch of a warp without noise: setup and the base step straight to the
// output, with the Classic application.  As walk_noise_batch.
template <bool CLASSIC>
__device__ __forceinline__ void walk_plain_batch(const LaunchArgs &g, const float4 *offsets, unsigned char *mine,
                                                 const float *tvals, const float *rvals, int lane, uint32_t batch,
                                                 int in_batch) {
    float4 *records = reinterpret_cast<float4 *>(mine);
    uint32_t *locals = reinterpret_cast<uint32_t *>(mine + (CLASSIC ? kWalkClassicRecordBytes : kWalkRecordBytes));
    const int P = static_cast<int>(g.p.cvs_per_strand);
    const bool counts = lane < in_batch;
    const WalkRoot root = walk_setup<false>(g, records, locals, lane,
                                            batch + (counts ? static_cast<uint32_t>(lane) : 0u), counts,
                                            static_cast<uint32_t>(P));
    if constexpr (CLASSIC) {
        walk_classic_setup(g, records, lane, root, locals[lane] & 0x7fffffffu, tvals, offsets);
    }
    __syncwarp();
    walk_base_direct<CLASSIC>(g, records, locals, tvals, rvals, offsets, lane, in_batch, P);
    __syncwarp();
    if constexpr (CLASSIC) {
        walk_classic_drop(g, records, lane, counts, locals[lane] & 0x7fffffffu, tvals, offsets, P);
        __syncwarp();
    }
}

} // namespace dev
} // namespace nxg
