// sg_pixel_kernels.cu — the per-pixel kernels: the integrator megakernel, the
// per-pixel path-replay adjoint and the segments between vertex checkpoints.
//
// The integrator: one thread owns one pixel, runs the dispatch's samples
// through trace() and folds the batch into a Kahan-compensated per-pixel sum.
// CTAs cover 16x16 pixel tiles and each warp an 8x4 sub-tile, so neighbouring
// lanes trace neighbouring pixels and take the same branches as long as
// possible. Compiled once per landscape and FP64-sites variant, as
// sg_wave_stages.cu.
#include "sg_wave_common.cuh"

namespace sg {

namespace {

__device__ __forceinline__ void flush_events(const Events &ev, unsigned long long *events) {
    const uint32_t v[kEventCount] = {ev.vertices,      ev.sphere_tests,      ev.sphere_hits, ev.ring_tests,
                                     ev.light_samples, ev.shadow_rays,       ev.ring_events, ev.surface_events,
                                     ev.rng_draws,     ev.terrain_nodes,     ev.terrain_triangles,
                                     ev.prop_boxes,    ev.prop_tests};
#pragma unroll
    for (int k = 0; k < kEventCount; ++k) {
        unsigned long long x = v[k];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
        if ((threadIdx.x & 31u) == 0u && events) atomicAdd(&events[k], x);
    }
}

// Resident CTAs per SM the integrator is compiled for (register budget
// 65536 / (256 * SG_TRACE_MIN_BLOCKS) per thread). Measured on the ring
// workload: 1 CTA/SM 1846, 2 CTAs 2465, 3 CTAs 2882, 4 CTAs 2981 Msamples/s —
// more resident warps hide instruction-fetch and dependency latency better
// than the extra registers save spills.
#ifndef SG_TRACE_MIN_BLOCKS
#define SG_TRACE_MIN_BLOCKS 4
#endif

template <bool C, bool L, bool F, bool A>
__global__ void __launch_bounds__(kThreads, SG_TRACE_MIN_BLOCKS) trace_kernel(const __grid_constant__ TraceParams P) {
    extern __shared__ float4 smem[];
    const Scene S = stage_scene(P, smem);
    Events ev{};
    const Counter<C, L, F> K{&ev};
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
    const uint32_t x = blockIdx.x * kTile + (warp & 1u) * 8u + (lane & 7u);
    const uint32_t y = blockIdx.y * kTile + (warp >> 1) * 4u + (lane >> 3);
    if (x < P.width && y < P.height) {
        const uint32_t pixel = y * P.width + x;
        const uint32_t z = P.s.counts[2];
        // Lanes of a warp trace the same sample index in lockstep: adjacent
        // pixels then sit at the same vertex type (camera ray, ring event,
        // bounce) far more often than with per-lane path regeneration, which
        // measured 20 % slower on the ring workload.
        float4 total = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        float3 sky = f3(0.0f, 0.0f, 0.0f);
        Path path;
        Forward<A> nograd;
        const Cull cull = camera_cull<C>(P, blockIdx.y * gridDim.x + blockIdx.x);
        for (uint32_t smp = 0; smp < z; ++smp) {
            start_path(path, &P.s, K, pixel, x, y, smp);
            // The camera ray takes the tile's cull masks, later rays none.
            if (!step(S, K, path, nograd, cull)) {
                while (!step(S, K, path, nograd)) {
                }
            }
            const float4 r = finish_path(path);
            total.x += r.x;
            total.y += r.y;
            total.z += r.z;
            total.w += r.w;
            sky = sky + path.backdrop;
        }
        if (P.sky_on) fold_backdrop(P, pixel, sky);
        // Progressive accumulation: the WGSL keeps a running mean
        // (pathtrace.wgsl:1662-1674); here the per-pixel sum is compensated
        // (Kahan) and the mean re-derived from it.
        const uint32_t old_count = P.s.counts[1];
        const float new_count = (float)(old_count + z);
        float4 sum, comp;
        if (old_count == 0u) {
            sum = total;
            comp = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        } else {
            sum = P.sum[pixel];
            comp = P.comp[pixel];
            float yv, t;
            yv = __fsub_rn(total.x, comp.x); t = __fadd_rn(sum.x, yv); comp.x = __fsub_rn(__fsub_rn(t, sum.x), yv); sum.x = t;
            yv = __fsub_rn(total.y, comp.y); t = __fadd_rn(sum.y, yv); comp.y = __fsub_rn(__fsub_rn(t, sum.y), yv); sum.y = t;
            yv = __fsub_rn(total.z, comp.z); t = __fadd_rn(sum.z, yv); comp.z = __fsub_rn(__fsub_rn(t, sum.z), yv); sum.z = t;
            yv = __fsub_rn(total.w, comp.w); t = __fadd_rn(sum.w, yv); comp.w = __fsub_rn(__fsub_rn(t, sum.w), yv); sum.w = t;
        }
        P.sum[pixel] = sum;
        P.comp[pixel] = comp;
        P.mean[pixel] = make_float4(__fdiv_rn(__fsub_rn(sum.x, comp.x), new_count),
                                    __fdiv_rn(__fsub_rn(sum.y, comp.y), new_count),
                                    __fdiv_rn(__fsub_rn(sum.z, comp.z), new_count),
                                    __fdiv_rn(__fsub_rn(sum.w, comp.w), new_count));
    }
    if constexpr (C) flush_events(ev, P.events);
}

// ---------------------------------------------------------------------------
// Path-replay adjoint
// ---------------------------------------------------------------------------
// One sample's derivative: pass 1 replays the path without derivatives and
// records what pass 2 needs to weigh each factor by the radiance gathered
// after it (sg_adjoint.cuh); pass 2 replays it again and scatters.
// A path whose ring-indirect cap does not bind ends after pass 1 (its
// deferred factors flushed); the others replay once more. `lanes`: the
// warp's lanes that run the same samples; they meet after each pass so that
// a warp replays one pass at a time (lanes left to drift between the two
// passes would run two copies of the integrator apart).
// Replays a checkpointed path from `path` until a scatter brings its depth
// to `end_depth`, where the next segment's record starts, or it ends.
template <bool L, bool F>
__device__ __forceinline__ void replay_segment(const Scene &S, Counter<false, L, F> K, Prb &G, Path &path,
                                               uint32_t end_depth, Cull first = kTestAll) {
    if (step(S, K, path, G, first) || path.depth >= end_depth) return;
    while (!step(S, K, path, G)) {
        if (path.depth >= end_depth) break;
    }
}

template <bool L, bool F>
__device__ __forceinline__ void adjoint_sample(const Scene &S, Counter<false, L, F> K, Prb &G, float3 w, uint32_t pixel,
                                               uint32_t x, uint32_t y, uint32_t smp, unsigned lanes,
                                               uint32_t segment_end, Cull cull) {
    bool again = true;
#pragma unroll 1
    for (int pass = 0; pass < 2; ++pass) {
        if (again) {
            Path path;
            start_path(path, S.s, K, pixel, x, y, smp);
            if (segment_end) {
                // A checkpointed sample: its first segment, once.
                replay_segment(S, K, G, path, segment_end, cull);
                again = false;
            } else {
                // The camera ray takes the tile's cull masks.
                if (!step(S, K, path, G, cull)) {
                    while (!step(S, K, path, G)) {
                    }
                }
                if (pass == 0) {
                    again = G.deferral_full || cap_binds(G, path.radiance);
                    if (again) pass2_setup(G, path.radiance, w);
                    else flush_deferred(G);
                }
            }
        }
        __syncwarp(lanes);
    }
}

// Resident CTAs per SM the adjoint is compiled for.
#ifndef SG_ADJOINT_MIN_BLOCKS
#define SG_ADJOINT_MIN_BLOCKS 2
#endif

template <bool L, bool F>
__global__ void __launch_bounds__(kThreads, SG_ADJOINT_MIN_BLOCKS)
    adjoint_kernel(const __grid_constant__ TraceParams P, const __grid_constant__ AdjointParams A) {
    extern __shared__ float4 smem[];
    // Dynamic shared memory: bodies and staged tables (stage_scene), the
    // inverse colours (2 float4 per body), then the gradient windows.
    const uint32_t n_bodies = P.s.counts[0];
    float4 *inv = smem + trace_smem_floats(P) / 4u;
    float *window = reinterpret_cast<float *>(inv + 2u * n_bodies);
    const uint32_t window_n = A.tau_window + A.color_window;
    for (uint32_t k = threadIdx.x; k < window_n; k += blockDim.x) window[k] = 0.0f;
    for (uint32_t k = threadIdx.x; k < n_bodies; k += blockDim.x) {
        const float4 m = P.bodies[k * kBodyVec4 + kMaterial], r = P.bodies[k * kBodyVec4 + kRingColor];
        inv[2u * k] = make_float4(inv_or_zero(m.x), inv_or_zero(m.y), inv_or_zero(m.z), 0.0f);
        inv[2u * k + 1u] = make_float4(inv_or_zero(r.x), inv_or_zero(r.y), inv_or_zero(r.z), 0.0f);
    }
    const Scene S = stage_scene(P, smem);  // synchronises the block
    const Counter<false, L, F> K{nullptr};
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
    const uint32_t x = blockIdx.x * kTile + (warp & 1u) * 8u + (lane & 7u);
    const uint32_t y = blockIdx.y * kTile + (warp >> 1) * 4u + (lane >> 3);
    float own[6u * kColorSlots];
#pragma unroll
    for (uint32_t k = 0; k < 6u * kColorSlots; ++k) own[k] = 0.0f;
    const uint32_t own_n = 6u * (n_bodies < kColorSlots ? n_bodies : kColorSlots);
    PrbLists lists;
    float4 local[kMaxLocal];
    Prb G;
    G.lists = &lists;
    G.local = local;
    G.local_stride = 1u;
    G.sink = GradSink{own, own_n, window, A.tau_window, window + A.tau_window, A.color_window, A.grad, 1u};
    G.inv = inv;
    G.dropped = 0;
    const bool inside = x < P.width && y < P.height;
    const uint32_t pixel = inside ? y * P.width + x : 0u;
    float3 w = f3(0.0f, 0.0f, 0.0f);
    if (inside) {
        const float4 d = A.dl_dimage[pixel];
        w = f3(d.x, d.y, d.z) * A.inv_samples;
    }
    const bool busy = w.x != 0.0f || w.y != 0.0f || w.z != 0.0f;
    const unsigned lanes = __ballot_sync(0xffffffffu, busy);
    const Cull cull = camera_cull<false>(P, blockIdx.y * gridDim.x + blockIdx.x);
    if (busy) {
        const uint32_t z = P.s.counts[2];
        const uint32_t pixels = P.width * P.height;
#pragma unroll 1
        for (uint32_t smp = 0; smp < z; ++smp) {
            // With the forward's checkpoints, a sample that has them (and no
            // binding cap) replays only up to its first one; the segment
            // kernel replays the rest.
            uint32_t segment_end = 0;
            if (A.ck.totals && A.ck.sample_base + smp < A.ck.samples) {
                const float4 t = A.ck.totals[(size_t)(A.ck.sample_base + smp) * pixels + pixel];
                if ((__float_as_uint(t.w) & 3u) == 1u) {
                    segment_setup(G, w, f3(t.x, t.y, t.z), f3(0.0f, 0.0f, 0.0f));
                    segment_end = A.ck.every;
                }
            }
            if (!segment_end) pass1_setup(G, w);
            adjoint_sample(S, K, G, w, pixel, x, y, smp, lanes, segment_end, cull);
        }
    }
    // Per-thread colour sums: reduce over the warp, then into the window.
#pragma unroll
    for (uint32_t k = 0; k < 6u * kColorSlots; ++k) {
        float v = own[k];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
        if (lane == 0u && v != 0.0f) {
            if (k < A.color_window) atomicAdd(window + A.tau_window + k, v);
            else atomicAdd(A.grad + kGradColor + k, v);
        }
    }
    __syncthreads();
    for (uint32_t k = threadIdx.x; k < window_n; k += blockDim.x) {
        const float v = window[k];
        if (v != 0.0f) atomicAdd(A.grad + (k < A.tau_window ? k : kGradColor + (k - A.tau_window)), v);
    }
    unsigned long long dropped = G.dropped;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) dropped += __shfl_down_sync(0xffffffffu, dropped, o);
    if (lane == 0u && dropped != 0ull && A.overflow) atomicAdd(A.overflow, dropped);
}

// The segments between vertex checkpoints: one thread per record of the
// forward (Checkpoints), replaying from the stored state with the weights of
// the path's known total until the next checkpoint depth or the path's end.
// Gradient sinks as in adjoint_kernel.
template <bool L, bool F>
__global__ void __launch_bounds__(kThreads, SG_ADJOINT_MIN_BLOCKS)
    segment_kernel(const __grid_constant__ TraceParams P, const __grid_constant__ AdjointParams A, uint32_t records) {
    extern __shared__ float4 smem[];
    const uint32_t n_bodies = P.s.counts[0];
    float4 *inv = smem + trace_smem_floats(P) / 4u;
    float *window = reinterpret_cast<float *>(inv + 2u * n_bodies);
    const uint32_t window_n = A.tau_window + A.color_window;
    for (uint32_t k = threadIdx.x; k < window_n; k += blockDim.x) window[k] = 0.0f;
    for (uint32_t k = threadIdx.x; k < n_bodies; k += blockDim.x) {
        const float4 m = P.bodies[k * kBodyVec4 + kMaterial], r = P.bodies[k * kBodyVec4 + kRingColor];
        inv[2u * k] = make_float4(inv_or_zero(m.x), inv_or_zero(m.y), inv_or_zero(m.z), 0.0f);
        inv[2u * k + 1u] = make_float4(inv_or_zero(r.x), inv_or_zero(r.y), inv_or_zero(r.z), 0.0f);
    }
    const Scene S = stage_scene(P, smem);  // synchronises the block
    const Counter<false, L, F> K{nullptr};
    const uint32_t lane = threadIdx.x & 31u;
    float own[6u * kColorSlots];
#pragma unroll
    for (uint32_t k = 0; k < 6u * kColorSlots; ++k) own[k] = 0.0f;
    const uint32_t own_n = 6u * (n_bodies < kColorSlots ? n_bodies : kColorSlots);
    PrbLists lists;
    float4 local[kMaxLocal];
    Prb G;
    G.lists = &lists;
    G.local = local;
    G.local_stride = 1u;
    G.sink = GradSink{own, own_n, window, A.tau_window, window + A.tau_window, A.color_window, A.grad, 1u};
    G.inv = inv;
    G.dropped = 0;
    const uint32_t pixels = P.width * P.height;
#pragma unroll 1
    for (uint32_t r = blockIdx.x * blockDim.x + threadIdx.x; r < records; r += gridDim.x * blockDim.x) {
        Path path;
        const uint3 key = load_checkpoint(A.ck, r, path);  // (pixel, sample, depth)
        path.backdrop = f3(0.0f, 0.0f, 0.0f);
        path.sample = 0u;
        const float4 t = A.ck.totals[(size_t)key.y * pixels + key.x];
        if (__float_as_uint(t.w) & 2u) continue;  // replayed from its seed
        const float4 d = A.dl_dimage[key.x];
        const float3 w = f3(d.x, d.y, d.z) * A.inv_samples;
        if (w.x == 0.0f && w.y == 0.0f && w.z == 0.0f) continue;
        segment_setup(G, w, f3(t.x, t.y, t.z), path.radiance);
        const uint32_t next = key.z + A.ck.every;
        replay_segment(S, K, G, path, next <= A.ck.max_depth ? next : 0xffffffffu);
    }
#pragma unroll
    for (uint32_t k = 0; k < 6u * kColorSlots; ++k) {
        float v = own[k];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
        if (lane == 0u && v != 0.0f) {
            if (k < A.color_window) atomicAdd(window + A.tau_window + k, v);
            else atomicAdd(A.grad + kGradColor + k, v);
        }
    }
    __syncthreads();
    for (uint32_t k = threadIdx.x; k < window_n; k += blockDim.x) {
        const float v = window[k];
        if (v != 0.0f) atomicAdd(A.grad + (k < A.tau_window ? k : kGradColor + (k - A.tau_window)), v);
    }
    unsigned long long dropped = G.dropped;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) dropped += __shfl_down_sync(0xffffffffu, dropped, o);
    if (lane == 0u && dropped != 0ull && A.overflow) atomicAdd(A.overflow, dropped);
}

}  // namespace

template <bool L, bool F>
PixelKernels pixel_kernels() {
    return PixelKernels{{(const void *)trace_kernel<false, L, F, false>, (const void *)trace_kernel<false, L, F, true>},
                        (const void *)trace_kernel<true, L, F, true>,
                        (const void *)adjoint_kernel<L, F>,
                        (const void *)segment_kernel<L, F>};
}
template PixelKernels pixel_kernels<SG_STAGE_L, SG_STAGE_F>();

}  // namespace sg
