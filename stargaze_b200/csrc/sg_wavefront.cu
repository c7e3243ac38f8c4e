// sg_wavefront.cu — the integrator in wavefront form.
//
// The per-pixel megakernel (sg_kernels.cu) keeps a whole path in registers
// and walks it to the end, so a warp's lanes idle while the longest path of
// the 32 finishes and every lane drags the code of every vertex kind
// through the instruction cache. Here a dispatch's samples become paths in
// a pool whose state lives in HBM (seven float4 planes per path, read and
// written as 16-byte vectors, consecutive paths in consecutive slots), and
// each iteration runs three small kernels over it:
//
//   extend    tops the pool up with new camera paths (16x16 pixel tiles,
//             8x4 per warp, as the megakernel orders its lanes), then finds
//             the closest hit, point disc and ring crossing of every live
//             path; splits the paths into a ring queue and a surface queue
//             and finishes those that escaped;
//   ring      ring events (next-event estimation through the slab, null or
//             scatter), for the ring queue only;
//   surface   emitter hits and surface vertices (next-event estimation,
//             ringshine, cosine bounce), for the surface queue only.
//
// The shade stages append surviving paths, compacted, to the other state
// buffer. Queues are appended with one atomic per CTA and round (warp
// ballots, then a CTA prefix), so the order within a CTA is the order of
// its input. A new camera path is built in registers and stored only if it
// survives its first extend. Finished paths write their radiance to a
// per-(sample, pixel) slot; resolve sums each pixel's samples in sample
// order and folds them into the compensated accumulation exactly as the
// megakernel does. Both integrators run the same per-path functions
// (sg_integrator.cuh) on the same random sequences; they differ only where
// the compiler fuses a shading multiply-add in one kernel and not in the
// other, a few ulps. Once few paths are left, finish runs each to its end in
// its own thread; the GPU itself decides when (finishes()). The stage kernels
// are in sg_wave_stages.cu.
#include <algorithm>

#include "sg_wave_common.cuh"

namespace sg {

namespace {

// Per pixel: the chunk's samples summed in sample order onto the running
// total, and on the last chunk the megakernel's compensated fold.
__global__ void __launch_bounds__(kThreads) wave_resolve(const __grid_constant__ TraceParams P,
                                                         const __grid_constant__ WaveParams W, int first, int last) {
    const uint32_t pixels = P.width * P.height;
    const uint32_t pixel = blockIdx.x * kThreads + threadIdx.x;
    await_previous();
    if (pixel >= pixels) return;
    float4 total = first ? make_float4(0.0f, 0.0f, 0.0f, 0.0f) : W.totals[pixel];
    // The samples of a tile that is not traced are zero.
    uint32_t samples = W.chunk_samples;
    if (W.skip_empty) {
        const uint2 m = P.camera_cull[(pixel / P.width / kTile) * W.tiles_x + pixel % P.width / kTile];
        if ((m.x | m.y) == 0u) samples = 0u;
    }
    for (uint32_t smp = 0; smp < samples; ++smp) {
        const float4 r = W.results[(size_t)smp * pixels + pixel];
        total.x += r.x;
        total.y += r.y;
        total.z += r.z;
        total.w += r.w;
    }
    if (W.sky_results) {
        float3 sky = first ? f3(0.0f, 0.0f, 0.0f) : xyz4(W.sky_totals[pixel]);
        for (uint32_t smp = 0; smp < W.chunk_samples; ++smp) sky = sky + xyz4(W.sky_results[(size_t)smp * pixels + pixel]);
        if (last) fold_backdrop(P, pixel, sky);
        else W.sky_totals[pixel] = pack3(sky, 0.0f);
    }
    if (!last) {
        W.totals[pixel] = total;
        return;
    }
    const uint32_t old_count = P.s.counts[1];
    const float new_count = (float)(old_count + P.s.counts[2]);
    float4 sum, comp;
    if (old_count == 0u) {
        sum = total;
        comp = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    } else {
        sum = P.sum[pixel];
        comp = P.comp[pixel];
        float yv, tt;
        yv = __fsub_rn(total.x, comp.x); tt = __fadd_rn(sum.x, yv); comp.x = __fsub_rn(__fsub_rn(tt, sum.x), yv); sum.x = tt;
        yv = __fsub_rn(total.y, comp.y); tt = __fadd_rn(sum.y, yv); comp.y = __fsub_rn(__fsub_rn(tt, sum.y), yv); sum.y = tt;
        yv = __fsub_rn(total.z, comp.z); tt = __fadd_rn(sum.z, yv); comp.z = __fsub_rn(__fsub_rn(tt, sum.z), yv); sum.z = tt;
        yv = __fsub_rn(total.w, comp.w); tt = __fadd_rn(sum.w, yv); comp.w = __fsub_rn(__fsub_rn(tt, sum.w), yv); sum.w = tt;
    }
    P.sum[pixel] = sum;
    P.comp[pixel] = comp;
    P.mean[pixel] = make_float4(__fdiv_rn(__fsub_rn(sum.x, comp.x), new_count),
                                __fdiv_rn(__fsub_rn(sum.y, comp.y), new_count),
                                __fdiv_rn(__fsub_rn(sum.z, comp.z), new_count),
                                __fdiv_rn(__fsub_rn(sum.w, comp.w), new_count));
}

// ---------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------
// Live paths at or below which, once every sample of the chunk is out, the
// rest of the chunk runs in wave_finish (1080p ring dispatch: 2^17 and 2^18
// measured alike, 2^19 and 2^20 0.5 % slower).
constexpr uint32_t kFinishPaths = 1u << 17;
// Samples of a chunk up to which the host enqueues a fixed number of
// iterations and the finish kernel for every path left: one iteration up to
// kSingleSamples, else two. How many paths that leaves depends on the view, which
// the host does not know, so the rule has to hold where every camera ray meets
// something, too. Celestial frames with rings or procedural surfaces keep more
// and dearer paths: there one iteration only up to kSingleLongTails, and with
// surfaces a third one above kTwoStyled, which finds nothing where the paths after
// the second were at most kFewPaths: the finish kernel has taken them then. (Plain
// rings go without: it would cost every wide view 8 us.) Above kDirectSamples the
// host asks.
// Eight bounces, us, the host loop | one iteration | two | three ("narrow": a
// tenth to a third of the field, where most rays meet something):
//                              2^18 samples          2^19             2^22
//   three spheres                    -        120 |  57 |  89    274 | - |  243
//   rings                      - | 166 | 172  240 | 262 | 208    735 | - |  679 |  693
//   rings, narrow              - | 235 | 198  311 | 443 | 279   1388 | - | 1579 | 1370
//   styled rings               - | 460 | 444  601 | 715 | 569   2264 | - | 2096 | 2107
//   styled rings, narrow       - | 485 | 550  765 | 813 | 730   2931 | - | 3389 | 2968
//   terrain                          -        618 | 476 | 497   2299 | - | 2213
//   terrain, narrow                  -        706 | 663 | 595   2717 | - | 2629
constexpr uint32_t kDirectSamples = 1u << 22;
constexpr uint32_t kSingleSamples = 1u << 19;
constexpr uint32_t kSingleLongTails = 1u << 18;
constexpr uint32_t kTwoStyled = 1u << 21;
constexpr uint32_t kFewPaths = 1u << 18;

cudaError_t run_iteration(const WaveStages &stages, TraceParams &p, WaveParams &w, uint32_t t, const int (&grid)[4],
                          const int (&threads)[4], size_t smem, cudaStream_t stream, StageMarks *m, bool overlap) {
    void *args[] = {&p, &w, &t};
    const void *fns[3] = {stages.extend, stages.ring, stages.surface};
    const int names[3] = {kStageExtend, kStageRing, kStageSurface};
    cudaError_t e;
    for (int k = 0; k < 3; ++k) {
        if ((e = mark(m, names[k], stream)) != cudaSuccess) return e;
        if ((e = launch_stage(fns[k], grid[k], threads[k], args, smem, stream, overlap)) != cudaSuccess) return e;
    }
    return mark(m, kStageGap, stream);
}

}  // namespace

size_t wave_state_bytes(uint32_t pool) {
    return (size_t)pool * sizeof(float4) * (2 * kWavePlanes + kWaveHitPlanes) + (size_t)pool * 2 * sizeof(uint32_t) +
           (kWaveCounterSets + 1u) * sizeof(WaveCounters);
}

size_t wave_result_bytes(uint32_t pixels, uint32_t chunk_samples) {
    return (size_t)pixels * sizeof(float4) * ((size_t)chunk_samples + 1u);
}

cudaError_t launch_wavefront(const TraceParams &params, WaveParams w, WaveProgress &progress, cudaStream_t stream,
                             WaveRun *run, StageMarks *marks) {
    TraceParams p = params;
    const uint32_t z = p.s.counts[2];
    const uint32_t pixels = p.width * p.height;
    *run = WaveRun{};
    if (marks) marks->used = 0;
    if (z == 0 || pixels == 0) return cudaSuccess;
    const bool land = p.s.g.ground_north[3] != 0.0f;
    // Checkpoints are stored for the frames the adjoint differentiates
    // (no air, no styles): variants 8-11.
    const bool ck = w.ck.records != nullptr;
    if (ck && (p.air_on || p.styled)) return cudaErrorInvalidValue;
    const bool air = p.air_on || p.styled;
    const WaveStages set = land ? (p.fp64_sites ? wave_stages<true, true>(air, ck) : wave_stages<true, false>(air, ck))
                                : (p.fp64_sites ? wave_stages<false, true>(air, ck) : wave_stages<false, false>(air, ck));
    const size_t smem = trace_smem_bytes(p);
    const void *fns[4] = {set.extend, set.ring, set.surface, set.finish};
    int grid[4] = {0, 0, 0, 0};
    const int threads[4] = {extend_threads(land, air), shade_threads(land, true), shade_threads(land, false), kThreads};
    for (int k = 0; k < 4; ++k) {
        if (!fns[k]) continue;
        const size_t bytes = smem;
        if (bytes > 48u * 1024u) {
            cudaError_t e = cudaFuncSetAttribute(fns[k], cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
            if (e != cudaSuccess) return e;
        }
        cudaError_t e = persistent_grid(fns[k], bytes, &grid[k], threads[k]);
        if (e != cudaSuccess) return e;
    }
    w.tiles_x = (p.width + kTile - 1) / kTile;
    w.tiles_y = (p.height + kTile - 1) / kTile;
    const uint32_t chunk = w.chunk_samples;
    const uint32_t per_sample = w.tiles_x * w.tiles_y * 256u;
    // A tile whose camera rays meet no body and no ring needs no paths where a
    // ray that escapes leaves nothing: no landscape, air, sky or stored totals.
    w.skip_empty = !land && !air && !p.sky_on && !w.ck.totals;
    // A chunk that does not fit the pool takes its tiles in a fixed order, so
    // that the same samples share its iterations (and their tails the finish
    // kernel) in every run.
    const bool ordered = (uint64_t)per_sample * std::min(chunk, z) > w.pool;
    if (cudaError_t e = cull_tiles(p, w, stream, run, ordered); e != cudaSuccess) return e;
    // A path ends within max_vertices * (bodies + 2) + 1 iterations, and an
    // iteration that takes no new sample has a full pool of paths that all
    // advance, so a chunk drains within (samples + 1) * (that + 1)
    // iterations: a host-side guard.
    const uint64_t cap = (uint64_t)p.s.counts[3] * (p.s.counts[0] + 2u) + 2u;
    for (uint32_t first = 0; first < z; first += chunk) {
        w.chunk_first = first;
        w.chunk_samples = std::min(chunk, z - first);
        const uint32_t samples = per_sample * w.chunk_samples;
        const uint64_t bound = ((uint64_t)samples + 1u) * cap;
        // (The first chunk's were cleared with the active-tile count.)
        cudaError_t e = cudaSuccess;
        if (first > 0u) e = cudaMemsetAsync(w.counters, 0, kWaveCounterSets * sizeof(WaveCounters), stream);
        if (e != cudaSuccess) return e;
        // A chunk that fits the pool has taken all its samples after one
        // iteration. Up to kDirectSamples of them, the host then asks nothing:
        // it enqueues one to three iterations and the finish kernel for whatever
        // paths are left. The finish and resolve kernels, and the stages of a
        // single iteration or a third, overlap their start with their predecessor's end:
        // 256x256 spheres, 1 sample, 52.2 -> 42.6 us, rings 124 -> 117 us. The
        // stages of larger dispatches lose by it (1001x563 rings, 7 samples,
        // 486 -> 506 us).
        const bool direct = set.finish && samples <= w.pool && samples <= kDirectSamples;
        const uint32_t single = w.long_tails && !land ? kSingleLongTails : kSingleSamples;
        const bool third = p.styled && !land && samples > kTwoStyled;
        const uint64_t direct_iterations = samples <= single ? 1u : third ? 3u : 2u;
        w.finish_paths = direct || !set.finish ? 0u : kFinishPaths;
        // Otherwise the host reads the start of iteration t - kLookahead while
        // the GPU runs the later ones; once one started empty the chunk has
        // drained (the iterations after it are empty launches). The finish
        // kernel follows every iteration that may have been the last to take
        // samples: the GPU itself decides whether few enough paths are left
        // (finishes()), so the tail does not wait for the host.
        uint64_t out_by = 0;  // the first iteration after which no sample may be left
        for (uint64_t t = 0;; ++t) {
            if (t >= bound) return cudaErrorLaunchTimeout;
            uint32_t it = (uint32_t)t;
            if (direct) w.finish_paths = t == 2u ? kFewPaths : 0u;  // what finish was given before iteration t
            e = run_iteration(set, p, w, it, grid, threads, smem, stream, marks,
                              direct && (direct_iterations == 1u || t == 2u));
            if (e != cudaSuccess) return e;
            run->kernels += 3;
            run->iterations += 1;
            const bool last = direct && t + 1u == direct_iterations;
            const bool few = direct && !last && t == 1u;
            if (last || few || (!direct && w.finish_paths > 0u && t >= out_by)) {
                if ((e = mark(marks, kStageFinish, stream)) != cudaSuccess) return e;
                uint32_t next_t = it + 1u, limit = last ? samples : few ? kFewPaths : w.finish_paths;
                void *args[] = {&p, &w, &next_t, &limit};
                const uint32_t blocks = std::min<uint32_t>(grid[3], (std::min(limit, samples) + kThreads - 1) / kThreads);
                e = launch_stage(set.finish, blocks, kThreads, args, smem, stream, true);
                if (e != cudaSuccess) return e;
                if ((e = mark(marks, kStageGap, stream)) != cudaSuccess) return e;
                run->kernels += 1;
            }
            if (last) break;
            if (direct) continue;
            if ((e = iteration_done(progress, t, stream)) != cudaSuccess) return e;
            if (t < kLookahead) continue;
            WaveStart start;
            if ((e = started(progress, t - kLookahead, &start)) != cudaSuccess) return e;
            if (start.kept == 0u && start.left == 0u) break;
            out_by = start.left > 0u ? t - kLookahead + (start.left - 1u) / w.pool : 0u;
        }
        const bool first_chunk = first == 0, last_chunk = first + w.chunk_samples >= z;
        if ((e = mark(marks, kStageResolve, stream)) != cudaSuccess) return e;
        int first_arg = first_chunk, last_arg = last_chunk;
        void *args[] = {&p, &w, &first_arg, &last_arg};
        e = launch_stage((const void *)wave_resolve, (pixels + kThreads - 1) / kThreads, kThreads, args, 0, stream, true);
        if (e != cudaSuccess) return e;
        if ((e = mark(marks, kStageGap, stream)) != cudaSuccess) return e;
        e = cudaGetLastError();
        if (e != cudaSuccess) return e;
        run->kernels += 1;
    }
    return cudaSuccess;
}

}  // namespace sg
