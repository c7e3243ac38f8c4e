// sg_wave_adjoint.cu — the staged adjoint's host side: buffers and the stage
// loop over the kernels of sg_wave_adjoint_stages.cu.
#include <algorithm>

#include "sg_wave_common.cuh"

namespace sg {

namespace {

// When the rest of the replay runs in adj_finish. On a landscape, and where that
// holds for all samples after the first iteration: once every sample is out and
// at most kFinishPaths paths are left, which the GPU itself decides (finishes()).
// In celestial frames such paths are mostly second replays with most of their
// length to go, and the finish kernel, divergent, is slower with tens of
// thousands of them than the stages: there it waits until the host has seen an
// iteration start with at most kSeenPaths, and one more has run. Backward alone,
// eight bounces, us; ring scene: 333x217, 7 samples, 909 (1017 when the GPU decided
// at 2^16), 1024x1024, 2 samples, 1479 (2110), 512x512, 16 samples, 2154 (2792), 64
// samples, 5692 (5756); with two bounces, whose replays are short, 512x512, 4
// samples, 759 (720). Terrain, 512x512, 4 samples: 1519 as it is, 1614 by the host.
constexpr uint32_t kFinishPaths = 1u << 16;
constexpr uint32_t kSeenPaths = 1u << 17;

}  // namespace

size_t adjoint_slot_bytes(uint32_t pool) {
    return (size_t)pool * (kAdjointSideVec4 * sizeof(float4) + 2u * sizeof(uint4) + sizeof(PrbLists)) +
           (size_t)pool * sizeof(uint32_t) + 4 * sizeof(uint32_t);
}

cudaError_t launch_adjoint_wavefront(const TraceParams &params, const AdjointParams &adjoint, WaveParams w,
                                     const AdjointWave &slots, WaveProgress &progress, cudaStream_t stream,
                                     WaveRun *run) {
    TraceParams p = params;
    AdjointParams a = adjoint;
    AdjointWave x = slots;
    *run = WaveRun{};
    const uint32_t z = p.s.counts[2];
    if (z == 0 || p.width == 0 || p.height == 0) return cudaSuccess;
    const bool land = p.s.g.ground_north[3] != 0.0f;
    const WaveStages set = land ? (p.fp64_sites ? adjoint_stages<true, true>() : adjoint_stages<true, false>())
                                : (p.fp64_sites ? adjoint_stages<false, true>() : adjoint_stages<false, false>());
    const void *fns[4] = {set.extend, set.ring, set.surface, set.finish};
    // After the adjoint's shared memory: the per-thread colour sums, and in
    // the shade stages the pending-factor lists (16-byte aligned).
    const size_t smem[2] = {
        adjoint_smem_bytes(p, a) + (size_t)6u * kColorSlots * kThreads * sizeof(float),
        adjoint_smem_bytes(p, a) + 16u + (size_t)6u * kColorSlots * kShadeThreads * sizeof(float) +
            (size_t)kMaxLocal * kShadeThreads * sizeof(float4)};
    int grid[4];
    for (int k = 0; k < 4; ++k) {
        const size_t bytes = smem[k == 0 ? 0 : 1];
        if (bytes > 48u * 1024u) {
            cudaError_t e = cudaFuncSetAttribute(fns[k], cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
            if (e != cudaSuccess) return e;
        }
        cudaError_t e = persistent_grid(fns[k], bytes, &grid[k], k == 0 ? kThreads : kShadeThreads);
        if (e != cudaSuccess) return e;
    }
    w.tiles_x = (p.width + kTile - 1) / kTile;
    w.tiles_y = (p.height + kTile - 1) / kTile;
    w.chunk_first = 0;
    w.chunk_samples = z;
    const uint32_t samples = w.tiles_x * w.tiles_y * 256u * z;
    // A sample replays at most twice, each replay ending within the
    // iteration bound; see launch_wavefront for the host-side guard.
    const uint64_t cap = 2ull * ((uint64_t)p.s.counts[3] * (p.s.counts[0] + 2u) + 2u);
    const uint64_t bound = ((uint64_t)samples + 1u) * cap;
    // A tile whose camera rays meet nothing has no gradient.
    w.skip_empty = !land;
    const bool whole = samples <= kFinishPaths && samples <= w.pool;
    const bool device_decides = land || whole;
    w.finish_paths = device_decides ? kFinishPaths : 0u;
    cudaError_t e = cull_tiles(p, w, stream, run, false);
    if (e != cudaSuccess) return e;
    // Every slot is free (both counters zero: allocation j < pool takes slot
    // j); the finish kernel of an earlier launch gave none of its slots back.
    if ((e = cudaMemsetAsync(x.free_ends, 0, 2 * sizeof(uint32_t), stream)) != cudaSuccess) return e;
    // The finish kernel for the paths live at the start of iteration t, if they
    // are at most `limit`.
    auto finish = [&](uint32_t t, uint32_t limit, uint32_t most) -> cudaError_t {
        WaveParams taken = w;
        taken.finish_paths = limit;
        void *args[] = {&p, &a, &taken, &x, &t};
        const uint32_t blocks = std::min<uint32_t>(grid[3], (std::min(most, samples) + kShadeThreads - 1) / kShadeThreads);
        run->kernels += 1;
        return cudaLaunchKernel(set.finish, dim3(blocks), dim3(kShadeThreads), args, smem[1], stream);
    };
    uint64_t out_by = 0;  // as in launch_wavefront
    for (uint64_t t = 0;; ++t) {
        if (t >= bound) return cudaErrorLaunchTimeout;
        uint32_t it = (uint32_t)t;
        void *args[] = {&p, &a, &w, &x, &it};
        for (int k = 0; k < 3; ++k) {
            e = cudaLaunchKernel(fns[k], dim3(grid[k]), dim3(k == 0 ? kThreads : kShadeThreads), args,
                                 smem[k == 0 ? 0 : 1], stream);
            if (e != cudaSuccess) return e;
        }
        run->kernels += 3;
        run->iterations += 1;
        if (device_decides && t >= out_by && (e = finish(it + 1u, kFinishPaths, kFinishPaths)) != cudaSuccess) return e;
        if (whole) break;
        if ((e = iteration_done(progress, t, stream)) != cudaSuccess) return e;
        if (t < kLookahead) continue;
        WaveStart start;
        if ((e = started(progress, t - kLookahead, &start)) != cudaSuccess) return e;
        if (start.kept == 0u && start.left == 0u) break;
        if (!device_decides && start.left == 0u && start.kept <= kSeenPaths) {
            // Every sample is out, and no later iteration holds more paths.
            if ((e = finish(it + 1u, samples, start.kept)) != cudaSuccess) return e;
            break;
        }
        out_by = start.left > 0u ? t - kLookahead + (start.left - 1u) / w.pool : 0u;
    }
    return cudaSuccess;
}

}  // namespace sg
