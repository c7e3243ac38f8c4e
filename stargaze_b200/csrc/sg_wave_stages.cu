// sg_wave_stages.cu — the wavefront integrator's stage kernels
// (sg_wavefront.cu drives them). Compiled once per landscape and FP64-sites
// variant (SG_STAGE_L, SG_STAGE_F: 0 or 1), so that the variants build in
// parallel.
// The stage kernels are small enough to inline the multi-site helpers and
// the derivative hooks that the per-pixel kernels keep out of line for
// their instruction footprint (measured on the ring workload: forward 6 %,
// adjoint 14 % faster inlined).
#define SG_HELPER __forceinline__
#define SG_ADJ_HOOK __forceinline__

#include "sg_wave_common.cuh"

namespace sg {

namespace {

// ---------------------------------------------------------------------------
// Stages
// ---------------------------------------------------------------------------
// A: the host air's code and the surface styles are compiled in (frames
// with air or styled bodies run these).
//
// Landscape frames under air are bound by instruction fetch (the query and the
// air march are far larger than the instruction caches): their CTAs are of 512
// threads and pass through the parts of an extend together. 640x360, 16
// samples: 256 threads 6.74 ms, the same with the barriers 6.02, 512 with them
// 5.76; 1024 without 5.83, with 6.00. The airless landscape, whose parts are
// smaller and whose paths then live across the barriers, measured slower with
// them (1080p, 32 samples: 47.6 against 49.2 ms) and with larger CTAs (48.5,
// 50.5), and with smaller ones or warps that append by themselves (49.7, 53.7).
template <bool L, bool F, bool A>
__global__ void __launch_bounds__(extend_threads(L, A), extend_blocks(L, A))
    wave_extend(const __grid_constant__ TraceParams P, const __grid_constant__ WaveParams W, uint32_t t) {
    extern __shared__ float4 smem[];
    constexpr int kB = extend_threads(L, A);
    // Celestial frames take several paths per append (their work per path
    // is even; SG_WAVE_EXTEND_ITEMS); landscape frames one, so that a CTA's
    // last round is small when traversal costs differ (measured with four:
    // rings 59.5 -> 56.5 ms per step, terrain 455 -> 531 ms). Landscape frames keep the append
    // barrier although their quadtree walks differ in length: writing a
    // per-path kind instead and building the queues in a kernel of their
    // own let the warps of a CTA drift apart, and the terrain step went
    // from 450 to 513 ms (the barrier keeps neighbouring pixels' walks
    // through the same quadtree nodes at the same time, in L1).
    constexpr uint32_t kItems = L ? 1u : SG_WAVE_EXTEND_ITEMS;
    __shared__ AppendK<2, kItems, kB> sm[2];
    const Scene S = stage_scene(P, smem);
    await_previous();
    WaveCounters *c = counters(W, t);
    // Paths the previous iteration kept occupy [0, kept); new samples of the
    // chunk fill the pool up to n.
    const uint32_t next = c->next, per_sample = padded_pixels(W);
    const uint32_t kept = finishes(W, c, per_sample, W.finish_paths) ? 0u : c->cont;
    const uint32_t left = per_sample * W.chunk_samples - next;
    const uint32_t take = min(W.pool - kept, left);
    const uint32_t n = kept + take;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        counters(W, t + 1u)->next = next + take;
        *counters(W, t + 2u) = WaveCounters{};
        W.progress[t % kProgressSlots] = make_uint2(kept, left);
    }
    if (blockIdx.x * kB * kItems >= n) return;
    const Counter<false, L, F> K{nullptr};
    Forward<A> nograd;
    float4 *st = W.state[t & 1u];
    float4 *H = W.hits;
    uint32_t round = 0;
    // Each round a thread extends kItems paths (i = base + k * kB +
    // threadIdx.x), then the CTA appends them to the queues at once.
    for (uint32_t base = blockIdx.x * kB * kItems; base < n; base += gridDim.x * kB * kItems, ++round) {
      uint32_t ring_bits = 0, surface_bits = 0;
#pragma unroll 1
      for (uint32_t item = 0; item < kItems; ++item) {
        const uint32_t i = base + item * kB + threadIdx.x;
        bool ring = false, surface = false;
        Path p;
        uint32_t slot = 0;
        const bool fresh = i >= kept;
        bool valid = i < n, was_in_air = false;
        Cull cull = kTestAll;
        if (valid) {
            if (fresh) {
                // Sample k of the chunk, numbered sample-major over the
                // padded tile grid; padding pixels are skipped.
                const uint32_t k = next + (i - kept);
                const uint32_t smp = k / per_sample;
                const uint32_t q = k - smp * per_sample;
                const uint32_t tile = camera_tile(W, q >> 8), within = q & 255u;
                const uint32_t warp = within >> 5, lane = within & 31u;
                const uint32_t x = (tile % W.tiles_x) * kTile + (warp & 1u) * 8u + (lane & 7u);
                const uint32_t y = (tile / W.tiles_x) * kTile + (warp >> 1) * 4u + (lane >> 3);
                valid = x < P.width && y < P.height;
                if (valid) {
                    const uint32_t pixel = y * P.width + x;
                    start_path(p, &P.s, K, pixel, x, y, W.chunk_first + smp);
                    slot = smp * P.width * P.height + pixel;
                    cull = camera_cull<false>(P, tile);
                }
            } else {
                slot = load_ray_part(st, W.pool, i, p);
            }
            // A continuation leaving the host air may be attenuated in
            // extend: it needs its throughput.
            was_in_air = A && !fresh && p.in_air;
            if (was_in_air) {
                const float4 c = st[2 * W.pool + i];
                p.throughput = xyz4(c);
                p.previous_pdf = c.w;
            }
        }
        Extension e;
        bool alive = false;
        if constexpr (L && A) {
            // A landscape under air: the bodies and the host sphere, the
            // terrain, the primitives, then the air march, each by the whole
            // CTA at a time.
            LandQuery land;
            land.open = false;
            if (valid) alive = extend_begin(S, K, p, nograd);
            if (alive) {
                e.hit = closest_body(S, K, p.ray, cull);
                land = landscape_begin(S, K, p.ray, 1.0e30f, false);
            }
            __syncthreads();
            if (land.open) landscape_terrain(S, K, land, false);
            __syncthreads();
            if (land.open) land.closest = landscape_props(S, K, land, false);
            __syncthreads();
            if (alive) {
                if (land.closest.t < e.hit.t)
                    e.hit = Hit{land.closest.t, land.closest.index, land.closest.delta, land.closest.n};
                extend_rest(S, K, p, nograd, e, cull);
            }
        } else {
            if (valid) alive = extend(S, K, p, nograd, e, cull);
        }
        if (valid) {
            ring = alive && e.ring.index != kMiss;
            surface = alive && !ring && e.hit.index != kMiss;
            if (ring || surface) {
                if (fresh) {
                    store_path(st, W.pool, i, p, slot);
                } else {
                    st[1 * W.pool + i] = pack3u(p.ray.d, p.rng);
                    st[6 * W.pool + i] = make_float4(iteration_word(p), depth_word(p), __uint_as_float(slot),
                                                     __uint_as_float(p.ckpt));
                    if (was_in_air) st[2 * W.pool + i] = pack3(p.throughput, p.previous_pdf);
                }
                if (ring) H[1 * W.pool + i] = pack3(e.ring.p, e.ring.t);
                else H[0 * W.pool + i] = pack3(e.hit.n, e.hit.t);
                H[2 * W.pool + i] = make_float4(__uint_as_float(e.hit.index), __uint_as_float(e.ring.index),
                                                e.hit.delta, e.disc_scale);
            } else {
                // Ended at the iteration bound, or escaped (then the sky
                // backdrop of an unscattered camera path, as
                // surface_vertex's miss). A new path's radiance is still
                // zero.
                if (!fresh) load_radiance_part(st, W.pool, i, p);
                if (alive && (P.sky_on || (A && p.sky_on_escape))) {
                    if (!fresh && !was_in_air) p.throughput = xyz4(st[2 * W.pool + i]);
                    // A sky-lit local surface's continuation sees the
                    // surface sky cache (pathtrace.wgsl:1497-1499).
                    if (A && p.sky_on_escape)
                        p.radiance = p.radiance + p.throughput * surface_sky_lookup(S, p.ray.d);
                    sky_miss(S, p);
                }
                W.results[slot] = finish_path(p);
                if (W.sky_results) W.sky_results[slot] = pack3(p.backdrop, 0.0f);
                if (W.ck.totals) checkpoint_total(W.ck, W.chunk_first, P.width * P.height, slot, p);
            }
        }
        ring_bits |= (ring ? 1u : 0u) << item;
        surface_bits |= (surface ? 1u : 0u) << item;
      }
      const uint32_t flags[2] = {ring_bits, surface_bits};
      uint32_t *const ctr[2] = {&c->ring, &c->surface};
      uint32_t q[2][kItems];
      block_append_k<2, kItems, kB>(sm[round & 1u], flags, ctr, q);
#pragma unroll
      for (uint32_t item = 0; item < kItems; ++item) {
        const uint32_t i = base + item * kB + threadIdx.x;
        if ((ring_bits >> item) & 1u) W.ring_queue[q[0][item]] = i;
        if ((surface_bits >> item) & 1u) W.surface_queue[q[1][item]] = i;
      }
    }
}

// Ring (R == true) or surface stage over its queue. CK: the forward stores
// vertex checkpoints (W.ck). The ring stage runs at 3 CTAs per SM (85
// registers, fewer spills: 13.07 → 12.81 ms per 1080p ring step; 2 CTAs
// measured 13.57), the surface stage at 4 (3 measured slower). On a landscape
// the surface stage, bound by instruction fetch, runs in CTAs of 512 threads:
// the append's barrier keeps twice as many warps in the same code (1080p, 32
// samples: 14.7 ms with 256 threads, 13.3 with 512, 13.5 with 1024); celestial
// frames, styled ones too, lose by it (styled viewer frame 0.37, 0.42, 0.48).
template <bool L, bool F, bool R, bool A, bool CK = false>
__global__ void __launch_bounds__(shade_threads(L, R), shade_blocks(L, R))
    wave_shade(const __grid_constant__ TraceParams P, const __grid_constant__ WaveParams W, uint32_t t) {
    extern __shared__ float4 smem[];
    constexpr int kB = shade_threads(L, R);
    constexpr int kQueues = CK ? 2 : 1;
    __shared__ Append<kQueues, kB> sm[2];
    const Scene S = stage_scene(P, smem);
    await_previous();
    WaveCounters *c = counters(W, t);
    const uint32_t n = R ? c->ring : c->surface;
    if (blockIdx.x * kB >= n) return;
    const Counter<false, L, F> K{nullptr};
    Stage<A> nograd;
    const float4 *st = W.state[t & 1u];
    float4 *out = W.state[(t + 1u) & 1u];
    const float4 *H = W.hits;
    const uint32_t *queue = R ? W.ring_queue : W.surface_queue;
    uint32_t round = 0;
    for (uint32_t base = blockIdx.x * kB; base < n; base += gridDim.x * kB, ++round) {
        const uint32_t j = base + threadIdx.x;
        bool keep = false, record = false;
        Path p;
        uint32_t slot = 0;
        if (j < n) {
            const uint32_t i = queue[j];
            slot = load_ray_part(st, W.pool, i, p);
            load_radiance_part(st, W.pool, i, p);
            load_shade_part(st, W.pool, i, p);
            const uint32_t depth_before = p.depth;
            const float4 h2 = H[2 * W.pool + i];
            bool ended;
            if constexpr (R) {
                const float4 h1 = H[1 * W.pool + i];
                const RingHit ring{h1.w, __float_as_uint(h2.y), xyz4(h1)};
                ended = ring_vertex(S, K, p, ring, nograd);
            } else {
                const float4 h0 = H[0 * W.pool + i];
                const Hit hit{h0.w, __float_as_uint(h2.x), h2.z, xyz4(h0)};
                ended = surface_vertex(S, K, p, hit, h2.w, nograd);
            }
            keep = !ended;
            if (ended) {
                W.results[slot] = finish_path(p);
                if (W.sky_results) W.sky_results[slot] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                if (W.ck.totals) checkpoint_total(W.ck, W.chunk_first, P.width * P.height, slot, p);
            }
            if constexpr (CK) {
                // A scatter brought the depth to a checkpoint depth.
                record = keep && p.depth != depth_before && p.depth % W.ck.every == 0u && p.depth <= W.ck.max_depth &&
                         checkpoint_sample(W.ck, W.chunk_first, P.width * P.height, slot) < W.ck.samples;
            }
        }
        if constexpr (CK) {
            const bool flags[2] = {keep, record};
            uint32_t *const ctr[2] = {&counters(W, t + 1u)->cont, W.ck.count};
            uint32_t q[2];
            block_append<2, kB>(sm[round & 1u], flags, ctr, q);
            if (record) {
                if (q[1] < W.ck.capacity) {
                    p.ckpt |= 1u;
                    const uint32_t pixels = P.width * P.height;
                    store_checkpoint(W.ck, q[1], p, slot % pixels, checkpoint_sample(W.ck, W.chunk_first, pixels, slot));
                } else {
                    p.ckpt |= 2u;
                }
            }
            if (keep) store_path(out, W.pool, q[0], p, slot);
        } else {
            const bool flags[1] = {keep};
            uint32_t *const ctr[1] = {&counters(W, t + 1u)->cont};
            uint32_t q[1];
            block_append<1, kB>(sm[round & 1u], flags, ctr, q);
            if (keep) store_path(out, W.pool, q[0], p, slot);
        }
    }
}

// The tail of a chunk: once every sample is out and few paths are left,
// stage iterations cost their launches and load chains (about 18 us) for a
// handful of paths each. Here every path live at the start of iteration t runs
// to its end in its own thread through the same per-path functions (step(), as
// the megakernel), and writes its result as the stages would. Unless samples
// are left or more than `limit` paths are live, which the GPU itself decides
// here (and extend of iteration t alike). Its loops are as divergent as the
// megakernel's: above a few hundred thousand paths the stages are faster
// (launch_wavefront has the figures).
template <bool L, bool F, bool A>
__global__ void __launch_bounds__(kThreads, SG_WAVE_SHADE_MIN_BLOCKS) wave_finish(const __grid_constant__ TraceParams P,
                                                                            const __grid_constant__ WaveParams W,
                                                                            uint32_t t, uint32_t limit) {
    extern __shared__ float4 smem[];
    const Scene S = stage_scene(P, smem);
    await_previous();
    if (!finishes(W, counters(W, t), padded_pixels(W), limit)) return;
    const uint32_t n = counters(W, t)->cont;
    if (blockIdx.x * kThreads >= n) return;
    const Counter<false, L, F> K{nullptr};
    Forward<A> nograd;
    const float4 *st = W.state[t & 1u];
#pragma unroll 1
    for (uint32_t i = blockIdx.x * kThreads + threadIdx.x; i < n; i += gridDim.x * kThreads) {
        Path p;
        const uint32_t slot = load_ray_part(st, W.pool, i, p);
        load_radiance_part(st, W.pool, i, p);
        load_shade_part(st, W.pool, i, p);
        p.backdrop = f3(0.0f, 0.0f, 0.0f);
        while (!step(S, K, p, nograd)) {
        }
        W.results[slot] = finish_path(p);
        if (W.sky_results) W.sky_results[slot] = pack3(p.backdrop, 0.0f);
        if (W.ck.totals) checkpoint_total(W.ck, W.chunk_first, P.width * P.height, slot, p);
    }
}

template <bool L, bool F, bool A, bool CK = false>
WaveStages stage_set() {
    return WaveStages{(const void *)wave_extend<L, F, A>, (const void *)wave_shade<L, F, true, A, CK>,
                      (const void *)wave_shade<L, F, false, A, CK>,
                      CK ? nullptr : (const void *)wave_finish<L, F, A>};
}

}  // namespace

template <bool L, bool F>
WaveStages wave_stages(bool air, bool checkpoints) {
    if (checkpoints) return stage_set<L, F, false, true>();
    return air ? stage_set<L, F, true>() : stage_set<L, F, false>();
}
template WaveStages wave_stages<SG_STAGE_L, SG_STAGE_F>(bool, bool);

}  // namespace sg
