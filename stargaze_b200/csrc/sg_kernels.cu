// sg_kernels.cu — probe kernels, the terrain cache, the camera-ray culling and
// the launches of the per-pixel kernels (sg_pixel_kernels.cu).
#include <algorithm>

#include "sg_wave_common.cuh"

namespace sg {

namespace {

__device__ __forceinline__ Ray load_ray(const sg_ray &in) {
    return Ray{f3(in.offset[0], in.offset[1], in.offset[2]), f3(in.direction[0], in.direction[1], in.direction[2]),
               in.anchor};
}

template <bool F>
__global__ void __launch_bounds__(kThreads) closest_hit_kernel(const __grid_constant__ TraceParams P,
                                                               const sg_ray *rays, sg_hit *hits, uint32_t n) {
    extern __shared__ float4 smem[];
    const Scene S = stage_scene(P, smem);
    const Counter<false, true, F> K{nullptr};
    const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    const sg_ray in = rays[k];
    const Ray r = load_ray(in);
    // An anchor outside the body table would index past the staged bodies.
    const bool valid = in.anchor == kMiss || in.anchor < P.s.counts[0];
    const Hit h = valid ? closest_hit(S, K, r) : Hit{1.0e30f, kMiss, 0.0f, f3(0.0f, 0.0f, 0.0f)};
    sg_hit out;
    out.distance = h.t;
    out.index = h.index;
    float3 nrm = f3(0.0f, 0.0f, 0.0f);
    if (h.index != kMiss) nrm = h.index >= kLocalBase ? h.n : sphere_normal(S, r, h.index, h.delta);
    out.normal[0] = nrm.x;
    out.normal[1] = nrm.y;
    out.normal[2] = nrm.z;
    hits[k] = out;
}

template <bool F>
__global__ void __launch_bounds__(kThreads) visibility_kernel(const __grid_constant__ TraceParams P,
                                                              const sg_ray *rays, const uint32_t *lights,
                                                              float *out, uint32_t n) {
    extern __shared__ float4 smem[];
    const Scene S = stage_scene(P, smem);
    const Counter<false, true, F> K{nullptr};
    const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    const sg_ray in = rays[k];
    const uint32_t light = lights[k];
    const bool valid = (in.anchor == kMiss || in.anchor < P.s.counts[0]) && light < P.s.counts[0];
    out[k] = valid ? light_visibility(S, K, load_ray(in), light) : 0.0f;
}

template <bool F>
__global__ void __launch_bounds__(kThreads) ring_probe_kernel(const __grid_constant__ TraceParams P,
                                                              const sg_ray *rays, uint32_t body, float *out,
                                                              uint32_t n) {
    extern __shared__ float4 smem[];
    const Scene S = stage_scene(P, smem);
    const Counter<false, true, F> K{nullptr};
    const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    const sg_ray in = rays[k];
    const Ray r = load_ray(in);
    float4 result = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (body < P.s.counts[0] && (in.anchor == kMiss || in.anchor < P.s.counts[0])) {
        const RingHit h = ring_hit(S, K, r, body);
        if (h.index != kMiss)
            result = make_float4(h.t, __fdiv_rn(length_rn(h.p), b_radius(S, body)), ring_transmission(S, r, h), 1.0f);
    }
    // Scalar stores: a caller's device pointer need only be 4-byte aligned.
    out[4 * k + 0] = result.x;
    out[4 * k + 1] = result.y;
    out[4 * k + 2] = result.z;
    out[4 * k + 3] = result.w;
}

__global__ void __launch_bounds__(kThreads) terrain_probe_kernel(const __grid_constant__ TraceParams P,
                                                                 const float *rays, float *out, uint32_t n) {
    const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    float4 result = make_float4(0.0f, 0.0f, 0.0f, 1.0e30f);
    if (P.terrain) {
        const float3 o = f3(rays[6 * k], rays[6 * k + 1], rays[6 * k + 2]);
        const float3 d = f3(rays[6 * k + 3], rays[6 * k + 4], rays[6 * k + 5]);
        result = terrain_query<false>(P.terrain, P.terrain_cells, P.s.g.ground_up[3],
                                      (P.s.g.ground_counts[2] & 255u) == 3u, o, d, 1.0e29f, false, nullptr);
    }
    out[4 * k + 0] = result.x;
    out[4 * k + 1] = result.y;
    out[4 * k + 2] = result.z;
    out[4 * k + 3] = result.w;
}

__global__ void ring_energy_kernel(float albedo, float tau, float mu, uint32_t steps, float *out) {
    // ring_tests.rs:365-377: unscattered transmission plus both scattered
    // hemispheres, midpoint rule in the incoming cosine.
    if (blockIdx.x != 0 || threadIdx.x != 0) return;
    const Optics o{f3(albedo, albedo, albedo), tau};
    float energy = expf(-tau / mu);
    for (uint32_t i = 0; i < steps; ++i) {
        const float mi = ((float)i + 0.5f) / (float)steps;
        const float3 sum = ring_bsdf(o, mu, mi) + ring_bsdf(o, mu, -mi);
        energy += sum.x * (kTau * mi / (float)steps);
    }
    *out = energy;
}

// FMA-chain throughput kernel: eight independent chains per thread keep
// every FP32 pipe busy; the result is kept live by an impossible store.
__global__ void __launch_bounds__(256) fma_peak_kernel(float seed, int iters, float *out) {
    float a0 = seed + (float)threadIdx.x, a1 = a0 + 1.0f, a2 = a0 + 2.0f, a3 = a0 + 3.0f;
    float a4 = a0 + 4.0f, a5 = a0 + 5.0f, a6 = a0 + 6.0f, a7 = a0 + 7.0f;
    const float b = 0.999999f, c = 1.0e-7f;
    for (int i = 0; i < iters; ++i) {
#pragma unroll
        for (int k = 0; k < 16; ++k) {
            a0 = fmaf(a0, b, c); a1 = fmaf(a1, b, c); a2 = fmaf(a2, b, c); a3 = fmaf(a3, b, c);
            a4 = fmaf(a4, b, c); a5 = fmaf(a5, b, c); a6 = fmaf(a6, b, c); a7 = fmaf(a7, b, c);
        }
    }
    const float s = ((a0 + a1) + (a2 + a3)) + ((a4 + a5) + (a6 + a7));
    if (s == 1234.5678f) out[0] = s;
}

// cache_terrain_geometry (terrain.wgsl:242-285): node boxes with curvature
// and a +-0.02 m margin, curved heights and normals (12+12-bit packed on
// grids over 1024 cells), in the records of t_root and below. Thread i writes
// node record i, leaf record i and the normal of vertex i. Strict arithmetic
// keeps the cache bit-identical to an IEEE evaluation, so traversal decisions
// match the oracle.
__device__ __forceinline__ float2 cached_range(const float *T, uint32_t cells, float scale, float r, uint32_t index,
                                               float lo_x, float lo_z, float hi_x, float hi_z) {
    const float near_x = clampf(0.0f, lo_x, hi_x), near_z = clampf(0.0f, lo_z, hi_z);
    const float far_x = fmaxf(fabsf(lo_x), fabsf(hi_x)), far_z = fmaxf(fabsf(lo_z), fabsf(hi_z));
    const float lower = __fsub_rn(__fadd_rn(__fmul_rn(T[t_bounds(cells) + index * 2u], scale),
                                            t_curvature(far_x, far_z, r)), 0.02f);
    const float upper = __fadd_rn(__fadd_rn(__fmul_rn(T[t_bounds(cells) + index * 2u + 1u], scale),
                                            t_curvature(near_x, near_z, r)), 0.02f);
    return make_float2(lower, upper);
}

__global__ void __launch_bounds__(256) terrain_cache_kernel(float *T, uint32_t cells, float r) {
    const uint32_t index = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t width = t_width(cells);
    const float scale = t_scale_r(r);
    if (index == 0u) {
        const float lo = t_coordinate(0u, cells, scale), hi = t_coordinate(cells, cells, scale);
        const float2 y = cached_range(T, cells, scale, r, 0u, lo, lo, hi, hi);
        float *c = T + t_root(cells);
        c[0] = lo, c[1] = y.x, c[2] = lo, c[3] = hi, c[4] = y.y, c[5] = hi;
    }
    if (index < t_inner(cells)) {
        const uint3 node = t_node(index, cells);
        float x[3], z[3];
        for (uint32_t k = 0; k < 3u; ++k) {
            x[k] = t_coordinate(node.x + k * (node.z / 2u), cells, scale);
            z[k] = t_coordinate(node.y + k * (node.z / 2u), cells, scale);
        }
        float2 y[4];
        for (uint32_t k = 0; k < 4u; ++k) {
            const uint32_t i = k & 1u, j = k >> 1;
            y[k] = cached_range(T, cells, scale, r, 4u * index + 1u + k, x[i], z[j], x[i + 1u], z[j + 1u]);
        }
        float4 *c = reinterpret_cast<float4 *>(T + t_node_records(cells)) + 4u * (size_t)index;
        c[0] = make_float4(x[0], x[1], x[2], z[0]);
        c[1] = make_float4(z[1], z[2], y[0].x, y[0].y);
        c[2] = make_float4(y[1].x, y[1].y, y[2].x, y[2].y);
        c[3] = make_float4(y[3].x, y[3].y, 0.0f, 0.0f);
    }
    if (index < t_leaves(cells)) {
        const uint3 node = t_node(t_inner(cells) + index, cells);
        float x[3], z[3], y[9];
        for (uint32_t k = 0; k < 3u; ++k) {
            x[k] = t_coordinate(node.x + k, cells, scale);
            z[k] = t_coordinate(node.y + k, cells, scale);
        }
        for (uint32_t k = 0; k < 9u; ++k) {
            const uint32_t i = k % 3u, j = k / 3u;
            y[k] = __fadd_rn(__fmul_rn(T[(node.y + j) * width + node.x + i], scale), t_curvature(x[i], z[j], r));
        }
        float4 *c = reinterpret_cast<float4 *>(T + t_leaf_records(cells)) + 4u * (size_t)index;
        c[0] = make_float4(x[0], x[1], x[2], z[0]);
        c[1] = make_float4(z[1], z[2], y[0], y[1]);
        c[2] = make_float4(y[2], y[3], y[4], y[5]);
        c[3] = make_float4(y[6], y[7], y[8], 0.0f);
    }
    if (index >= t_vertices(cells)) return;
    const uint32_t x = index % width, z = index / width;
    const float px = t_coordinate(x, cells, scale), pz = t_coordinate(z, cells, scale);
    const float denom =
        __fsqrt_rn(fmaxf(__fsub_rn(__fmul_rn(r, r), __fadd_rn(__fmul_rn(px, px), __fmul_rn(pz, pz))), 1.0f));
    const float gx = __fdiv_rn(px, denom), gz = __fdiv_rn(pz, denom);
    float3 normal;
    if (t_compact(cells)) {
        const uint32_t lox = x > 0u ? x - 1u : 0u, loz = z > 0u ? z - 1u : 0u;
        const uint32_t hix = x + 1u < cells ? x + 1u : cells, hiz = z + 1u < cells ? z + 1u : cells;
        const float dx = __fdiv_rn(__fsub_rn(T[z * width + hix], T[z * width + lox]),
                                   __fdiv_rn(__fsub_rn(t_coordinate(hix, cells, scale), t_coordinate(lox, cells, scale)), scale));
        const float dz = __fdiv_rn(__fsub_rn(T[hiz * width + x], T[loz * width + x]),
                                   __fdiv_rn(__fsub_rn(t_coordinate(hiz, cells, scale), t_coordinate(loz, cells, scale)), scale));
        normal = f3(__fadd_rn(-dx, gx), 1.0f, __fadd_rn(-dz, gz));
    } else {
        const uint32_t vertices = t_vertices(cells);
        normal = f3(__fadd_rn(-T[vertices + index], gx), 1.0f, __fadd_rn(-T[2u * vertices + index], gz));
    }
    normal = mul_rn(normal, __fdiv_rn(1.0f, length_rn(normal)));
    float *v = T + t_normals(cells) + (size_t)index * t_normal_stride(cells);
    if (t_compact(cells)) {
        // WGSL round() is round-half-to-even, as rintf.
        const float ux = rintf(__fmul_rn(clampf(__fadd_rn(__fmul_rn(normal.x, 0.5f), 0.5f), 0.0f, 1.0f), 4095.0f));
        const float uz = rintf(__fmul_rn(clampf(__fadd_rn(__fmul_rn(normal.z, 0.5f), 0.5f), 0.0f, 1.0f), 4095.0f));
        v[0] = (float)((uint32_t)ux | ((uint32_t)uz << 12));
    } else {
        v[0] = normal.x;
        v[1] = normal.y;
        v[2] = normal.z;
    }
}

}  // namespace

size_t terrain_source_floats(uint32_t cells) { return (size_t)t_source(cells); }
size_t terrain_floats(uint32_t cells) { return t_floats(cells); }

cudaError_t launch_terrain_cache(float *terrain, uint32_t cells, float radius_m, cudaStream_t stream) {
    const uint32_t threads = t_vertices(cells) > t_nodes(cells) ? t_vertices(cells) : t_nodes(cells);
    terrain_cache_kernel<<<(threads + 255u) / 256u, 256, 0, stream>>>(terrain, cells, radius_m);
    return cudaGetLastError();
}

cudaError_t launch_fma_peak(int blocks, int iters, float *out, cudaStream_t stream) {
    fma_peak_kernel<<<blocks, 256, 0, stream>>>(1.0f, iters, out);
    return cudaGetLastError();
}

// cache_surface_sky (terrain.wgsl:286-302): texel (x, y) holds the air's
// in-scatter along the local direction at azimuth 2 pi (x + 0.5) / 16 and
// elevation sine (y + 0.5) / 8, seen from the camera, with the random state
// the reference seeds per texel. Zero without terrain. Built with the
// settings of an accumulation's first dispatch (counts.y = 0).
template <bool F>
__global__ void __launch_bounds__(kThreads) sky_cache_kernel(const __grid_constant__ TraceParams P, float4 *out) {
    extern __shared__ float4 smem[];
    const Scene S = stage_scene(P, smem);
    const uint32_t index = threadIdx.x;
    if (index >= kSkyTexels) return;
    float3 light = f3(0.0f, 0.0f, 0.0f);
    if (P.s.g.atmo_params[3] > 0.5f && P.s.g.ground_counts[1] != 0u) {
        const uint32_t x = index % 16u, y = index / 16u;
        const float mu = ((float)y + 0.5f) / 8.0f;
        const float phi = kTau * ((float)x + 0.5f) / 16.0f;
        const float r = sqrtf(1.0f - mu * mu);
        const float3 dir = from_ground(S, f3(r * cosf(phi), mu, r * sinf(phi)));
        const Counter<false, true, F> K{nullptr};
        light = atmosphere(S, K, f3(0.0f, 0.0f, 0.0f), dir, 1.0e30f, hash_u32(index ^ 0x91ce452du), 0u).inscatter;
    }
    out[index] = make_float4(light.x, light.y, light.z, 0.0f);
}

size_t trace_smem_bytes(const TraceParams &p) {
    return (size_t)p.s.counts[0] * kBodyVec4 * sizeof(float4) + (size_t)p.staged_table_floats * sizeof(float);
}

static cudaError_t set_smem(const void *fn, size_t bytes) {
    if (bytes <= 48u * 1024u) return cudaSuccess;
    return cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
}

// Launch one instantiation of a kernel with `smem` bytes of dynamic shared
// memory and 256-thread CTAs.
template <typename... K, typename... A>
static cudaError_t launch_variant(void (*kernel)(K...), dim3 grid, size_t smem, cudaStream_t stream, A &&...args) {
    cudaError_t e = set_smem((const void *)kernel, smem);
    if (e != cudaSuccess) return e;
    kernel<<<grid, kThreads, smem, stream>>>(args...);
    return cudaGetLastError();
}

// The per-pixel kernels of the frame's variant.
static PixelKernels kernels_of(const TraceParams &p) {
    if (p.s.g.ground_north[3] != 0.0f) return p.fp64_sites ? pixel_kernels<true, true>() : pixel_kernels<true, false>();
    return p.fp64_sites ? pixel_kernels<false, true>() : pixel_kernels<false, false>();
}

cudaError_t launch_trace(const TraceParams &p, bool count_events, cudaStream_t stream) {
    const size_t smem = trace_smem_bytes(p);
    const dim3 grid((p.width + kTile - 1) / kTile, (p.height + kTile - 1) / kTile);
    // The landscape instantiation only for frames that enable it: the
    // celestial one carries neither its registers nor its code.
    // Frames with host air or styled bodies run the instantiations that
    // carry that code; the event-counting ones always do (gated at run time
    // there).
    const PixelKernels k = kernels_of(p);
    const void *fn = count_events ? k.counted : k.trace[p.air_on || p.styled ? 1 : 0];
    cudaError_t e = set_smem(fn, smem);
    if (e != cudaSuccess) return e;
    TraceParams params = p;
    void *args[] = {&params};
    return cudaLaunchKernel(fn, grid, dim3(kThreads), args, smem, stream);
}

cudaError_t launch_sky_cache(const TraceParams &p, float4 *out, cudaStream_t stream) {
    const size_t smem = trace_smem_bytes(p);
    if (p.fp64_sites) return launch_variant(sky_cache_kernel<true>, dim3(1), smem, stream, p, out);
    return launch_variant(sky_cache_kernel<false>, dim3(1), smem, stream, p, out);
}

size_t adjoint_smem_bytes(const TraceParams &p, const AdjointParams &a) {
    return trace_smem_bytes(p) + (size_t)p.s.counts[0] * 2u * sizeof(float4) +
           (size_t)(a.tau_window + a.color_window) * sizeof(float);
}

cudaError_t launch_adjoint(const TraceParams &p, const AdjointParams &a, cudaStream_t stream) {
    const size_t smem = adjoint_smem_bytes(p, a);
    const dim3 grid((p.width + kTile - 1) / kTile, (p.height + kTile - 1) / kTile);
    const void *fn = kernels_of(p).adjoint;
    cudaError_t e = set_smem(fn, smem);
    if (e != cudaSuccess) return e;
    TraceParams params = p;
    AdjointParams adjoint = a;
    void *args[] = {&params, &adjoint};
    return cudaLaunchKernel(fn, grid, dim3(kThreads), args, smem, stream);
}

// A tile's camera rays: the cone of half-angle alpha about the unit direction
// `axis` (alpha already carries the 1e-3 rad margin below), and its corners'
// unnormalised directions (x, y, -1) in order around the tile.
struct TileCone {
    double3 axis;
    double cos_a, sin_a;
    double cx[4], cy[4];
    bool valid;  // a cone below 90 degrees, all finite: else every body is kept
};

__device__ __forceinline__ double dot3(double3 a, double3 b) { return a.x * b.x + a.y * b.y + a.z * b.z; }

// Whether no ray of the tile can meet a sphere of radius `rho` at `c` (telescope
// space, camera at the origin): the directions that hit an external sphere form
// the cone of half-angle asin(rho / |c|) about c. Radius and angles carry
// margins (1e-3 relative, 1e-3 rad) far above the f32 error of the exact
// intersection tests, so a true here is a certain miss there. With the camera
// within the margin of the surface (an observer on the ground), the tile is
// culled only when the exact test's own f32 value of |c|^2 - r^2, the same for
// every camera ray, is positive (`outside`) and every ray points more than
// 90 degrees and the margin away from the centre: that test's early out.
__device__ __forceinline__ bool cone_misses_sphere(const TileCone &t, double3 c, double rho, bool outside) {
    const double dist = sqrt(dot3(c, c)), r = rho * (1.0 + 1.0e-3);
    const double cos_g = dot3(t.axis, c) / dist;
    if (!(dist > r)) return outside && cos_g < -t.sin_a;
    const double sin_b = r / dist, cos_b = sqrt(1.0 - sin_b * sin_b);
    return t.sin_a * cos_b + t.cos_a * sin_b > 0.0 && cos_g < t.cos_a * cos_b - t.sin_a * sin_b;
}

// Whether no ray of the tile can cross the annulus [inner, outer] about c in
// the plane of normal n. A tile whose rays all cross the plane on one side of
// the camera maps to a convex quadrilateral of the plane: its radii lie between
// its distance from c and its farthest corner's. Margins: 1e-3 of the radii
// and 1e-4 of the centre's distance, over plane angles above 0.01, where the
// f32 error of the exact test's crossing is below 1e-4 of that distance.
__device__ __forceinline__ bool tile_misses_annulus(const TileCone &t, double3 c, double3 n, double inner, double outer) {
    const double nn = dot3(n, n);
    if (!(nn > 0.0)) return false;
    const double scale = 1.0 / sqrt(nn);
    n = make_double3(n.x * scale, n.y * scale, n.z * scale);
    const double h = dot3(n, c), dist = sqrt(dot3(c, c)), slack = 1.0e-4 * dist;
    double den[4], longest = 0.0, steepest = 1.0e300;
    bool positive = true, negative = true;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        den[k] = n.x * t.cx[k] + n.y * t.cy[k] - n.z;
        longest = fmax(longest, t.cx[k] * t.cx[k] + t.cy[k] * t.cy[k] + 1.0);
        steepest = fmin(steepest, fabs(den[k]));
        positive = positive && den[k] > 0.0;
        negative = negative && den[k] < 0.0;
    }
    if (!(positive || negative) || !(steepest > 0.01 * sqrt(longest))) return false;
    double3 p[4];
    double farthest = 0.0;
    bool behind = true, ahead = true;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const double s = h / den[k];
        const double along = s * sqrt(t.cx[k] * t.cx[k] + t.cy[k] * t.cy[k] + 1.0);
        behind = behind && along < -1.0e-3 * dist;
        ahead = ahead && s > 0.0;
        p[k] = make_double3(s * t.cx[k] - c.x, s * t.cy[k] - c.y, -s - c.z);
        farthest = fmax(farthest, dot3(p[k], p[k]));
    }
    if (behind) return true;
    if (!ahead) return false;
    if (sqrt(farthest) < inner * (1.0 - 1.0e-3) - slack) return true;
    double nearest = 1.0e300;
    bool left = true, right = true;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const double3 a = p[k], b = p[(k + 1) & 3];
        const double3 e = make_double3(b.x - a.x, b.y - a.y, b.z - a.z);
        const double w = n.x * (a.y * b.z - a.z * b.y) + n.y * (a.z * b.x - a.x * b.z) + n.z * (a.x * b.y - a.y * b.x);
        left = left && w >= 0.0;
        right = right && w <= 0.0;
        const double u = fmin(fmax(-dot3(a, e) / fmax(dot3(e, e), 1.0e-300), 0.0), 1.0);
        const double3 q = make_double3(a.x + u * e.x, a.y + u * e.y, a.z + u * e.z);
        nearest = fmin(nearest, dot3(q, q));
    }
    return !left && !right && sqrt(nearest) > outer * (1.0 + 1.0e-3) + slack;
}

// `group` lanes per 16x16 tile, one per body (the power of two at or above
// their number): the bodies (their point discs included) and the rings a
// camera ray of the tile may meet. A camera ray of pixel (x, y) has ndc in
// [2x/W - 1, 2(x+1)/W - 1] x [1 - 2(y+1)/H, 1 - 2y/H] (camera_direction,
// pathtrace.wgsl:1619-1626); the tile's rays lie in the cone about its centre
// ray through its farthest corner. With `active`, the tiles that can meet
// anything (every tile, without `skip_empty`) are appended to it, their number
// added to *count (zero before the launch); tiles of one warp keep their order.
// Two thirds of the camera rays of a celestial frame meet nothing. Without the
// paths of such tiles, and with the annulus in place of its bounding sphere and
// the horizon of the ground the observer stands on, a 1920x1080, 64-sample
// dispatch of the ring scene went from 13.8 to 11.0 ms, a 256x256 one of the
// three-sphere scene from 345 to 285 us. Latency bounds the kernel itself: a
// few hundred double operations per lane.
__global__ void __launch_bounds__(128) camera_cull_kernel(const __grid_constant__ TraceParams P, uint2 *out,
                                                          uint32_t *active, uint32_t *count, bool skip_empty,
                                                          uint32_t group, uint32_t tiles_x, uint32_t tiles) {
    const uint32_t thread = blockIdx.x * blockDim.x + threadIdx.x, lane = threadIdx.x & 31u;
    const uint32_t tile = thread / group, i = thread % group;
    const uint32_t n = P.s.counts[0];
    bool body = false, ring = false;
    if (tile < tiles && i < n) {
        const uint32_t tx = tile % tiles_x, ty = tile / tiles_x;
        const double w = P.s.g.viewport[0], h = P.s.g.viewport[1];
        const double tangent = P.s.g.cam_forward[3], aspect = P.s.g.viewport[3];
        const double x0 = (2.0 * (tx * kTile) / w - 1.0) * tangent * aspect;
        const double x1 = (2.0 * fmin((double)(tx * kTile + kTile), w) / w - 1.0) * tangent * aspect;
        const double y0 = (1.0 - 2.0 * fmin((double)(ty * kTile + kTile), h) / h) * tangent;
        const double y1 = (1.0 - 2.0 * (ty * kTile) / h) * tangent;
        TileCone t;
        t.cx[0] = x0, t.cx[1] = x1, t.cx[2] = x1, t.cx[3] = x0;
        t.cy[0] = y0, t.cy[1] = y0, t.cy[2] = y1, t.cy[3] = y1;
        const double ax = 0.5 * (x0 + x1), ay = 0.5 * (y0 + y1), al = 1.0 / sqrt(ax * ax + ay * ay + 1.0);
        t.axis = make_double3(ax * al, ay * al, -al);
        double c = 1.0;
        t.valid = true;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const double v = (t.cx[k] * t.axis.x + t.cy[k] * t.axis.y - t.axis.z) /
                             sqrt(t.cx[k] * t.cx[k] + t.cy[k] * t.cy[k] + 1.0);
            t.valid = t.valid && v > 0.0 && v < 1.0 + 1.0e-9;
            c = fmin(c, v);
        }
        // alpha + 1e-3 rad.
        const double s = sqrt(fmax(1.0 - c * c, 0.0));
        constexpr double kMarginCos = 0.9999995000000417, kMarginSin = 9.999998333333417e-4;
        t.cos_a = c * kMarginCos - s * kMarginSin;
        t.sin_a = s * kMarginCos + c * kMarginSin;
        const float4 hi = P.bodies[i * kBodyVec4 + kCenter], lo = P.bodies[i * kBodyVec4 + kLow];
        const double3 centre = make_double3((double)hi.x + lo.x, (double)hi.y + lo.y, (double)hi.z + lo.z);
        const double dist = sqrt(dot3(centre, centre));
        // point_disc_hit draws an unresolved body as a disc of at least
        // `angle` radians (pathtrace.wgsl:1308-1333).
        const double pixel = 2.0 * tangent / fmax(h, 1.0);
        const double angle = fmin(fmax((double)kPointDiscRadius, 0.7 * pixel), (double)kStarDotPixels * pixel);
        const double radius = hi.w, drawn = fmax(radius, angle * dist);
        const float3 oc = add_rn(xyz(hi), xyz(lo));  // relative_center of a camera ray
        const bool outside = drawn == radius && __fsub_rn(dot_rn(oc, oc), __fmul_rn(hi.w, hi.w)) > 0.0f;
        body = !(t.valid && cone_misses_sphere(t, centre, drawn, outside));
        const float4 plane = P.bodies[i * kBodyVec4 + kRingPlane], params = P.bodies[i * kBodyVec4 + kRingParams];
        // The annulus lies inside the sphere of its outer radius.
        if (params.x > plane.w && params.y > 0.0f)
            ring = !(t.valid && (cone_misses_sphere(t, centre, (double)params.x * radius, false) ||
                                 tile_misses_annulus(t, centre, make_double3(plane.x, plane.y, plane.z),
                                                     (double)plane.w * radius, (double)params.x * radius)));
    }
    const uint32_t shift = lane & ~(group - 1u), field = group == 32u ? 0xffffffffu : (1u << group) - 1u;
    const uint32_t bodies = (__ballot_sync(0xffffffffu, body) >> shift) & field;
    const uint32_t rings = (__ballot_sync(0xffffffffu, ring) >> shift) & field;
    const bool leader = i == 0u && tile < tiles;
    if (leader) out[tile] = make_uint2(bodies, rings);
    if (!active) return;
    const bool taken = leader && (!skip_empty || (bodies | rings) != 0u);
    const uint32_t taken_lanes = __ballot_sync(0xffffffffu, taken);
    uint32_t at = 0u;
    if (lane == 0u && taken_lanes) at = atomicAdd(count, __popc(taken_lanes));
    at = __shfl_sync(0xffffffffu, at, 0);
    if (taken) active[at + __popc(taken_lanes & ((1u << lane) - 1u))] = tile;
}

// The list of camera_cull_kernel in raster order, by one CTA.
__global__ void __launch_bounds__(1024) tile_list_kernel(const uint2 *masks, uint32_t *active, uint32_t *count,
                                                         bool skip_empty, uint32_t tiles) {
    __shared__ uint32_t warp_counts[32];
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    uint32_t listed = 0u;
    for (uint32_t base = 0; base < tiles; base += 1024u) {
        const uint32_t tile = base + threadIdx.x;
        bool taken = false;
        if (tile < tiles) {
            const uint2 m = masks[tile];
            taken = !skip_empty || (m.x | m.y) != 0u;
        }
        const uint32_t lanes = __ballot_sync(0xffffffffu, taken);
        if (lane == 0u) warp_counts[warp] = __popc(lanes);
        __syncthreads();
        uint32_t before = 0u, total = 0u;
        for (uint32_t w = 0; w < 32u; ++w) {
            if (w == warp) before = total;
            total += warp_counts[w];
        }
        if (taken) active[listed + before + __popc(lanes & ((1u << lane) - 1u))] = tile;
        listed += total;
        __syncthreads();
    }
    if (threadIdx.x == 0u) *count = listed;
}

cudaError_t launch_camera_cull(const TraceParams &p, uint2 *out, uint32_t *active, uint32_t *count, bool skip_empty,
                               bool ordered, cudaStream_t stream) {
    const uint32_t tiles_x = (p.width + kTile - 1) / kTile, tiles = tiles_x * ((p.height + kTile - 1) / kTile);
    const uint32_t n = p.s.counts[0];
    if (n == 0u || n > 32u || tiles == 0u) return cudaErrorInvalidValue;
    uint32_t group = 1u;
    while (group < n) group *= 2u;
    const uint64_t threads = (uint64_t)tiles * group;
    camera_cull_kernel<<<(uint32_t)((threads + 127u) / 128u), 128, 0, stream>>>(p, out, ordered ? nullptr : active, count,
                                                                                skip_empty, group, tiles_x, tiles);
    if (ordered && active) tile_list_kernel<<<1, 1024, 0, stream>>>(out, active, count, skip_empty, tiles);
    return cudaGetLastError();
}

cudaError_t launch_checkpoint_segments(const TraceParams &p, const AdjointParams &a, uint32_t records,
                                       cudaStream_t stream) {
    if (records == 0) return cudaSuccess;
    const size_t smem = adjoint_smem_bytes(p, a);
    const void *fn = kernels_of(p).segments;
    int grid = 0;
    cudaError_t e = set_smem(fn, smem);
    if (e == cudaSuccess) e = persistent_grid(fn, smem, &grid);
    if (e != cudaSuccess) return e;
    grid = (int)std::min<uint32_t>((uint32_t)grid, (records + kThreads - 1) / kThreads);
    TraceParams params = p;
    AdjointParams adjoint = a;
    void *args[] = {&params, &adjoint, &records};
    return cudaLaunchKernel(fn, dim3(grid), dim3(kThreads), args, smem, stream);
}

cudaError_t launch_closest_hit(const TraceParams &p, const sg_ray *rays, sg_hit *hits, uint32_t n,
                               cudaStream_t stream) {
    if (n == 0) return cudaSuccess;
    const size_t smem = trace_smem_bytes(p);
    const dim3 grid((n + kThreads - 1) / kThreads);
    if (p.fp64_sites) return launch_variant(closest_hit_kernel<true>, grid, smem, stream, p, rays, hits, n);
    return launch_variant(closest_hit_kernel<false>, grid, smem, stream, p, rays, hits, n);
}

cudaError_t launch_light_visibility(const TraceParams &p, const sg_ray *rays, const uint32_t *lights,
                                    float *out, uint32_t n, cudaStream_t stream) {
    if (n == 0) return cudaSuccess;
    const size_t smem = trace_smem_bytes(p);
    const dim3 grid((n + kThreads - 1) / kThreads);
    if (p.fp64_sites) return launch_variant(visibility_kernel<true>, grid, smem, stream, p, rays, lights, out, n);
    return launch_variant(visibility_kernel<false>, grid, smem, stream, p, rays, lights, out, n);
}

cudaError_t launch_ring_probe(const TraceParams &p, const sg_ray *rays, uint32_t body, float *out,
                              uint32_t n, cudaStream_t stream) {
    if (n == 0) return cudaSuccess;
    const size_t smem = trace_smem_bytes(p);
    const dim3 grid((n + kThreads - 1) / kThreads);
    if (p.fp64_sites) return launch_variant(ring_probe_kernel<true>, grid, smem, stream, p, rays, body, out, n);
    return launch_variant(ring_probe_kernel<false>, grid, smem, stream, p, rays, body, out, n);
}

cudaError_t launch_terrain_probe(const TraceParams &p, const float *rays, float *out, uint32_t n,
                                 cudaStream_t stream) {
    if (n == 0) return cudaSuccess;
    terrain_probe_kernel<<<(n + kThreads - 1) / kThreads, kThreads, 0, stream>>>(p, rays, out, n);
    return cudaGetLastError();
}

cudaError_t launch_ring_energy(float albedo, float tau, float mu, uint32_t steps, float *out,
                               cudaStream_t stream) {
    ring_energy_kernel<<<1, 32, 0, stream>>>(albedo, tau, mu, steps, out);
    return cudaGetLastError();
}

}  // namespace sg
