// Wavefront path tracer: the reference's PathIntegrator::Radiance bounce loop
// (Core/Integrator/PathIntegrator.cpp:44-367) restated as queue-driven
// kernels over SoA path state:
//
//   k_camera   one camera ray per (pixel, sample) of the wave
//              (BaseRenderer::RenderRegion, Core/Renderer/BaseRenderer.cpp:62-169;
//               PerspectiveCamera::GetRay, Core/Camera/PerspectiveCamera.cpp:44-60)
//   k_extend   closest hit of every queued ray (the traversal of trace.cuh)
//   k_shade    emission at depth 0, NEE toward every quad light but the hit one
//              (IIntegrator::SampleAllLights / EstimateDirectLighting,
//               Core/Integrator/Integrator.cpp:114-185; DiffuseAreaLight,
//               Core/Light/DiffuseAreaLight.cpp:52-69), BSDF sample, throughput,
//              Russian roulette after depth 3, spawn offset along the
//              geometric normal; pushes shadow rays and continuations with
//              warp-aggregated atomics (the queue compaction)
//   k_shadow   any hit of every shadow segment; unoccluded contributions are
//              added to the pixel
//   k_resolve  pixel sums / spp
//
// Random numbers come from a counter-based hash of (seed, pixel, sample,
// depth, dimension) instead of the reference's shared Mersenne twister, so
// images agree with the reference statistically, not bit for bit.
#include "bvh8.cuh"
#include "render.cuh"
#include "trace.cuh"
#include "mlp.cuh"
#include "devinfo.cuh"

#include <algorithm>
#include <cfloat>

namespace ilg {

namespace {

constexpr float kInvPi = 0.318309886183790671538f;
constexpr float kTwoPi = 6.28318530717958647692f;

__device__ __forceinline__ uint64_t mix64(uint64_t x)
{
    x += 0x9E3779B97F4A7C15ull;
    x = (x ^ (x >> 30)) * 0xBF58476D1CE4E5B9ull;
    x = (x ^ (x >> 27)) * 0x94D049BB133111EBull;
    return x ^ (x >> 31);
}

// uniform float in [0, 1) for one (path, dimension)
__device__ __forceinline__ float rnd(uint64_t key, uint32_t dim)
{
    return (float)(uint32_t)(mix64(key + (uint64_t)dim * 0xD1B54A32D192ED03ull) >> 40) * 0x1p-24f;
}

__device__ __forceinline__ uint64_t path_key(uint32_t seed, uint64_t path_global)
{
    return mix64(path_global ^ ((uint64_t)seed * 0xA24BAED4963EE407ull));
}

// dimensions: per depth d, base 32*d: lights 2l, 2l+1 (l < 8); bsdf 20, 21, 22; roulette 23
constexpr uint32_t kDimCam = 0xFFFFFF00u;
__device__ __forceinline__ uint32_t dim_of(uint32_t depth, uint32_t k) { return depth * 32u + k; }

__device__ __forceinline__ float3 operator+(float3 a, float3 b) { return make_float3(a.x + b.x, a.y + b.y, a.z + b.z); }
__device__ __forceinline__ float3 operator-(float3 a, float3 b) { return make_float3(a.x - b.x, a.y - b.y, a.z - b.z); }
__device__ __forceinline__ float3 operator*(float3 a, float s) { return make_float3(a.x * s, a.y * s, a.z * s); }
__device__ __forceinline__ float3 operator*(float3 a, float3 b) { return make_float3(a.x * b.x, a.y * b.y, a.z * b.z); }
__device__ __forceinline__ float dot3(float3 a, float3 b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
__device__ __forceinline__ float3 cross3(float3 a, float3 b)
{
    return make_float3(a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x);
}
__device__ __forceinline__ float3 normalize3(float3 a) { return a * rsqrtf(dot3(a, a)); }
__device__ __forceinline__ bool is_black(float3 a) { return a.x == 0.f && a.y == 0.f && a.z == 0.f; }

// OrthonormalBasis::InitFromW, Core/Geometry/Basis.cpp:85-99
__device__ __forceinline__ void onb_from_w(float3 w, float3 &u, float3 &v)
{
    if (fabsf(w.x) > fabsf(w.y)) {
        float inv = 1.f / sqrtf(w.x * w.x + w.z * w.z);
        v = make_float3(-w.z * inv, 0.f, w.x * inv);
    } else {
        float inv = 1.f / sqrtf(w.y * w.y + w.z * w.z);
        v = make_float3(0.f, w.z * inv, -w.y * inv);
    }
    u = cross3(w, v);
}

// warp-aggregated queue push: returns this lane's slot (or 0xffffffff if !want)
__device__ __forceinline__ uint32_t push_slot(bool want, uint32_t *count)
{
    const uint32_t mask = __ballot_sync(__activemask(), want);
    if (!want) return 0xffffffffu;
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t leader = __ffs(mask) - 1u;
    uint32_t base = 0;
    if (lane == leader) base = atomicAdd(count, (uint32_t)__popc(mask));
    base = __shfl_sync(mask, base, leader);
    return base + __popc(mask & ((1u << lane) - 1u));
}

__device__ __forceinline__ void add_pixel(float4 *accum, uint32_t pixel, float3 c)
{
    atomicAdd(accum + pixel, make_float4(c.x, c.y, c.z, 0.f));  // one vector reduction
}

// scene of a global path index (the scenes' path ranges are consecutive)
__device__ __forceinline__ uint32_t scene_of(const RenderDev &R, uint64_t g)
{
    uint32_t lo = 0, hi = R.n_scenes;
    while (hi - lo > 1) {
        const uint32_t mid = (lo + hi) >> 1;
        if (R.scenes[mid].path_begin <= g) lo = mid;
        else hi = mid;
    }
    return lo;
}

// path identity inside its scene: (pixel, sample-sequence key)
// (pixel = index in the rendered region, image coordinates x, y). The key
// depends on the image pixel and the sample only, so a region renders exactly
// the paths the whole image renders there.
__device__ __forceinline__ void path_ident(const SceneRec &S, uint64_t g, uint32_t &pixel, uint64_t &key,
                                           uint32_t &x, uint32_t &y)
{
    const uint64_t local = g - S.path_begin;
    uint64_t sample;
    if (local >> 32) {
        sample = local / S.wh;
        pixel = (uint32_t)(local - sample * S.wh);
    } else {  // (a 64-bit division is some 100 instructions)
        const uint32_t s = (uint32_t)local / S.wh;
        sample = s;
        pixel = (uint32_t)local - s * S.wh;
    }
    x = S.region_x + pixel % S.region_w;
    y = S.region_y + pixel / S.region_w;
    key = path_key(S.seed, sample * S.full_wh + (uint64_t)y * S.width + x);
}

// The first ray of global path g of scene S: the caller's ray
// (IIntegrator::Radiance(..., ray, ...), whose first intersection uses the
// ray's own [Min, Max]) or a camera ray.
__device__ __forceinline__ void first_ray(const SceneRec &S, uint64_t g, uint32_t &pixel, uint64_t &key, float4 &o,
                                          float4 &d)
{
    uint32_t x, y;
    path_ident(S, g, pixel, key, x, y);
    if (S.ray_o) {
        o = S.ray_o[pixel];
        d = S.ray_d[pixel];
        return;
    }
    // BoxFilter shifts the [0,1) sample by -0.5 (Core/Filter/BoxFilter.cpp:20-28)
    const float xi1 = rnd(key, kDimCam) - 0.5f, xi2 = rnd(key, kDimCam + 1) - 0.5f;
    const float fx = x * S.rcp_w + xi1 * S.rcp_w, fy = y * S.rcp_h + xi2 * S.rcp_h;
    const float3 target = S.corner + S.across * fx + S.up * fy;
    const float3 dd = normalize3(target - S.centre);
    o = make_float4(S.centre.x, S.centre.y, S.centre.z, 0.f);
    d = make_float4(dd.x, dd.y, dd.z, FLT_MAX);
}

__global__ void k_camera(RenderDev R, uint32_t n_paths, uint64_t wave_begin)
{
    const uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p == 0) R.count[0] = n_paths;  // the wave's first extend queue is every path
    if (p >= n_paths) return;
    const uint64_t g = wave_begin + p;
    const uint32_t sid = scene_of(R, g);
    const SceneRec &S = R.scenes[sid];
    uint32_t pixel;
    uint64_t key;
    first_ray(S, g, pixel, key, R.q_o[0][p], R.q_d[0][p]);
    R.q_path[0][p] = p;
    if (R.n_scenes > 1u) R.path_scene[p] = sid;
    R.beta[p] = make_float4(1.f, 1.f, 1.f, 0.f);
    if (R.cache_depth) {
        uint32_t slot = 0xffffffffu;
        if (mix64(key ^ 0x5851F42D4C957F2Dull) % R.train_every == 0) {
            const uint32_t s = atomicAdd(R.train_count, 1u);
            if (s < R.train_cap) slot = s;
        }
        R.train_slot[p] = slot;
    }
}

// Adds contribution c, found at vertex `vert` of a training path, to the
// targets of that path's recorded vertices 1..vert (each in units of the
// radiance leaving its own vertex: divided by the throughput there).
__device__ __forceinline__ void credit(const RenderDev &R, uint32_t slot, uint32_t vert, float3 c)
{
    const uint32_t stride = R.depth_max + 1;
    for (uint32_t k = 1; k <= vert && k <= R.depth_max; k++) {
        const uint32_t ri = R.rec_of[slot * stride + k];
        if (ri == 0xffffffffu || ri >= R.rec_cap) continue;
        const float4 b = R.rec_beta[ri];
        atomicAdd(&R.rec_tgt[3 * ri], c.x / fmaxf(b.x, 1e-8f));
        atomicAdd(&R.rec_tgt[3 * ri + 1], c.y / fmaxf(b.y, 1e-8f));
        atomicAdd(&R.rec_tgt[3 * ri + 2], c.z / fmaxf(b.z, 1e-8f));
    }
}

__device__ __forceinline__ void write_features(float *f, const RenderDev &R, float3 p, float3 wo, float3 n,
                                               const Mat &m)
{
    f[0] = (p.x - R.scene_lo.x) * R.scene_inv_ext.x;
    f[1] = (p.y - R.scene_lo.y) * R.scene_inv_ext.y;
    f[2] = (p.z - R.scene_lo.z) * R.scene_inv_ext.z;
    f[3] = wo.x; f[4] = wo.y; f[5] = wo.z;
    f[6] = n.x; f[7] = n.y; f[8] = n.z;
    const bool ggx = m.kind == 1u;
    f[9] = ggx ? m.alpha : 1.f;
    const float3 a = ggx ? m.f0 : m.albedo;
    f[10] = a.x; f[11] = a.y; f[12] = a.z;
    f[13] = f[14] = f[15] = 0.f;
}

// Sum over the warp of counts below 2^32.
__device__ __forceinline__ unsigned long long warp_sum(uint32_t v)
{
    return ((unsigned long long)__reduce_add_sync(0xffffffffu, v >> 16) << 16) +
           __reduce_add_sync(0xffffffffu, v & 0xffffu);
}

// Work counters of a counted render: R.stats[k0] += rays, [k0 + 1] += node
// records read, [k0 + 2] += triangle records tested. All threads of the block
// call it, once; one atomic per block and counter (with one per warp, 4096
// rays' extension kernel took 14.5 us, of which 3 waited for them).
__device__ __forceinline__ void count_work(const RenderDev &R, int k0, bool ray, uint32_t nn, uint32_t nt)
{
    __shared__ unsigned long long s_work[3];
    if (threadIdx.x < 3u) s_work[threadIdx.x] = 0ull;
    __syncthreads();
    const uint32_t rays = __popc(__ballot_sync(0xffffffffu, ray));
    const unsigned long long wn = warp_sum(nn), wt = warp_sum(nt);
    if ((threadIdx.x & 31u) == 0u && rays) {
        atomicAdd(&s_work[0], (unsigned long long)rays);
        atomicAdd(&s_work[1], wn);
        atomicAdd(&s_work[2], wt);
    }
    __syncthreads();
    if (threadIdx.x < 3u && s_work[0]) atomicAdd(R.stats + k0 + threadIdx.x, s_work[threadIdx.x]);
}

// An unoccluded shadow segment adds its contribution to its pixel (and to
// Direct when tagged), and credits the training record it belongs to.
__device__ __forceinline__ void shadow_unoccluded(const RenderDev &R, uint32_t i)
{
    const float4 c = R.s_c[i];
    const uint32_t bits = __float_as_uint(c.w);
    add_pixel(R.accum, bits & 0x7fffffffu, make_float3(c.x, c.y, c.z));
    if (bits >> 31) add_pixel(R.accum_direct, bits & 0x7fffffffu, make_float3(c.x, c.y, c.z));
    if (R.cache_depth) {
        const uint32_t meta = R.s_meta[i];
        if (meta != 0xffffffffu) credit(R, meta >> 8, meta & 0xffu, make_float3(c.x, c.y, c.z));
    }
}

template <bool kStats>
__global__ void __launch_bounds__(256, 4) k_extend(RenderDev R, int cur)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    const bool live = i < R.count[cur];
    if (!kStats && !live) return;
    uint32_t nn = 0, nt = 0;
    if (live) {
        const float4 o = R.q_o[cur][i], d = R.q_d[cur][i];
        const SceneRec &S = R.scenes[R.n_scenes > 1u ? R.path_scene[R.q_path[cur][i]] : 0u];
        int best;
        float bt, bu, bv;
        trace_one<false, kStats>(S.nodes, S.tris, S.n_nodes, S.n_tris, R.min_dir, o, d, best, bt, bu, bv, R.err, nn, nt);
        R.hit_tri[i] = best;
        R.hit_t[i] = bt;
    }
    if (kStats) count_work(R, 0, live, nn, nt);
}

// GGX conductor (Trowbridge-Reitz D, Smith G1 separable, Schlick F), sampled
// with the visible-normal distribution (Heitz 2018). Local frame: z = normal.
__device__ __forceinline__ float ggx_d(float3 h, float a)
{
    const float a2 = a * a;
    const float t = h.x * h.x / a2 + h.y * h.y / a2 + h.z * h.z;
    return 1.f / (3.14159265358979f * a2 * t * t);
}
__device__ __forceinline__ float ggx_g1(float3 w, float a)
{
    const float z2 = w.z * w.z;
    if (z2 <= 0.f) return 0.f;
    const float t2 = (w.x * w.x + w.y * w.y) * a * a / z2;
    return 2.f / (1.f + sqrtf(1.f + t2));
}
__device__ __forceinline__ float3 schlick(float3 f0, float c)
{
    const float m = 1.f - fminf(fmaxf(c, 0.f), 1.f);
    const float m5 = m * m * m * m * m;
    return f0 + (make_float3(1.f, 1.f, 1.f) - f0) * m5;
}
__device__ __forceinline__ float3 ggx_f(float3 wo, float3 wi, float3 f0, float a)
{
    if (wo.z <= 0.f || wi.z <= 0.f) return make_float3(0.f, 0.f, 0.f);
    const float3 h = normalize3(wo + wi);
    const float g = ggx_g1(wo, a) * ggx_g1(wi, a);
    return schlick(f0, dot3(wi, h)) * (ggx_d(h, a) * g / (4.f * wo.z * wi.z));
}
__device__ __forceinline__ float ggx_pdf(float3 wo, float3 wi, float a)
{
    if (wo.z <= 0.f || wi.z <= 0.f) return 0.f;
    const float3 h = normalize3(wo + wi);
    // pdf of the visible normal h, times the reflection Jacobian 1 / (4 wo.h)
    return ggx_g1(wo, a) * fmaxf(dot3(wo, h), 0.f) * ggx_d(h, a) / wo.z / (4.f * dot3(wo, h));
}
__device__ __forceinline__ float3 ggx_sample_vndf(float3 wo, float a, float u1, float u2)
{
    const float3 vh = normalize3(make_float3(a * wo.x, a * wo.y, wo.z));
    const float lensq = vh.x * vh.x + vh.y * vh.y;
    const float3 t1 = lensq > 0.f ? make_float3(-vh.y, vh.x, 0.f) * rsqrtf(lensq) : make_float3(1.f, 0.f, 0.f);
    const float3 t2 = cross3(vh, t1);
    const float r = sqrtf(u1);
    float s, c;
    sincosf(kTwoPi * u2, &s, &c);
    const float p1 = r * c;
    float p2 = r * s;
    const float sh = 0.5f * (1.f + vh.z);
    p2 = (1.f - sh) * sqrtf(fmaxf(0.f, 1.f - p1 * p1)) + sh * p2;
    const float3 nh = t1 * p1 + t2 * p2 + vh * sqrtf(fmaxf(0.f, 1.f - p1 * p1 - p2 * p2));
    const float3 h = normalize3(make_float3(a * nh.x, a * nh.y, fmaxf(0.f, nh.z)));
    const float3 wi = h * (2.f * dot3(wo, h)) - wo;
    return wi;
}

// BSDF::F for one material in the local frame (Core/Material/BSDF.cpp:214-234:
// reflection lobes only count when wi.z > 0)
// BSDF value for a direction pair; the specular materials (mirror, glass)
// are zero for every pair, as their BxDFs' F is (SpecularReflection::F,
// SpecularTransmission::F).
__device__ __forceinline__ float3 bsdf_f(const Mat &m, float3 wo, float3 wi)
{
    if (m.kind == 1u) return ggx_f(wo, wi, m.f0, m.alpha);
    if (m.kind == 0u && wi.z > 0.f) return m.albedo * kInvPi;
    return make_float3(0.f, 0.f, 0.f);
}

// Specular sampling of the reference's MirrorMaterial and GlassMaterial in
// the local frame (z = normal). Mirror: SpecularReflection::SampleF
// (Core/Material/SpecularReflectionBxDF.cpp:26-33): wi = (-wo.x, -wo.y,
// wo.z), pdf 1, f = reflectivity / |wi.z|. Glass: BSDF::SampleF
// (Core/Material/BSDF.cpp:141-211) picks one of its two BxDFs with the 1D
// sample (index (int)(w * 2) % 2: 0 = SpecularTransmission with the
// transmittance, 1 = SpecularReflection with the reflectivity) and halves
// the pdf; SpecularTransmission::SampleF
// (Core/Material/SpecularTransmissionBxDF.cpp:24-58) refracts by the ratio
// of indices with no Fresnel weight, and total internal reflection gives
// f = 0 (the path ends). `transmit` tells the caller to offset the next ray
// origin below the surface (PathIntegrator.cpp:184-187).
__device__ __forceinline__ void sample_specular(const Mat &m, float3 wo, float w, float3 &wi, float3 &f, float &pdf,
                                                bool &transmit)
{
    transmit = false;
    const float3 zero = make_float3(0.f, 0.f, 0.f);
    if (m.kind == 2u || (int)(w * 2.f) % 2 == 1) {
        wi = make_float3(-wo.x, -wo.y, wo.z);
        f = m.albedo * (1.f / fabsf(wi.z));
        pdf = m.kind == 2u ? 1.f : 0.5f;
        return;
    }
    // glass, transmission: m.alpha holds eta_i / eta_t
    const bool entering = wo.z > 0.f;
    const float eta = entering ? m.alpha : 1.f / m.alpha;
    const float sin_i2 = 1.f - wo.z * wo.z;
    const float sin_t2 = sin_i2 * eta * eta;
    pdf = 0.5f;
    if (sin_t2 > 1.f) {
        wi = zero;
        f = zero;
        return;
    }
    float cos_t = sqrtf(fmaxf(0.f, 1.f - sin_t2));
    if (entering) cos_t = -cos_t;
    wi = make_float3(eta * -wo.x, eta * -wo.y, cos_t);
    f = m.f0 * (1.f / fabsf(cos_t));
    transmit = true;
}

// One light sample of next-event estimation at a shading point
// (IIntegrator::EstimateDirectLighting, Core/Integrator/Integrator.cpp:114-139,
// with the light's SampleRadiance): light l's shadow segment and the
// contribution it adds when unoccluded; false when the sample adds nothing.
// The shading frame is (U, V, W) with W the shading normal; wo_l is the
// outgoing direction in it.
__device__ __forceinline__ bool light_sample(const SceneRec &S, uint32_t l, uint64_t key, uint32_t depth, float3 p,
                                             float3 U, float3 V, float3 W, float3 wo_l, const Mat &m, float3 beta,
                                             float4 &so, float4 &sd, float3 &c)
{
    const Light &L = S.lights[l];
    const float u = rnd(key, dim_of(depth, 2 * l)), v = rnd(key, dim_of(depth, 2 * l + 1));
    if (L.kind == kLightInfinite) {
        // InfiniteAreaLight::SampleRadiance (InfiniteAreaLight.cpp:73-83):
        // a direction in the cone cos(theta) >= 1e-4 about the shading
        // normal (Montecarlo::UniformSampleCone, Montecarlo.h:74-80), the
        // light's intensity with no division by the pdf, a shadow ray
        // over [1e-4, FLT_MAX] from the point itself
        const float ct = (1.f - u) + u * 1e-4f;
        const float st = sqrtf(1.f - ct * ct);
        float sp, cp;
        sincosf(kTwoPi * v, &sp, &cp);
        const float3 wi = U * (cp * st) + V * (sp * st) + W * ct;
        const float3 wi_l = make_float3(dot3(U, wi), dot3(V, wi), dot3(W, wi));
        c = beta * L.emit * fmaxf(0.f, dot3(wi, W)) * bsdf_f(m, wo_l, wi_l);
        if (is_black(c)) return false;
        so = make_float4(p.x, p.y, p.z, 1e-4f);
        sd = make_float4(wi.x, wi.y, wi.z, FLT_MAX);
        return true;
    }
    float3 P, nl;
    if (L.kind == kLightMesh) {
        // ITriangleMesh::SamplePoint (Core/Shape/TriangleMesh.cpp:142-161):
        // a triangle picked uniformly by index (not by area), a uniform
        // point on it (IndexedTriangle::SamplePoint, Montecarlo.h:59-64),
        // its normal (p3 - p1) x (p2 - p1) turned to face the shaded
        // point; the pdf is 1 / the mesh's whole area (DiffuseAreaLight.cpp:36-40)
        const uint32_t k = min((uint32_t)((float)L.tri_count * rnd(key, dim_of(depth, 24 + l))),
                               L.tri_count - 1u);
        const uint32_t *tv = S.idx + 3ull * (L.first_tri + k);
        const float *a = S.pos + 3ull * tv[0], *b = S.pos + 3ull * tv[1], *cc = S.pos + 3ull * tv[2];
        const float3 p1 = make_float3(a[0], a[1], a[2]), p2 = make_float3(b[0], b[1], b[2]),
                     p3 = make_float3(cc[0], cc[1], cc[2]);
        const float su = sqrtf(u);
        const float b1 = 1.f - su, b2 = v * su;
        P = p1 * b1 + p2 * b2 + p3 * (1.f - b1 - b2);
        nl = normalize3(cross3(p3 - p1, p2 - p1));
        if (dot3(P - p, nl) > 0.f) nl = nl * -1.f;
    } else {
        // Quad::SamplePoint (Core/Shape/Quad.cpp:144-153): a bilinear
        // patch over the reference's tessellation vertices
        P = L.p[0] + (L.p[2] - L.p[0]) * u + (L.p[3] - L.p[2]) * v +
            (L.p[0] - L.p[2] + L.p[1] - L.p[3]) * (u * v);
        nl = L.n;
    }
    float3 win = p - P;
    const float dist2 = dot3(win, win);
    win = normalize3(win);
    const float cl = fmaxf(0.f, dot3(win, nl));
    const float3 Ls = L.emit * (cl * L.area / dist2);
    if (is_black(Ls)) return false;
    const float3 wi = win * -1.f;
    const float3 wi_l = make_float3(dot3(U, wi), dot3(V, wi), dot3(W, wi));
    c = beta * Ls * (fmaxf(0.f, dot3(wi, W))) * bsdf_f(m, wo_l, wi_l);
    if (is_black(c)) return false;
    const float3 seg = P - p;
    so = make_float4(p.x, p.y, p.z, S.eps);
    sd = make_float4(seg.x, seg.y, seg.z, 1.f - S.eps);
    return true;
}

// The path's next ray (PathIntegrator.cpp:141-187): a BSDF sample
// (BSDF::SampleF, Core/Material/BSDF.cpp:141-211), the throughput update,
// Russian roulette after depth 3 and the spawn offset along the geometric
// normal (below the surface for a transmitted ray). False when the path
// ends here; beta is updated when it continues.
__device__ __forceinline__ bool continue_path(const SceneRec &S, uint64_t key, uint32_t depth, const Mat &m,
                                              bool specular, float3 p, float3 ng, float3 U, float3 V, float3 W,
                                              float3 wo_l, float3 &beta, float4 &no, float4 &nd)
{
    const float u1 = rnd(key, dim_of(depth, 20)), u2 = rnd(key, dim_of(depth, 21));
    float3 wi_l, f;
    float pdf;
    bool transmit = false;
    if (specular) {
        sample_specular(m, wo_l, rnd(key, dim_of(depth, 22)), wi_l, f, pdf, transmit);
    } else if (m.kind == 1u) {
        wi_l = ggx_sample_vndf(wo_l, m.alpha, u1, u2);
        pdf = ggx_pdf(wo_l, wi_l, m.alpha);
        f = ggx_f(wo_l, wi_l, m.f0, m.alpha);
    } else {
        // Lambertian::SampleF (Core/Material/LambertianBxDF.cpp:27-37)
        const float r = sqrtf(u1);
        float s, c;
        sincosf(kTwoPi * u2, &s, &c);
        wi_l = make_float3(r * c, r * s, sqrtf(1.f - u1));
        if (wo_l.z < 0.f) wi_l.z = -wi_l.z;
        pdf = fabsf(wi_l.z) * kInvPi;
        f = bsdf_f(m, wo_l, wi_l);
    }
    if (is_black(f) || !(pdf > 0.f)) return false;
    const float3 wi = U * wi_l.x + V * wi_l.y + W * wi_l.z;
    float3 b = beta * f * (fabsf(dot3(wi, W)) / pdf);
    if (depth > 3) {
        const float q = fminf(0.5f, 0.212671f * b.x + 0.715160f * b.y + 0.072169f * b.z);
        if (rnd(key, dim_of(depth, 23)) > q) return false;
        b = b * (1.f / q);
    }
    beta = b;
    // a transmitted ray starts below the surface (PathIntegrator.cpp:184-187)
    const float3 org = p + ng * (transmit ? -S.eps : S.eps);
    no = make_float4(org.x, org.y, org.z, S.eps);
    nd = make_float4(wi.x, wi.y, wi.z, FLT_MAX);
    return true;
}

// kCache: a render with the radiance cache. kOne: a render of one scene (no
// scene index to load before everything else). The kernel waits on chains of
// dependent loads (ray -> path -> scene -> hit triangle -> material), so what
// it needs is warps in flight: the plain one-scene form takes a third fewer
// registers and two loads less in the chain than the general one.
template <bool kCache, bool kOne>
__global__ void __launch_bounds__(256) k_shade(RenderDev R, int cur, uint32_t depth, uint64_t wave_begin)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    const int nxt = cur ^ 1;
    bool cont = false;
    float4 no = make_float4(0.f, 0.f, 0.f, 0.f), nd = no;
    uint32_t path = 0;
    uint32_t pixel = 0;
    bool query = false;           // rendering path stopping into the cache here
    float4 qb = make_float4(0.f, 0.f, 0.f, 0.f);
    float qf[kMlpRaw];
    uint32_t tslot = 0xffffffffu;  // training slot of this path
    uint32_t qmeta = 0xffffffffu;  // the query's training tail, if it is one
    uint32_t sid = 0;

    if (i < R.count[cur]) {
        path = R.q_path[cur][i];
        if (kCache) tslot = R.train_slot[path];
        if (!kOne) sid = R.path_scene[path];
        const SceneRec &S = R.scenes[sid];
        const float4 o = R.q_o[cur][i], d = R.q_d[cur][i];
        const int ti = R.hit_tri[i];
        uint64_t key;
        uint32_t px, py;
        path_ident(S, wave_begin + path, pixel, key, px, py);
        pixel += S.pixel_base;
        // A training path's pixel takes the cache's value at the cache vertex,
        // as a rendering path's does; what its tail adds from there on (light
        // samples at that vertex and beyond, escapes after it) only trains the
        // cache and goes to the discard slot past the last pixel.
        const uint32_t image_pixel = pixel;
        if (kCache && tslot != 0xffffffffu &&
            (ti >= 0 ? depth >= R.cache_depth : depth > R.cache_depth))
            pixel = R.discard_pixel;
        const float4 beta4 = R.beta[path];
        float3 beta = make_float3(beta4.x, beta4.y, beta4.z);
        const bool after_specular = beta4.w != 0.f;  // the previous bounce was a specular one
        float3 add = make_float3(0.f, 0.f, 0.f);

        if (ti < 0) {
            // escape: constant environment (zero for the reference's area-light scenes)
            add = beta * S.sky;
            // the reference's infinite lights, seen by a camera ray or after a
            // specular bounce (PathIntegrator.cpp:84-92 and :194-198)
            if ((depth == 0 || after_specular) && S.inf_escape > 0.f) add = add + beta * S.inf_escape;
            if (kCache && tslot != 0xffffffffu && depth >= 2 && !is_black(add)) credit(R, tslot, depth - 1, add);
        } else if (depth <= S.max_depth) {
            const Tri tr = S.tris[ti];
            const uint32_t attr = tr.id.y;
            const uint32_t mat_id = attr & 0xffffu, light_id = attr >> 16;
            const Mat m = S.mats[mat_id < S.n_mats ? mat_id : 0];
            const float3 ng = normalize3(make_float3(tr.a.w, tr.b.w, tr.c.w));
            const float t = R.hit_t[i];
            const float3 dd = make_float3(d.x, d.y, d.z);
            const float3 p = make_float3(o.x + t * d.x, o.y + t * d.y, o.z + t * d.z);
            const float3 wo = normalize3(dd) * -1.f;
            // flat shading: the shading normal is the face normal
            const float3 W = ng;
            float3 U, V;
            onb_from_w(W, U, V);
            const float3 wo_l = make_float3(dot3(U, wo), dot3(V, wo), dot3(W, wo));

            // emission at depth 0 or right after a specular bounce
            // (PathIntegrator.cpp:126-128), one-sided (DiffuseAreaLight::Radiance,
            // DiffuseAreaLight.cpp:47-50)
            if ((depth == 0 || after_specular) && light_id != 0xffffu && light_id < S.n_lights &&
                dot3(W, wo) > 0.f) {
                const float3 e = beta * S.lights[light_id].emit;
                add = add + e;
                if (kCache && tslot != 0xffffffffu && depth >= 2) credit(R, tslot, depth - 1, e);
            }
            // RadianceContext::Albedo = the first hit's Material::Rho
            // (PathIntegrator.cpp:121): the reflectance; for the GGX conductor
            // its F0; for glass the sum over its two BxDFs (BSDF::Rho,
            // Core/Material/BSDF.cpp:123-139)
            if (depth == 0 && R.accum_albedo)
                add_pixel(R.accum_albedo, pixel,
                          m.kind == 1u ? m.f0 : (m.kind == 3u ? m.albedo + m.f0 : m.albedo));
            const bool specular = m.kind >= 2u;

            const bool at_cache = kCache && depth < S.max_depth && depth == R.cache_depth;
            // a training path with a short tail stops into the cache too; the
            // cache's answer there completes the targets of its records
            // (self-training), not its pixel
            const bool at_tail = kCache && depth < S.max_depth && R.train_tail && tslot != 0xffffffffu &&
                                 depth == R.cache_depth + R.train_tail;
            if (at_cache) {
                // the cache supplies the radiance leaving this vertex to the pixel
                query = true;
                write_features(qf, R, p, wo, W, m);
                qb = make_float4(beta.x, beta.y, beta.z, __uint_as_float(image_pixel));
            }
            if (at_tail) {
                query = true;
                qmeta = (tslot << 8) | depth;
                write_features(qf, R, p, wo, W, m);
                qb = make_float4(beta.x, beta.y, beta.z, __uint_as_float(R.discard_pixel));
            }
            if ((at_cache && tslot == 0xffffffffu) || at_tail) {
                // the path stops here
            } else if (depth < S.max_depth) {
                if (kCache && tslot != 0xffffffffu && depth >= 1) {
                    // training record of this vertex; its target fills in as the tail is traced
                    const uint32_t ri = atomicAdd(R.rec_count, 1u);
                    uint32_t stored = 0xffffffffu;
                    if (ri < R.rec_cap) {
                        float f[kMlpRaw];
                        write_features(f, R, p, wo, W, m);
#pragma unroll
                        for (int k = 0; k < kMlpRaw; k++) R.rec_feat[(size_t)ri * kMlpRaw + k] = f[k];
                        R.rec_beta[ri] = make_float4(beta.x, beta.y, beta.z, 0.f);
                        R.rec_tgt[3 * ri] = R.rec_tgt[3 * ri + 1] = R.rec_tgt[3 * ri + 2] = 0.f;
                        stored = ri;
                    }
                    R.rec_of[tslot * (R.depth_max + 1) + depth] = stored;
                }
                // next-event estimation toward every light but the one hit (a
                // specular BSDF's F is zero for every light direction); each
                // sample goes to the shadow queue as it is made
                for (uint32_t l = 0; l < S.n_lights && l < kMaxLights && !specular; l++) {
                    if (l == light_id) continue;
                    float4 so, sd;
                    float3 sc;
                    const bool ok = light_sample(S, l, key, depth, p, U, V, W, wo_l, m, beta, so, sd, sc);
                    const uint32_t s = push_slot(ok, R.sh_count);
                    if (ok) {
                        if (s < R.sh_capacity) {
                            R.s_o[s] = so;
                            R.s_d[s] = sd;
                            // bit 31 marks a light sample of the first vertex (Direct)
                            const uint32_t tag = (depth == 0 && R.accum_direct) ? 0x80000000u : 0u;
                            R.s_c[s] = make_float4(sc.x, sc.y, sc.z, __uint_as_float(pixel | tag));
                            if (!kOne) R.s_sid[s] = sid;
                            if (kCache)
                                R.s_meta[s] = tslot == 0xffffffffu ? 0xffffffffu : ((tslot << 8) | depth);
                        } else {
                            atomicOr(R.err, 16u);
                        }
                    }
                }

                if (continue_path(S, key, depth, m, specular, p, ng, U, V, W, wo_l, beta, no, nd)) {
                    cont = true;
                    R.beta[path] = make_float4(beta.x, beta.y, beta.z, specular ? 1.f : 0.f);
                }
            }
        }
        if (!is_black(add)) {
            add_pixel(R.accum, pixel, add);
            // what the first vertex adds is RadianceContext::Direct (PathIntegrator.cpp:102)
            if (depth == 0 && R.accum_direct) add_pixel(R.accum_direct, pixel, add);
        }
    }

    const uint32_t slot = push_slot(cont, &R.count[nxt]);
    if (cont) {
        if (slot < R.capacity) {
            R.q_o[nxt][slot] = no;
            R.q_d[nxt][slot] = nd;
            R.q_path[nxt][slot] = path;
        } else {
            atomicOr(R.err, 8u);
        }
    }
    if (kCache) {
        const uint32_t q = push_slot(query, R.qry_count);
        if (query) {
            if (q < R.capacity) {
#pragma unroll
                for (int k = 0; k < kMlpRaw; k++) R.qry_feat[(size_t)q * kMlpRaw + k] = qf[k];
                R.qry_beta[q] = qb;
                R.qry_meta[q] = qmeta;
            } else {
                atomicOr(R.err, 32u);
            }
        }
    }
}

// pixel += throughput * max(cache output, 0) for every cache query of the
// wave; a training tail's answer goes to its path's records instead (its
// pixel is the discard slot)
__global__ void k_cache_apply(RenderDev R)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= *R.qry_count || i >= R.capacity) return;
    const float4 b = R.qry_beta[i];
    const float3 y = make_float3(fmaxf(R.qry_out[3 * i], 0.f), fmaxf(R.qry_out[3 * i + 1], 0.f),
                                 fmaxf(R.qry_out[3 * i + 2], 0.f));
    const float3 c = make_float3(b.x * y.x, b.y * y.y, b.z * y.z);
    add_pixel(R.accum, __float_as_uint(b.w), c);
    if (R.train_tail) {
        const uint32_t meta = R.qry_meta[i];
        if (meta != 0xffffffffu) credit(R, meta >> 8, meta & 0xffu, c);
    }
}

template <bool kStats>
__global__ void __launch_bounds__(256, 4) k_shadow(RenderDev R)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    const bool live = i < *R.sh_count;
    if (!kStats && !live) return;
    uint32_t nn = 0, nt = 0;
    int best = -2;
    if (live) {
        const float4 o = R.s_o[i], d = R.s_d[i];
        const SceneRec &S = R.scenes[R.n_scenes > 1u ? R.s_sid[i] : 0u];
        float bt, bu, bv;
        trace_one<true, kStats>(S.nodes, S.tris, S.n_nodes, S.n_tris, R.min_dir, o, d, best, bt, bu, bv, R.err, nn, nt);
    }
    if (kStats) count_work(R, 3, live, nn, nt);
    if (live && best == -1) shadow_unoccluded(R, i);
}

// ---------------------------------------------------------------------------
// Persistent forms of k_extend and k_shadow over trace_persistent, so the
// incoherent bounce and shadow rays do not leave lanes waiting on the longest
// ray of a warp. Rays of one warp may belong to different scenes of a batch;
// each lane traverses its own scene's tree. Seven blocks an SM (72 registers):
// measured on the 5.2 M-triangle field at 1920x1080, 4 samples, depth 12: six
// blocks 16.9 ms, seven 15.7, eight (spilling) 16.3; 18.5 with the previous
// traversal.
// ---------------------------------------------------------------------------
__device__ __forceinline__ void bind_scene(TraceScene &T, const SceneRec &S)
{
    T.nodes = S.nodes;
    T.tris = S.tris;
    T.n_nodes = S.n_nodes;
    T.n_tris = S.n_tris;
}

// kOne: a render of one scene, whose tree then stays in uniform registers
// instead of six registers a lane (and two dependent loads a ray).
template <bool kAnyHit, bool kOne>
__device__ __forceinline__ void wave_trace_dyn(const RenderDev &R, uint32_t n, uint32_t *next, int cur)
{
    __shared__ uint2 sstack[kShortStack * kStackColumns];  // launched with kStackColumns threads a block
    uint2 lstack[kMaxStack - kShortStack];
    const SplitStack stack{sstack + threadIdx.x, lstack};
    TraceScene scene{nullptr, nullptr, 0u, 0u};
    if (kOne) bind_scene(scene, R.scenes[0]);
    uint32_t id = 0;
    trace_persistent<kAnyHit, false, false, kRefillLanes>(
        stack, scene, n, plane_magic(n), next, R.err, nullptr,
        [&](uint32_t k, RayState &r, TraceScene &T) {
            id = k;
            if (!kOne) bind_scene(T, R.scenes[kAnyHit ? R.s_sid[id] : R.path_scene[R.q_path[cur][id]]]);
            if (kAnyHit) ray_init(r, R.s_o[id], R.s_d[id], T.n_nodes, R.min_dir);
            else ray_init(r, R.q_o[cur][id], R.q_d[cur][id], T.n_nodes, R.min_dir);
        },
        [&](const RayState &r) {
            if (kAnyHit) {
                if (r.best == -1) shadow_unoccluded(R, id);
            } else {
                R.hit_tri[id] = r.best;
                R.hit_t[id] = r.best >= 0 ? r.tcur : __int_as_float(0x7f800000);
            }
        });
}

// The shadow rays of depth d and the extension rays of depth d + 1 in one
// persistent launch: both come from k_shade at depth d and neither reads
// what the other writes (shadow rays add to the pixel sums and training
// targets, extension rays write hit records), so one traversal loop
// (trace_persistent<kMixed>) takes the extension rays first, then the shadow rays:
// twice the rays in flight and one launch tail instead of two. `cur` is the
// queue the extension rays are in.
template <bool kOne>
__global__ void __launch_bounds__(kStackColumns, 7) k_trace_mixed(RenderDev R, int cur, uint32_t *next)
{
    __shared__ uint2 sstack[kShortStack * kStackColumns];  // launched with kStackColumns threads a block
    uint2 lstack[kMaxStack - kShortStack];
    const SplitStack stack{sstack + threadIdx.x, lstack};
    const uint32_t n_ext = min(R.count[cur], R.capacity), n_sh = min(*R.sh_count, R.sh_capacity);
    TraceScene scene{nullptr, nullptr, 0u, 0u};
    if (kOne) bind_scene(scene, R.scenes[0]);
    uint32_t id = 0;
    trace_persistent<false, false, true, kRefillLanes>(
        stack, scene, n_ext + n_sh, plane_magic(n_ext), next, R.err, nullptr,
        [&](uint32_t k, RayState &r, TraceScene &T) {
            const bool shadow = k >= n_ext;
            id = shadow ? k - n_ext : k;
            if (!kOne) bind_scene(T, R.scenes[shadow ? R.s_sid[id] : R.path_scene[R.q_path[cur][id]]]);
            if (shadow) ray_init(r, R.s_o[id], R.s_d[id], T.n_nodes, R.min_dir);
            else ray_init(r, R.q_o[cur][id], R.q_d[cur][id], T.n_nodes, R.min_dir);
            r.any = shadow;
        },
        [&](const RayState &r) {
            if (r.any) {
                if (r.best == -1) shadow_unoccluded(R, id);
            } else {
                R.hit_tri[id] = r.best;
                R.hit_t[id] = r.best >= 0 ? r.tcur : __int_as_float(0x7f800000);
            }
        });
}

template <bool kOne>
__global__ void __launch_bounds__(kStackColumns, 7) k_extend_dyn(RenderDev R, int cur, uint32_t *next)
{
    wave_trace_dyn<false, kOne>(R, min(R.count[cur], R.capacity), next, cur);
}

template <bool kOne>
__global__ void __launch_bounds__(kStackColumns, 7) k_shadow_dyn(RenderDev R, uint32_t *next)
{
    wave_trace_dyn<true, kOne>(R, min(*R.sh_count, R.sh_capacity), next, 0);
}

// ---------------------------------------------------------------------------
// The whole render as one persistent launch. Each warp owns kPathSlots paths,
// twice its lanes, and three lists of its own: rays to trace (closest-hit and
// shadow rays), paths whose ray has hit and that wait to be shaded, and the
// lanes' rays in flight. Idle lanes take rays from the first list; when it
// runs short, 32 waiting paths are shaded together: each adds what its vertex
// emits, appends a shadow ray per light sample and its next ray, and a path
// that ended is replaced by a new one, of any scene of the batch, from a
// device counter. With two paths a lane there are always 32 to shade or a ray
// for every lane, so both the traversal loop and the shading code run with
// full warps, and no warp waits for another.
//
// A ray in flight is parked in shared memory while its warp shades, so the
// kernel fits 80 to 96 registers. Measured on a B200, 12 scenes of up to 128 K
// triangles / the 5.2 M-triangle field at 1920x1080x4: one path a lane, shading
// once three quarters of the warp had stopped tracing, 19.4 / 29.6 ms; with
// the pool 11.9 / 19.8 (spilling at 96 registers), 9.2 / 17.1 parked, 9.4 /
// 15.9 at 80 registers; 128 paths a warp gain nothing. The wavefront takes
// 10.2 / 17.6.
//
// The sample sequence, the shading code (light_sample, continue_path) and the
// traversal are the wavefront's, so every path is the wavefront path of the
// same index and the images agree up to the order of the float additions into
// each pixel. Plain renders only: no radiance cache, no Direct / Albedo
// outputs, no work counters.
//
// kOrdered, for renders with one sample a pixel: a pixel then has one path, and
// its sum the path's own order: what vertex d emits, its light samples light
// by light, what vertex d + 1 emits. So two calls give the same bits, as a
// wavefront does that adds to a pixel once a launch. A path is shaded when all
// its rays are back, and adds its light samples then instead of as they
// arrive. Measured on a B200, added as they arrive / ordered: box scene 64x64
// at 1 sample 124 / 135 us, 512x512 281 / 327, 5.2 M-triangle field 960x540
// 1606 / 1899; as a wavefront 227, 348 and 2303. With eight lights the waiting
// costs more: box 256x256 561 us ordered, 362 as a wavefront.
// ---------------------------------------------------------------------------
constexpr int kPersistThreads = 128;
constexpr uint32_t kPathSlots = 64;
constexpr int kNewPath = -3;  // hit of a slot that waits for a path
constexpr int kEndedPath = -4;  // hit of a slot whose path ended with shadow rays under way (kOrdered)

// One warp's part of the pool, in device memory: the paths, then a stack of
// rays. A shading step runs when fewer than 32 rays are left and appends at
// most 32 x (1 + lights).
struct WarpPool {
    float4 *beta;          // throughput, w = the previous bounce was specular
    uint4 *id;             // sample key (x, y), pixel, scene | depth << 16
    float4 *hit_o, *hit_d; // the finished ray: origin, t; direction, triangle
    float4 *ray_o, *ray_d, *ray_c;  // ray; shadow rays: contribution, pixel
    uint32_t *ray_m;       // scene | slot << 16; bit 31: a shadow ray (kOrdered: | light << 24)
    float4 *lit;           // kOrdered: the contributions of a slot's shadow rays, a light each
};
__host__ __device__ constexpr size_t pool_bytes(uint32_t lights, bool ordered)
{
    return kPathSlots * 64u + 32u * (2u + lights) * 52u + (ordered ? kPathSlots * lights * 16u : 0u);
}
__device__ __forceinline__ WarpPool warp_pool(unsigned char *base, uint32_t lights)
{
    const uint32_t rays = 32u * (2u + lights);
    float4 *f = reinterpret_cast<float4 *>(base);
    WarpPool P;
    P.beta = f;
    P.id = reinterpret_cast<uint4 *>(f + kPathSlots);
    P.hit_o = f + 2 * kPathSlots;
    P.hit_d = f + 3 * kPathSlots;
    P.ray_o = f + 4 * kPathSlots;
    P.ray_d = P.ray_o + rays;
    P.ray_c = P.ray_d + rays;
    P.ray_m = reinterpret_cast<uint32_t *>(P.ray_c + rays);
    P.lit = reinterpret_cast<float4 *>(P.ray_m + rays);
    return P;
}

// A lane's ray in flight, kept in shared memory while its warp shades: the
// shading code needs the registers.
constexpr int kParkedWords = 20;
struct Parked {
    uint32_t w[kParkedWords][kPersistThreads];
};
__device__ __forceinline__ void park(Parked &s, const RayState &r)
{
    const uint32_t v[kParkedWords] = {
        __float_as_uint(r.ox), __float_as_uint(r.oy), __float_as_uint(r.oz), __float_as_uint(r.dx), __float_as_uint(r.dy),
        __float_as_uint(r.dz), __float_as_uint(r.tmin), __float_as_uint(r.tcur), r.ng_base, r.ng_hits, r.tg_base,
        r.tg_slots, r.tg_hits, r.tq_base, r.tq_slots, r.tq_hits, r.budget, (uint32_t)r.sp, (uint32_t)r.best, r.any};
#pragma unroll
    for (int k = 0; k < kParkedWords; k++) s.w[k][threadIdx.x] = v[k];
}
__device__ __forceinline__ void unpark(const Parked &s, RayState &r, float min_dir)
{
    auto u = [&](int k) { return s.w[k][threadIdx.x]; };
    auto f = [&](int k) { return __uint_as_float(s.w[k][threadIdx.x]); };
    ray_init(r, make_float4(f(0), f(1), f(2), f(6)), make_float4(f(3), f(4), f(5), f(7)), 0u, min_dir);
    r.ng_base = u(8);
    r.ng_hits = u(9);
    r.tg_base = u(10);
    r.tg_slots = u(11);
    r.tg_hits = u(12);
    r.tq_base = u(13);
    r.tq_slots = u(14);
    r.tq_hits = u(15);
    r.budget = u(16);
    r.sp = (int)u(17);
    r.best = (int)u(18);
    r.any = u(19) != 0u;
}

template <bool kOne, bool kOrdered>
__global__ void __launch_bounds__(kPersistThreads, kOne ? 6 : 5)
    k_render_persistent(RenderDev R, uint64_t total, unsigned long long *next, unsigned char *pool, uint32_t lights)
{
    constexpr uint32_t kFull = 0xffffffffu;
    __shared__ uint2 sstack[kShortStack * kStackColumns];
    __shared__ float4 s_shadow[kPersistThreads];               // the lane's shadow ray: contribution, pixel
    __shared__ uint8_t s_wait[kPersistThreads / 32][kPathSlots];  // slots of the paths to shade
    __shared__ Parked s_park;
    // kOrdered: a slot's rays under way, and which of its light samples are lit
    __shared__ uint32_t s_pending[kOrdered ? kPersistThreads / 32 : 1][kPathSlots];
    __shared__ uint32_t s_lit[kOrdered ? kPersistThreads / 32 : 1][kPathSlots];
    uint2 lstack[kMaxStack - kShortStack];
    const SplitStack stack{sstack + threadIdx.x, lstack};
    const uint32_t lane = threadIdx.x & 31u, below = (1u << lane) - 1u, magic = plane_magic(R.n_scenes);
    uint8_t *wait = s_wait[threadIdx.x >> 5];
    uint32_t *pending = s_pending[kOrdered ? threadIdx.x >> 5 : 0], *lit_mask = s_lit[kOrdered ? threadIdx.x >> 5 : 0];
    const WarpPool P = warp_pool(
        pool + (size_t)(blockIdx.x * (kPersistThreads / 32) + (threadIdx.x >> 5)) * pool_bytes(lights, kOrdered), lights);
    for (uint32_t k = lane; k < kPathSlots; k += 32u) {
        wait[k] = (uint8_t)k;
        P.hit_d[k] = make_float4(0.f, 0.f, 0.f, __int_as_float(kNewPath));
        if (kOrdered) pending[k] = lit_mask[k] = 0u;
    }
    __syncwarp();
    uint32_t n_wait = kPathSlots, n_rays = 0;  // warp-uniform, as is exhausted
    bool exhausted = false;
    TraceScene scene{nullptr, nullptr, 0u, 0u};
    if (kOne) bind_scene(scene, R.scenes[0]);
    RayState r;
    ray_init(r, make_float4(0.f, 0.f, 0.f, 0.f), make_float4(0.f, 0.f, 1.f, 0.f), 0u, 1.f);
    ray_stop(r);
    r.any = false;
    bool has = false;
    uint32_t meta = 0;  // of the lane's ray

    // Appends a ray for every lane of the warp that wants one.
    auto push = [&](bool want, float4 o, float4 d, float4 c, uint32_t m) {
        const uint32_t lanes = __ballot_sync(kFull, want);
        if (want) {
            const uint32_t at = n_rays + __popc(lanes & below);
            P.ray_o[at] = o;
            P.ray_d[at] = d;
            if (!kOrdered && m >> 31) P.ray_c[at] = c;
            P.ray_m[at] = m;
        }
        n_rays += __popc(lanes);
    };

    // Shades the last min(32, n_wait) waiting paths.
    auto shade = [&]() {
        const uint32_t m = min(32u, n_wait);
        n_wait -= m;
        bool live = lane < m, cont = false, lit = false;
        const uint32_t slot = live ? wait[n_wait + lane] : 0u;
        float4 no = make_float4(0.f, 0.f, 0.f, 0.f), nd = no;
        float3 beta = make_float3(1.f, 1.f, 1.f);
        uint64_t key = 0;
        uint32_t pixel = 0, sid = 0, depth = 0, light_id = 0xffffu, n_lights = 0;
        Mat mat;
        float3 p, W = make_float3(0.f, 0.f, 1.f), U = W, V = W, wo_l = W;
        bool specular = false;
        int ti = kNewPath;
        uint32_t rays = 0;  // kOrdered: the slot's new rays
        if (live) {
            const float4 hd = P.hit_d[slot];
            ti = __float_as_int(hd.w);
            if (ti != kNewPath) {
                const float4 ho = P.hit_o[slot], b4 = P.beta[slot];
                const uint4 id = P.id[slot];
                key = (uint64_t)id.x | (uint64_t)id.y << 32;
                pixel = id.z;
                sid = kOne ? 0u : id.w & 0xffffu;
                depth = id.w >> 16;
                beta = make_float3(b4.x, b4.y, b4.z);
                const bool after_specular = b4.w != 0.f;
                const SceneRec &S = R.scenes[sid];
                if (kOrdered) {  // the vertex before this one
                    for (uint32_t l = 0, lit_of = lit_mask[slot]; lit_of >> l; l++) {
                        if (!(lit_of >> l & 1u)) continue;
                        const float4 c = P.lit[slot * lights + l];
                        add_pixel(R.accum, pixel, make_float3(c.x, c.y, c.z));
                    }
                    lit_mask[slot] = 0u;
                }
                float3 add = make_float3(0.f, 0.f, 0.f);
                if (ti == -1) {
                    add = beta * S.sky;
                    if ((depth == 0 || after_specular) && S.inf_escape > 0.f) add = add + beta * S.inf_escape;
                } else if (ti >= 0 && depth <= S.max_depth) {
                    const Tri tr = S.tris[ti];
                    const uint32_t mat_id = tr.id.y & 0xffffu;
                    light_id = tr.id.y >> 16;
                    mat = S.mats[mat_id < S.n_mats ? mat_id : 0];
                    W = normalize3(make_float3(tr.a.w, tr.b.w, tr.c.w));
                    const float t = ho.w;
                    p = make_float3(ho.x + t * hd.x, ho.y + t * hd.y, ho.z + t * hd.z);
                    const float3 wo = normalize3(make_float3(hd.x, hd.y, hd.z)) * -1.f;
                    onb_from_w(W, U, V);
                    wo_l = make_float3(dot3(U, wo), dot3(V, wo), dot3(W, wo));
                    if ((depth == 0 || after_specular) && light_id != 0xffffu && light_id < S.n_lights &&
                        dot3(W, wo) > 0.f)
                        add = add + beta * S.lights[light_id].emit;
                    if (depth < S.max_depth) {
                        specular = mat.kind >= 2u;
                        lit = !specular;
                        n_lights = min(S.n_lights, kMaxLights);
                        cont = true;
                    }
                }
                if (!is_black(add)) add_pixel(R.accum, pixel, add);
            }
        }
        for (uint32_t l = 0; __any_sync(kFull, lit && l < n_lights); l++) {
            float4 so = no, sd = no;
            float3 c = make_float3(0.f, 0.f, 0.f);
            const bool ok = lit && l < n_lights && l != light_id &&
                            light_sample(R.scenes[sid], l, key, depth, p, U, V, W, wo_l, mat, beta, so, sd, c);
            const float4 cp = make_float4(c.x, c.y, c.z, __uint_as_float(pixel));
            if (kOrdered && ok) {
                P.lit[slot * lights + l] = cp;
                rays++;
            }
            push(ok, so, sd, cp, 0x80000000u | sid | (kOrdered ? slot << 16 | l << 24 : 0u));
        }
        if (cont)
            cont = continue_path(R.scenes[sid], key, depth, mat, specular, p, W, U, V, W, wo_l, beta, no, nd);
        float flag = specular ? 1.f : 0.f;
        depth++;
        // ended paths (and slots that had none) take new ones
        // (kOrdered: once their last light samples are added)
        const bool ended = live && !cont, stay = kOrdered && ended && rays != 0u;
        if (stay) P.hit_d[slot].w = __int_as_float(kEndedPath);
        const uint32_t need = __ballot_sync(kFull, ended && !stay);
        if (need && !exhausted) {
            unsigned long long base = 0;
            if (lane == 0u) base = atomicAdd(next, (unsigned long long)__popc(need));
            base = __shfl_sync(kFull, base, 0);
            exhausted = base + __popc(need) >= total;
            const uint64_t g = base + __popc(need & below);
            if (ended && !stay && g < total) {
                sid = kOne ? 0u : scene_of(R, g);
                const SceneRec &S = R.scenes[sid];
                first_ray(S, g, pixel, key, no, nd);
                pixel += S.pixel_base;
                beta = make_float3(1.f, 1.f, 1.f);
                flag = 0.f;
                depth = 0;
                cont = true;
            }
        }
        if (cont) {
            P.beta[slot] = make_float4(beta.x, beta.y, beta.z, flag);
            P.id[slot] = make_uint4((uint32_t)key, (uint32_t)(key >> 32), pixel, sid | depth << 16);
        }
        if (kOrdered && live) pending[slot] = rays + (cont ? 1u : 0u);
        push(cont, no, nd, no, sid | slot << 16);
        __syncwarp();
    };

    while (true) {
        const uint32_t idle = __ballot_sync(kFull, r.tg_hits == 0u && !ray_has_nodes(r));
        if (__popc(idle) >= kRefillLanes || idle == kFull) {
            // results of the finished rays
            const bool mine = (idle >> lane) & 1u, done = mine && has, closest = done && !(meta >> 31);
            const uint32_t slot = meta >> 16 & (kPathSlots - 1u);
            if (closest) {
                P.hit_o[slot] = make_float4(r.ox, r.oy, r.oz, r.tcur);
                P.hit_d[slot] = make_float4(r.dx, r.dy, r.dz, __int_as_float(r.best));
            } else if (done && r.best == -1) {
                if (kOrdered) {
                    atomicOr(&lit_mask[slot], 1u << (meta >> 24 & 7u));
                } else {
                    const float4 c = s_shadow[threadIdx.x];
                    add_pixel(R.accum, __float_as_uint(c.w), make_float3(c.x, c.y, c.z));
                }
            }
            // kOrdered: the last of a slot's rays to finish
            const bool to_shade = kOrdered ? done && atomicSub(&pending[slot], 1u) == 1u : closest;
            const uint32_t hits = __ballot_sync(kFull, to_shade);
            if (to_shade) wait[n_wait + __popc(hits & below)] = (uint8_t)slot;
            if (mine) has = false;
            n_wait += __popc(hits);
            __syncwarp();
            // rays for the idle lanes: shade while they run short, with full
            // warps unless few rays are in flight
            const uint32_t want = __popc(idle);
            if (n_rays < want && n_wait > 0u && (n_wait >= 32u || want > 24u)) {
                park(s_park, r);
                __syncwarp();
                do shade();
                while (n_rays < want && n_wait > 0u && (n_wait >= 32u || want > 24u));
                unpark(s_park, r, R.min_dir);
                if (!kOne) bind_scene(scene, R.scenes[meta & 0xffffu]);
            }
            const uint32_t rank = __popc(idle & below), take = min(want, n_rays);
            if (mine && rank < take) {
                const uint32_t at = n_rays - 1u - rank;
                const float4 o = P.ray_o[at], d = P.ray_d[at];
                meta = P.ray_m[at];
                if (!kOne) bind_scene(scene, R.scenes[meta & 0xffffu]);
                ray_init(r, o, d, scene.n_nodes, R.min_dir);
                r.any = (meta >> 31) != 0u;
                if (!kOrdered && r.any) s_shadow[threadIdx.x] = P.ray_c[at];
                has = true;
            }
            n_rays -= take;
            if (take == 0u && idle == kFull) break;  // no ray, and so no path left to shade
        }
        __syncwarp();
        if (r.tq_hits == 0u && ray_has_nodes(r)) ray_node(r, stack, scene.nodes, scene.n_nodes, magic, R.err);
        while (true) {
            const uint32_t tri = __ballot_sync(kFull, r.tg_hits != 0u);
            const uint32_t node = __ballot_sync(kFull, r.tq_hits == 0u && ray_has_nodes(r));
            if (tri == 0u || (__popc(tri) < kTriLanes && __popc(node) >= kNodeLanes)) break;
            if (r.tg_hits) ray_tri<false, false, false, false, true>(r, scene.tris, scene.n_tris, R.err);
        }
    }
}

__global__ void k_resolve(const float4 *__restrict__ accum, uint32_t wh, float scale, float *__restrict__ out)
{
    const uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= wh) return;
    const float4 a = accum[p];
    out[3 * p] = a.x * scale;
    out[3 * p + 1] = a.y * scale;
    out[3 * p + 2] = a.z * scale;
}

__global__ void k_tri_attr(Tri *__restrict__ tris, uint32_t n, const uint32_t *__restrict__ mat_ids,
                           const uint32_t *__restrict__ light_of_prim)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const uint32_t p = tris[i].id.x;
    tris[i].id.y = (mat_ids ? (mat_ids[p] & 0xffffu) : 0u) | (light_of_prim[p] << 16);
}

__global__ void k_light_of_prim(uint32_t *lop, uint32_t n_prims, const uint2 *range, uint32_t n_lights)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n_prims) return;
    uint32_t id = 0xffffu;
    for (uint32_t l = 0; l < n_lights; l++)
        if (i - range[l].x < range[l].y) id = l;
    lop[i] = id;
}

__global__ void k_tri_area(const float *__restrict__ pos, const uint32_t *__restrict__ idx, uint32_t first,
                           uint32_t count, float *__restrict__ area)
{
    const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= count) return;
    const uint32_t *tv = idx + 3ull * (first + k);
    const float *a = pos + 3ull * tv[0], *b = pos + 3ull * tv[1], *c = pos + 3ull * tv[2];
    const float3 e1 = make_float3(b[0] - a[0], b[1] - a[1], b[2] - a[2]);
    const float3 e2 = make_float3(c[0] - a[0], c[1] - a[1], c[2] - a[2]);
    const float3 n = cross3(e1, e2);
    area[k] = sqrtf(dot3(n, n)) * 0.5f;
}

inline uint32_t blocks_for(uint64_t n, uint32_t t) { return (uint32_t)((n + t - 1) / t); }

// Grid of a persistent kernel of 128-thread blocks over at most n items.
inline uint32_t persistent_blocks(uint64_t n)
{
    const int sms = current_sm_count();
    const uint32_t b = blocks_for(n, 128);
    const uint32_t cap = (uint32_t)sms * 16u;
    return b < 1u ? 1u : (b < cap ? b : cap);
}

}  // namespace

cudaError_t triangle_areas(const float *pos, const uint32_t *idx, uint32_t first, uint32_t count, float *area,
                           cudaStream_t st)
{
    if (count == 0) return cudaSuccess;
    k_tri_area<<<blocks_for(count, 256), 256, 0, st>>>(pos, idx, first, count, area);
    return cudaGetLastError();
}

cudaError_t build_tri_attr(Tri *tris, uint32_t n_tris, const uint32_t *mat_ids,
                           const uint2 *light_range, uint32_t n_lights, uint32_t *light_of_prim,
                           cudaStream_t st)
{
    k_light_of_prim<<<blocks_for(n_tris, 256), 256, 0, st>>>(light_of_prim, n_tris, light_range, n_lights);
    k_tri_attr<<<blocks_for(n_tris, 256), 256, 0, st>>>(tris, n_tris, mat_ids, light_of_prim);
    return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// Hash-grid radiance cache: a non-learned stand-in for the network, the
// baseline the learned cache is measured against. A cell is a voxel of the
// scene's bounding box (256 per axis) crossed with the normal's dominant
// axis and sign (6) and the octant of the outgoing direction (8); it holds
// the running mean of the training records that fell in it. Lookup is
// open addressing over kHashCacheCells cells, 8 probes; a query that finds
// no filled cell answers 0.
// ---------------------------------------------------------------------------
__device__ __forceinline__ unsigned long long hc_key(const float *f)
{
    const uint32_t x = (uint32_t)fminf(fmaxf(f[0] * 256.f, 0.f), 255.f);
    const uint32_t y = (uint32_t)fminf(fmaxf(f[1] * 256.f, 0.f), 255.f);
    const uint32_t z = (uint32_t)fminf(fmaxf(f[2] * 256.f, 0.f), 255.f);
    const float ax = fabsf(f[6]), ay = fabsf(f[7]), az = fabsf(f[8]);
    const uint32_t axis = ax >= ay && ax >= az ? 0u : (ay >= az ? 1u : 2u);
    const uint32_t nsign = (axis == 0u ? f[6] : axis == 1u ? f[7] : f[8]) < 0.f ? 1u : 0u;
    const uint32_t oct = (f[3] < 0.f ? 1u : 0u) | (f[4] < 0.f ? 2u : 0u) | (f[5] < 0.f ? 4u : 0u);
    return (unsigned long long)x | ((unsigned long long)y << 8) | ((unsigned long long)z << 16) |
           ((unsigned long long)(axis * 2u + nsign) << 24) | ((unsigned long long)oct << 27);
}

__device__ __forceinline__ uint32_t hc_slot(unsigned long long key, uint32_t mask)
{
    unsigned long long h = key * 0x9E3779B97F4A7C15ull;
    h ^= h >> 29;
    return (uint32_t)h & mask;
}

__global__ void k_hc_update(RenderDev R)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= min(*R.rec_count, R.rec_cap)) return;
    const float *f = R.rec_feat + (size_t)i * kMlpRaw;
    const unsigned long long key = hc_key(f) + 1ull;
    const uint32_t mask = kHashCacheCells - 1u;
    uint32_t s = hc_slot(key, mask);
    for (int probe = 0; probe < 8; probe++, s = (s + 1u) & mask) {
        const unsigned long long prev = atomicCAS(R.hc_keys + s, 0ull, key);
        if (prev == 0ull || prev == key) {
            float *v = reinterpret_cast<float *>(R.hc_vals + s);
            atomicAdd(v, fmaxf(R.rec_tgt[3 * i], 0.f));
            atomicAdd(v + 1, fmaxf(R.rec_tgt[3 * i + 1], 0.f));
            atomicAdd(v + 2, fmaxf(R.rec_tgt[3 * i + 2], 0.f));
            atomicAdd(v + 3, 1.f);
            return;
        }
    }
    // all 8 probed cells hold other keys: the record is dropped (and counted)
    atomicAdd(R.hc_dropped, 1u);
}

__global__ void k_hc_query(RenderDev R, uint32_t cap)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= *R.qry_count || i >= cap) return;
    const float *f = R.qry_feat + (size_t)i * kMlpRaw;
    const unsigned long long key = hc_key(f) + 1ull;
    const uint32_t mask = kHashCacheCells - 1u;
    uint32_t s = hc_slot(key, mask);
    float3 y = make_float3(0.f, 0.f, 0.f);
    for (int probe = 0; probe < 8; probe++, s = (s + 1u) & mask) {
        const unsigned long long k = R.hc_keys[s];
        if (k == 0ull) break;
        if (k == key) {
            const float4 v = R.hc_vals[s];
            if (v.w > 0.f) y = make_float3(v.x / v.w, v.y / v.w, v.z / v.w);
            break;
        }
    }
    R.qry_out[3 * i] = y.x;
    R.qry_out[3 * i + 1] = y.y;
    R.qry_out[3 * i + 2] = y.z;
}

cudaError_t hash_cache_update(const RenderDev &R, cudaStream_t st)
{
    k_hc_update<<<blocks_for(R.rec_cap, 256), 256, 0, st>>>(R);
    return cudaGetLastError();
}

cudaError_t render_wave(const RenderDev &R, uint32_t n_paths, uint64_t wave_begin, cudaStream_t st,
                        const MlpDev *cache, uint32_t block)
{
    const uint32_t T = block;
    cudaError_t e;
    if ((e = cudaMemsetAsync(R.count, 0, 2 * sizeof(uint32_t), st)) != cudaSuccess) return e;
    if (R.cache_depth) {
        if ((e = cudaMemsetAsync(R.train_count, 0, sizeof(uint32_t), st)) != cudaSuccess) return e;
        if ((e = cudaMemsetAsync(R.qry_count, 0, sizeof(uint32_t), st)) != cudaSuccess) return e;
        if ((e = cudaMemsetAsync(R.rec_of, 0xff, sizeof(uint32_t) * R.train_cap * (R.depth_max + 1), st)) !=
            cudaSuccess)
            return e;
    }
    k_camera<<<blocks_for(n_paths, 128), 128, 0, st>>>(R, n_paths, wave_begin);  // also sets count[0]
    int cur = 0;
    // with short training tails every path has stopped by the tail vertex
    const uint32_t tail = R.cache_depth + R.train_tail;
    const uint32_t last = (R.cache_depth && R.train_tail && cache) ? std::min(R.depth_max, tail) : R.depth_max;
    // persistent traversal: the shadow rays of depth d and the extension rays
    // of depth d + 1 go in one launch (k_trace_mixed)
    const bool merge = R.persistent && !R.stats, one = R.n_scenes == 1u;
    bool traced = false;  // this depth's extension rays were traced with the previous depth's shadow rays
    for (uint32_t depth = 0; depth <= last; depth++) {
        if (!traced) {
            if ((e = cudaMemsetAsync(R.count + (cur ^ 1), 0, sizeof(uint32_t), st)) != cudaSuccess) return e;
            if ((e = cudaMemsetAsync(R.sh_count, 0, sizeof(uint32_t), st)) != cudaSuccess) return e;
            if (R.stats) {
                k_extend<true><<<blocks_for(n_paths, T), T, 0, st>>>(R, cur);
            } else if (!R.persistent) {
                k_extend<false><<<blocks_for(n_paths, T), T, 0, st>>>(R, cur);
            } else {
                if ((e = cudaMemsetAsync(R.count + 6, 0, sizeof(uint32_t), st)) != cudaSuccess) return e;
                (one ? k_extend_dyn<true> : k_extend_dyn<false>)<<<persistent_blocks(n_paths), kStackColumns, 0, st>>>(
                    R, cur, R.count + 6);
            }
        }
        traced = false;
        (R.cache_depth ? (one ? k_shade<true, true> : k_shade<true, false>)
                       : (one ? k_shade<false, true> : k_shade<false, false>))<<<blocks_for(n_paths, T), T, 0, st>>>(
            R, cur, depth, wave_begin);
        if (R.cache_depth && cache && (depth == R.cache_depth || (R.train_tail && depth == tail))) {
            if (R.hc_keys)
                k_hc_query<<<blocks_for(n_paths, 256), 256, 0, st>>>(R, R.capacity);
            else if ((e = mlp_infer(*cache, R.qry_feat, n_paths, R.qry_out, st, R.qry_count)) != cudaSuccess)
                return e;
            k_cache_apply<<<blocks_for(n_paths, 128), 128, 0, st>>>(R);
            if ((e = cudaMemsetAsync(R.qry_count, 0, sizeof(uint32_t), st)) != cudaSuccess) return e;
        }
        if (depth < last && merge) {
            if ((e = cudaMemsetAsync(R.count + 6, 0, sizeof(uint32_t), st)) != cudaSuccess) return e;
            (one ? k_trace_mixed<true> : k_trace_mixed<false>)<<<persistent_blocks((uint64_t)n_paths + R.sh_capacity),
                                                                 kStackColumns, 0, st>>>(R, cur ^ 1, R.count + 6);
            // the queues the next k_shade appends to, now that they are consumed
            if ((e = cudaMemsetAsync(R.count + cur, 0, sizeof(uint32_t), st)) != cudaSuccess) return e;
            if ((e = cudaMemsetAsync(R.sh_count, 0, sizeof(uint32_t), st)) != cudaSuccess) return e;
            traced = true;
        } else if (depth < last) {
            if (R.stats) {
                k_shadow<true><<<blocks_for((uint64_t)R.sh_capacity, T), T, 0, st>>>(R);
            } else if (!R.persistent) {
                k_shadow<false><<<blocks_for((uint64_t)R.sh_capacity, T), T, 0, st>>>(R);
            } else {
                if ((e = cudaMemsetAsync(R.count + 7, 0, sizeof(uint32_t), st)) != cudaSuccess) return e;
                (one ? k_shadow_dyn<true> : k_shadow_dyn<false>)<<<persistent_blocks(R.sh_capacity), kStackColumns, 0,
                                                                   st>>>(R, R.count + 7);
            }
        }
        if ((e = cudaGetLastError()) != cudaSuccess) return e;
        cur ^= 1;
    }
    return cudaSuccess;
}

// The one-launch renderer's form for a render.
using PersistentKernel = void (*)(RenderDev, uint64_t, unsigned long long *, unsigned char *, uint32_t);
static PersistentKernel persistent_kernel(bool one, bool ordered)
{
    if (ordered) return one ? k_render_persistent<true, true> : k_render_persistent<false, true>;
    return one ? k_render_persistent<true, false> : k_render_persistent<false, false>;
}

// Its blocks on the current device, at most.
static cudaError_t persistent_grid(uint64_t total, PersistentKernel kernel, uint32_t &blocks)
{
    int per_sm = 0;
    const cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kPersistThreads, 0);
    if (e != cudaSuccess) return e;
    // small renders: a path a lane rather than two, on more SMs
    const uint64_t want = (total + kPersistThreads - 1) / kPersistThreads;
    const uint64_t cap = (uint64_t)current_sm_count() * (uint64_t)(per_sm > 0 ? per_sm : 1);
    blocks = (uint32_t)(want < cap ? (want > 0 ? want : 1) : cap);
    return cudaSuccess;
}

cudaError_t render_persistent_bytes(const RenderDev &R, uint64_t total, uint32_t lights, bool ordered, size_t &bytes)
{
    uint32_t blocks = 0;
    const cudaError_t e = persistent_grid(total, persistent_kernel(R.n_scenes == 1u, ordered), blocks);
    bytes = (size_t)blocks * (kPersistThreads / 32) * pool_bytes(lights, ordered);
    return e;
}

cudaError_t render_persistent(const RenderDev &R, uint64_t total, uint32_t lights, bool ordered,
                              unsigned long long *next, unsigned char *pool, cudaStream_t st)
{
    cudaError_t e = cudaMemsetAsync(next, 0, sizeof(unsigned long long), st);
    if (e != cudaSuccess) return e;
    const PersistentKernel kernel = persistent_kernel(R.n_scenes == 1u, ordered);
    uint32_t blocks = 0;
    if ((e = persistent_grid(total, kernel, blocks)) != cudaSuccess) return e;
    kernel<<<blocks, kPersistThreads, 0, st>>>(R, total, next, pool, lights);
    return cudaGetLastError();
}

cudaError_t render_resolve(const float4 *accum, uint32_t wh, float scale, float *out, cudaStream_t st)
{
    k_resolve<<<blocks_for(wh, 256), 256, 0, st>>>(accum, wh, scale, out);
    return cudaGetLastError();
}

}  // namespace ilg
