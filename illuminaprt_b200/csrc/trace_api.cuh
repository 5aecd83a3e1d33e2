// Host-side launch interface of the traversal kernels.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

#include "bvh8.cuh"

namespace ilg {

struct SceneView {
    const Node8 *nodes;
    const Tri *tris;
    uint32_t n_nodes, n_tris;
    float min_dir;  // min_direction of the scene
};

cudaError_t launch_closest(const SceneView &s, const float4 *ro, const float4 *rd, uint32_t n, int32_t *prim,
                           float *t, float *u, float *v, uint32_t *err, unsigned long long *stats, cudaStream_t st);
cudaError_t launch_any(const SceneView &s, const float4 *ro, const float4 *rd, uint32_t n, uint8_t *occ,
                       uint32_t *err, cudaStream_t st);

// Queries that ignore the input triangles [skip_lo, skip_lo + skip_n).
cudaError_t launch_closest_skip(const SceneView &s, const float4 *ro, const float4 *rd, uint32_t n,
                                uint32_t skip_lo, uint32_t skip_n, int32_t *prim, float *t, float *u, float *v,
                                uint32_t *err, cudaStream_t st);
cudaError_t launch_any_skip(const SceneView &s, const float4 *ro, const float4 *rd, uint32_t n, uint32_t skip_lo,
                            uint32_t skip_n, uint8_t *occ, uint32_t *err, cudaStream_t st);

// Watertight test (persistent kernels); raw = three float4 vertices per
// triangle record, made by build_raw_tris from the input mesh.
cudaError_t launch_closest_wt(const SceneView &s, const float4 *raw, const float4 *ro, const float4 *rd, uint32_t n,
                              int32_t *prim, float *t, float *u, float *v, uint32_t *next, uint32_t *err,
                              cudaStream_t st);
cudaError_t launch_any_wt(const SceneView &s, const float4 *raw, const float4 *ro, const float4 *rd, uint32_t n,
                          uint8_t *occ, uint32_t *next, uint32_t *err, cudaStream_t st);
cudaError_t build_raw_tris(const Tri *tris, const uint32_t *idx, const float *pos, uint32_t n, float4 *raw,
                           cudaStream_t st);

// Batches of at most kSmallBatch rays take the eight-lanes-a-ray kernel.
// Measured on a B200 against the persistent kernel, diffuse rays over 4 K / 1 M
// triangles: 1,000 rays 21 / 41 us against 46 / 85, 16,000 27 / 54 against
// 48 / 86, 32,000 35 / 73 against 55 / 98, 64,000 57 / 116 against 56 / 122,
// 128,000 99 / 200 against 78 / 146; camera rays gain up to 128,000.
constexpr uint32_t kSmallBatch = 40960u;
// Host batches of at most this many rays are read and answered in place.
// Measured on a B200, closest / any hit of diffuse rays from host arrays, staged
// copies against in place: over 4 K triangles 1,000 rays 98 / 52 us against
// 44 / 36, 16,384 152 / 90 against 91 / 77, 32,000 196 / 123 against 160 / 132; over
// 1 M triangles 16,384 181 / 109 against 120 / 91, 32,000 236 / 148 against 199 / 160:
// any hits, with a byte a ray to bring back, break even at 25,000.
constexpr uint32_t kSmallHostBatch = 16384u;
// A small batch whose rays and 16-byte hit records (prim, t, u, v) are in host
// memory that the device can address; *host_err is set when the context's
// error word is (raw: the watertight test's vertices, or null).
cudaError_t launch_small_host(const SceneView &s, const float4 *raw, const float4 *ro, const float4 *rd, uint32_t n,
                              int4 *hits, uint32_t *host_err, bool any, uint32_t *err, cudaStream_t st);

// Loads the code of the closest-hit kernels on the current device
// (kernels load lazily on first launch otherwise, which may allocate).
cudaError_t preload_closest_dyn();

// Persistent variants with dynamic ray fetch; `next` is a device counter word.
cudaError_t launch_closest_dyn(const SceneView &s, const float4 *ro, const float4 *rd, uint32_t n, int32_t *prim,
                               float *t, float *u, float *v, uint32_t *next, uint32_t *err, cudaStream_t st);
cudaError_t launch_any_dyn(const SceneView &s, const float4 *ro, const float4 *rd, uint32_t n, uint8_t *occ,
                           uint32_t *next, uint32_t *err, cudaStream_t st);

}  // namespace ilg
