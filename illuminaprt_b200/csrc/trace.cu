// Batched closest-hit / any-hit kernels over the 8-wide BVH.
#include "trace.cuh"
#include "trace_api.cuh"
#include "devinfo.cuh"

#include <algorithm>

namespace ilg {

namespace {

// One ray a thread: the excluding and the counted queries. Eight blocks an SM
// (64 registers; 70 without the bound: 1 M excluding rays 2 to 3 % slower).
template <bool kStats, bool kSkip = false>
__global__ void __launch_bounds__(128, 8) k_closest(const Node8 *__restrict__ nodes, const Tri *__restrict__ tris,
                                                 uint32_t n_nodes_total, uint32_t n_tris_total, float min_dir,
                                                 const float4 *__restrict__ ro, const float4 *__restrict__ rd,
                                                 uint32_t n, int32_t *__restrict__ prim, float *__restrict__ tout,
                                                 float *__restrict__ uout, float *__restrict__ vout,
                                                 uint32_t *__restrict__ err, unsigned long long *__restrict__ stats,
                                                 uint32_t skip_lo = 0, uint32_t skip_n = 0)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float4 o = __ldcs(ro + i), d = __ldcs(rd + i);
    int best;
    float bt, bu, bv;
    uint32_t nn = 0, nt = 0;
    trace_one<false, kStats, kSkip>(nodes, tris, n_nodes_total, n_tris_total, min_dir, o, d, best, bt, bu, bv, err, nn, nt,
                                    Skip{skip_lo, skip_n});
    __stcs(prim + i, best >= 0 ? (int32_t)__ldg(&tris[best].id.x) : (best == -2 ? -2 : -1));
    __stcs(tout + i, bt);
    __stcs(uout + i, bu);
    __stcs(vout + i, bv);
    if (kStats) {
        atomicAdd(&stats[0], nn);
        atomicAdd(&stats[1], nt);
    }
}

template <bool kSkip = false>
__global__ void __launch_bounds__(128) k_any(const Node8 *__restrict__ nodes, const Tri *__restrict__ tris,
                                             uint32_t n_nodes_total, uint32_t n_tris_total, float min_dir,
                                             const float4 *__restrict__ ro, const float4 *__restrict__ rd,
                                             uint32_t n, uint8_t *__restrict__ occ, uint32_t *__restrict__ err,
                                             uint32_t skip_lo = 0, uint32_t skip_n = 0)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float4 o = __ldcs(ro + i), d = __ldcs(rd + i);
    int best;
    float bt, bu, bv;
    uint32_t nn = 0, nt = 0;
    trace_one<true, false, kSkip>(nodes, tris, n_nodes_total, n_tris_total, min_dir, o, d, best, bt, bu, bv, err, nn, nt,
                                  Skip{skip_lo, skip_n});
    occ[i] = best >= 0 ? 1 : 0;
}

// Persistent closest / any hit with dynamic ray fetch (see trace.cuh);
// kWT: the watertight triangle test over `raw`. Eight blocks an SM (64
// registers): seven ran 5 % and nine, spilling, 11 % slower.
template <bool kAnyHit, bool kWT = false>
__global__ void __launch_bounds__(128, 8) k_trace_dyn(const Node8 *__restrict__ nodes, const Tri *__restrict__ tris,
                                                   uint32_t n_nodes_total, uint32_t n_tris_total, float min_dir,
                                                   const float4 *__restrict__ ro,
                                                   const float4 *__restrict__ rd, uint32_t n,
                                                   int32_t *__restrict__ prim, float *__restrict__ tout,
                                                   float *__restrict__ uout, float *__restrict__ vout,
                                                   uint8_t *__restrict__ occ, uint32_t *__restrict__ next,
                                                   uint32_t *__restrict__ err, const float4 *__restrict__ raw = nullptr)
{
    static_assert(kStackColumns == 128, "k_trace_dyn runs 128 threads a block");
    __shared__ uint2 sstack[kShortStack * kStackColumns];
    uint2 lstack[kMaxStack - kShortStack];
    const SplitStack stack{sstack + threadIdx.x, lstack};
    TraceScene scene{nodes, tris, n_nodes_total, n_tris_total};
    uint32_t id = 0;
    trace_persistent<kAnyHit, kWT, false, kRefillLanesQuery>(
        stack, scene, n, plane_magic(n_nodes_total), next, err, raw,
        [&](uint32_t k, RayState &r, TraceScene &) {
            id = k;
            ray_init<kWT>(r, __ldcs(ro + k), __ldcs(rd + k), n_nodes_total, min_dir);
        },
        [&](const RayState &r) {
            if (kAnyHit) {
                occ[id] = r.best >= 0 ? 1 : 0;
            } else {
                __stcs(prim + id, r.best >= 0 ? (int32_t)__ldg(&tris[r.best].id.x) : (r.best == -2 ? -2 : -1));
                __stcs(tout + id, r.best >= 0 ? r.tcur : __int_as_float(0x7f800000));
                __stcs(uout + id, r.best >= 0 ? r.bu : 0.f);
                __stcs(vout + id, r.best >= 0 ? r.bv : 0.f);
            }
        });
}

int sm_count() { return current_sm_count(); }

// ---------------------------------------------------------------------------
// Small batches: eight lanes a ray. A batch that leaves most of the GPU empty
// takes as long as its longest ray, a chain of node visits; with a ray a lane
// each visit issues 230 instructions and waits for the warp's other rays'
// triangles. Here a lane tests one child of the ray's node and one of its
// pending triangles, so a visit is some 70 instructions and one round of
// loads. Nodes and triangles are met in the order of the other kernels, with
// the same arithmetic, so the hits are the same: lanes test triangles against
// the window before the first of them, then the hits among them are taken in
// order, each against the window the one before left.
// ---------------------------------------------------------------------------
constexpr int kCoopThreads = 64;

// Where a small batch's results go: the caller's arrays, or one 16-byte record
// a ray (prim, t, u, v; any hit: prim = 0 / 1) in host memory the device
// writes directly, with a word that is set when the context has an error to
// report.
struct SmallOut {
    int32_t *prim;
    float *t, *u, *v;
    uint8_t *occ;
    int4 *host;
    uint32_t *host_err;
};

template <bool kAnyHit, bool kWT>
__global__ void __launch_bounds__(kCoopThreads) k_trace_coop(const Node8 *__restrict__ nodes,
                                                             const Tri *__restrict__ tris, uint32_t n_nodes_total,
                                                             uint32_t n_tris_total, float min_dir,
                                                             const float4 *__restrict__ ro,
                                                             const float4 *__restrict__ rd, uint32_t n, SmallOut out,
                                                             uint32_t *__restrict__ err,
                                                             const float4 *__restrict__ raw)
{
    constexpr uint32_t kFull = 0xffffffffu;
    __shared__ uint2 s_stack[kCoopThreads / 8][kMaxStack];
    const uint32_t lane = threadIdx.x & 31u, l = lane & 7u, shift = lane & 24u;
    uint2 *stack = s_stack[threadIdx.x >> 3];
    const uint32_t id = (blockIdx.x * kCoopThreads + threadIdx.x) >> 3;
    auto ballot8 = [&](bool v) { return __ballot_sync(kFull, v) >> shift & 0xffu; };
    const bool has = id < n;
    RayState r;
    r.ng_hits = 0u;
    r.sp = 0;
    r.best = -1;
    if (has) ray_init<kWT>(r, ro[id], rd[id], n_nodes_total, min_dir);
    const uint32_t px = r.ix >= 0.f ? 0u : 8u, py = r.iy >= 0.f ? 0u : 8u, pz = r.iz >= 0.f ? 0u : 8u;
    // (an earlier launch's error is this call's to report too)
    if (out.host_err && id == 0 && l == 0 && *err) *out.host_err = 1u;
    while (true) {
        const bool visit = has && ray_has_nodes(r);
        if (!__any_sync(kFull, visit)) break;
        uint32_t tg_base = 0, tg_slots = 0, tg_hits = 0;
        bool miss = true;
        float4 q0 = make_float4(0.f, 0.f, 0.f, 0.f), q1 = q0;
        uint32_t slots = 0;
        if (visit && !(r.ng_hits & kSlotInner)) {
            const uint2 e = stack[--r.sp];
            r.ng_base = e.x;
            r.ng_hits = e.y;
        }
        __syncwarp();  // the ray's lanes have read the entry that the first of them may write again below
        if (visit) {
            const uint32_t bit = 31u - __clz(r.ng_hits & kSlotInner);
            r.ng_hits &= ~(1u << bit);
            const uint32_t slot4 = (bit & 28u) ^ r.oct4;
            const uint32_t node_idx = r.ng_base + __popc(r.ng_hits & 0x11111111u & ((1u << slot4) - 1u));
            const bool rest = (r.ng_hits & kSlotInner) != 0u;
            const uint32_t bad = (r.budget-- == 0u ? 4u : 0u) | (node_idx >= n_nodes_total ? 2u : 0u) |
                                 (rest && r.sp >= kMaxStack ? 1u : 0u);
            if (bad) {
                if (l == 0u) atomicOr(err, bad);
                r.best = -2;
                ray_stop(r);
            } else {
                if (rest) {
                    if (l == 0u) stack[r.sp] = make_uint2(r.ng_base, r.ng_hits);
                    r.sp++;
                }
                const Node8 &nd = nodes[node_idx];
                q0 = __ldg(reinterpret_cast<const float4 *>(nd.q));
                q1 = __ldg(reinterpret_cast<const float4 *>(nd.q + 1));
                slots = __ldg(&nd.q[5].x);
                const uint8_t *pl = reinterpret_cast<const uint8_t *>(nd.q + 2) + l;
                const float nx = (float)(32768 + __ldg(pl + px)), fx = (float)(32768 + __ldg(pl + (8u ^ px)));
                const float ny = (float)(32768 + __ldg(pl + 16 + py)), fy = (float)(32768 + __ldg(pl + 16 + (8u ^ py)));
                const float nz = (float)(32768 + __ldg(pl + 32 + pz)), fz = (float)(32768 + __ldg(pl + 32 + (8u ^ pz)));
                // node_misses, one slot
                auto axis = [](float org, float o, float inv, float step, float pn, float pf, float &tn, float &tf) {
                    const float a = (org - o) * inv, s = step * inv;
                    const float a0 = fmaf(-32768.f, s, a);
                    tn = fmaf(pn, s * 0.9999980f, a0 * 0.9999980f);
                    tf = fmaf(pf, s, a0);
                };
                float tnx, tny, tnz, tfx, tfy, tfz;
                axis(q0.x, r.ox, r.ix, q1.x, nx, fx, tnx, tfx);
                axis(q0.y, r.oy, r.iy, q1.y, ny, fy, tny, tfy);
                axis(q0.z, r.oz, r.iz, q1.z, nz, fz, tnz, tfz);
                const float tn = max3(tnx, tny, fmaxf(tnz, r.tmin)), tf = min3(tfx, tfy, fminf(tfz, r.tcur));
                miss = (__float_as_uint(tf - tn) >> 31) != 0u;
            }
        }
        {
            // bit 3 of nibble s = slot s missed
            uint32_t m = ballot8(miss);
            m = (m | m << 12) & 0x000f000fu;
            m = (m | m << 6) & 0x03030303u;
            m = (m | m << 3) & 0x11111111u;
            m <<= 3;
            if (visit && r.best != -2) {
                const uint32_t inner = slots & kSlotInner;
                r.ng_base = __float_as_uint(q0.w);
                r.ng_hits = octant_order(inner & ~m, r.oct4) | (inner >> 3);
                tg_base = __float_as_uint(q1.w);
                tg_slots = slots & kSlotTris;
                tg_hits = ~(m - (m >> 3)) & tg_slots;
            }
        }
        // eight pending triangles at a time
        while (__any_sync(kFull, tg_hits != 0u)) {
            uint32_t x = tg_hits;
#pragma unroll
            for (uint32_t j = 0; j < 7u; j++) x = j < l ? x & (x - 1u) : x;
            const uint32_t b = x & (0u - x);  // this lane's triangle, 0 when there is none
            const uint32_t ti = tg_base + __popc(tg_slots & (b - 1u));
            const bool bad = b != 0u && ti >= n_tris_total;
            float th = 0.f, bh = 0.f, gh = 0.f;
            bool hit = false;
            if (b != 0u && !bad) {
                if (kWT) {
                    const float4 *vp = raw + 3ull * ti;
                    hit = watertight(__ldg(vp), __ldg(vp + 1), __ldg(vp + 2), r.ox, r.oy, r.oz, r.sh, r.whi, th, bh, gh);
                } else {
                    float4 ta, tb;
                    load32(&tris[ti].a, ta, tb);
                    hit = shirley(ta, tb, __ldg(&tris[ti].c), r.ox, r.oy, r.oz, r.dx, r.dy, r.dz, r.whi, th, bh, gh);
                }
            }
            if (ballot8(bad)) {
                if (bad) atomicOr(err, 2u);
                r.best = -2;
                ray_stop(r);
                tg_hits = 0u;
                hit = false;
            }
            while (true) {
                const uint32_t hits = ballot8(hit);
                if (!__any_sync(kFull, hits != 0u)) break;
                const uint32_t first = hits ? __ffs(hits) - 1u : 0u;
                const float t1 = __shfl_sync(kFull, th, shift + first), b1 = __shfl_sync(kFull, bh, shift + first),
                            g1 = __shfl_sync(kFull, gh, shift + first);
                const uint32_t i1 = __shfl_sync(kFull, ti, shift + first);
                if (hits) {
                    r.best = (int)i1;
                    if (kAnyHit) {
                        ray_stop(r);
                        tg_hits = 0u;
                        hit = false;
                    } else {
                        r.tcur = t1;
                        r.bu = b1;
                        r.bv = g1;
                        r.whi = window_hi(t1);
                        hit = hit && l > first && th <= r.whi;
                    }
                }
            }
            // the eight tested are done
#pragma unroll
            for (int j = 0; j < 8; j++) tg_hits &= tg_hits - 1u;
        }
        __syncwarp();  // the stack entry is read by the other lanes
    }
    if (!has || l != 0u) return;
    const int32_t prim = r.best >= 0 ? (int32_t)__ldg(&tris[r.best].id.x) : (r.best == -2 ? -2 : -1);
    const float t = r.best >= 0 ? r.tcur : __int_as_float(0x7f800000);
    const float u = r.best >= 0 ? r.bu : 0.f, v = r.best >= 0 ? r.bv : 0.f;
    if (out.host) {
        out.host[id] = kAnyHit ? make_int4(r.best >= 0 ? 1 : 0, 0, 0, 0)
                               : make_int4(prim, __float_as_int(t), __float_as_int(u), __float_as_int(v));
        if (r.best == -2) *out.host_err = 1u;
    } else if (kAnyHit) {
        out.occ[id] = r.best >= 0 ? 1 : 0;
    } else {
        out.prim[id] = prim;
        out.t[id] = t;
        out.u[id] = u;
        out.v[id] = v;
    }
}

// Whether a batch is small enough for eight lanes a ray.
bool small_batch(uint32_t n) { return n <= kSmallBatch; }

template <bool kAnyHit, bool kWT>
cudaError_t launch_coop(const SceneView &s, const float4 *raw, const float4 *ro, const float4 *rd, uint32_t n,
                        const SmallOut &out, uint32_t *err, cudaStream_t st)
{
    k_trace_coop<kAnyHit, kWT><<<(n + kCoopThreads / 8 - 1) / (kCoopThreads / 8), kCoopThreads, 0, st>>>(
        s.nodes, s.tris, s.n_nodes, s.n_tris, s.min_dir, ro, rd, n, out, err, raw);
    return cudaGetLastError();
}

}  // namespace

cudaError_t launch_small_host(const SceneView &s, const float4 *raw, const float4 *ro, const float4 *rd, uint32_t n,
                              int4 *hits, uint32_t *host_err, bool any, uint32_t *err, cudaStream_t st)
{
    const SmallOut out{nullptr, nullptr, nullptr, nullptr, nullptr, hits, host_err};
    if (any) return raw ? launch_coop<true, true>(s, raw, ro, rd, n, out, err, st)
                        : launch_coop<true, false>(s, raw, ro, rd, n, out, err, st);
    return raw ? launch_coop<false, true>(s, raw, ro, rd, n, out, err, st)
               : launch_coop<false, false>(s, raw, ro, rd, n, out, err, st);
}

cudaError_t preload_closest_dyn()
{
    cudaFuncAttributes a;
    cudaError_t e = cudaFuncGetAttributes(&a, (const void *)k_trace_coop<false, false>);
    if (e != cudaSuccess) return e;
    return cudaFuncGetAttributes(&a, (const void *)k_trace_dyn<false>);
}

cudaError_t launch_closest_dyn(const SceneView &s, const float4 *ro, const float4 *rd, uint32_t n, int32_t *prim,
                               float *t, float *u, float *v, uint32_t *next, uint32_t *err, cudaStream_t st)
{
    if (n == 0) return cudaSuccess;
    if (small_batch(n))
        return launch_coop<false, false>(s, nullptr, ro, rd, n, SmallOut{prim, t, u, v, nullptr, nullptr, nullptr}, err, st);
    cudaError_t e = cudaMemsetAsync(next, 0, sizeof(uint32_t), st);
    if (e != cudaSuccess) return e;
    const uint32_t blocks = std::min<uint32_t>((n + 127) / 128, (uint32_t)sm_count() * 16u);
    k_trace_dyn<false><<<blocks, 128, 0, st>>>(s.nodes, s.tris, s.n_nodes, s.n_tris, s.min_dir, ro, rd, n, prim, t,
                                               u, v, nullptr, next, err);
    return cudaGetLastError();
}

cudaError_t launch_any_dyn(const SceneView &s, const float4 *ro, const float4 *rd, uint32_t n, uint8_t *occ,
                           uint32_t *next, uint32_t *err, cudaStream_t st)
{
    if (n == 0) return cudaSuccess;
    if (small_batch(n))
        return launch_coop<true, false>(s, nullptr, ro, rd, n, SmallOut{nullptr, nullptr, nullptr, nullptr, occ, nullptr, nullptr}, err, st);
    cudaError_t e = cudaMemsetAsync(next, 0, sizeof(uint32_t), st);
    if (e != cudaSuccess) return e;
    const uint32_t blocks = std::min<uint32_t>((n + 127) / 128, (uint32_t)sm_count() * 16u);
    k_trace_dyn<true><<<blocks, 128, 0, st>>>(s.nodes, s.tris, s.n_nodes, s.n_tris, s.min_dir, ro, rd, n, nullptr,
                                              nullptr, nullptr, nullptr, occ, next, err);
    return cudaGetLastError();
}

cudaError_t launch_closest_wt(const SceneView &s, const float4 *raw, const float4 *ro, const float4 *rd, uint32_t n,
                              int32_t *prim, float *t, float *u, float *v, uint32_t *next, uint32_t *err,
                              cudaStream_t st)
{
    if (n == 0) return cudaSuccess;
    if (small_batch(n))
        return launch_coop<false, true>(s, raw, ro, rd, n, SmallOut{prim, t, u, v, nullptr, nullptr, nullptr}, err, st);
    cudaError_t e = cudaMemsetAsync(next, 0, sizeof(uint32_t), st);
    if (e != cudaSuccess) return e;
    const uint32_t blocks = std::min<uint32_t>((n + 127) / 128, (uint32_t)sm_count() * 16u);
    k_trace_dyn<false, true><<<blocks, 128, 0, st>>>(s.nodes, s.tris, s.n_nodes, s.n_tris, s.min_dir, ro, rd, n,
                                                     prim, t, u, v, nullptr, next, err, raw);
    return cudaGetLastError();
}

cudaError_t launch_any_wt(const SceneView &s, const float4 *raw, const float4 *ro, const float4 *rd, uint32_t n,
                          uint8_t *occ, uint32_t *next, uint32_t *err, cudaStream_t st)
{
    if (n == 0) return cudaSuccess;
    if (small_batch(n))
        return launch_coop<true, true>(s, raw, ro, rd, n, SmallOut{nullptr, nullptr, nullptr, nullptr, occ, nullptr, nullptr}, err, st);
    cudaError_t e = cudaMemsetAsync(next, 0, sizeof(uint32_t), st);
    if (e != cudaSuccess) return e;
    const uint32_t blocks = std::min<uint32_t>((n + 127) / 128, (uint32_t)sm_count() * 16u);
    k_trace_dyn<true, true><<<blocks, 128, 0, st>>>(s.nodes, s.tris, s.n_nodes, s.n_tris, s.min_dir, ro, rd, n,
                                                    nullptr, nullptr, nullptr, nullptr, occ, next, err, raw);
    return cudaGetLastError();
}

// Three float4 vertices per triangle record, in record order: the input
// vertices of the record's triangle, copied bit for bit.
__global__ void k_raw_tris(const Tri *__restrict__ tris, const uint32_t *__restrict__ idx,
                           const float *__restrict__ pos, uint32_t n, float4 *__restrict__ raw)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const uint32_t p = tris[i].id.x;
#pragma unroll
    for (int c = 0; c < 3; c++) {
        const uint32_t v = idx[3ull * p + c];
        raw[3ull * i + c] = make_float4(pos[3ull * v], pos[3ull * v + 1], pos[3ull * v + 2], 0.f);
    }
}

cudaError_t build_raw_tris(const Tri *tris, const uint32_t *idx, const float *pos, uint32_t n, float4 *raw,
                           cudaStream_t st)
{
    if (n == 0) return cudaSuccess;
    k_raw_tris<<<(n + 255) / 256, 256, 0, st>>>(tris, idx, pos, n, raw);
    return cudaGetLastError();
}

cudaError_t launch_closest(const SceneView &s, const float4 *ro, const float4 *rd, uint32_t n, int32_t *prim,
                           float *t, float *u, float *v, uint32_t *err, unsigned long long *stats, cudaStream_t st)
{
    if (n == 0) return cudaSuccess;
    const uint32_t T = 128;
    const uint32_t blocks = (n + T - 1) / T;
    if (stats)
        k_closest<true><<<blocks, T, 0, st>>>(s.nodes, s.tris, s.n_nodes, s.n_tris, s.min_dir, ro, rd, n, prim, t, u, v, err, stats);
    else
        k_closest<false><<<blocks, T, 0, st>>>(s.nodes, s.tris, s.n_nodes, s.n_tris, s.min_dir, ro, rd, n, prim, t, u, v, err, nullptr);
    return cudaGetLastError();
}

cudaError_t launch_any(const SceneView &s, const float4 *ro, const float4 *rd, uint32_t n, uint8_t *occ,
                       uint32_t *err, cudaStream_t st)
{
    if (n == 0) return cudaSuccess;
    const uint32_t T = 128;
    k_any<false><<<(n + T - 1) / T, T, 0, st>>>(s.nodes, s.tris, s.n_nodes, s.n_tris, s.min_dir, ro, rd, n, occ, err);
    return cudaGetLastError();
}

cudaError_t launch_closest_skip(const SceneView &s, const float4 *ro, const float4 *rd, uint32_t n,
                                uint32_t skip_lo, uint32_t skip_n, int32_t *prim, float *t, float *u, float *v,
                                uint32_t *err, cudaStream_t st)
{
    if (n == 0) return cudaSuccess;
    const uint32_t T = 128;
    k_closest<false, true><<<(n + T - 1) / T, T, 0, st>>>(s.nodes, s.tris, s.n_nodes, s.n_tris, s.min_dir, ro, rd, n,
                                                          prim, t, u, v, err, nullptr, skip_lo, skip_n);
    return cudaGetLastError();
}

cudaError_t launch_any_skip(const SceneView &s, const float4 *ro, const float4 *rd, uint32_t n, uint32_t skip_lo,
                            uint32_t skip_n, uint8_t *occ, uint32_t *err, cudaStream_t st)
{
    if (n == 0) return cudaSuccess;
    const uint32_t T = 128;
    k_any<true><<<(n + T - 1) / T, T, 0, st>>>(s.nodes, s.tris, s.n_nodes, s.n_tris, s.min_dir, ro, rd, n, occ, err,
                                               skip_lo, skip_n);
    return cudaGetLastError();
}

}  // namespace ilg
