// Closest-hit and any-hit traversal of the 8-wide BVH (replaces the reference's
// per-ray CPU walks: BasicSpace::Intersects -> KDTreeMesh::Intersect_New /
// BVHMesh::Intersect -> IndexedTriangle::Intersects; BasicSpace.cpp:58-115,
// KDTreeMesh.cpp:313-577, BVHMesh.cpp:143-198, IndexedTriangle.cpp:92-290).
//
// One ray per thread. The stack holds node groups (first child node index,
// remaining children and internal-child bits), one entry per level at most; the
// children of a node are intersected together from one 96-byte record and
// visited in octant order. A hit shrinks the ray's Max exactly as the
// reference does, so the triangle window `t > Max - 1e-5` and the result are
// the reference's, up to which of two hits less than 1e-5 apart is visited
// first.
#pragma once

#include "bvh8.cuh"

namespace ilg {

// Input triangles [lo, lo + n) that a query ignores (the reference's
// `p_pExclude` primitive after its triangles were flattened into one range).
struct Skip {
    uint32_t lo, n;
};

// ---------------------------------------------------------------------------
// Traversal state machine shared by every kernel
// ---------------------------------------------------------------------------

// The traversal stack: a plain uint2 array (local memory), or split in two,
// its first kShortStack entries in shared memory (one column per thread of a
// kStackColumns-thread block: entry i of a thread at s[i * kStackColumns]) and
// the rest in local memory. The BVH8 of a few million triangles is 7 to 9
// levels deep, so the local part is rarely touched; shared memory keeps the
// entries out of the L1 lines that node and triangle loads stream through
// (measured on a B200: 3 % more incoherent rays per second on the 1 M
// triangle heightfield).
constexpr int kShortStack = 8;
constexpr int kStackColumns = 128;
struct SplitStack {
    uint2 *s;  // this thread's column of the block's shared array
    uint2 *l;  // entries kShortStack .. kMaxStack - 1
};
__device__ __forceinline__ void stack_put(uint2 *a, int i, uint2 e) { a[i] = e; }
__device__ __forceinline__ uint2 stack_get(uint2 *a, int i) { return a[i]; }
__device__ __forceinline__ void stack_put(const SplitStack &t, int i, uint2 e)
{
    if (i < kShortStack) t.s[i * kStackColumns] = e;
    else t.l[i - kShortStack] = e;
}
__device__ __forceinline__ uint2 stack_get(const SplitStack &t, int i)
{
    return i < kShortStack ? t.s[i * kStackColumns] : t.l[i - kShortStack];
}

struct RayState {
    float ox, oy, oz, dx, dy, dz;
    float ix, iy, iz;
    float tmin, tcur, whi;
    uint32_t oct4;  // 4 x (7 - the direction's octant)
    // node group: first child, and a nibble per slot: bit 3 of nibble
    // (slot ^ oct4 / 4) = an internal child still to visit, bit 0 of nibble
    // slot = an internal child (for the children's addresses)
    uint32_t ng_base, ng_hits;
    // triangle group: first record, the node's triangle bits, those to test
    uint32_t tg_base, tg_slots, tg_hits;
    // a second one behind it (persistent kernels; see trace_persistent)
    uint32_t tq_base, tq_slots, tq_hits;
    uint32_t budget;
    int sp;
    int best;
    float bu, bv;
    Shear sh;  // watertight test only
    bool any;  // kMixed traversals: this ray is an any-hit (shadow) ray
};

template <bool kWT = false>
__device__ __forceinline__ void ray_init(RayState &r, float4 o, float4 d, uint32_t n_nodes_total, float min_dir)
{
    if (kWT) r.sh = shear_of(d.x, d.y, d.z);
    r.ox = o.x; r.oy = o.y; r.oz = o.z; r.dx = d.x; r.dy = d.y; r.dz = d.z;
    r.ix = copysignf(__frcp_rn(fmaxf(fabsf(d.x), min_dir)), d.x);
    r.iy = copysignf(__frcp_rn(fmaxf(fabsf(d.y), min_dir)), d.y);
    r.iz = copysignf(__frcp_rn(fmaxf(fabsf(d.z), min_dir)), d.z);
    const uint32_t oct = (d.x < 0.f ? 1u : 0u) | (d.y < 0.f ? 2u : 0u) | (d.z < 0.f ? 4u : 0u);
    r.oct4 = 4u * (7u - oct);
    r.tmin = o.w;
    r.tcur = d.w;
    r.whi = window_hi(r.tcur);
    r.ng_base = 0;
    r.ng_hits = (8u << r.oct4) | 1u;
    r.tg_base = r.tg_slots = 0;
    r.tg_hits = r.tq_hits = 0;
    r.budget = n_nodes_total + 1u;
    r.sp = 0;
    r.best = -1;
    r.bu = r.bv = 0.f;
}

// 32 aligned bytes in one load.
__device__ __forceinline__ void load32(const uint4 *p, uint4 &a, uint4 &b)
{
    asm("ld.global.nc.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=r"(a.x), "=r"(a.y), "=r"(a.z), "=r"(a.w), "=r"(b.x), "=r"(b.y), "=r"(b.z), "=r"(b.w)
        : "l"(p));
}

__device__ __forceinline__ void load32(const float4 *p, float4 &a, float4 &b)
{
    asm("ld.global.nc.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=f"(a.x), "=f"(a.y), "=f"(a.z), "=f"(a.w), "=f"(b.x), "=f"(b.y), "=f"(b.z), "=f"(b.w)
        : "l"(p));
}

// Two floats in one 64-bit register pair, for the packed FP32 arithmetic.
__device__ __forceinline__ uint64_t f2(float lo, float hi)
{
    uint64_t v;
    asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(lo), "f"(hi));
    return v;
}
__device__ __forceinline__ uint64_t f2bits(uint32_t lo, uint32_t hi)
{
    uint64_t v;
    asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "r"(lo), "r"(hi));
    return v;
}
__device__ __forceinline__ void unf2(uint64_t v, float &lo, float &hi)
{
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b)
{
    uint64_t d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c)
{
    uint64_t d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
// (NaN operands are ignored, as fmaxf / fminf do)
__device__ __forceinline__ float max3(float a, float b, float c)
{
    float d;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}
__device__ __forceinline__ float min3(float a, float b, float c)
{
    float d;
    asm("min.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}

// The slots of a node whose boxes the ray misses inside [tmin, tcur]: bit 3
// of the slot's nibble is set (the other bits are not meaningful).
//
// The kernel is bound by instruction issue, and byte-to-float conversions
// run on the slowest pipe (one per 8 cycles and scheduler), so this is built
// for few instructions on the wide pipes: a plane byte becomes the float
// 32768 + byte with one byte permute, its offset is folded into the plane
// equation's constant, near and far plane go through one packed FMA, and
// eight funnel shifts collect the signs of far - near (positive for a NaN,
// so an undefined axis never culls). The near plane is pulled in by a factor
// 1 - 2e-6 against rounding of large plane distances; what the offset costs
// in rounding is below 1/128 of a quantisation step, of which every box has a
// whole one to spare on each side; min_direction keeps it finite.
// `magic` is 0x47000000, as a value the compiler does not know: with the
// constant in sight it replaces each permute by two logic operations.
__device__ __forceinline__ uint32_t node_misses(const RayState &r, uint4 q0, uint4 q1, uint4 q2, uint4 q3, uint4 q4,
                                                uint32_t magic)
{
    auto axis = [&](uint32_t org, float o, float inv, uint32_t step, uint64_t &b, uint64_t &c) {
        const float a = (__uint_as_float(org) - o) * inv, s = __uint_as_float(step) * inv;
        const float a0 = fmaf(-32768.f, s, a);
        b = f2(s * 0.9999980f, s);
        c = f2(a0 * 0.9999980f, a0);
    };
    uint64_t bx, by, bz, cx, cy, cz;
    axis(q0.x, r.ox, r.ix, q1.x, bx, cx);
    axis(q0.y, r.oy, r.iy, q1.y, by, cy);
    axis(q0.z, r.oz, r.iz, q1.z, bz, cz);
    const bool px = r.ix >= 0.f, py = r.iy >= 0.f, pz = r.iz >= 0.f;
    const uint32_t nx[2] = {px ? q2.x : q2.z, px ? q2.y : q2.w}, fx[2] = {px ? q2.z : q2.x, px ? q2.w : q2.y};
    const uint32_t ny[2] = {py ? q3.x : q3.z, py ? q3.y : q3.w}, fy[2] = {py ? q3.z : q3.x, py ? q3.w : q3.y};
    const uint32_t nz[2] = {pz ? q4.x : q4.z, pz ? q4.y : q4.w}, fz[2] = {pz ? q4.z : q4.x, pz ? q4.w : q4.y};
    uint32_t miss = 0;
#pragma unroll
    for (int s = 7; s >= 0; s--) {
        const uint32_t sel = 0x7604u | ((uint32_t)(s & 3) << 4);  // bytes {0x00, plane, 0x00, 0x47}
        auto plane = [&](uint32_t w) { return __byte_perm(w, magic, sel); };
        float tnx, tny, tnz, tfx, tfy, tfz;
        unf2(fma2(f2bits(plane(nx[s >> 2]), plane(fx[s >> 2])), bx, cx), tnx, tfx);
        unf2(fma2(f2bits(plane(ny[s >> 2]), plane(fy[s >> 2])), by, cy), tny, tfy);
        unf2(fma2(f2bits(plane(nz[s >> 2]), plane(fz[s >> 2])), bz, cz), tnz, tfz);
        const float tn = max3(tnx, tny, fmaxf(tnz, r.tmin));
        const float tf = min3(tfx, tfy, fminf(tfz, r.tcur));
        miss = __funnelshift_l(__float_as_uint(tf - tn), miss, 4);
    }
    return miss;
}

// Moves bit 3 of every nibble s to nibble s ^ (oct4 / 4).
__device__ __forceinline__ uint32_t octant_order(uint32_t x, uint32_t oct4)
{
    x = __byte_perm(x, 0u, 0x3210u ^ ((oct4 >> 3) * 0x1111u));  // bytes (slot pairs)
    const uint32_t y = ((x << 4) & 0x80808080u) | ((x >> 4) & 0x08080808u);
    return (oct4 & 4u) ? y : x;
}

// The byte permute's constant (see node_misses), made from a number below 2^31
// that the compiler does not know: a tree's nodes, a render's scenes, the rays of
// a wave's queue (their buffers of 80 bytes a ray bound them).
__device__ __forceinline__ uint32_t plane_magic(uint32_t count) { return 0x47000000u | (count >> 31); }

// Ends the ray's traversal with r.best as it stands (-2 after an error).
__device__ __forceinline__ void ray_stop(RayState &r)
{
    r.ng_hits = 0;
    r.tg_hits = r.tq_hits = 0;
    r.sp = 0;
}

__device__ __forceinline__ bool ray_has_nodes(const RayState &r) { return (r.ng_hits & kSlotInner) != 0u || r.sp > 0; }

// Visits the next node in the ray's order (there is one: ray_has_nodes) and
// queues its hit triangles behind those still to test. At most one group of
// triangles may be pending (r.tq_hits == 0), without kQueue none (r.tg_hits == 0).
template <bool kStats = false, bool kQueue = true, class Stack = uint2 *>
__device__ __forceinline__ void ray_node(RayState &r, Stack stack, const Node8 *__restrict__ nodes,
                                         uint32_t n_nodes_total, uint32_t magic, uint32_t *__restrict__ err,
                                         uint32_t *n_nodes = nullptr)
{
    if (!(r.ng_hits & kSlotInner)) {
        const uint2 e = stack_get(stack, --r.sp);
        r.ng_base = e.x;
        r.ng_hits = e.y;
    }
    const uint32_t bit = 31u - __clz(r.ng_hits & kSlotInner);
    r.ng_hits &= ~(1u << bit);
    const uint32_t slot4 = (bit & 28u) ^ r.oct4;  // 4 x the slot
    const uint32_t node_idx = r.ng_base + __popc(r.ng_hits & 0x11111111u & ((1u << slot4) - 1u));
    const bool rest = (r.ng_hits & kSlotInner) != 0u;
    const uint32_t bad = (r.budget-- == 0u ? 4u : 0u) | (node_idx >= n_nodes_total ? 2u : 0u) |
                         (rest && r.sp >= kMaxStack ? 1u : 0u);
    if (bad) {
        atomicOr(err, bad);
        r.best = -2;
        ray_stop(r);
        return;
    }
    if (rest) stack_put(stack, r.sp++, make_uint2(r.ng_base, r.ng_hits));
    uint4 q0, q1, q2, q3, q4, q5;
    load32(nodes[node_idx].q, q0, q1);
    load32(nodes[node_idx].q + 2, q2, q3);
    load32(nodes[node_idx].q + 4, q4, q5);
    if (kStats) (*n_nodes)++;
    const uint32_t miss = node_misses(r, q0, q1, q2, q3, q4, magic) & kSlotInner;
    const uint32_t inner = q5.x & kSlotInner, slots = q5.x & kSlotTris;
    r.ng_base = q0.w;
    r.ng_hits = octant_order(inner & ~miss, r.oct4) | (inner >> 3);
    const uint32_t hit = ~(miss - (miss >> 3));  // bits 0..2 of a hit slot's nibble
    if (!kQueue || r.tg_hits == 0u) {
        r.tg_base = q1.w;
        r.tg_slots = slots;
        r.tg_hits = hit & slots;
    } else {
        r.tq_base = q1.w;
        r.tq_slots = slots;
        r.tq_hits = hit & slots;
    }
}

// Tests the next pending triangle (there is one: r.tg_hits != 0). Any hit
// (kAnyHit, or kMixed with r.any) ends the traversal; a closest hit shrinks
// the ray.
// kWT selects the watertight triangle test over `raw` (three float4
// vertices per triangle record) instead of the reference's Shirley test.
// kMixed: closest- and any-hit rays share one instance (r.any chooses per ray).
template <bool kAnyHit, bool kStats = false, bool kSkip = false, bool kWT = false, bool kMixed = false,
          bool kQueue = true>
__device__ __forceinline__ void ray_tri(RayState &r, const Tri *__restrict__ tris, uint32_t n_tris_total,
                                        uint32_t *__restrict__ err, uint32_t *n_tris = nullptr,
                                        Skip skip = Skip{0u, 0u}, const float4 *__restrict__ raw = nullptr)
{
    const uint32_t b = r.tg_hits & (0u - r.tg_hits);
    const uint32_t ti = r.tg_base + __popc(r.tg_slots & (b - 1u));
    r.tg_hits ^= b;
    if (kQueue && r.tg_hits == 0u) {
        r.tg_base = r.tq_base;
        r.tg_slots = r.tq_slots;
        r.tg_hits = r.tq_hits;
        r.tq_hits = 0u;
    }
    if (ti >= n_tris_total) {
        atomicOr(err, 2u);
        r.best = -2;
        ray_stop(r);
        return;
    }
    if (kStats) (*n_tris)++;
    float th, bh, gh;
    bool hit;
    if (kWT) {
        const float4 *vp = raw + 3ull * ti;
        hit = watertight(__ldg(vp), __ldg(vp + 1), __ldg(vp + 2), r.ox, r.oy, r.oz, r.sh, r.whi, th, bh, gh);
    } else {
        float4 ta, tb, tc, id;
        load32(&tris[ti].a, ta, tb);
        if (kSkip) {  // (the id's sector is the third edge's: both halves of the record are under way before it is looked at)
            load32(&tris[ti].c, tc, id);
            if (__float_as_uint(id.x) - skip.lo < skip.n) return;
        } else {
            tc = __ldg(&tris[ti].c);
        }
        hit = shirley(ta, tb, tc, r.ox, r.oy, r.oz, r.dx, r.dy, r.dz, r.whi, th, bh, gh);
    }
    if (hit) {
        r.best = (int)ti;
        if (kAnyHit || (kMixed && r.any)) {
            ray_stop(r);
        } else {
            r.bu = bh;
            r.bv = gh;
            r.tcur = th;
            r.whi = window_hi(r.tcur);
        }
    }
}

// Whole traversal of one ray (one ray per thread), a node's triangles right
// after the node. Its counters stay below the records there are (< 2^31).
template <bool kAnyHit, bool kStats, bool kSkip = false>
__device__ __forceinline__ void trace_one(const Node8 *__restrict__ nodes, const Tri *__restrict__ tris,
                                          uint32_t n_nodes_total, uint32_t n_tris_total, float min_dir,
                                          float4 o, float4 d, int &best, float &bt, float &bu, float &bv,
                                          uint32_t *__restrict__ err, uint32_t &n_nodes, uint32_t &n_tris,
                                          Skip skip = Skip{0u, 0u})
{
    uint2 stack[kMaxStack];
    RayState r;
    ray_init(r, o, d, n_nodes_total, min_dir);
    const uint32_t magic = plane_magic(n_nodes_total);
    while (ray_has_nodes(r)) {
        ray_node<kStats, false>(r, stack, nodes, n_nodes_total, magic, err, &n_nodes);
        while (r.tg_hits)
            ray_tri<kAnyHit, kStats, kSkip, false, false, false>(r, tris, n_tris_total, err, &n_tris, skip);
    }
    best = r.best;
    bt = r.best >= 0 ? r.tcur : __int_as_float(0x7f800000);
    bu = r.best >= 0 ? r.bu : 0.f;
    bv = r.best >= 0 ? r.bv : 0.f;
}

// ---------------------------------------------------------------------------
// Persistent traversal with dynamic ray fetch: each warp keeps its lanes busy
// by handing idle lanes new rays from a global counter (Aila & Laine 2009,
// "Understanding the efficiency of ray traversal on GPUs").
//
// A node visit costs a warp some 230 instructions however many of its lanes
// take part, a triangle test some 85. Nearly every lane wants a node at any
// time, but only one in six has a triangle to test (1 M-triangle heightfield,
// diffuse bounce rays: node visits ran with 26 of 32 lanes, triangle tests,
// done right after the node, with 5, at 1.9 tests a visit). So triangle tests
// wait until kTriLanes lanes have one, or fewer than kNodeLanes lanes can
// visit a node: a lane goes on with nodes while one group of triangles waits,
// and keeps a second group behind it (tests then run with 13 lanes, 0.65 a
// visit; a ray visits 2 % more nodes). Triangles are tested in the order
// their nodes were visited, and a triangle that an earlier hit would have
// culled is rejected by the shrunken window, so the hits are the same as with
// tests at once.
//
// Measured on a B200, 4.2 M bounce / camera rays of that mesh and 1.0 M
// occlusion segments of a 168 K-triangle one: 1648 / 521 / 276 us with tests
// at once, 80-byte nodes in five loads and converted planes (758 M warp
// instructions for 2.1 M bounce rays); 1510 / 520 / 255 with the planes by
// byte permutes and packed FMAs (658 M); 1402 / 475 / 268 with deferred tests
// (548 M); 1278 / 418 / 228 with 96-byte nodes in three loads. Thresholds
// (kTriLanes, kNodeLanes, refill): 12, 12, 8 1474 us where 6, 16, 4 took 1587,
// 16, 16, 8 1521 and 12, 16, 12 1508.
//
// `fetch(k, r, S)` starts ray k < n in r (and its scene in S), `done(r)` takes
// the result of the lane's ray; both run for several lanes at a time, when
// kRefill lanes are idle. `next` is a device counter, zero at the launch;
// magic: plane_magic.
// ---------------------------------------------------------------------------
constexpr int kTriLanes = 12;
constexpr int kNodeLanes = 12;
constexpr int kRefillLanesQuery = 8;
constexpr int kRefillLanes = 8;

struct TraceScene {
    const Node8 *nodes;
    const Tri *tris;
    uint32_t n_nodes, n_tris;
};

template <bool kAnyHit, bool kWT, bool kMixed, int kRefill, class Stack, class Fetch, class Done>
__device__ __forceinline__ void trace_persistent(Stack stack, TraceScene &S, uint32_t n, uint32_t magic,
                                                 uint32_t *__restrict__ next,
                                                 uint32_t *__restrict__ err, const float4 *__restrict__ raw,
                                                 Fetch fetch, Done done)
{
    const uint32_t lane = threadIdx.x & 31u;
    bool exhausted = n == 0u;  // warp-uniform
    RayState r;
    r.ng_hits = r.tg_hits = r.tq_hits = 0u;
    r.sp = 0;
    bool has = false;  // the lane holds a ray, in flight or finished
    while (true) {
        const uint32_t idle = __ballot_sync(0xffffffffu, r.tg_hits == 0u && !ray_has_nodes(r));
        if (__popc(idle) >= kRefill || idle == 0xffffffffu) {
            if (exhausted) {
                if (idle == 0xffffffffu) break;
            } else {
                const bool take = (idle >> lane) & 1u;
                if (take && has) done(r);
                uint32_t base = 0;
                if (lane == 0u) base = atomicAdd(next, (uint32_t)__popc(idle));
                base = __shfl_sync(0xffffffffu, base, 0);
                exhausted = base >= n;
                if (take) {
                    const uint32_t k = base + __popc(idle & ((1u << lane) - 1u));
                    has = k < n;
                    if (has) fetch(k, r, S);
                }
            }
        }
        __syncwarp();  // lanes with a new ray and lanes without visit their nodes together
        if (r.tq_hits == 0u && ray_has_nodes(r)) ray_node(r, stack, S.nodes, S.n_nodes, magic, err);
        while (true) {
            const uint32_t tri = __ballot_sync(0xffffffffu, r.tg_hits != 0u);
            const uint32_t node = __ballot_sync(0xffffffffu, r.tq_hits == 0u && ray_has_nodes(r));
            if (tri == 0u || (__popc(tri) < kTriLanes && __popc(node) >= kNodeLanes)) break;
            if (r.tg_hits) ray_tri<kAnyHit, false, false, kWT, kMixed>(r, S.tris, S.n_tris, err, nullptr,
                                                                       Skip{0u, 0u}, raw);
        }
    }
    if (has) done(r);
}

}  // namespace ilg
