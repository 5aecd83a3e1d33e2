// Device build of the 8-wide BVH (replaces the reference's per-mesh CPU tree
// builders, KDTreeMesh::Compile / BVHMesh::Compile, KDTreeMesh.cpp:114-275 and
// BVHMesh.cpp:78-107, which take ~6-20 s per million triangles on one core).
//
// Pipeline, all on the context's stream:
//   1. k_tri_bounds   per-triangle AABB + centroid, scene centroid bounds
//   2. k_morton       30-bit Morton code of each centroid
//   3. radix sort     (code, triangle) pairs (CUB)
//   4. k_karras       binary radix tree over the sorted codes (Karras 2012),
//                     duplicate codes split by index
//   5. k_treelet      bottom-up AABBs and subtree triangle counts, one atomic
//                     arrival counter per node, and treelet restructuring for
//                     least SAH cost (Karras & Aila 2013)
//   5c. k_collapse_cost  bottom-up SAH costs of the binary subtrees as 1..8
//                     roots of an 8-wide node (Ylitie et al. 2017)
//   6. k_collapse     level by level: each work item turns one binary node
//                     into one 8-wide node (its children: the roots the
//                     step 5c costs chose; a root is a leaf or a node),
//                     orders the slots by octant, quantises the child boxes
//                     to 8 bits against the node origin, and writes the
//                     triangle records of its leaf children.
#include "bvh8.cuh"
#include "build.cuh"
#include "devinfo.cuh"

#include <cub/device/device_radix_sort.cuh>

#include <algorithm>
#include <cfloat>
#include <climits>
#include <cmath>
#include <utility>

namespace ilg {

namespace {

__device__ __forceinline__ uint32_t float_flip(float f)
{
    uint32_t u = __float_as_uint(f);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float float_unflip(uint32_t u)
{
    return __uint_as_float((u & 0x80000000u) ? (u & 0x7fffffffu) : ~u);
}

__device__ __forceinline__ uint32_t expand_bits10(uint32_t v)
{
    v &= 0x3ffu;
    v = (v * 0x00010001u) & 0xFF0000FFu;
    v = (v * 0x00000101u) & 0x0F00F00Fu;
    v = (v * 0x00000011u) & 0xC30C30C3u;
    v = (v * 0x00000005u) & 0x49249249u;
    return v;
}

struct Box {
    float3 lo, hi;
};

__device__ __forceinline__ float area(const float3 &lo, const float3 &hi)
{
    float dx = fmaxf(hi.x - lo.x, 0.f), dy = fmaxf(hi.y - lo.y, 0.f), dz = fmaxf(hi.z - lo.z, 0.f);
    return dx * dy + dy * dz + dz * dx;
}

// ---------------------------------------------------------------- step 1 ----
__global__ void k_tri_bounds(const float *__restrict__ pos, uint32_t n_verts, const uint32_t *__restrict__ idx,
                             uint32_t n, float4 *__restrict__ tlo, float4 *__restrict__ thi,
                             uint32_t *__restrict__ cbounds /* ordered maxima of -min xyz, max xyz; zeroed */,
                             uint32_t *__restrict__ err)
{
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    float3 clo = make_float3(FLT_MAX, FLT_MAX, FLT_MAX), chi = make_float3(-FLT_MAX, -FLT_MAX, -FLT_MAX);
    if (i < n) {
        uint32_t a = idx[3 * i], b = idx[3 * i + 1], c = idx[3 * i + 2];
        if (a >= n_verts || b >= n_verts || c >= n_verts) {
            atomicOr(err, 1u);
            a = b = c = 0;
        }
        float3 p0 = make_float3(pos[3 * a], pos[3 * a + 1], pos[3 * a + 2]);
        float3 p1 = make_float3(pos[3 * b], pos[3 * b + 1], pos[3 * b + 2]);
        float3 p2 = make_float3(pos[3 * c], pos[3 * c + 1], pos[3 * c + 2]);
        float3 lo = make_float3(fminf(p0.x, fminf(p1.x, p2.x)), fminf(p0.y, fminf(p1.y, p2.y)),
                                fminf(p0.z, fminf(p1.z, p2.z)));
        float3 hi = make_float3(fmaxf(p0.x, fmaxf(p1.x, p2.x)), fmaxf(p0.y, fmaxf(p1.y, p2.y)),
                                fmaxf(p0.z, fmaxf(p1.z, p2.z)));
        tlo[i] = make_float4(lo.x, lo.y, lo.z, 0.f);
        thi[i] = make_float4(hi.x, hi.y, hi.z, 0.f);
        clo = make_float3(0.5f * (lo.x + hi.x), 0.5f * (lo.y + hi.y), 0.5f * (lo.z + hi.z));
        chi = clo;
    }
    // block reduce over ordered integers, then one atomic per block and bound
    // (one per warp kept 8 K warps waiting on six addresses: 34 us for 262 K
    // triangles, 9 us so)
    __shared__ uint32_t s_bound[6];
    if (threadIdx.x < 6) s_bound[threadIdx.x] = 0u;
    __syncthreads();
    const uint32_t key[6] = {~float_flip(clo.x), ~float_flip(clo.y), ~float_flip(clo.z),
                             float_flip(chi.x),  float_flip(chi.y),  float_flip(chi.z)};
#pragma unroll
    for (int k = 0; k < 6; k++) {
        const uint32_t m = __reduce_max_sync(0xffffffffu, key[k]);
        if ((threadIdx.x & 31) == 0) atomicMax(&s_bound[k], m);
    }
    __syncthreads();
    if (threadIdx.x < 6) atomicMax(&cbounds[threadIdx.x], s_bound[threadIdx.x]);
}

// ---------------------------------------------------------------- step 2 ----
__global__ void k_morton(const float4 *__restrict__ tlo, const float4 *__restrict__ thi, uint32_t n,
                         const uint32_t *__restrict__ cbounds, uint32_t *__restrict__ keys,
                         uint32_t *__restrict__ vals)
{
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    float3 lo = make_float3(float_unflip(~cbounds[0]), float_unflip(~cbounds[1]), float_unflip(~cbounds[2]));
    float3 hi = make_float3(float_unflip(cbounds[3]), float_unflip(cbounds[4]), float_unflip(cbounds[5]));
    float4 a = tlo[i], b = thi[i];
    float cx = 0.5f * (a.x + b.x), cy = 0.5f * (a.y + b.y), cz = 0.5f * (a.z + b.z);
    float ex = hi.x - lo.x, ey = hi.y - lo.y, ez = hi.z - lo.z;
    float nx = ex > 0.f ? (cx - lo.x) / ex : 0.f;
    float ny = ey > 0.f ? (cy - lo.y) / ey : 0.f;
    float nz = ez > 0.f ? (cz - lo.z) / ez : 0.f;
    uint32_t ix = (uint32_t)fminf(fmaxf(nx * 1024.f, 0.f), 1023.f);
    uint32_t iy = (uint32_t)fminf(fmaxf(ny * 1024.f, 0.f), 1023.f);
    uint32_t iz = (uint32_t)fminf(fmaxf(nz * 1024.f, 0.f), 1023.f);
    keys[i] = (expand_bits10(ix) << 2) | (expand_bits10(iy) << 1) | expand_bits10(iz);
    vals[i] = i;
}

// ---------------------------------------------------------------- step 4 ----
// Internal node i of n-1; children encoded >= 0 internal, < 0 leaf ~sorted_pos.
__device__ __forceinline__ int delta(const uint32_t *keys, int n, int i, int j)
{
    if (j < 0 || j >= n) return -1;
    uint32_t a = keys[i], b = keys[j];
    if (a == b) return 32 + __clz((uint32_t)i ^ (uint32_t)j);
    return __clz(a ^ b);
}

__global__ void k_karras(const uint32_t *__restrict__ keys, int n, int2 *__restrict__ child,
                         int *__restrict__ parent_int, int *__restrict__ parent_leaf)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n - 1) return;
    int dl = delta(keys, n, i, i - 1), dr = delta(keys, n, i, i + 1);
    int d = dr > dl ? 1 : -1;
    int dmin = d > 0 ? dl : dr;
    int lmax = 2;
    while (lmax < (1 << 30) && delta(keys, n, i, i + lmax * d) > dmin) lmax <<= 1;
    int l = 0;
    for (int t = lmax >> 1; t >= 1; t >>= 1)
        if (delta(keys, n, i, i + (l + t) * d) > dmin) l += t;
    int j = i + l * d;
    int dnode = delta(keys, n, i, j);
    int s = 0;
    int len = l;
    int t = (len + 1) >> 1;
    for (int it = 0; it < 64 && t >= 1; it++) {  // t halves (rounding up) to 1; the cap is only a guard
        if (delta(keys, n, i, i + (s + t) * d) > dnode) s += t;
        if (t == 1) break;
        t = (t + 1) >> 1;
    }
    int gamma = i + s * d + min(d, 0);
    const int first = min(i, j), last = max(i, j);
    int left = (first == gamma) ? ~gamma : gamma;
    int right = (last == gamma + 1) ? ~(gamma + 1) : gamma + 1;
    child[i] = make_int2(left, right);
    if (i == 0) parent_int[0] = -1;  // the root ends every bottom-up walk
    if (left >= 0) parent_int[left] = i; else parent_leaf[~left] = i;
    if (right >= 0) parent_int[right] = i; else parent_leaf[~right] = i;
}

// ---------------------------------------------------------------- step 5 ----
// Boxes and counts, and treelet restructuring (Karras & Aila 2013, "Fast
// parallel construction of high-quality bounding volume hierarchies"), in
// bottom-up passes over the binary tree. At each internal node p, once both of
// its subtrees are final, the treelet of p (p and the internal nodes below it found by
// repeatedly opening the treelet leaf of largest surface area, until
// kTreeletLeaves leaves) is rebuilt with the topology of least SAH cost over
// those leaves, found by dynamic programming over the leaves' subsets. The
// treelet keeps its node indices and its root's box; only the topology
// below the root changes. The passes also leave every internal node's
// triangle count in cnt (the collapse reads it).
// SAH cost model: internal node kSahCi x its area, triangle kSahCt x its area.
constexpr int kTreeletLeaves = 7;
// passes of the restructuring; measured on a B200 (1 M-triangle heightfield,
// coherent / incoherent Mrays/s): none 5835 / 2043, 1 pass 6686 / 2250,
// 2 passes 6928 / 2319, 3 passes 6988 / 2331
constexpr int kTreeletPasses = 2;
constexpr float kSahCi = 1.2f, kSahCt = 1.0f;

// Half the surface area of a box, and of a subset of a treelet's leaves. Which
// of two topologies of almost equal cost wins depends on the last bit, so
// every rounding of the costs is spelled out here: the tree of a mesh does
// not change with how the compiler contracts the sums around it.
__device__ __forceinline__ float box_area(const float3 &lo, const float3 &hi)
{
    const float dx = fmaxf(hi.x - lo.x, 0.f), dy = fmaxf(hi.y - lo.y, 0.f), dz = fmaxf(hi.z - lo.z, 0.f);
    return fmaf(dz, dx, fmaf(dx, dy, __fmul_rn(dy, dz)));
}
__device__ __forceinline__ float subset_area(const float3 &lo, const float3 &hi)
{
    const float dx = fmaxf(hi.x - lo.x, 0.f), dy = fmaxf(hi.y - lo.y, 0.f), dz = fmaxf(hi.z - lo.z, 0.f);
    return fmaf(dz, dx, fmaf(dy, dz, __fmul_rn(dx, dy)));
}

// Arrives at a binary node; true for the second of its two arrivals, which
// sees everything written before the first. The counter wraps back to 0 for
// the next pass. (One acquire-release atomic: with a full fence on either
// side the walk up the tree spent most of its time in fences.)
__device__ __forceinline__ bool second_arrival(uint32_t *count)
{
    uint32_t old;
    asm volatile("atom.inc.acq_rel.gpu.global.u32 %0, [%1], 1;" : "=r"(old) : "l"(count) : "memory");
    return old != 0u;
}

__device__ __forceinline__ void handle_box(int c, const uint32_t *sorted_tri, const float4 *tlo, const float4 *thi,
                                           const float4 *nlo, const float4 *nhi, float3 &lo, float3 &hi)
{
    float4 a, b;
    if (c >= 0) { a = __ldcg(&nlo[c]); b = __ldcg(&nhi[c]); }
    else { const uint32_t t = sorted_tri[~c]; a = tlo[t]; b = thi[t]; }
    lo = make_float3(a.x, a.y, a.z);
    hi = make_float3(b.x, b.y, b.z);
}

// The 127 non-empty subsets of the 7 treelet leaves ordered by size (7 of
// size 1, 21 of size 2, 35, 35, 21, 7, 1), and where each size starts.
struct SubsetTable {
    uint8_t s[127];
    uint8_t start[8];
};
constexpr SubsetTable make_subset_table()
{
    SubsetTable t{};
    int k = 0;
    for (int size = 1; size <= kTreeletLeaves; size++) {
        t.start[size - 1] = (uint8_t)k;
        for (int S = 1; S < (1 << kTreeletLeaves); S++)
        {
            int bits = 0;
            for (int b = 0; b < kTreeletLeaves; b++) bits += (S >> b) & 1;
            if (bits == size) t.s[k++] = (uint8_t)S;
        }
    }
    t.start[kTreeletLeaves] = (uint8_t)k;
    return t;
}
__constant__ SubsetTable c_subsets = make_subset_table();

constexpr int kTreeletThreads = 128;
constexpr int kTreeletWarps = kTreeletThreads / 32;

struct TreeletShared {
    float copt[1 << kTreeletLeaves];     // least cost of each subset of the leaves
    float area[1 << kTreeletLeaves];     // the area of its box
    uint8_t split[1 << kTreeletLeaves];  // the part with the lowest leaf of its best split
    float box[kTreeletLeaves][6];
    int leaf[kTreeletLeaves], count[kTreeletLeaves];
    int inner[kTreeletLeaves - 1];       // the treelet's internal nodes, its root first
    int subset[kTreeletLeaves - 1];      // the new topology: internal node i's leaves
    int2 kids[kTreeletLeaves - 1];
};

// Bit patterns of non-negative floats order like the floats. The least cost
// over the lanes of `group` and, among equal ones, the largest Q: the split
// that a loop over Q downwards finds first.
__device__ __forceinline__ void best_split(uint32_t group, float &cost, int &Q)
{
    const uint32_t bits = __float_as_uint(cost);
    const uint32_t least = __reduce_min_sync(group, bits);
    Q = (int)__reduce_max_sync(group, bits == least ? (uint32_t)Q : 0u);
    cost = __uint_as_float(least);
}

// Inserts a zero bit at position b of x.
__device__ __forceinline__ int open_bit(int x, int b) { return ((x >> b) << (b + 1)) | (x & ((1 << b) - 1)); }

// Bound by the dependent loads and the shared-memory search of each warp's
// chain of treelets, not by memory traffic. Measured on a B200, the two passes
// over 262 K triangles (with the boxes' pass before the first): 2.28 ms with
// one lane walking the treelet and solving sizes 6 and 7, 0.94 ms so; the
// whole build, with the scratch kept and the eight-lane collapse (0.45 ->
// 0.12 ms), 12.0 -> 1.24 ms, and 18.0 -> 2.6 ms for 1 M triangles.
//
// One warp rebuilds the treelet of root p (box area areap). Lane k < 7 holds
// leaf k: its handle, box, cost and count, loaded together when the leaf
// enters the treelet, so opening a node costs two dependent loads. The
// subsets' box areas are found four a lane; then the subsets of one size are
// solved per round: one lane a subset up to size 5, four lanes a subset at
// size 6 (31 splits each) and the whole warp at size 7 (63 splits). The new
// topology, if cheaper, is laid out by lane 0 and written by six lanes.
// Every cost is the same sum of the same floats whichever lane finds it.
// p's count and cost are final. All 32 lanes call this together.
__device__ void treelet_warp(int p, float areap, const uint32_t *sorted_tri, const float4 *tlo, const float4 *thi,
                             int2 *child, int *parent_int, int *parent_leaf, float4 *nlo, float4 *nhi, int *cnt,
                             float *cost, TreeletShared &s)
{
    constexpr uint32_t kFull = 0xffffffffu;
    constexpr int kAll = (1 << kTreeletLeaves) - 1;
    const int lane = threadIdx.x & 31;
    __syncwarp();  // behind the leader's arrival, which saw the subtree below p final
    int h = 0, count = 1;
    float3 lo = make_float3(0.f, 0.f, 0.f), hi = lo;
    float a = -1.f, c = 0.f;
    auto take = [&](int handle) {  // this lane's leaf
        h = handle;
        handle_box(h, sorted_tri, tlo, thi, nlo, nhi, lo, hi);
        a = box_area(lo, hi);
        count = h >= 0 ? __ldcg(&cnt[h]) : 1;
        c = h >= 0 ? __ldcg(&cost[h]) : kSahCt * a;
    };
    int2 kids = __ldcg(&child[p]);
    if (lane < 2) take(lane ? kids.y : kids.x);
    float cur = kSahCi * areap;
    int inner = p;  // lane i: internal node i of the treelet
    for (int n_l = 2; n_l < kTreeletLeaves; n_l++) {
        // the leaf of largest area that is a node, the first of equal ones
        const uint32_t key = lane < n_l && h >= 0 && a >= 0.f ? __float_as_uint(a) + 1u : 0u;
        const uint32_t best = __reduce_max_sync(kFull, key);
        if (best == 0u) return;  // (not reached: p has >= 7 triangles)
        const int w = __ffs(__ballot_sync(kFull, key == best)) - 1;
        const int open = __shfl_sync(kFull, h, w);
        if (lane == n_l - 1) inner = open;
        cur = fmaf(kSahCi, __uint_as_float(best - 1u), cur);
        kids = __ldcg(&child[open]);
        if (lane == w || lane == n_l) take(lane == w ? kids.x : kids.y);
    }
    if (lane < kTreeletLeaves) {
        float *b = s.box[lane];
        b[0] = lo.x; b[1] = lo.y; b[2] = lo.z; b[3] = hi.x; b[4] = hi.y; b[5] = hi.z;
        s.copt[1 << lane] = c;
        s.leaf[lane] = h;
        s.count[lane] = count;
        if (lane < kTreeletLeaves - 1) s.inner[lane] = inner;
    }
    __syncwarp();
#pragma unroll
    for (int k = 0; k < kTreeletLeaves; k++) cur += s.copt[1 << k];
    auto join = [&](float3 &l, float3 &u, int k) {
        const float *b = s.box[k];
        l = make_float3(fminf(l.x, b[0]), fminf(l.y, b[1]), fminf(l.z, b[2]));
        u = make_float3(fmaxf(u.x, b[3]), fmaxf(u.y, b[4]), fmaxf(u.z, b[5]));
    };
    {
        float3 l = make_float3(FLT_MAX, FLT_MAX, FLT_MAX), u = make_float3(-FLT_MAX, -FLT_MAX, -FLT_MAX);
#pragma unroll
        for (int k = 0; k < 5; k++)
            if (lane >> k & 1) join(l, u, k);
#pragma unroll
        for (int j = 0; j < 4; j++) {
            float3 l2 = l, u2 = u;
            if (j & 1) join(l2, u2, 5);
            if (j & 2) join(l2, u2, 6);
            s.area[lane + 32 * j] = subset_area(l2, u2);
        }
    }
    __syncwarp();
    // splits low | Q against S ^ low ^ Q, for Q downwards over the proper
    // subsets of S without its lowest leaf
    for (int size = 2; size <= 5; size++) {
        for (int j = c_subsets.start[size - 1] + lane; j < c_subsets.start[size]; j += 32) {
            const int S = c_subsets.s[j], low = S & -S, R = S ^ low;
            float best = FLT_MAX;
            int bq = 0;
            for (int Q = (R - 1) & R;; Q = (Q - 1) & R) {
                const float cc = s.copt[low | Q] + s.copt[R ^ Q];
                if (cc < best) { best = cc; bq = Q; }
                if (Q == 0) break;
            }
            s.copt[S] = fmaf(kSahCi, s.area[S], best);
            s.split[S] = (uint8_t)(low | bq);
        }
        __syncwarp();
    }
    if (lane < 28) {  // size 6: all leaves but e
        const uint32_t group = 15u << (lane & 28);
        const int e = lane >> 2, S = kAll ^ (1 << e), low = S & -S, R = S ^ low;
        float best = FLT_MAX;
        int bq = 0;
        for (int i = 30 - (lane & 3); i >= 0; i -= 4) {
            // bits of i to the places of R: 0..6 without 0 and e (e == 0: without 0 and 1)
            const int Q = e == 0 ? i << 2 : open_bit(i << 1, e);
            const float cc = s.copt[low | Q] + s.copt[R ^ Q];
            if (cc < best) { best = cc; bq = Q; }
        }
        best_split(group, best, bq);
        if ((lane & 3) == 0) {
            s.copt[S] = fmaf(kSahCi, s.area[S], best);
            s.split[S] = (uint8_t)(low | bq);
        }
    }
    __syncwarp();
    float all;
    {
        const int R = kAll ^ 1;
        float best = FLT_MAX;
        int bq = 0;
#pragma unroll
        for (int j = 1; j >= 0; j--) {
            const int Q = 2 * (lane + 32 * j);
            if (Q == R) continue;
            const float cc = s.copt[1 | Q] + s.copt[R ^ Q];
            if (cc < best) { best = cc; bq = Q; }
        }
        best_split(kFull, best, bq);
        all = fmaf(kSahCi, s.area[kAll], best);
        if (lane == 0) {
            s.copt[kAll] = all;
            s.split[kAll] = (uint8_t)(1 | bq);
        }
    }
    if (!(all < cur * 0.9999f)) {
        __syncwarp();
        return;
    }
    if (lane == 0) {
        int used = 1;
        s.subset[0] = kAll;
        for (int i = 0; i < kTreeletLeaves - 1; i++) {
            const int S = s.subset[i];
            int hs[2];
#pragma unroll
            for (int q = 0; q < 2; q++) {
                const int P = q ? S ^ s.split[S] : s.split[S];
                if ((P & (P - 1)) == 0) {
                    hs[q] = s.leaf[__ffs(P) - 1];
                } else {
                    s.subset[used] = P;
                    hs[q] = s.inner[used++];
                }
            }
            s.kids[i] = make_int2(hs[0], hs[1]);
        }
    }
    __syncwarp();
    if (lane < kTreeletLeaves - 1) {
        const int node = s.inner[lane], S = s.subset[lane];
        const int2 k2 = s.kids[lane];
        if (k2.x >= 0) __stcg(&parent_int[k2.x], node);
        else __stcg(&parent_leaf[~k2.x], node);
        if (k2.y >= 0) __stcg(&parent_int[k2.y], node);
        else __stcg(&parent_leaf[~k2.y], node);
        __stcg(&child[node], k2);
        __stcg(&cost[node], s.copt[S]);
        if (lane) {
            float3 l = make_float3(FLT_MAX, FLT_MAX, FLT_MAX), u = make_float3(-FLT_MAX, -FLT_MAX, -FLT_MAX);
            int cn = 0;
#pragma unroll
            for (int k = 0; k < kTreeletLeaves; k++) {
                if (!(S >> k & 1)) continue;
                join(l, u, k);
                cn += s.count[k];
            }
            __stcg(&nlo[node], make_float4(l.x, l.y, l.z, 0.f));
            __stcg(&nhi[node], make_float4(u.x, u.y, u.z, 0.f));
            __stcg(&cnt[node], cn);
        }
    }
    __syncwarp();  // before the leader's arrival at p's parent, which releases these writes
}

// The bottom-up pass: every lane with a leaf walks up from it; a lane whose
// node has both subtrees final (second arrival) sets the node's box
// (kBoxes: the first pass), count and cost, and the warp then rebuilds, one
// after another, the treelets of the nodes its lanes hold that have >=
// kTreeletLeaves triangles. Lanes stay in the loop until the whole warp is
// done (the treelet work uses all 32). The arrival counters wrap back to 0.
template <bool kBoxes>
__global__ void __launch_bounds__(kTreeletThreads) k_treelet(int n, const uint32_t *__restrict__ sorted_tri,
                                                             const float4 *__restrict__ tlo,
                                                             const float4 *__restrict__ thi, int2 *child,
                                                             int *parent_int, int *parent_leaf,
                                                             uint32_t *__restrict__ arrivals, float4 *nlo,
                                                             float4 *nhi, int *cnt, float *cost, int restructure,
                                                             int leaves)
{
    __shared__ TreeletShared shared[kTreeletWarps];
    const int w = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31, i = (blockIdx.x * kTreeletWarps + w) * leaves + lane;
    bool alive = lane < leaves && i < n;
    int p = alive ? parent_leaf[i] : -1;
    for (int guard = 0; guard <= n; guard++) {
        bool ready = false;
        float ap = 0.f;
        if (alive && (p < 0 || p >= n - 1)) alive = false;
        if (alive) {
            if (!second_arrival(&arrivals[p])) {
                alive = false;
            } else {
                const int2 c = __ldcg(&child[p]);
                int cp = 0;
                float part[2];
                float3 plo = make_float3(FLT_MAX, FLT_MAX, FLT_MAX), phi = make_float3(-FLT_MAX, -FLT_MAX, -FLT_MAX);
#pragma unroll
                for (int q = 0; q < 2; q++) {
                    const int h = q ? c.y : c.x;
                    if (kBoxes || h < 0) {
                        float3 lo, hi;
                        handle_box(h, sorted_tri, tlo, thi, nlo, nhi, lo, hi);
                        if (kBoxes) {
                            plo = make_float3(fminf(plo.x, lo.x), fminf(plo.y, lo.y), fminf(plo.z, lo.z));
                            phi = make_float3(fmaxf(phi.x, hi.x), fmaxf(phi.y, hi.y), fmaxf(phi.z, hi.z));
                        }
                        part[q] = kSahCt * box_area(lo, hi);
                    }
                    if (h >= 0) part[q] = __ldcg(&cost[h]);
                    cp += h >= 0 ? __ldcg(&cnt[h]) : 1;
                }
                if (kBoxes) {
                    __stcg(&nlo[p], make_float4(plo.x, plo.y, plo.z, 0.f));
                    __stcg(&nhi[p], make_float4(phi.x, phi.y, phi.z, 0.f));
                } else {
                    handle_box(p, sorted_tri, tlo, thi, nlo, nhi, plo, phi);
                }
                ap = box_area(plo, phi);
                __stcg(&cnt[p], cp);
                __stcg(&cost[p], __fadd_rn(fmaf(kSahCi, ap, part[0]), part[1]));
                ready = restructure && cp >= kTreeletLeaves;
            }
        }
        unsigned todo = __ballot_sync(0xffffffffu, ready);
        while (todo) {
            const int leader = __ffs(todo) - 1;
            todo &= todo - 1;
            const int q = __shfl_sync(0xffffffffu, p, leader);
            const float qa = __shfl_sync(0xffffffffu, ap, leader);
            treelet_warp(q, qa, sorted_tri, tlo, thi, child, parent_int, parent_leaf, nlo, nhi, cnt, cost, shared[w]);
        }
        if (alive) p = __ldcg(&parent_int[p]);
        if (!__any_sync(0xffffffffu, alive)) break;
    }
}

// ------------------------------------------------------------- step 5c ----
// Which binary nodes become 8-wide nodes, and which leaves, for least SAH
// cost (the dynamic program of Ylitie, Karras & Laine 2017, "Efficient
// incoherent ray traversal on GPUs through compressed wide BVHs", without its
// leaf reordering): bottom-up, for each binary node n and i = 1..8, the least
// cost of the subtree of n as at most i roots under an 8-wide parent. One
// root is n itself, as a leaf (<= kLeafMax triangles: its area x kColTri x
// its triangles) or as an 8-wide node (its area x kColNode + the least cost
// of its subtree below as at most 8 roots); more roots split the subtree
// between n's two children. Decisions per node (dpd, 16 bytes): [0] n as one
// root is a leaf (1) or an 8-wide node (0); [j - 1], j = 2..8: the left
// child's share of a j-root split; [8 + i - 1]: the roots (1 = n itself, or
// the split j) that give the least cost with at most i roots.
constexpr float kColNode = 1.0f, kColTri = 0.3f;

__device__ __forceinline__ void root_costs(int h, const uint32_t *sorted_tri, const float4 *tlo, const float4 *thi,
                                           const float *dpc, float (&c)[8])
{
    if (h < 0) {
        const uint32_t t = sorted_tri[~h];
        const float4 lo = tlo[t], hi = thi[t];
        const float a = kColTri * area(make_float3(lo.x, lo.y, lo.z), make_float3(hi.x, hi.y, hi.z));
#pragma unroll
        for (int i = 0; i < 8; i++) c[i] = a;
    } else {
        const float4 *src = reinterpret_cast<const float4 *>(dpc + 8 * (size_t)h);
        const float4 x = __ldcg(src), y = __ldcg(src + 1);
        c[0] = x.x; c[1] = x.y; c[2] = x.z; c[3] = x.w; c[4] = y.x; c[5] = y.y; c[6] = y.z; c[7] = y.w;
    }
}

__global__ void __launch_bounds__(128) k_collapse_cost(int n, const uint32_t *__restrict__ sorted_tri,
                                                       const float4 *__restrict__ tlo, const float4 *__restrict__ thi,
                                                       const int2 *__restrict__ child, const int *__restrict__ parent_int,
                                                       const int *__restrict__ parent_leaf,
                                                       uint32_t *__restrict__ arrivals, const float4 *__restrict__ nlo,
                                                       const float4 *__restrict__ nhi, const int *__restrict__ cnt,
                                                       float *dpc, uint8_t *__restrict__ dpd)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    int p = parent_leaf[i];
    for (int guard = 0; p >= 0 && p < n - 1 && guard < n; guard++) {
        if (!second_arrival(&arrivals[p])) return;
        const int2 c = child[p];
        float ca[8], cb[8];
        root_costs(c.x, sorted_tri, tlo, thi, dpc, ca);
        root_costs(c.y, sorted_tri, tlo, thi, dpc, cb);
        uint8_t dec[16];
        float split[8];  // [j - 1]: least cost of j roots split between the children
#pragma unroll
        for (int j = 2; j <= 8; j++) {
            float best = FLT_MAX;
            int bk = 1;
#pragma unroll
            for (int k = 1; k < j; k++) {
                const float v = ca[k - 1] + cb[j - k - 1];
                if (v < best) { best = v; bk = k; }
            }
            split[j - 1] = best;
            dec[j - 1] = (uint8_t)bk;
        }
        const float4 lo = nlo[p], hi = nhi[p];
        const float a = area(make_float3(lo.x, lo.y, lo.z), make_float3(hi.x, hi.y, hi.z));
        const int np = cnt[p];
        const float as_leaf = np <= kLeafMax ? kColTri * a * (float)np : FLT_MAX;
        const float as_node = kColNode * a + split[7];
        float cost[8];
        cost[0] = fminf(as_leaf, as_node);
        dec[0] = as_leaf <= as_node ? 1u : 0u;
        dec[8] = 1;
#pragma unroll
        for (int k = 2; k <= 8; k++) {
            cost[k - 1] = cost[k - 2];
            dec[8 + k - 1] = dec[8 + k - 2];
            if (split[k - 1] < cost[k - 1]) {
                cost[k - 1] = split[k - 1];
                dec[8 + k - 1] = (uint8_t)k;
            }
        }
        float4 *dst = reinterpret_cast<float4 *>(dpc + 8 * (size_t)p);
        __stcg(dst, make_float4(cost[0], cost[1], cost[2], cost[3]));
        __stcg(dst + 1, make_float4(cost[4], cost[5], cost[6], cost[7]));
        uint4 d;
        memcpy(&d, dec, 16);
        *reinterpret_cast<uint4 *>(dpd + 16 * (size_t)p) = d;
        p = parent_int[p];
    }
}

// ---------------------------------------------------------------- step 6 ----
struct Work {
    int bin;       // binary node: >= 0 internal, < 0 leaf ~sorted_pos (only for n == 1)
    uint32_t node; // 8-wide node index to fill
};

static_assert(sizeof(Work) == 8, "work item is 8 bytes");

__device__ __forceinline__ void child_box(int c, const uint32_t *sorted_tri, const float4 *tlo, const float4 *thi,
                                          const float4 *nlo, const float4 *nhi, float3 &lo, float3 &hi)
{
    float4 a, b;
    if (c >= 0) { a = nlo[c]; b = nhi[c]; }
    else { uint32_t t = sorted_tri[~c]; a = tlo[t]; b = thi[t]; }
    lo = make_float3(a.x, a.y, a.z);
    hi = make_float3(b.x, b.y, b.z);
}

// triangles below handle c (an internal node's count from k_treelet)
__device__ __forceinline__ int child_count(int c, const int *cnt) { return c >= 0 ? cnt[c] : 1; }

// whether root handle c becomes an 8-wide node (else a leaf child)
__device__ __forceinline__ bool is_node_root(int c, const uint8_t *dpd) { return c >= 0 && dpd[16 * (size_t)c] == 0; }

// The sorted positions of the triangles below handle c, which holds at most
// kLeafMax of them, left to right. Returns how many.
__device__ __forceinline__ int leaf_tris(int c, const int2 *child, int (&out)[kLeafMax])
{
    int st[2 * kLeafMax], sp = 0, m = 0;
    st[sp++] = c;
    for (int it = 0; it < 4 * kLeafMax && sp > 0; it++) {
        const int x = st[--sp];
        if (x < 0) {
            if (m < kLeafMax) out[m++] = ~x;
        } else if (sp + 2 <= 2 * kLeafMax) {
            const int2 cc = child[x];
            st[sp++] = cc.y;
            st[sp++] = cc.x;
        }
    }
    return m;
}

// The record of input triangle t.
__device__ __forceinline__ void write_tri(Tri *dst, uint32_t t, const float *__restrict__ pos,
                                          const uint32_t *__restrict__ idx)
{
    const uint32_t a = idx[3 * t], b = idx[3 * t + 1], c = idx[3 * t + 2];
    const float v0x = pos[3 * a], v0y = pos[3 * a + 1], v0z = pos[3 * a + 2];
    const float e1x = __fsub_rn(pos[3 * b], v0x), e1y = __fsub_rn(pos[3 * b + 1], v0y),
                e1z = __fsub_rn(pos[3 * b + 2], v0z);
    const float e2x = __fsub_rn(pos[3 * c], v0x), e2y = __fsub_rn(pos[3 * c + 1], v0y),
                e2z = __fsub_rn(pos[3 * c + 2], v0z);
    const float nx = __fsub_rn(__fmul_rn(e1y, e2z), __fmul_rn(e1z, e2y));
    const float ny = __fsub_rn(__fmul_rn(e1z, e2x), __fmul_rn(e1x, e2z));
    const float nz = __fsub_rn(__fmul_rn(e1x, e2y), __fmul_rn(e1y, e2x));
    dst->a = make_float4(v0x, v0y, v0z, nx);
    dst->b = make_float4(e1x, e1y, e1z, ny);
    dst->c = make_float4(e2x, e2y, e2z, nz);
    dst->id = make_uint4(t, 0u, 0u, 0u);
}

// Quantisation step for one axis: the smallest power of two 2^e with
// extent / 2^e <= 255 - 2 (one step of slack each side), and never below
// `min_step` so that a step stays many float ulps wide.
__device__ __forceinline__ int quant_exp(float extent, float min_step)
{
    float target = fmaxf(extent / 253.0f, min_step);
    int e;
    frexpf(target, &e);  // target = m * 2^e, m in [0.5, 1)  ->  2^e >= target
    e = max(e, -120);
    e = min(e, 127);
    return e;
}

__device__ __forceinline__ float exp2i(int e) { return ldexpf(1.0f, e); }

// One 8-wide node per group of eight lanes. The levels are short chains of
// dependent loads, not much work: with one thread a node (which kept the
// children, their scores and the slots in local memory) a level took 40 to
// 50 us whatever its size.
constexpr int kCollapseThreads = 128;

__global__ void __launch_bounds__(kCollapseThreads)
    k_collapse(const Work *__restrict__ in, const uint32_t *__restrict__ in_count, Work *__restrict__ out,
               uint32_t *__restrict__ out_count, uint32_t out_cap, const int2 *__restrict__ child,
               const int *__restrict__ cnt, const uint8_t *__restrict__ dpd, const float4 *__restrict__ nlo,
               const float4 *__restrict__ nhi, const uint32_t *__restrict__ sorted_tri, const float4 *__restrict__ tlo,
               const float4 *__restrict__ thi, const float *__restrict__ pos, const uint32_t *__restrict__ idx,
               Node8 *__restrict__ nodes, uint32_t *__restrict__ node_count, uint32_t node_cap, Tri *__restrict__ tris,
               uint32_t *__restrict__ tri_count, uint32_t tri_cap, float min_step, uint32_t *__restrict__ levels,
               uint32_t *__restrict__ err)
{
    constexpr uint32_t kFull = 0xffffffffu;
    constexpr int kNone = INT_MIN;
    __shared__ uint32_t s_planes[kCollapseThreads / 8][12];  // per group: the node's plane bytes
    __shared__ uint8_t s_at[kCollapseThreads];               // per group: the child in each slot
    const int lane = threadIdx.x & 31, l = lane & 7, shift = lane & 24, group = threadIdx.x >> 3;
    uint8_t *planes = reinterpret_cast<uint8_t *>(s_planes[group]);
    // The host does not know how many items a level has: the grid strides
    // over them. A level without items ends the build.
    const uint32_t items = min(*in_count, out_cap);
    if (blockIdx.x == 0 && threadIdx.x == 0 && items) *levels += 1u;
    const uint32_t per_block = kCollapseThreads / 8, stride = gridDim.x * per_block;
    for (uint32_t w0 = blockIdx.x * per_block; w0 < items; w0 += stride) {
        const uint32_t w = w0 + group;
        const bool live = w < items;
        const Work job = live ? in[w] : Work{~0, 0u};
        auto sum8 = [&](uint32_t v) {
            for (int o = 1; o < 8; o <<= 1) v += __shfl_xor_sync(kFull, v, o);
            return v;
        };
        auto min8 = [&](float v) {
            for (int o = 1; o < 8; o <<= 1) v = fminf(v, __shfl_xor_sync(kFull, v, o));
            return v;
        };
        auto ballot8 = [&](bool v) { return __ballot_sync(kFull, v) >> shift & 0xffu; };

        // The roots the collapse costs chose for the subtree below this
        // node, left to right: a handle h that may spread over r roots starts
        // at a lane and owns it and the r - 1 behind; a split into k and
        // j - k roots leaves the left part there and puts the right part k
        // lanes on.
        int h = kNone, roots = 0;
        if (live && job.bin < 0 && l == 0) h = job.bin;  // single-triangle scene
        if (live && job.bin >= 0) {
            const int2 c = child[job.bin];
            const int k8 = dpd[16 * (size_t)job.bin + 7];
            if (l == 0) { h = c.x; roots = k8; }
            if (l == k8) { h = c.y; roots = 8 - k8; }
        }
        for (int round = 0; round < 8; round++) {
            int j = 1, k = 0;
            int2 c = make_int2(0, 0);
            if (h >= 0) {
                const uint4 d = *reinterpret_cast<const uint4 *>(dpd + 16 * (size_t)h);
                c = child[h];
                auto byte = [&](int b) {
                    const uint32_t word = b < 8 ? (b < 4 ? d.x : d.y) : (b < 12 ? d.z : d.w);
                    return (int)(word >> (8 * (b & 3)) & 0xffu);
                };
                j = byte(8 + roots - 1);
                if (j > 1) k = byte(j - 1);
            }
            const bool split = j > 1;
            if (!__any_sync(kFull, split)) break;
            const uint32_t owners = ballot8(h != kNone);
            // the lane that owns this one, and whether its right part starts here
            const int owner = 31 - __clz((owners & ((2u << l) - 1u)) | 1u);
            const int ok = __shfl_sync(kFull, split ? k : 0, shift + owner);
            const int oj = __shfl_sync(kFull, j, shift + owner), oy = __shfl_sync(kFull, c.y, shift + owner);
            if (split) {
                h = c.x;
                roots = k;
            } else if (h == kNone && ok > 0 && owner + ok == l) {
                h = oy;
                roots = oj - ok;
            }
        }
        // child k = the k-th owner: its box, kind and triangles
        const uint32_t owners = ballot8(h != kNone);
        const int m = __popc(owners);
        const bool has = l < m;
        if (h != kNone) s_at[threadIdx.x - l + __popc(owners & ((1u << l) - 1u))] = (uint8_t)l;
        __syncwarp();
        h = __shfl_sync(kFull, h, shift + (has ? s_at[threadIdx.x] : 0));
        float3 clo = make_float3(FLT_MAX, FLT_MAX, FLT_MAX), chi = make_float3(-FLT_MAX, -FLT_MAX, -FLT_MAX);
        bool node = false;
        int n_tris = 0;
        if (has) {
            child_box(h, sorted_tri, tlo, thi, nlo, nhi, clo, chi);
            node = is_node_root(h, dpd);
            n_tris = node ? 0 : child_count(h, cnt);
        }
        const float3 plo = make_float3(min8(clo.x), min8(clo.y), min8(clo.z));
        const float3 phi = make_float3(-min8(-chi.x), -min8(-chi.y), -min8(-chi.z));

        // Slots: slot s is the corner with bit k set = positive along axis k.
        // The best remaining (child, slot) pair takes its slot, the first in
        // (child, slot) order of equal ones.
        int slot = -1;
        {
            const float3 pc = make_float3(0.5f * (plo.x + phi.x), 0.5f * (plo.y + phi.y), 0.5f * (plo.z + phi.z));
            const float3 c = make_float3(0.5f * (clo.x + chi.x) - pc.x, 0.5f * (clo.y + chi.y) - pc.y,
                                         0.5f * (clo.z + chi.z) - pc.z);
            uint32_t used = 0;
            for (int it = 0; it < 8; it++) {
                // 0 = no candidate; a NaN score ranks below every other
                uint32_t best = 0;
                int bs = 0;
                if (has && slot < 0) {
#pragma unroll
                    for (int s = 0; s < 8; s++) {
                        if (used >> s & 1u) continue;
                        // (+ 0 turns -0 into +0, which compare equal)
                        const float score = ((s & 1) ? c.x : -c.x) + ((s & 2) ? c.y : -c.y) + ((s & 4) ? c.z : -c.z) + 0.f;
                        const uint32_t key = score == score ? max(float_flip(score), 2u) : 1u;
                        if (key > best) { best = key; bs = s; }
                    }
                }
                uint32_t top = best;
                for (int o = 1; o < 8; o <<= 1) top = max(top, __shfl_xor_sync(kFull, top, o));
                const uint32_t winners = ballot8(best == top && top != 0u);
                const int who = winners ? __ffs(winners) - 1 : 0;
                const int ws = __shfl_sync(kFull, bs, shift + who);
                if (winners) used |= 1u << ws;
                if (winners && l == who) slot = ws;
                if (!__any_sync(kFull, winners != 0u)) break;
            }
        }

        // node and triangle records: one allocation a group
        const uint32_t n_int = __popc(ballot8(node)), n_leaf = sum8((uint32_t)n_tris);
        uint32_t child_base = 0, tri_base = 0, queue = 0;
        if (live && l == 0 && n_int) child_base = atomicAdd(node_count, n_int);
        if (live && l == 1 && n_leaf) tri_base = atomicAdd(tri_count, n_leaf);
        if (live && l == 2 && n_int) queue = atomicAdd(out_count, n_int);
        child_base = __shfl_sync(kFull, child_base, shift);
        tri_base = __shfl_sync(kFull, tri_base, shift + 1);
        queue = __shfl_sync(kFull, queue, shift + 2);
        const uint32_t full = (child_base + n_int > node_cap ? 2u : 0u) | (tri_base + n_leaf > tri_cap ? 4u : 0u) |
                              (queue + n_int > out_cap ? 8u : 0u);
        if (full && live && l == 0) atomicOr(err, full);
        const bool write = live && !full;

        // quantisation frame: origin one step below the union so that
        // floor() never goes negative
        const int ex = quant_exp(phi.x - plo.x, min_step), ey = quant_exp(phi.y - plo.y, min_step),
                  ez = quant_exp(phi.z - plo.z, min_step);
        const float sx = exp2i(ex), sy = exp2i(ey), sz = exp2i(ez);
        const float3 org = make_float3(plo.x - sx, plo.y - sy, plo.z - sz);

        // lane s: the child in slot s
        __syncwarp();
        s_at[threadIdx.x] = 0xff;
        __syncwarp();
        if (slot >= 0) s_at[threadIdx.x - l + slot] = (uint8_t)l;
        __syncwarp();
        const uint32_t k = s_at[threadIdx.x];
        const bool filled = k != 0xffu;
        const int from = shift + (filled ? (int)k : l);
        h = __shfl_sync(kFull, h, from);
        node = __shfl_sync(kFull, (int)node, from) && filled;
        n_tris = __shfl_sync(kFull, n_tris, from);
        if (!filled) n_tris = 0;
        clo = make_float3(__shfl_sync(kFull, clo.x, from), __shfl_sync(kFull, clo.y, from), __shfl_sync(kFull, clo.z, from));
        chi = make_float3(__shfl_sync(kFull, chi.x, from), __shfl_sync(kFull, chi.y, from), __shfl_sync(kFull, chi.z, from));
        const uint32_t inner = ballot8(node);
        uint32_t tri_off = (uint32_t)n_tris;  // inclusive prefix sum over the slots
        for (int o = 1; o < 8; o <<= 1) {
            const uint32_t up = __shfl_up_sync(kFull, tri_off, o, 8);
            if (l >= o) tri_off += up;
        }
        tri_off -= (uint32_t)n_tris;
        // conservative 8-bit box: floor/ceil in double (exact for float
        // inputs), one extra step of slack each side
        auto low = [&](float v, float o, float s) {
            return filled ? (uint8_t)fmin(fmax(floor(((double)v - o) / s) - 1, 0.0), 255.0) : (uint8_t)0;
        };
        auto high = [&](float v, float o, float s) {
            return filled ? (uint8_t)fmin(fmax(ceil(((double)v - o) / s) + 1, 0.0), 255.0) : (uint8_t)0;
        };
        planes[l] = low(clo.x, org.x, sx);
        planes[8 + l] = high(chi.x, org.x, sx);
        planes[16 + l] = low(clo.y, org.y, sy);
        planes[24 + l] = high(chi.y, org.y, sy);
        planes[32 + l] = low(clo.z, org.z, sz);
        planes[40 + l] = high(chi.z, org.z, sz);
        const uint32_t slots = sum8((node ? 8u : (1u << n_tris) - 1u) << (4 * l));
        __syncwarp();
        if (write && l < 6) {
            uint4 q;
            if (l == 0) {
                q = make_uint4(__float_as_uint(org.x), __float_as_uint(org.y), __float_as_uint(org.z), child_base);
            } else if (l == 1) {
                q = make_uint4((uint32_t)(ex + 127) << 23, (uint32_t)(ey + 127) << 23, (uint32_t)(ez + 127) << 23,
                               tri_base);
            } else if (l == 5) {
                q = make_uint4(slots, 0u, 0u, 0u);
            } else {
                const uint32_t *b = s_planes[group] + 4 * (l - 2);
                q = make_uint4(b[0], b[1], b[2], b[3]);
            }
            nodes[job.node].q[l] = q;
        }
        if (write && node) {
            const uint32_t nth = __popc(inner & ((1u << l) - 1u));
            out[queue + nth] = Work{h, child_base + nth};
        }
        if (write && n_tris) {
            int at[kLeafMax];
            leaf_tris(h, child, at);
#pragma unroll
            for (int q = 0; q < kLeafMax; q++)
                if (q < n_tris) write_tri(tris + tri_base + tri_off + q, sorted_tri[at[q]], pos, idx);
        }
        __syncwarp();  // the planes are read before the next item's are written
    }
}

__global__ void k_root(Work *q, int n, uint32_t *counters)
{
    q[0] = Work{n > 1 ? 0 : ~0, 0u};
    counters[0] = 1;  // the root node
    counters[4] = 1;  // level 0's work item
}

inline uint32_t div_up(uint64_t a, uint32_t b) { return (uint32_t)((a + b - 1) / b); }

__global__ void k_nodes_to_file(const Node8 *__restrict__ in, uint32_t n, FileNode8 *__restrict__ out)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = to_file(in[i]);
}

__global__ void k_nodes_from_file(const FileNode8 *__restrict__ in, uint32_t n, Node8 *__restrict__ out)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = from_file(in[i]);
}

__global__ void k_tris_to_file(const Tri *__restrict__ in, uint32_t n, FileTri *__restrict__ out,
                               uint32_t *__restrict__ prim)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const Tri t = in[i];
    out[i] = FileTri{t.a, t.b, t.c};
    prim[i] = t.id.x;
}

__global__ void k_tris_from_file(const FileTri *__restrict__ in, const uint32_t *__restrict__ prim, uint32_t n,
                                 Tri *__restrict__ out)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const FileTri t = in[i];
    out[i] = Tri{t.a, t.b, t.c, make_uint4(prim[i], 0u, 0u, 0u)};
}

}  // namespace

cudaError_t records_to_file(const Node8 *nodes, uint32_t n, FileNode8 *out, cudaStream_t st)
{
    k_nodes_to_file<<<div_up(n, 128), 128, 0, st>>>(nodes, n, out);
    return cudaGetLastError();
}

cudaError_t records_to_file(const Tri *tris, uint32_t n, FileTri *out, uint32_t *prim, cudaStream_t st)
{
    k_tris_to_file<<<div_up(n, 128), 128, 0, st>>>(tris, n, out, prim);
    return cudaGetLastError();
}

cudaError_t records_from_file(const FileNode8 *in, uint32_t n, Node8 *nodes, cudaStream_t st)
{
    k_nodes_from_file<<<div_up(n, 128), 128, 0, st>>>(in, n, nodes);
    return cudaGetLastError();
}

cudaError_t records_from_file(const FileTri *in, const uint32_t *prim, uint32_t n, Tri *tris, cudaStream_t st)
{
    k_tris_from_file<<<div_up(n, 128), 128, 0, st>>>(in, prim, n, tris);
    return cudaGetLastError();
}

// ---------------------------------------------------------------------------
#define ILG_CK(call)                                                                       \
    do {                                                                                   \
        cudaError_t e_ = (call);                                                           \
        if (e_ != cudaSuccess) {                                                           \
            snprintf(err, err_len, "%s: %s (%s:%d)", #call, cudaGetErrorString(e_), __FILE__, __LINE__); \
            return 3;                                                                      \
        }                                                                                  \
    } while (0)

int bvh_build(BuildBuffers &B, const float *d_pos, uint32_t n_verts, const uint32_t *d_idx, uint32_t n,
              cudaStream_t st, BuildResult &res, char *err, size_t err_len)
{
    if (n == 0) {
        snprintf(err, err_len, "ilg_build: empty mesh");
        return 1;
    }
    // scratch sizing
    size_t sort_tmp = 0;
    ILG_CK(cub::DeviceRadixSort::SortPairs(nullptr, sort_tmp, (uint32_t *)nullptr, (uint32_t *)nullptr,
                                           (uint32_t *)nullptr, (uint32_t *)nullptr, (int)n, 0, 30, st));
    const uint32_t node_cap = n;           // 8-wide nodes never exceed the triangle count
    const uint32_t tri_cap = n;
    const uint32_t queue_cap = n + 1;
    ILG_CK(B.reserve(n, sort_tmp, node_cap, queue_cap));

    ILG_CK(cudaMemsetAsync(B.counters, 0, BuildBuffers::kCounters * sizeof(uint32_t), st));
    const uint32_t T = 256;
    k_tri_bounds<<<div_up(n, T), T, 0, st>>>(d_pos, n_verts, d_idx, n, B.tlo, B.thi, B.cbounds, B.err);
    k_morton<<<div_up(n, T), T, 0, st>>>(B.tlo, B.thi, n, B.cbounds, B.keys, B.vals);
    ILG_CK(cudaGetLastError());
    ILG_CK(cub::DeviceRadixSort::SortPairs(B.sort_tmp, sort_tmp, B.keys, B.keys_alt, B.vals, B.vals_alt, (int)n, 0,
                                           30, st));
    if (n > 1) {
        k_karras<<<div_up(n - 1, T), T, 0, st>>>(B.keys_alt, (int)n, B.child, B.parent_int, B.parent_leaf);
        ILG_CK(cudaMemsetAsync(B.arrivals, 0, sizeof(uint32_t) * (n - 1), st));
        // Leaves a warp starts from: it rebuilds the treelets of its lanes
        // one after another, so small meshes take fewer, for shorter chains
        // on more SMs; enough warps to fill the GPU anyway take all 32 (1 M
        // triangles: 4 leaves 4.4 ms, 8 3.8, 16 3.4, 32 3.2 for the build).
        int leaves = 32;
        while (leaves > 4 && n / (uint32_t)leaves < (uint32_t)current_sm_count() * 24u) leaves /= 2;
        const uint32_t tblocks = div_up(n, kTreeletWarps * (uint32_t)leaves);
        for (int pass = 0; pass < (res.treelets ? kTreeletPasses : 1); pass++) {
            (pass == 0 ? k_treelet<true> : k_treelet<false>)<<<tblocks, kTreeletThreads, 0, st>>>(
                (int)n, B.vals_alt, B.tlo, B.thi, B.child, B.parent_int, B.parent_leaf, B.arrivals, B.nlo, B.nhi,
                B.cnt, B.cost, res.treelets ? 1 : 0, leaves);
            ILG_CK(cudaGetLastError());
        }
        k_collapse_cost<<<div_up(n, 128), 128, 0, st>>>((int)n, B.vals_alt, B.tlo, B.thi, B.child, B.parent_int,
                                                        B.parent_leaf, B.arrivals, B.nlo, B.nhi, B.cnt, B.dpc, B.dpd);
        ILG_CK(cudaGetLastError());
    }
    k_root<<<1, 1, 0, st>>>((Work *)B.qa_raw, (int)n, B.counters);
    ILG_CK(cudaGetLastError());

    // Levels go to the stream kLevelBatch at a time (a tree of a few million
    // triangles has 7 to 10), each over as many items as the previous one
    // made; the host looks at the counters once a batch.
    constexpr int kLevelBatch = 12;
    const float min_step = res.min_step;
    Work *qin = (Work *)B.qa_raw, *qout = (Work *)B.qb_raw;
    const uint32_t blocks = std::min<uint32_t>(div_up(n, kCollapseThreads / 8), (uint32_t)current_sm_count() * 16u);
    uint32_t h[BuildBuffers::kCounters];
    for (int level = 0;;) {
        for (int k = 0; k < kLevelBatch && level < kMaxLevels; k++, level++) {
            k_collapse<<<blocks, kCollapseThreads, 0, st>>>(qin, B.counters + 4 + level, qout, B.counters + 5 + level, queue_cap,
                                              B.child, B.cnt, B.dpd, B.nlo, B.nhi, B.vals_alt, B.tlo, B.thi, d_pos,
                                              d_idx, B.nodes, B.counters + 0, node_cap, B.tris, B.counters + 1,
                                              tri_cap, min_step, B.counters + 2, B.err);
            std::swap(qin, qout);
        }
        ILG_CK(cudaGetLastError());
        ILG_CK(cudaMemcpyAsync(h, B.counters, sizeof(h), cudaMemcpyDeviceToHost, st));
        ILG_CK(cudaStreamSynchronize(st));
        if (h[4 + level] == 0) break;
        if (level >= kMaxLevels) {
            snprintf(err, err_len, "ilg_build: collapse did not converge");
            return 5;
        }
    }
    const uint32_t herr = h[3], depth = h[2];
    if (herr & 1u) {
        snprintf(err, err_len, "ilg_build: triangle index out of range of the vertex array");
        return 1;
    }
    if (herr) {
        snprintf(err, err_len, "ilg_build: capacity exceeded (flags 0x%x)", herr);
        return 5;
    }
    if (h[1] != n) {
        snprintf(err, err_len, "ilg_build: %u triangle records written for %u triangles", h[1], n);
        return 5;
    }
    res.n_nodes = h[0];
    res.n_tris = h[1];
    res.depth = depth;
    return 0;
}

}  // namespace ilg
