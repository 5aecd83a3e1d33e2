// Device data layout of the 8-wide BVH and the reference-compatible triangle
// test shared by the build and the traversal kernels.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

namespace ilg {

// ---------------------------------------------------------------------------
// Node record: 96 bytes, 32-byte aligned, read with three 256-bit loads.
//   q0: origin.xyz (float bits), w = first child node
//   q1: quantisation step per axis (float bits of powers of two), w = first
//       triangle record
//   q2: x/y = qlo.x[0..7], z/w = qhi.x[0..7]   (one byte per slot)
//   q3: same for y, q4: same for z
//   q5: x = slots word, the rest 0
// The lanes of a warp visit different nodes, so each of a lane's loads costs
// L1 a cycle of its own: as five 16-byte loads of an 80-byte record the node
// fetches kept L1's data pipe 70 % busy; in three loads the record is read in
// three cycles a lane, and it covers three 32-byte sectors either way.
// Slots word: one nibble per slot. 0 = empty slot; 8 = internal child;
// 1, 3 or 7 = a leaf with 1, 2 or 3 triangles (one bit each). The triangles
// of a node's leaves are stored contiguously in slot order, so the triangle
// of bit b is record first_triangle + popc(slots & 0x77777777 & ((1 << b) - 1)).
// The traversal gets a node's hit children and hit triangles from one AND
// with a mask that has a whole nibble per hit slot.
// Internal children of a node are stored contiguously in slot order, so the
// child in slot s is node first_child + popc(slots & 0x88888888 & ((8 << 4 s) - 1)).
// Slots are assigned so that a ray in octant o visits children in
// descending order of (slot ^ (7 - o)), which approximates front to back.
// ---------------------------------------------------------------------------
struct __align__(32) Node8 {
    uint4 q[6];
};
static_assert(sizeof(Node8) == 96, "node record must be 96 bytes");

// Node record of a scene file: 80 bytes.
//   q0: origin.xyz, w = ex | ey << 8 | ez << 16 | imask << 24 (e* are the
//       biased exponents of the quantisation steps, imask bit s = slot s holds
//       an internal child)
//   q1: x = first child node, y = first triangle record,
//       z = meta[0..3], w = meta[4..7]
//   q2..q4: the plane bytes, as above
// meta byte of a slot: 0 = empty; 0x80 = internal child; otherwise a leaf
// with count (1..3) in bits 5-6 and the offset of its first triangle from the
// node's first triangle record (0..23) in bits 0-4.
struct __align__(16) FileNode8 {
    uint4 q[5];
};
static_assert(sizeof(FileNode8) == 80, "file node record must be 80 bytes");

// Triangle record: 64 bytes, 32-byte aligned, read with two loads.
//   a = (v0.x, v0.y, v0.z, n.x), b = (e1.xyz, n.y), c = (e2.xyz, n.z)
//   id = (index in the input mesh, material (low 16 bits) | light (high 16,
//         0xffff none; written by build_tri_attr before a render), 0, 0)
// with e1 = v1 - v0, e2 = v2 - v0, n = e1 x e2 evaluated exactly as the
// reference does (IndexedTriangle.cpp:44-45, :103), one rounding per op.
struct __align__(32) Tri {
    float4 a, b, c;
    uint4 id;
};
static_assert(sizeof(Tri) == 64, "triangle record must be 64 bytes");

// Triangle record of a scene file: 48 bytes (the input indices follow as an
// array of their own).
struct __align__(16) FileTri {
    float4 a, b, c;
};
static_assert(sizeof(FileTri) == 48, "file triangle record must be 48 bytes");

constexpr int kMaxStack = 64;      // traversal stack entries (node groups)
// triangles per leaf child; measured on a B200 with the treelet-restructured
// tree (1 M-triangle heightfield, coherent / incoherent Mrays/s; 21 M-triangle
// field, 960x540x16 ms): 1: 6790 / 2254, 25.6; 2: 7100 / 2357, 26.0;
// 3: 6920 / 2316, 26.7
constexpr int kLeafMax = 2;
constexpr uint32_t kSlotInner = 0x88888888u, kSlotTris = 0x77777777u;
constexpr uint32_t kMetaInternal = 0x80u;  // scene file

__host__ __device__ inline FileNode8 to_file(const Node8 &n)
{
    FileNode8 f;
    uint32_t imask = 0, off = 0;
    uint64_t meta = 0;
    for (int s = 0; s < 8; s++) {
        const uint32_t nib = (n.q[5].x >> (4 * s)) & 15u;
        const uint32_t count = nib == 7u ? 3u : (nib == 3u ? 2u : (nib == 1u ? 1u : 0u));
        if (nib == 8u) {
            imask |= 1u << s;
            meta |= (uint64_t)kMetaInternal << (8 * s);
        } else if (count) {
            meta |= (uint64_t)((count << 5) | off) << (8 * s);
        }
        off += count;
    }
    f.q[0] = uint4{n.q[0].x, n.q[0].y, n.q[0].z,
                   n.q[1].x >> 23 | (n.q[1].y >> 23) << 8 | (n.q[1].z >> 23) << 16 | imask << 24};
    f.q[1] = uint4{n.q[0].w, n.q[1].w, (uint32_t)meta, (uint32_t)(meta >> 32)};
    for (int a = 0; a < 3; a++) f.q[2 + a] = n.q[2 + a];
    return f;
}

// Whether a file's record is one that to_file writes: triangle offsets that
// follow from the counts, an imask that agrees with the slots.
inline bool canonical(const FileNode8 &f)
{
    uint32_t off = 0;
    for (int s = 0; s < 8; s++) {
        const uint32_t m = ((s < 4 ? f.q[1].z : f.q[1].w) >> (8 * (s & 3))) & 0xffu, count = m >> 5 & 3u;
        const bool inner = m == kMetaInternal;
        if (inner != ((f.q[0].w >> (24 + s) & 1u) != 0u)) return false;
        if (inner || m == 0u) continue;
        if (count == 0u || m != (count << 5 | off)) return false;
        off += count;
    }
    return true;
}

__host__ __device__ inline Node8 from_file(const FileNode8 &f)
{
    uint32_t slots = 0;
    for (int s = 0; s < 8; s++) {
        const uint32_t m = ((s < 4 ? f.q[1].z : f.q[1].w) >> (8 * (s & 3))) & 0xffu;
        slots |= (m == kMetaInternal ? 8u : (1u << ((m >> 5) & 3u)) - 1u) << (4 * s);
    }
    const uint32_t e = f.q[0].w;
    Node8 n;
    n.q[0] = uint4{f.q[0].x, f.q[0].y, f.q[0].z, f.q[1].x};
    n.q[1] = uint4{(e & 0xffu) << 23, (e >> 8 & 0xffu) << 23, (e >> 16 & 0xffu) << 23, f.q[1].y};
    for (int a = 0; a < 3; a++) n.q[2 + a] = f.q[2 + a];
    n.q[5] = uint4{slots, 0u, 0u, 0u};
    return n;
}

// The smallest direction component that the box test divides by, for a scene
// with coordinates up to max_abs: 1e-20, and more in scenes above 8e14 units,
// where a quantisation step (at most 2^-5.9 max_abs) times 32768 and the
// reciprocal (see node_misses) would pass FLT_MAX and every box be missed.
// 2^-116 max_abs keeps that product below 2^126; a ray that it tilts is off by
// a whole step only at distances of 2^90 steps.
inline float min_direction(float max_abs) { return max_abs * 0x1p-116f > 1e-20f ? max_abs * 0x1p-116f : 1e-20f; }

// Lower bound of the reference's triangle window, `t < 1e-5` evaluated in
// double (IndexedTriangle.cpp:115): for a float t this is t < the smallest
// float >= 1e-5, i.e. 0x3727C5AD.
__device__ __forceinline__ float window_lo() { return __int_as_float(0x3727C5AD); }

// Upper bound: `t > Max - 1e-5` in double holds for a float t exactly when
// t > (Max - 1e-5) rounded down to float.
__device__ __forceinline__ float window_hi(float tmax)
{
    return __double2float_rd(__dsub_rn((double)tmax, 1e-5));
}

// Shirley-form test of IndexedTriangle::Intersects (IndexedTriangle.cpp:92-128)
// with every product and sum rounded separately (no contraction), so that t,
// beta and gamma are bit-identical to the reference compiled without FMA.
// `hi` is window_hi(current Max).
__device__ __forceinline__ bool shirley(float4 ta, float4 tb, float4 tc, float ox, float oy, float oz, float dx, float dy,
                                        float dz, float hi, float &t_out, float &b_out, float &g_out)
{
    const float nx = ta.w, ny = tb.w, nz = tc.w;
    const float den = __fadd_rn(__fadd_rn(__fmul_rn(nx, dx), __fmul_rn(ny, dy)), __fmul_rn(nz, dz));
    const float rcp = __frcp_rn(den);  // correctly rounded, as the division 1 / den is
    const float ex = __fsub_rn(ta.x, ox), ey = __fsub_rn(ta.y, oy), ez = __fsub_rn(ta.z, oz);
    const float num = __fadd_rn(__fadd_rn(__fmul_rn(nx, ex), __fmul_rn(ny, ey)), __fmul_rn(nz, ez));
    const float t = __fmul_rn(num, rcp);
    if (t > hi || t < window_lo()) return false;
    // interm = d x edge2
    const float ix = __fsub_rn(__fmul_rn(dy, ez), __fmul_rn(dz, ey));
    const float iy = __fsub_rn(__fmul_rn(dz, ex), __fmul_rn(dx, ez));
    const float iz = __fsub_rn(__fmul_rn(dx, ey), __fmul_rn(dy, ex));
    const float beta =
        __fmul_rn(__fadd_rn(__fadd_rn(__fmul_rn(ix, tc.x), __fmul_rn(iy, tc.y)), __fmul_rn(iz, tc.z)), -rcp);
    if (beta < 0.0f) return false;
    const float gamma =
        __fmul_rn(__fadd_rn(__fadd_rn(__fmul_rn(ix, tb.x), __fmul_rn(iy, tb.y)), __fmul_rn(iz, tb.z)), rcp);
    if (__fadd_rn(beta, gamma) > 1.0f || gamma < 0.0f) return false;
    // A NaN t (origin in the triangle's plane, direction parallel to it)
    // passes the reference's comparisons and poisons its ray.Max; it is
    // rejected here instead.
    if (!(t <= hi)) return false;
    t_out = t;
    b_out = beta;
    g_out = gamma;
    return true;
}

// ---------------------------------------------------------------------------
// Watertight test (Woop, Benthin and Wald 2013, "Watertight Ray/Triangle
// Intersection", JCGT 2(1)): the triangle is sheared into the ray's frame
// (the ray's largest direction component becomes z) and the three 2D edge
// functions U, V, W are evaluated from the vertices themselves, so two
// triangles that share an edge evaluate it with the same numbers and a ray
// through it cannot slip between them. Edge functions that come out exactly
// zero are recomputed in double. Every operation is rounded separately. The
// rejection window is the reference's (t < 1e-5 or t > Max - 1e-5); beta
// and gamma are the weights of v1 and v2, as in the reference.
// ---------------------------------------------------------------------------
struct Shear {
    uint32_t kx, ky, kz;
    float sx, sy, sz;
};

__device__ __forceinline__ float pick(float x, float y, float z, uint32_t k) { return k == 0u ? x : (k == 1u ? y : z); }

__device__ __forceinline__ Shear shear_of(float dx, float dy, float dz)
{
    const float ax = fabsf(dx), ay = fabsf(dy), az = fabsf(dz);
    Shear s;
    s.kz = ax >= ay ? (ax >= az ? 0u : 2u) : (ay >= az ? 1u : 2u);
    s.kx = s.kz == 2u ? 0u : s.kz + 1u;
    s.ky = s.kx == 2u ? 0u : s.kx + 1u;
    const float dkz = pick(dx, dy, dz, s.kz);
    if (dkz < 0.f) {
        const uint32_t k = s.kx;
        s.kx = s.ky;
        s.ky = k;
    }
    s.sx = __fdiv_rn(pick(dx, dy, dz, s.kx), dkz);
    s.sy = __fdiv_rn(pick(dx, dy, dz, s.ky), dkz);
    s.sz = __fdiv_rn(1.0f, dkz);
    return s;
}

// v0, v1, v2: the triangle's own vertices (w unused).
__device__ __forceinline__ bool watertight(float4 v0, float4 v1, float4 v2, float ox, float oy, float oz,
                                           const Shear &sh, float hi, float &t_out, float &b_out, float &g_out)
{
    const float a0 = __fsub_rn(v0.x, ox), a1 = __fsub_rn(v0.y, oy), a2 = __fsub_rn(v0.z, oz);
    const float b0 = __fsub_rn(v1.x, ox), b1 = __fsub_rn(v1.y, oy), b2 = __fsub_rn(v1.z, oz);
    const float c0 = __fsub_rn(v2.x, ox), c1 = __fsub_rn(v2.y, oy), c2 = __fsub_rn(v2.z, oz);
    const float akz = pick(a0, a1, a2, sh.kz), bkz = pick(b0, b1, b2, sh.kz), ckz = pick(c0, c1, c2, sh.kz);
    const float Ax = __fsub_rn(pick(a0, a1, a2, sh.kx), __fmul_rn(sh.sx, akz));
    const float Ay = __fsub_rn(pick(a0, a1, a2, sh.ky), __fmul_rn(sh.sy, akz));
    const float Bx = __fsub_rn(pick(b0, b1, b2, sh.kx), __fmul_rn(sh.sx, bkz));
    const float By = __fsub_rn(pick(b0, b1, b2, sh.ky), __fmul_rn(sh.sy, bkz));
    const float Cx = __fsub_rn(pick(c0, c1, c2, sh.kx), __fmul_rn(sh.sx, ckz));
    const float Cy = __fsub_rn(pick(c0, c1, c2, sh.ky), __fmul_rn(sh.sy, ckz));
    float U = __fsub_rn(__fmul_rn(Cx, By), __fmul_rn(Cy, Bx));
    float V = __fsub_rn(__fmul_rn(Ax, Cy), __fmul_rn(Ay, Cx));
    float W = __fsub_rn(__fmul_rn(Bx, Ay), __fmul_rn(By, Ax));
    if (U == 0.f || V == 0.f || W == 0.f) {
        U = __double2float_rn(__dsub_rn(__dmul_rn(Cx, By), __dmul_rn(Cy, Bx)));
        V = __double2float_rn(__dsub_rn(__dmul_rn(Ax, Cy), __dmul_rn(Ay, Cx)));
        W = __double2float_rn(__dsub_rn(__dmul_rn(Bx, Ay), __dmul_rn(By, Ax)));
    }
    if ((U < 0.f || V < 0.f || W < 0.f) && (U > 0.f || V > 0.f || W > 0.f)) return false;
    const float det = __fadd_rn(__fadd_rn(U, V), W);
    if (det == 0.f) return false;
    const float Az = __fmul_rn(sh.sz, akz), Bz = __fmul_rn(sh.sz, bkz), Cz = __fmul_rn(sh.sz, ckz);
    const float T = __fadd_rn(__fadd_rn(__fmul_rn(U, Az), __fmul_rn(V, Bz)), __fmul_rn(W, Cz));
    const float rcp = __frcp_rn(det);
    const float t = __fmul_rn(T, rcp);
    if (!(t <= hi) || t < window_lo()) return false;
    t_out = t;
    b_out = __fmul_rn(V, rcp);
    g_out = __fmul_rn(W, rcp);
    return true;
}

}  // namespace ilg
