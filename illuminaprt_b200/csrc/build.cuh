// Buffers and entry point of the device BVH build (build.cu).
#pragma once

#include <cstddef>
#include <cstdint>
#include <cstdio>
#include <cuda_runtime.h>

#include <type_traits>

#include "bvh8.cuh"

namespace ilg {

// Grow-only device allocation owned by a context.
template <class T>
struct DevBuf {
    T *ptr = nullptr;
    size_t cap = 0;  // elements
    cudaError_t reserve(size_t n)
    {
        if (n <= cap) return cudaSuccess;
        if (ptr) cudaFree(ptr);
        ptr = nullptr;
        cap = 0;
        cudaError_t e = cudaMalloc((void **)&ptr, (n ? n : 1) * sizeof(T));
        if (e == cudaSuccess) cap = n;
        return e;
    }
    void release()
    {
        if (ptr) cudaFree(ptr);
        ptr = nullptr;
        cap = 0;
    }
};

// Levels of 8-wide nodes the collapse can count (a tree has far fewer).
constexpr int kMaxLevels = 208;

struct BuildBuffers {
    // scratch (valid only during a build), carved out of one allocation: a
    // build made of 25 of them spent three quarters of its time in cudaMalloc
    // and cudaFree (262 K triangles: 12.0 ms, of which 3.1 ms on the device)
    DevBuf<unsigned char> scratch_b;
    int builds = 0;  // builds of the context so far (2: more)
    // outputs (the built scene)
    DevBuf<Node8> nodes_b;
    DevBuf<Tri> tris_b;

    float4 *tlo, *thi, *nlo, *nhi;
    uint32_t *keys, *keys_alt, *vals, *vals_alt, *arrivals, *cbounds, *counters, *err;
    int2 *child;
    int *parent_int, *parent_leaf, *cnt;
    float *cost, *dpc;  // dpc: 8 collapse costs a binary node
    uint8_t *dpd;       // 16 collapse decisions a binary node
    void *sort_tmp;
    void *qa_raw, *qb_raw;  // two 8-byte work-item queues
    Node8 *nodes;
    Tri *tris;

    // counters: [0] nodes, [1] triangle records, [2] levels, [3] error flags,
    // [4 + l] work items of level l, then the 6 centroid bounds
    static constexpr size_t kCounters = 4 + kMaxLevels + 1 + 6;

    cudaError_t reserve(size_t n, size_t sort_bytes, size_t node_cap, size_t queue_cap)
    {
        size_t total = 0;
        for (int pass = 0; pass < 2; pass++) {
            unsigned char *base = scratch_b.ptr;
            total = 0;
            auto take = [&](auto *&p, size_t count) {
                using T = std::remove_reference_t<decltype(*p)>;
                if (pass) p = reinterpret_cast<T *>(base + total);
                total += (count * sizeof(T) + 255) / 256 * 256;
            };
            take(tlo, n); take(thi, n); take(nlo, n); take(nhi, n);
            take(dpc, 8 * n); take(dpd, 16 * n); take(child, n);
            take(keys, n); take(keys_alt, n); take(vals, n); take(vals_alt, n); take(arrivals, n);
            take(parent_int, n); take(parent_leaf, n); take(cnt, n); take(cost, n);
            take(counters, kCounters);
            uint64_t *qa, *qb;  // work items, 8 bytes each
            unsigned char *st;
            take(qa, queue_cap); take(qb, queue_cap); take(st, sort_bytes);
            if (pass) {
                qa_raw = qa; qb_raw = qb; sort_tmp = st; err = counters + 3; cbounds = counters + 4 + kMaxLevels + 1;
            } else {
                cudaError_t e = scratch_b.reserve(total);
                if (e != cudaSuccess) return e;
            }
        }
        cudaError_t e;
        if ((e = nodes_b.reserve(node_cap)) != cudaSuccess) return e;
        if ((e = tris_b.reserve(n)) != cudaSuccess) return e;
        nodes = nodes_b.ptr; tris = tris_b.ptr;
        return cudaSuccess;
    }

    // After a build: a context that builds again and again keeps scratch of up
    // to 256 MB (1.4 M triangles, 180 bytes each) for its next build; its first
    // build, which may be its only one, a failed one and larger ones give it
    // back at once.
    void release_scratch(bool built)
    {
        if (!built || builds == 0 || scratch_b.cap > ((size_t)256 << 20)) scratch_b.release();
        if (built && builds < 2) builds++;
    }

    void release_all()
    {
        scratch_b.release();
        nodes_b.release(); tris_b.release();
    }
};

struct BuildResult {
    float min_step = 0.f;   // in: smallest quantisation step (world units)
    bool treelets = true;   // in: restructure the binary tree by treelets before the collapse
    uint32_t n_nodes = 0;   // out
    uint32_t n_tris = 0;    // out
    uint32_t depth = 0;     // out
};

// Records of a built scene to those of a scene file and back, on the device.
cudaError_t records_to_file(const Node8 *nodes, uint32_t n, FileNode8 *out, cudaStream_t st);
cudaError_t records_to_file(const Tri *tris, uint32_t n, FileTri *out, uint32_t *prim, cudaStream_t st);
cudaError_t records_from_file(const FileNode8 *in, uint32_t n, Node8 *nodes, cudaStream_t st);
cudaError_t records_from_file(const FileTri *in, const uint32_t *prim, uint32_t n, Tri *tris, cudaStream_t st);

// Returns 0 on success, else an ilg_status code with `err` filled in.
int bvh_build(BuildBuffers &B, const float *d_pos, uint32_t n_verts, const uint32_t *d_idx, uint32_t n,
              cudaStream_t st, BuildResult &res, char *err, size_t err_len);

}  // namespace ilg
