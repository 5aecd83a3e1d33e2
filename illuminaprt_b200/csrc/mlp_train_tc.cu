// Radiance-cache training on the 5th-generation tensor cores.
//
// k_mlp_train_tc: one CTA of 512 threads per SM takes 128-row tiles of the
// batch through
//   * the forward pass: the encoded input X and the hidden activations
//     H_0..H_4 (ReLU, rounded to BF16) stay in shared memory as K-major
//     A tiles, every layer one tcgen05.mma group (M = 128, K = 96 or 64,
//     N = 64 or 16) against the forward weight copy, accumulated in TMEM;
//   * the loss: the relative L2 loss of the three outputs (y held constant
//     in the denominator) and dL/dy, rounded to BF16 as dZ_5;
//   * the backward pass: dH_{l-1} = dZ_l W_l^T as one MMA group per layer
//     against the backward weight copy (W_l as N = in x K = out), masked by
//     H_{l-1} > 0 and rounded to BF16 as dZ_{l-1};
//   * the weight gradients: dW_l = H_{l-1}^T dZ_l as MMAs over the tile's
//     128 rows with both operands read MN-major from the very tiles above (an
//     8 x 8 core matrix with the features contiguous is K-major for the
//     layers and MN-major for their transposes). Each layer's sum has its own
//     TMEM columns, grows over the CTA's tiles and is added to the FP32
//     gradient once, at the end, in 16-byte vector atomics. These MMAs go out
//     behind the layer's own and run under its epilogue; dZ alternates between
//     two tiles for that.
// Only dZ_0 leaves the CTA (column-major, for the grid's gradient).
//
// Bound by a tile's serial chain: encode, eleven layers of barrier, issue,
// MMA, wait, load, convert and store. Four threads share a row (its TMEM lane
// can be read by the four warps of one lane quarter) to shorten every link.
// Measured on a B200, gradients of 16,384 rows with the hash grid: 67.8 us with
// a thread a row, weights copied through registers and the activations written
// out for a second kernel that summed the weight gradients a K step at a time
// (53.8 with both of those kernels pipelined but apart); 43.3 us so, of which the
// encoding was about a quarter and the weight gradient's atomics 4 (39.5 since,
// by the grid's kernel and the clears).
//
// The arithmetic is the warp-level kernels' (mlp.cu): BF16 operands at the
// same points, FP32 accumulation. Every mbarrier wait is bounded and raises
// an error bit instead of hanging; TMEM is allocated once per CTA and freed
// on exit.
#include "devinfo.cuh"
#include "mlp.cuh"
#include "umma.cuh"

namespace ilg {

namespace {

using namespace umma;

constexpr int kTrRows = 128;
constexpr int kTrSplit = 4;                      // threads a row: 16 of a layer's 64 columns each
constexpr int kTrThreads = kTrRows * kTrSplit;
static_assert(kMlpHid == 16 * kTrSplit && kMlpIn / 8 == 3 * kTrSplit, "columns of a row's threads");
// TMEM columns: the layers' accumulator, then dW_0..dW_4, then dW_5
constexpr uint32_t kTrTmemCols = 512;
__host__ __device__ constexpr uint32_t dw_col(int l) { return 64u + 64u * (uint32_t)l; }
static_assert(dw_col(kMlpLayers - 1) + 16 <= kTrTmemCols, "TMEM columns");
constexpr size_t kTrWf = ((kUmmaElems * 2 + 1023) / 1024) * 1024;     // forward weights
constexpr size_t kTrWb = ((kUmmaBwdElems * 2 + 1023) / 1024) * 1024;  // backward weights
constexpr size_t kTrX = (size_t)kTrRows * kMlpIn * 2;                 // X tile
constexpr size_t kTrH = (size_t)kTrRows * kMlpHid * 2;                // one hidden tile, one dZ tile
constexpr size_t kTrSmem = kTrWf + kTrWb + kTrX + 7 * kTrH;
static_assert(kTrSmem <= 227 * 1024, "shared memory of the training kernel");
static_assert(kTrX % 1024 == 0 && kTrH % 1024 == 0, "tile alignment");

// One layer's MMAs, D (TMEM, 128 x N) = A (128 x K) B^T (B: N x K), both
// K-major tiles of 8-row x 16-byte core matrices; issued by one thread and
// committed to `bar`.
template <int K, int N>
__device__ __forceinline__ void issue_layer(uint32_t tmem, uint32_t a_addr, uint32_t b_addr, uint32_t bar)
{
    const uint64_t da = umma_desc(a_addr, 128, (K / 8) * 128), db = umma_desc(b_addr, 128, (K / 8) * 128);
#pragma unroll
    for (int s = 0; s < K / 16; s++)  // 256 bytes on, in units of 16
        mma_bf16(tmem, da + 16u * s, db + 16u * s, umma_idesc(kTrRows, N), s > 0 ? 1u : 0u);
    mma_commit(bar);
}

// dW (TMEM, in x N) += A^T B over the tile's 128 rows: A the K-major tile of
// a layer's input (kIn features), B the one of its dZ (kOut columns), both
// read MN-major: 128 bytes to the next 8 features, a row of core matrices to
// the next 8 rows. M is 128 whatever kIn: the features past it are what lies
// behind (shared memory of this CTA) and fill lanes that nothing reads.
template <int kIn, int kOut>
__device__ __forceinline__ void issue_dw(uint32_t tmem, uint32_t a_addr, uint32_t b_addr, bool add)
{
    constexpr uint32_t a_rows = (kIn / 8) * 128, b_rows = (kOut / 8) * 128;
    constexpr uint32_t idesc = umma_idesc(128, kOut) | 1u << 15 | 1u << 16;  // A and B MN-major
    const uint64_t da = umma_desc(a_addr, a_rows, 128), db = umma_desc(b_addr, b_rows, 128);
#pragma unroll
    for (int s = 0; s < kTrRows / 16; s++)
        mma_bf16(tmem, da + s * (2 * a_rows / 16), db + s * (2 * b_rows / 16), idesc, (s > 0 || add) ? 1u : 0u);
}

// `bytes` (a multiple of 16, both addresses aligned to it) from global to
// shared memory by the copy engine, counted on `bar`.
__device__ __forceinline__ void bulk_load(uint32_t dst, const void *src, uint32_t bytes, uint32_t bar)
{
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
                 "l"(src), "r"(bytes), "r"(bar)
                 : "memory");
}

__global__ void __launch_bounds__(kTrThreads, 1) k_mlp_train_tc(const MlpDev M, const float *__restrict__ raw,
                                                                const float *__restrict__ target, uint32_t n,
                                                                const TrainRows rows)
{
    n = rows_of(n, rows);
    if (blockIdx.x * kTrRows >= n) return;
    // counts the Adam step whose kernel comes next
    if (rows.count && blockIdx.x == 0 && threadIdx.x == 0) *M.step += 1u;
    extern __shared__ __align__(1024) unsigned char smem[];
    unsigned char *wf_s = smem, *wb_s = smem + kTrWf, *x_s = wb_s + kTrWb, *h_s = x_s + kTrX, *dz_s = h_s + 5 * kTrH;
    __shared__ __align__(8) uint64_t bar, wbar, drain;
    __shared__ uint32_t tmem_base_s;

    const int warp = threadIdx.x >> 5, part = threadIdx.x / kTrRows, tid = threadIdx.x % kTrRows;
    const uint32_t bar_a = smem_u32(&bar), wbar_a = smem_u32(&wbar);
    const uint32_t wf_a = smem_u32(wf_s), wb_a = smem_u32(wb_s), x_a = smem_u32(x_s), h_a = smem_u32(h_s);
    const uint32_t dz_a = smem_u32(dz_s);
    if (threadIdx.x == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar_a) : "memory");
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(wbar_a) : "memory");
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&drain)) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        // the weights arrive while the first tile is encoded
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(wbar_a),
                     "r"((uint32_t)(kUmmaElems + kUmmaBwdElems) * 2u)
                     : "memory");
        bulk_load(wf_a, M.wu, kUmmaElems * 2, wbar_a);
        bulk_load(wb_a, M.wv, kUmmaBwdElems * 2, wbar_a);
    }
    if (warp == 0) {
        __syncwarp();
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_s)),
                     "r"(kTrTmemCols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    fence_before_sync();
    __syncthreads();
    fence_after_sync();
    const uint32_t tmem = tmem_base_s;
    const uint32_t taddr = tmem + ((uint32_t)((warp & 3) * 32) << 16) + 16u * part;  // this thread's 16 columns
    const size_t cap = M.cap;
    const float inv_count = 1.f / (3.f * (float)n);
    uint32_t phase = 0;
    bool ok = true;
    float loss = 0.f;

    // Every thread's part of the A tile in place; false when a wait of any
    // thread ran out before.
    auto ready = [&]() {
        fence_async_smem();
        fence_before_sync();
        ok = __syncthreads_and(ok) != 0;
        fence_after_sync();
        return ok;
    };
    // waits for the layer's MMAs (a wait that runs out sets the error bit)
    auto wait_layer = [&]() {
        if (!mbar_wait(bar_a, phase)) {
            atomicOr(M.err, kErrWait);
            ok = false;
        }
        phase ^= 1u;
        fence_after_sync();
    };
    // this thread's 16 accumulator values
    auto load_acc = [&](float (&v)[16]) {
        tmem_ld16(taddr, v);
        tmem_wait_ld(v);
    };
    auto put16 = [&](unsigned char *tile, const float (&v)[16]) {
        put_chunk(tile, tid, 2 * part, kMlpHid, v);
        put_chunk(tile, tid, 2 * part + 1, kMlpHid, v + 8);
    };

    const uint32_t n_tiles = (n + kTrRows - 1) / kTrRows;
    for (uint32_t tile = blockIdx.x; tile < n_tiles; tile += gridDim.x) {
        const uint32_t row = tile * kTrRows + tid;
        const bool live = row < n, add = tile != blockIdx.x;
        // the encoded input: the A tile of layer 0. Each of the row's threads takes every fourth 8-column chunk (with
        // the hash grid: four levels and two chunks of the rest).
        {
            float f[kMlpRaw];
            const float4 *src = reinterpret_cast<const float4 *>(raw + (size_t)row * kMlpRaw);
#pragma unroll
            for (int k = 0; k < 4; k++) {
                const float4 q = live ? src[k] : make_float4(0.f, 0.f, 0.f, 0.f);
                f[4 * k] = q.x;
                f[4 * k + 1] = q.y;
                f[4 * k + 2] = q.z;
                f[4 * k + 3] = q.w;
            }
            int c = part;
            if (M.encoding == kEncHashGrid) {
                float v[8];
#pragma unroll
                for (int e = 0; e < 8; e += 2) {  // the loads of the four levels go out together
                    const float2 p = grid_features(M, 4 * part + e / 2, f[0], f[1], f[2]);
                    v[e] = live ? p.x : 0.f;
                    v[e + 1] = live ? p.y : 0.f;
                }
                put_chunk(x_s, tid, c, kMlpIn, v);
                c += kTrSplit;
            }
#pragma unroll 1
            for (; c < kMlpIn / 8; c += kTrSplit) {
                float v[8];
#pragma unroll
                for (int e = 0; e < 8; e += 2) {
                    const float2 p = encode_pair(f, 8 * c + e, M);
                    v[e] = live ? p.x : 0.f;
                    v[e + 1] = live ? p.y : 0.f;
                }
                put_chunk(x_s, tid, c, kMlpIn, v);
            }
        }
        if (!mbar_wait(wbar_a, 0u)) {  // the weights (a tile after the first finds them there)
            atomicOr(M.err, kErrWait);
            ok = false;
        }
        // forward
#pragma unroll 1
        for (int l = 0; l < kMlpLayers - 1; l++) {
            if (!ready()) break;
            if (threadIdx.x == 0) {
                if (l == 0)
                    issue_layer<kMlpIn, kMlpHid>(tmem, x_a, wf_a, bar_a);
                else
                    issue_layer<kMlpHid, kMlpHid>(tmem, h_a + (uint32_t)((l - 1) * kTrH),
                                                  wf_a + 2u * (umma_off(1) + (l - 1) * kMlpHid * kMlpHid), bar_a);
            }
            wait_layer();
            float v[16];
            load_acc(v);
#pragma unroll
            for (int e = 0; e < 16; e++) v[e] = fmaxf(v[e], 0.f);
            put16(h_s + (size_t)l * kTrH, v);
        }
        // the output layer, the loss and dL/dy (mean over rows and RGB of
        // (y - t)^2 / (y^2 + 0.01)): one thread a row
        if (!ready()) break;
        if (threadIdx.x == 0)
            issue_layer<kMlpHid, umma_n(kMlpLayers - 1)>(tmem, h_a + (uint32_t)(4 * kTrH),
                                                         wf_a + 2u * umma_off(kMlpLayers - 1), bar_a);
        wait_layer();
        if (part == 0) {
            float y[16], d[16];
            load_acc(y);
#pragma unroll
            for (int e = 0; e < 16; e++) d[e] = 0.f;
#pragma unroll
            for (int c = 0; c < 3; c++) {
                if (live) {
                    const float t = target[(size_t)row * 3 + c];
                    const float den = y[c] * y[c] + 0.01f;
                    const float diff = y[c] - t;
                    loss += diff * diff / den;
                    d[c] = 2.f * diff / den * inv_count;
                }
            }
            // dZ_5 as the A tile of the first backward layer (K = 16)
            put_chunk(dz_s + kTrH, tid, 0, 16, d);
            put_chunk(dz_s + kTrH, tid, 1, 16, d + 8);
        }
        // backward: dZ_{l-1} = (dZ_l W_l^T) * (H_{l-1} > 0), dZ_l in tile l & 1
#pragma unroll 1
        for (int l = kMlpLayers - 1; l >= 1; l--) {
            if (!ready()) break;
            if (threadIdx.x == 0) {
                const uint32_t a = dz_a + (l & 1) * (uint32_t)kTrH, h = h_a + (uint32_t)((l - 1) * kTrH);
                if (l == kMlpLayers - 1) {
                    issue_layer<umma_bk(kMlpLayers - 1), kMlpHid>(tmem, a, wb_a + 2u * umma_boff(kMlpLayers - 1), bar_a);
                    issue_dw<kMlpHid, umma_n(kMlpLayers - 1)>(tmem + dw_col(l), h, a, add);
                } else {
                    issue_layer<kMlpHid, kMlpHid>(tmem, a, wb_a + 2u * (uint32_t)((l - 1) * kMlpHid * kMlpHid), bar_a);
                    issue_dw<kMlpHid, kMlpHid>(tmem + dw_col(l), h, a, add);
                }
            }
            wait_layer();
            const unsigned char *ht = h_s + (size_t)(l - 1) * kTrH;
            float v[16];
            load_acc(v);
#pragma unroll
            for (int h = 0; h < 2; h++) {
                // this row's 8 activations of chunk 2 * part + h (the K-major tile's 16-byte row piece)
                const uint4 hv = *reinterpret_cast<const uint4 *>(ht + (size_t)(tid / 8) * (kMlpHid / 8) * 128 +
                                                                  (size_t)(2 * part + h) * 128 + (tid % 8) * 16);
                const uint32_t w4[4] = {hv.x, hv.y, hv.z, hv.w};
#pragma unroll
                for (int e = 0; e < 4; e++) {
                    if (!((w4[e] & 0x7fffu) != 0u && !(w4[e] & 0x8000u))) v[8 * h + 2 * e] = 0.f;
                    if (!((w4[e] >> 16 & 0x7fffu) != 0u && !(w4[e] & 0x80000000u))) v[8 * h + 2 * e + 1] = 0.f;
                }
            }
            put16(dz_s + ((l - 1) & 1) * kTrH, v);
            if (l == 1 && live && M.encoding == kEncHashGrid) {
#pragma unroll
                for (int e = 0; e < 16; e++) M.dzcm[(size_t)(16 * part + e) * cap + row] = __float2bfloat16_rn(v[e]);
            }
        }
        if (!ready()) break;
        if (threadIdx.x == 0) {
            issue_dw<kMlpIn, kMlpHid>(tmem + dw_col(0), x_a, dz_a, add);
            mma_commit(bar_a);
        }
        wait_layer();  // all of the tile's MMAs: its shared memory is free again
    }
    ok = __syncthreads_and(ok) != 0;
    fence_after_sync();
    if (ok) {
        // row `tid` of each dW_l, this thread's 16 columns of it
#pragma unroll 1
        for (int k = 0; k < kMlpLayers; k++) {  // neighbouring CTAs begin with different layers
            const int l = (int)((blockIdx.x + k) % kMlpLayers);
            const int in = mlp_in(l), out = mlp_out(l);
            if ((warp & 3) * 32 >= in || 16 * part >= out) continue;  // whole warps
            float v[16];
            tmem_ld16(taddr + dw_col(l), v);
            tmem_wait_ld(v);
            float *g = M.grad + mlp_off(l) + (size_t)tid * out + 16 * part;
#pragma unroll
            for (int e = 0; e < 16; e += 4)  // four columns in one vector atomic (sm_90 and later)
                if (16 * part + e < out)
                    atomicAdd(reinterpret_cast<float4 *>(g + e), make_float4(v[e], v[e + 1], v[e + 2], v[e + 3]));
        }
    } else if (threadIdx.x == 0) {
        mbar_wait(wbar_a, 0u);  // nothing may arrive in shared memory after the block has gone
        mma_drain(smem_u32(&drain));
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) loss += __shfl_xor_sync(0xffffffffu, loss, o);
    if ((threadIdx.x & 31) == 0 && loss != 0.f) atomicAdd(M.loss, loss / (3.f * (float)n));
    fence_before_sync();
    __syncthreads();
    fence_after_sync();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTrTmemCols) : "memory");
}

}  // namespace

cudaError_t mlp_train_tc(const MlpDev &M, const float *raw, const float *target, uint32_t n, cudaStream_t st,
                         const TrainRows &rows)
{
    if (n == 0) return cudaSuccess;
    if ((uintptr_t)raw & 15u) return cudaErrorMisalignedAddress;  // rows are read as 16-byte vectors
    const uint32_t n_pad = (n + 15) / 16 * 16;
    if (n_pad > M.cap) return cudaErrorInvalidValue;
    cudaError_t e = ensure_dynamic_smem((const void *)k_mlp_train_tc, (int)kTrSmem);
    if (e != cudaSuccess) return e;
    const uint32_t tiles = (n + kTrRows - 1) / kTrRows;
    const uint32_t sms = (uint32_t)current_sm_count();
    k_mlp_train_tc<<<tiles < sms ? tiles : sms, kTrThreads, kTrSmem, st>>>(M, raw, target, n, rows);
    return cudaGetLastError();
}

}  // namespace ilg
