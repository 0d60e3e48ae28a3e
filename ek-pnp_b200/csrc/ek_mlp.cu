// ek_mlp.cu -- the learned warm start (new; the reference has none): a
// 4 -> 256 -> 256 -> 256 -> 512 MLP with SiLU, trained and evaluated on the
// GPU by hand-written kernels.
//
//   GEMMs      C = A B^T on the 5th-generation tensor cores: BF16 operands
//              brought by TMA into a ring of shared-memory stages (K-major,
//              128-byte swizzle), tcgen05.mma issued by one thread into an
//              FP32 accumulator in tensor memory as each K chunk lands,
//              completion through tcgen05.commit on an mbarrier (bounded
//              waits), tcgen05.ld and a fused epilogue (bias, SiLU, SiLU
//              derivative, BF16 and transposed BF16 stores).
//   training   per iteration: batch gather, 4 forward GEMMs, MSE loss and its
//              gradient, 3 backward-data GEMMs with 4 weight-gradient GEMMs and
//              bias gradients beside them, Adam on FP32 master weights, BF16 casts --
//              16 launches, captured once in a CUDA graph and replayed.
// Weights are used in BF16 with FP32 accumulation; the FP32 master copy, the
// Adam moments and the gradients live in one flat buffer laid out per layer
// as W (out x in, row-major, layer-0 inputs padded from 4 to 16) then b.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <random>
#include <string>
#include <vector>

#include "ek_ctx.h"
#include "ek_tc.cuh"

using bf16 = __nv_bfloat16;

namespace {

constexpr int TM = 128;  // rows of a CTA tile (the MMA's M)
constexpr int KC = 64;   // K elements staged per round
constexpr int NT_MAX = 128;
constexpr int NL = 4;
constexpr int IN = 4, INP = 16, HID = 256, OUT = 512;
constexpr int DIM_IN[NL] = {INP, HID, HID, HID};
constexpr int DIM_OUT[NL] = {HID, HID, HID, OUT};

enum Epi { EPI_F32 = 0, EPI_FWD_HIDDEN = 1, EPI_FWD_OUT = 2, EPI_BWD_HIDDEN = 3 };

struct GemmArgs {
    CUtensorMap ta;  // A: M x K BF16, boxes of TM rows x KC columns
    CUtensorMap tb;  // B: N x K BF16, boxes of nt rows x KC columns
    int m, n, k, nt, stages, zoff;
    float *c;       // EPI_F32 / EPI_FWD_OUT: M x N fp32, row stride ldc
    int ldc;
    bool c_vec;     // c and ldc allow 16-byte stores
    const float *bias;
    float *z;       // EPI_FWD_HIDDEN: pre-activations out (may be null); EPI_BWD_HIDDEN: pre-activations in
    int ldz;
    bf16 *h;        // BF16 result, row stride ldh
    int ldh;
    bf16 *ht;       // BF16 transposed result, row stride ldht (may be null in EPI_FWD_HIDDEN)
    int ldht;
    int *err;
    long long wait_cycles;  // bound of each wait for the MMAs of a K chunk
};

__device__ __forceinline__ float silu(float z) { return z / (1.0f + expf(-z)); }
__device__ __forceinline__ float silu_grad(float z) {
    const float s = 1.0f / (1.0f + expf(-z));
    return s * (1.0f + z * (1.0f - s));
}

// One 128 x nt tile of C = A B^T per CTA.
//
// What bounds it: latency.  The network's GEMMs are small (256 x 256 x 256:
// 0.02 us of tensor time), so a launch is one round trip for the operands,
// the MMAs, and the epilogue's stores.  Hence
//  * narrow tiles (tile_columns), so that a GEMM spreads over tens of CTAs;
//  * operands by TMA (one box a K chunk and operand, 128-byte swizzle), up to
//    MAX_STAGES chunks in flight (all of K <= 512): 16-byte cp.async copies
//    by 256 threads took 4.5 us to bring in 64 KB of A;
//  * programmatic dependent launch, with the operand that the kernel just
//    before did not write (B: weights, or activations of the forward pass)
//    and the pre-activations fetched before the wait;
//  * an epilogue through shared memory with 16 warps, so that global stores
//    are runs of 8- and 16-byte vectors and the SiLUs of a tile take one round
//    (each thread storing its own row's elements one by one was most of a
//    launch: 45 us for a hidden layer of 256 rows).
//
// K is cut into chunks of KC = one 128-byte swizzle row; chunk c is staged in
// ring slot c % stages (A: TM rows, then B: nt rows).  One thread issues the
// copies (a "full" mbarrier a slot counts their bytes), the tcgen05.mma
// instructions of each chunk as it lands, and a commit to the slot's "empty"
// mbarrier where the slot is refilled; the last commit goes to `done`.  Every
// wait is bounded.
constexpr int GT = 512;  // threads
constexpr int MAX_STAGES = 8;
constexpr int STAGE_A = TM * KC * 2;
__host__ __device__ constexpr int stage_bytes(int nt) { return STAGE_A + nt * KC * 2; }
// Epilogue tiles, over the ring once the MMAs are done: the accumulator, FP32
// TM x (nt + 4), and the BF16 result transposed, nt x (TM + 4); the pitches
// keep their accesses on distinct banks (two lanes a bank for the transposed
// one).  EPI_BWD_HIDDEN has a tile of pre-activations after the ring.
constexpr int TT_PITCH = TM + 4;
__host__ __device__ constexpr int epi_f32_bytes(int nt) { return TM * (nt + 4) * 4; }
__host__ __device__ constexpr int epi_bytes(int nt) { return epi_f32_bytes(nt) + nt * TT_PITCH * 2; }
constexpr int SMEM_MAX = 216 * 1024;
__host__ constexpr int ring_stages(int nt, int k) {
    int st = (k + KC - 1) / KC;
    if (st > MAX_STAGES) st = MAX_STAGES;
    while (st * stage_bytes(nt) + epi_f32_bytes(nt) > SMEM_MAX) --st;
    return st;
}
// The ring's bytes (the epilogue's where they are more), then the pre-activations.
__host__ constexpr int ring_bytes(int nt, int k) {
    const int ring = ring_stages(nt, k) * stage_bytes(nt), epi = epi_bytes(nt);
    return ring > epi ? ring : epi;
}
static_assert(ring_bytes(NT_MAX, 8 * KC) + epi_f32_bytes(NT_MAX) <= SMEM_MAX && ring_bytes(NT_MAX, 16) <= SMEM_MAX,
              "the widest tile fits");

// Box of chunk c (columns c KC ..., rows row0 ...) of an operand; columns
// past K read as zero.
__device__ __forceinline__ void tma_chunk(uint32_t dst, const CUtensorMap *map, int c, int row0, uint64_t *bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(dst),
        "l"(map), "r"(c * KC), "r"(row0), "r"(ek::tc::smem_u32(bar))
        : "memory");
}

__device__ __forceinline__ uint32_t pack_bf16(bf16 lo, bf16 hi) {
    return (uint32_t)__bfloat16_as_ushort(lo) | ((uint32_t)__bfloat16_as_ushort(hi) << 16);
}

template <int EPI>
__global__ void __launch_bounds__(GT) mlp_gemm(const __grid_constant__ GemmArgs g) {
    extern __shared__ __align__(1024) uint8_t stage_mem[];
    __shared__ __align__(8) uint64_t full[MAX_STAGES], empty[MAX_STAGES], done;
    __shared__ uint32_t tmem_base;
    __shared__ int gave_up;
    __shared__ __align__(16) float sbias[NT_MAX];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int nt = g.nt, lg = 31 - __clz(nt), stages = g.stages;  // nt a power of two (tile_columns)
    const int m0 = blockIdx.x * TM, n0 = blockIdx.y * nt;
    const uint32_t tmem_cols = nt < 32 ? 32 : nt;
    const int nk = (g.k + KC - 1) / KC, sbytes = stage_bytes(nt), pre = min(nk, stages);
    const uint32_t ring = ek::tc::smem_u32(stage_mem);
    if (tid == 0) {
        for (int b = 0; b < stages; ++b) {
            ek::tc::mbar_init(&full[b], 1);
            ek::tc::mbar_init(&empty[b], 1);
        }
        ek::tc::mbar_init(&done, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        // B of the first chunks: not written by the kernel just before this one
        for (int c = 0; c < pre; ++c) {
            ek::tc::mbar_expect_tx(&full[c], (uint32_t)sbytes);
            tma_chunk(ring + c * sbytes + STAGE_A, &g.tb, c, n0, &full[c]);
        }
    }
    if (warp == 1) {
        ek::tc::tmem_alloc(&tmem_base, tmem_cols);
        ek::tc::tmem_relinquish();
    }
    float *const zt = reinterpret_cast<float *>(stage_mem + g.zoff);
    if (EPI == EPI_BWD_HIDDEN) {  // the tile's pre-activations (of the forward pass)
        for (int v = tid; v < (TM * nt) >> 2; v += GT) {
            const int r = v >> (lg - 2), c = (v << 2) & (nt - 1);
            *reinterpret_cast<float4 *>(zt + r * (nt + 4) + c) =
                *reinterpret_cast<const float4 *>(g.z + (size_t)(m0 + r) * g.ldz + n0 + c);
        }
    }
    if ((EPI == EPI_FWD_HIDDEN || EPI == EPI_FWD_OUT) && tid < nt) sbias[tid] = g.bias[n0 + tid];
    ek::pdl_wait();
    if (tid == 0)
        for (int c = 0; c < pre; ++c) tma_chunk(ring + c * sbytes, &g.ta, c, m0, &full[c]);
    ek::tc::fence_before_sync();
    __syncthreads();
    ek::tc::fence_after_sync();
    const uint32_t tmem = tmem_base;
    if (tid == 0) {
        const uint32_t idesc = ek::tc::idesc_bf16_f32(TM, nt);
        bool ok = true;
        int i = 0, issued = pre;  // chunks consumed, chunks whose copies were issued
        for (; i < nk; ++i) {
            const int st = i % stages;
            const uint32_t ph = (uint32_t)(i / stages) & 1u;
            ok = ek::tc::mbar_wait_bounded(&full[st], ph, g.wait_cycles);
            if (!ok) break;
            const uint32_t a0 = ring + st * sbytes, b0 = a0 + STAGE_A;
            const int kk = min(KC, g.k - i * KC);
            for (int kq = 0; kq < kk / 16; ++kq)  // 16 K-elements: 32 bytes along the swizzled row
                ek::tc::mma_bf16(tmem, ek::tc::smem_desc_sw128(a0 + kq * 32), ek::tc::smem_desc_sw128(b0 + kq * 32), idesc,
                                 (i > 0 || kq > 0) ? 1u : 0u);
            if (i + stages < nk) {
                // the slot is refilled once the MMAs that read it have completed
                ek::tc::mma_commit(&empty[st]);
                ok = ek::tc::mbar_wait_bounded(&empty[st], ph, g.wait_cycles);
                if (!ok) {
                    ++i;
                    break;
                }
                ek::tc::mbar_expect_tx(&full[st], (uint32_t)sbytes);
                tma_chunk(ring + st * sbytes, &g.ta, i + stages, m0, &full[st]);
                tma_chunk(ring + st * sbytes + STAGE_A, &g.tb, i + stages, n0, &full[st]);
                ++issued;
            }
        }
        // `done` tracks all MMAs issued; after a wait that gave up, the copies
        // and MMAs still in flight get one more wait, at the default bound,
        // before the shared and tensor memory go
        ek::tc::mma_commit(&done);
        if (ok) ok = ek::tc::mbar_wait_bounded(&done, 0, g.wait_cycles);
        if (!ok) {
            for (; i < issued; ++i)
                ek::tc::mbar_wait_bounded(&full[i % stages], (uint32_t)(i / stages) & 1u, ek::tc::WAIT_CYCLES_DEFAULT);
            ek::tc::mbar_wait_bounded(&done, 0, ek::tc::WAIT_CYCLES_DEFAULT);
            atomicOr(g.err, 1);
        }
        gave_up = !ok;
    }
    __syncthreads();
    ek::tc::fence_after_sync();
    if (!gave_up) {
        // the accumulator through shared memory: warps w, w + 4, ... hold the
        // same 32 rows (a warp reads the tensor-memory lanes of its index mod
        // 4) and take every fourth group of 8 columns
        const int fp = nt + 4;
        float *ft = reinterpret_cast<float *>(stage_mem);
        bf16 *tt = reinterpret_cast<bf16 *>(stage_mem + epi_f32_bytes(nt));
        const uint32_t trow = tmem + ((uint32_t)((warp & 3) * 32) << 16);
        float *fr = ft + ((warp & 3) * 32 + lane) * fp;
        for (int j = (warp >> 2) * 8; j < nt; j += GT / 16) {
            float v[8];
            ek::tc::tmem_ld8(trow + j, v);
            *reinterpret_cast<float4 *>(fr + j) = make_float4(v[0], v[1], v[2], v[3]);
            *reinterpret_cast<float4 *>(fr + j + 4) = make_float4(v[4], v[5], v[6], v[7]);
        }
        __syncthreads();
        // four columns of a row a thread and round; one small loop body (the
        // code is fetched cold by every launch)
#pragma unroll 1
        for (int e = tid; e < (TM * nt) >> 2; e += GT) {
            const int r = e >> (lg - 2), c = (e << 2) & (nt - 1);
            float4 v = *reinterpret_cast<const float4 *>(ft + r * fp + c);
            if (EPI == EPI_FWD_OUT || EPI == EPI_FWD_HIDDEN) {
                const float4 b = *reinterpret_cast<const float4 *>(sbias + c);
                v = make_float4(v.x + b.x, v.y + b.y, v.z + b.z, v.w + b.w);
            }
            if (EPI == EPI_F32 || EPI == EPI_FWD_OUT) {
                float *o = g.c + (size_t)(m0 + r) * g.ldc + n0 + c;
                if (EPI == EPI_FWD_OUT || g.c_vec) {
                    *reinterpret_cast<float4 *>(o) = v;
                } else {  // a caller's matrix with an odd row stride or address
                    o[0] = v.x;
                    o[1] = v.y;
                    o[2] = v.z;
                    o[3] = v.w;
                }
            } else {
                float w[4] = {v.x, v.y, v.z, v.w};
                bf16 h[4];
                if (EPI == EPI_BWD_HIDDEN) {
                    const float4 z = *reinterpret_cast<const float4 *>(zt + r * fp + c);
                    const float zz[4] = {z.x, z.y, z.z, z.w};
#pragma unroll
                    for (int i = 0; i < 4; ++i) h[i] = __float2bfloat16_rn(w[i] * silu_grad(zz[i]));
                } else {
                    if (g.z) *reinterpret_cast<float4 *>(g.z + (size_t)(m0 + r) * g.ldz + n0 + c) = v;
#pragma unroll
                    for (int i = 0; i < 4; ++i) h[i] = __float2bfloat16_rn(silu(w[i]));
                }
                *reinterpret_cast<uint2 *>(g.h + (size_t)(m0 + r) * g.ldh + n0 + c) =
                    make_uint2(pack_bf16(h[0], h[1]), pack_bf16(h[2], h[3]));
#pragma unroll
                for (int i = 0; i < 4; ++i) tt[(c + i) * TT_PITCH + r] = h[i];
            }
        }
        if ((EPI == EPI_FWD_HIDDEN && g.ht) || EPI == EPI_BWD_HIDDEN) {
            __syncthreads();
            for (int v = tid; v < nt * (TM / 4); v += GT) {
                const int c = v / (TM / 4), r = (v % (TM / 4)) * 4;
                *reinterpret_cast<uint2 *>(g.ht + (size_t)(n0 + c) * g.ldht + m0 + r) =
                    *reinterpret_cast<const uint2 *>(tt + c * TT_PITCH + r);
            }
        }
    }
    ek::tc::fence_before_sync();
    __syncthreads();
    if (warp == 1) ek::tc::tmem_dealloc(tmem, tmem_cols);
}

// Batch rows idx[offset .. offset+B) of the data set: X (padded to 16 inputs,
// BF16, and transposed), targets T (FP32).  offset = (*step - *base) * B, or 0.
__global__ void gather_batch(const float *__restrict__ xs, const float *__restrict__ ts, const int *__restrict__ idx,
                             const int64_t *__restrict__ step, const int64_t *__restrict__ base, int B,
                             bf16 *__restrict__ x, bf16 *__restrict__ xt, float *__restrict__ t) {
    ek::pdl_wait();
    const int64_t off = step ? (*step - *base) * B : 0;
    const int b = blockIdx.x;
    const int src = idx[off + b];
    for (int j = threadIdx.x; j < OUT; j += blockDim.x) t[(size_t)b * OUT + j] = ts[(size_t)src * OUT + j];
    if (threadIdx.x < INP) {
        const float v = threadIdx.x < IN ? xs[(size_t)src * IN + threadIdx.x] : 0.0f;
        const bf16 h = __float2bfloat16_rn(v);
        x[(size_t)b * INP + threadIdx.x] = h;
        xt[(size_t)threadIdx.x * B + b] = h;
    }
}

// Inputs of the evaluation: n x 4 FP32 rows -> BF16 rows padded to 16 inputs,
// zero rows up to the end of the last tile; one thread a row.
__global__ void pad_inputs(const float4 *__restrict__ x, int n, int rows, uint4 *__restrict__ xb) {
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= rows) return;
    const float4 v = r < n ? x[r] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    xb[2 * r] = make_uint4(pack_bf16(__float2bfloat16_rn(v.x), __float2bfloat16_rn(v.y)),
                           pack_bf16(__float2bfloat16_rn(v.z), __float2bfloat16_rn(v.w)), 0u, 0u);
    xb[2 * r + 1] = make_uint4(0u, 0u, 0u, 0u);
}

// MSE over B x 512 outputs: dY = 2 (Y - T) / (B 512) (BF16, and transposed);
// the loss of the iteration is added to loss[*step - *base].  A block takes a
// 32 x 64 tile, transposed through shared memory so that both results are
// stored in runs (one row a block with scattered transposed stores: 5.3 us
// against 3.3 us at 256 rows, B200).
__global__ void __launch_bounds__(256) mse_grad(const float *y, const float *__restrict__ t, int B,
                                                bf16 *__restrict__ dy, bf16 *__restrict__ dyt,
                                                double *__restrict__ loss, const int64_t *__restrict__ step,
                                                const int64_t *__restrict__ base) {
    __shared__ bf16 tile[64][32 + 2];
    __shared__ double red[8];
    const int b0 = blockIdx.x * 32, j0 = blockIdx.y * 64;
    const float scale = 2.0f / ((float)B * (float)OUT);
    double acc = 0.0;
    // the thread's 8 elements: targets (of the gather, kernels ago) before the wait,
    // outputs (of the kernel before) after it, all of them before the first store
    const size_t o0 = (size_t)(b0 + (threadIdx.x >> 6)) * OUT + j0 + (threadIdx.x & 63);
    float tv[8], yv[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) tv[e] = __ldg(t + o0 + (size_t)(e * 4) * OUT);
    ek::pdl_wait();
#pragma unroll
    for (int e = 0; e < 8; ++e) yv[e] = ek::ld_fresh(y + o0 + (size_t)(e * 4) * OUT);
#pragma unroll
    for (int e = 0; e < 8; ++e) {
        const int r = e * 4 + (threadIdx.x >> 6), c = threadIdx.x & 63;
        const size_t o = o0 + (size_t)(e * 4) * OUT;
        const float d = yv[e] - tv[e];
        acc += (double)d * (double)d;
        const bf16 g = __float2bfloat16_rn(scale * d);
        dy[o] = g;
        tile[c][r] = g;
    }
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
    __syncthreads();
#pragma unroll
    for (int e = 0; e < 8; ++e) {
        const int c = e * 8 + (threadIdx.x >> 5), r = threadIdx.x & 31;
        dyt[(size_t)(j0 + c) * B + b0 + r] = tile[c][r];
    }
    if (threadIdx.x == 0) {
        double s = 0.0;
        for (int w = 0; w < 8; ++w) s += red[w];
        const int64_t slot = step ? (*step - *base) : 0;
        atomicAdd(loss + slot, s / ((double)B * OUT));
    }
}

struct BiasSeg {
    const bf16 *dzt[NL];  // (out x B) transposed deltas
    float *db[NL];
    int rows[NL];
};

// db[n] = sum over the batch of dZ[:, n]: one warp per output n.
__global__ void bias_grads(const BiasSeg s, int B) {
    const int w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    int l = 0, n = w;
    while (l < NL && n >= s.rows[l]) n -= s.rows[l++];
    if (l >= NL) return;
    const bf16 *r = s.dzt[l] + (size_t)n * B;
    float acc = 0.0f;
    for (int b = lane; b < B; b += 32) acc += __bfloat162float(r[b]);
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
    if (lane == 0) s.db[l][n] = acc;
}

// Adam on the flat FP32 parameters, four a thread; step count t = *step + 1.
// The two bias corrections (FP64 powers) are computed by two threads of the
// block: in every thread they were half the kernel's time. An ordinary launch:
// it waits for both streams of the backward pass.
__global__ void __launch_bounds__(256) adam_update(float4 *__restrict__ p, const float4 *__restrict__ g,
                                                   float4 *__restrict__ m, float4 *__restrict__ v, int64_t n4, float lr,
                                                   float b1, float b2, float eps, const int64_t *__restrict__ step) {
    __shared__ float corr[2];
    if (threadIdx.x < 64 && (threadIdx.x & 31) == 0) {
        const double t = (double)(*step + 1);
        corr[threadIdx.x >> 5] = (float)(1.0 - pow((double)(threadIdx.x ? b2 : b1), t));
    }
    __syncthreads();
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n4) return;
    const float c1 = corr[0], c2 = corr[1];
    const float4 gv = g[i];
    float4 mv = m[i], vv = v[i], pv = p[i];
    auto one = [&](float gi, float &m1, float &v1, float &p1) {
        const float mi = b1 * m1 + (1.0f - b1) * gi;
        const float vi = b2 * v1 + (1.0f - b2) * gi * gi;
        m1 = mi;
        v1 = vi;
        p1 -= lr * (mi / c1) / (sqrtf(vi / c2) + eps);
    };
    one(gv.x, mv.x, vv.x, pv.x);
    one(gv.y, mv.y, vv.y, pv.y);
    one(gv.z, mv.z, vv.z, pv.z);
    one(gv.w, mv.w, vv.w, pv.w);
    m[i] = mv;
    v[i] = vv;
    p[i] = pv;
}

struct CastSeg {
    const float *w[NL];
    bf16 *wb[NL];
    bf16 *wt[NL];
    int out[NL], in[NL];
};

// Blocks of cast_weights: 32 x 32 tiles of every layer (32 x 16 of layer 0).
constexpr int cast_tiles(int l) { return (DIM_OUT[l] / 32) * ((DIM_IN[l] + 31) / 32); }
constexpr int CAST_BLOCKS = cast_tiles(0) + cast_tiles(1) + cast_tiles(2) + cast_tiles(3);

// BF16 copies W (out x in) and W^T (in x out) of every layer, one tile a block,
// transposed through shared memory (scattered transposed stores: 10.5 us
// against 3.5 us on B200); one thread advances the step counter (after Adam,
// before the next gather).
__global__ void __launch_bounds__(256) cast_weights(const CastSeg s, int64_t *__restrict__ step) {
    __shared__ bf16 tile[32][32 + 2];
    int l = 0, e = blockIdx.x;
    while (e >= (s.out[l] / 32) * ((s.in[l] + 31) / 32)) e -= (s.out[l] / 32) * ((s.in[l] + 31) / 32), ++l;
    const int in = s.in[l], out = s.out[l], per = (in + 31) / 32;
    const int o0 = (e / per) * 32, c0 = (e % per) * 32, w = min(32, in - c0);
    ek::pdl_wait();
    if (blockIdx.x == 0 && threadIdx.x == 0 && step) ++*step;
    const int c = threadIdx.x & 31;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const int r = q * 8 + (threadIdx.x >> 5);
        if (c < w) {
            const bf16 h = __float2bfloat16_rn(s.w[l][(size_t)(o0 + r) * in + c0 + c]);
            s.wb[l][(size_t)(o0 + r) * in + c0 + c] = h;
            tile[c][r] = h;
        }
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const int r = q * 8 + (threadIdx.x >> 5);
        if (r < w) s.wt[l][(size_t)(c0 + r) * out + o0 + c] = tile[r][c];
    }
}

}  // namespace

struct ek_mlp {
    int B = 256;
    cudaStream_t stream = nullptr;
    cudaStream_t side = nullptr;              // weight and bias gradients, beside the backward chain
    cudaEvent_t ready[4] = {}, joined = nullptr;  // delta of layer 3, 2, 1, 0 written; the gradients done
    int64_t nparam = 0;
    int64_t off_w[NL], off_b[NL];
    float *p = nullptr, *g = nullptr, *m = nullptr, *v = nullptr;  // flat FP32
    bf16 *wb[NL] = {}, *wt[NL] = {};
    bf16 *x = nullptr, *xt = nullptr;
    float *t = nullptr, *y = nullptr;
    float *z[3] = {};
    bf16 *h[3] = {}, *ht[3] = {};   // outputs of hidden layers 0..2
    bf16 *dz[3] = {}, *dzt[3] = {};
    bf16 *dy = nullptr, *dyt = nullptr;
    // data set and iteration state
    float *xs = nullptr, *ts = nullptr;
    int64_t nrows = 0;
    int *idx = nullptr;
    double *loss = nullptr;
    int64_t *step = nullptr, *base = nullptr;
    int64_t host_step = 0;
    std::mt19937_64 rng;
    std::vector<int> perm;          // permutation of the current epoch
    int *err = nullptr;
    long long wait_cycles = ek::tc::WAIT_CYCLES_DEFAULT;
    cudaGraphExec_t graph = nullptr;
    float graph_lr = -1.0f;
    int64_t launches = 0;
    // evaluation (ek_mlp_forward): rows in flight at once, kept between calls
    // and grown to the largest call so far, at most EVAL_ROWS rows
    int64_t eval_cap = 0;
    float *ey = nullptr, *ex = nullptr;      // outputs (rows x 512; the allocation), inputs (rows x 4)
    bf16 *exb = nullptr, *eh[2] = {};        // padded BF16 inputs, two hidden layers' activations
};

namespace {

int cuda_err(cudaError_t e, const char *what) {
    return ek::ctx_fail(e == cudaErrorMemoryAllocation ? EK_ERR_NOMEM : EK_ERR_CUDA,
                        (std::string(what) + ": " + cudaGetErrorString(e)).c_str());
}
#define EK_MCUDA(call, what)                              \
    do {                                                  \
        cudaError_t e_ = (call);                          \
        if (e_ != cudaSuccess) return cuda_err(e_, what); \
    } while (0)

// The GEMM's ring of stages is dynamic shared memory above the 48 KB
// default: allow it for every epilogue on the current device, before any
// launch (and outside any stream capture).
cudaError_t gemm_set_attributes() {
    const void *fns[] = {(const void *)mlp_gemm<EPI_F32>, (const void *)mlp_gemm<EPI_FWD_HIDDEN>,
                         (const void *)mlp_gemm<EPI_FWD_OUT>, (const void *)mlp_gemm<EPI_BWD_HIDDEN>};
    for (const void *f : fns) {
        const cudaError_t e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_MAX);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

// Columns of a CTA's tile: the widest of 128, 64, 32, 16 that divides n and
// still gives every SM a tile, else 16 (the smallest share of the epilogue a
// CTA can have; A is fetched again by every CTA of a row of tiles, from L2).
int tile_columns(int m, int n) {
    for (int nt = NT_MAX; nt > 16; nt /= 2)
        if (n % nt == 0 && (m / TM) * (n / nt) >= 148) return nt;
    return 16;
}

// pdl: programmatic launch; an ordinary one where another stream is waited for too.
template <int EPI>
cudaError_t gemm(const GemmArgs &a, cudaStream_t s, bool pdl = true) {
    const size_t smem = (size_t)a.zoff + (EPI == EPI_BWD_HIDDEN ? epi_f32_bytes(a.nt) : 0);
    if (!pdl) {
        mlp_gemm<EPI><<<dim3(a.m / TM, a.n / a.nt), GT, smem, s>>>(a);
        return cudaGetLastError();
    }
    return ek::launch_pdl(mlp_gemm<EPI>, dim3(a.m / TM, a.n / a.nt), dim3(GT), smem, s, a);
}

// g: the launch's arguments, the tensor maps of both operands among them.
cudaError_t gemm_args(GemmArgs &g, const bf16 *a, int lda, const bf16 *b, int ldb, int m, int n, int k, int *err,
                      long long wait_cycles = ek::tc::WAIT_CYCLES_DEFAULT) {
    g = GemmArgs{};
    g.wait_cycles = wait_cycles;
    g.m = m;
    g.n = n;
    g.k = k;
    g.nt = tile_columns(m, n);
    g.stages = ring_stages(g.nt, k);
    g.zoff = ring_bytes(g.nt, k);
    g.c_vec = true;
    g.err = err;
    const cudaError_t e = ek::make_matrix_tensor_map(a, m, k, lda, TM, KC, &g.ta);
    return e != cudaSuccess ? e : ek::make_matrix_tensor_map(b, n, k, ldb, g.nt, KC, &g.tb);
}

// Forward of the current batch (x): Z, H of the hidden layers and Y.
int forward(ek_mlp *q) {
    const int B = q->B;
    const bf16 *in = q->x;
    int ldin = INP;
    for (int l = 0; l < 3; ++l) {
        GemmArgs a;
        EK_MCUDA(gemm_args(a, in, ldin, q->wb[l], DIM_IN[l], B, HID, DIM_IN[l], q->err, q->wait_cycles), "operand maps");
        a.bias = q->p + q->off_b[l];
        a.z = q->z[l];
        a.ldz = HID;
        a.h = q->h[l];
        a.ldh = HID;
        a.ht = q->ht[l];
        a.ldht = B;
        EK_MCUDA(gemm<EPI_FWD_HIDDEN>(a, q->stream), "forward GEMM");
        in = q->h[l];
        ldin = HID;
    }
    GemmArgs a;
    EK_MCUDA(gemm_args(a, in, HID, q->wb[3], HID, B, OUT, HID, q->err, q->wait_cycles), "operand maps");
    a.bias = q->p + q->off_b[3];
    a.c = q->y;
    a.ldc = OUT;
    EK_MCUDA(gemm<EPI_FWD_OUT>(a, q->stream), "output GEMM");
    q->launches += 4;
    return EK_OK;
}

// Loss gradient, backward GEMMs and bias gradients into q->g.
int backward(ek_mlp *q, bool counted) {
    const int B = q->B;
    EK_MCUDA(ek::launch_pdl(mse_grad, dim3(B / 32, OUT / 64), dim3(256), 0, q->stream, q->y, q->t, B, q->dy, q->dyt,
                            q->loss, counted ? q->step : nullptr, counted ? q->base : nullptr),
             "loss kernel");
    // The weight and bias gradients run on a second stream beside the chain of
    // deltas: no kernel of the chain reads them, none of them fills more than a
    // fraction of the SMs, and each costs a launch's latency when it is waited
    // for (an iteration of 256 rows on B200: 66 us one after the other, 55 us
    // so). Adam waits for both streams.
    auto fork = [&](int i) -> cudaError_t {
        cudaError_t e = cudaEventRecord(q->ready[i], q->stream);
        return e == cudaSuccess ? cudaStreamWaitEvent(q->side, q->ready[i], 0) : e;
    };
    EK_MCUDA(fork(0), "gradient stream");
    // layer 3: dW3 = dY^T H2, dZ2 = (dY W3) * silu'(Z2)
    {
        GemmArgs a;
        EK_MCUDA(gemm_args(a, q->dyt, B, q->ht[2], B, OUT, HID, B, q->err, q->wait_cycles), "operand maps");
        a.c = q->g + q->off_w[3];
        a.ldc = HID;
        EK_MCUDA(gemm<EPI_F32>(a, q->side, false), "weight-gradient GEMM");
    }
    const bf16 *up = q->dy;
    int ldup = OUT;
    for (int l = 2; l >= 0; --l) {
        // dZ_l = (dZ_{l+1} W_{l+1}) * silu'(Z_l)
        GemmArgs a;
        EK_MCUDA(gemm_args(a, up, ldup, q->wt[l + 1], DIM_OUT[l + 1], B, HID, DIM_OUT[l + 1], q->err, q->wait_cycles), "operand maps");
        a.z = q->z[l];
        a.ldz = HID;
        a.h = q->dz[l];
        a.ldh = HID;
        a.ht = q->dzt[l];
        a.ldht = B;
        EK_MCUDA(gemm<EPI_BWD_HIDDEN>(a, q->stream), "backward GEMM");
        EK_MCUDA(fork(3 - l), "gradient stream");
        // dW_l = dZ_l^T H_{l-1} (H_{-1} = X)
        const bf16 *hin_t = l > 0 ? q->ht[l - 1] : q->xt;
        GemmArgs w;
        EK_MCUDA(gemm_args(w, q->dzt[l], B, hin_t, B, HID, DIM_IN[l], B, q->err, q->wait_cycles), "operand maps");
        w.c = q->g + q->off_w[l];
        w.ldc = DIM_IN[l];
        EK_MCUDA(l > 0 ? gemm<EPI_F32>(w, q->side, false) : gemm<EPI_F32>(w, q->stream), "weight-gradient GEMM");
        up = q->dz[l];
        ldup = HID;
    }
    BiasSeg s{};
    int rows = 0;
    for (int l = 0; l < NL; ++l) {
        s.dzt[l] = l < 3 ? q->dzt[l] : q->dyt;
        s.db[l] = q->g + q->off_b[l];
        s.rows[l] = DIM_OUT[l];
        rows += DIM_OUT[l];
    }
    bias_grads<<<(rows * 32 + 255) / 256, 256, 0, q->side>>>(s, B);
    EK_MCUDA(cudaGetLastError(), "bias gradients");
    EK_MCUDA(cudaEventRecord(q->joined, q->side), "gradient stream");
    EK_MCUDA(cudaStreamWaitEvent(q->stream, q->joined, 0), "gradient stream");
    q->launches += 9;
    return EK_OK;
}

int cast_all(ek_mlp *q, bool advance) {
    CastSeg s{};
    for (int l = 0; l < NL; ++l) {
        s.w[l] = q->p + q->off_w[l];
        s.wb[l] = q->wb[l];
        s.wt[l] = q->wt[l];
        s.out[l] = DIM_OUT[l];
        s.in[l] = DIM_IN[l];
    }
    EK_MCUDA(ek::launch_pdl(cast_weights, dim3(CAST_BLOCKS), dim3(256), 0, q->stream, s, advance ? q->step : nullptr),
             "weight casts");
    ++q->launches;
    return EK_OK;
}

int train_iteration(ek_mlp *q, float lr) {
    // an ordinary launch: it reads the step count that the iteration before ends with
    gather_batch<<<q->B, 256, 0, q->stream>>>(q->xs, q->ts, q->idx, q->step, q->base, q->B, q->x, q->xt, q->t);
    EK_MCUDA(cudaGetLastError(), "batch gather");
    ++q->launches;
    int rc = forward(q);
    if (rc == EK_OK) rc = backward(q, true);
    if (rc != EK_OK) return rc;
    const int64_t n4 = q->nparam / 4;  // every layer's weights and biases come in fours
    adam_update<<<(unsigned)((n4 + 255) / 256), 256, 0, q->stream>>>((float4 *)q->p, (const float4 *)q->g, (float4 *)q->m,
                                                                    (float4 *)q->v, n4, lr, 0.9f, 0.999f, 1e-8f, q->step);
    EK_MCUDA(cudaGetLastError(), "Adam");
    ++q->launches;
    return cast_all(q, true);
}

// Evaluation workspace for at least `rows` rows (rounded up to whole tiles).
constexpr int64_t EVAL_ROWS = 8192;
int eval_reserve(ek_mlp *q, int64_t rows) {
    const int64_t cap = (rows + TM - 1) / TM * TM;
    if (cap <= q->eval_cap) return EK_OK;
    EK_MCUDA(cudaStreamSynchronize(q->stream), "evaluation workspace");
    // one allocation: outputs, inputs, then the BF16 activations (row sizes are multiples of 16 bytes)
    q->eval_cap = 0;
    cudaFree(q->ey);
    q->ey = nullptr;
    EK_MCUDA(cudaMalloc(&q->ey, (size_t)cap * (OUT * 4 + IN * 4 + INP * 2 + 2 * HID * 2)), "evaluation workspace");
    q->ex = q->ey + (size_t)cap * OUT;
    q->exb = (bf16 *)(q->ex + (size_t)cap * IN);
    q->eh[0] = q->exb + (size_t)cap * INP;
    q->eh[1] = q->eh[0] + (size_t)cap * HID;
    q->eval_cap = cap;
    return EK_OK;
}

int check_err(ek_mlp *q) {
    int v = 0;
    EK_MCUDA(cudaMemcpyAsync(&v, q->err, sizeof(int), cudaMemcpyDeviceToHost, q->stream), "error word");
    EK_MCUDA(cudaStreamSynchronize(q->stream), "error word");
    if (v) {
        EK_MCUDA(cudaMemsetAsync(q->err, 0, sizeof(int), q->stream), "error word");
        return ek::ctx_fail(EK_ERR_TIMEOUT, "a bounded wait for the tensor cores gave up");
    }
    return EK_OK;
}

}  // namespace

extern "C" {

int ek_mlp_create(int32_t batch, uint64_t seed, ek_mlp **out) {
    if (!out || batch <= 0 || batch % TM) return ek::ctx_fail(EK_ERR_INVALID, "batch must be a positive multiple of 128");
    *out = nullptr;
    EK_MCUDA(gemm_set_attributes(), "GEMM attributes");
    ek_mlp *q = new ek_mlp();
    q->B = batch;
    q->rng.seed(seed);
    int64_t off = 0;
    for (int l = 0; l < NL; ++l) {
        q->off_w[l] = off;
        off += (int64_t)DIM_OUT[l] * DIM_IN[l];
        q->off_b[l] = off;
        off += DIM_OUT[l];
    }
    q->nparam = off;
    const int B = batch;
    struct A { void **p; size_t bytes; };
    std::vector<A> al = {
        {(void **)&q->p, (size_t)off * 4}, {(void **)&q->g, (size_t)off * 4}, {(void **)&q->m, (size_t)off * 4},
        {(void **)&q->v, (size_t)off * 4},
        {(void **)&q->x, (size_t)B * INP * 2}, {(void **)&q->xt, (size_t)B * INP * 2},
        {(void **)&q->t, (size_t)B * OUT * 4}, {(void **)&q->y, (size_t)B * OUT * 4},
        {(void **)&q->dy, (size_t)B * OUT * 2}, {(void **)&q->dyt, (size_t)B * OUT * 2},
        {(void **)&q->step, 8}, {(void **)&q->base, 8}, {(void **)&q->err, 4},
    };
    for (int l = 0; l < NL; ++l) {
        al.push_back({(void **)&q->wb[l], (size_t)DIM_OUT[l] * DIM_IN[l] * 2});
        al.push_back({(void **)&q->wt[l], (size_t)DIM_OUT[l] * DIM_IN[l] * 2});
    }
    for (int l = 0; l < 3; ++l) {
        al.push_back({(void **)&q->z[l], (size_t)B * HID * 4});
        al.push_back({(void **)&q->h[l], (size_t)B * HID * 2});
        al.push_back({(void **)&q->ht[l], (size_t)B * HID * 2});
        al.push_back({(void **)&q->dz[l], (size_t)B * HID * 2});
        al.push_back({(void **)&q->dzt[l], (size_t)B * HID * 2});
    }
    cudaError_t e = cudaStreamCreateWithFlags(&q->stream, cudaStreamNonBlocking);
    if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&q->side, cudaStreamNonBlocking);
    for (cudaEvent_t &ev : q->ready)
        if (e == cudaSuccess) e = cudaEventCreateWithFlags(&ev, cudaEventDisableTiming);
    if (e == cudaSuccess) e = cudaEventCreateWithFlags(&q->joined, cudaEventDisableTiming);
    for (auto &a : al) {
        if (e == cudaSuccess) e = cudaMalloc(a.p, a.bytes);
        if (e == cudaSuccess) e = cudaMemsetAsync(*a.p, 0, a.bytes, q->stream);
    }
    if (e != cudaSuccess) {
        ek_mlp_destroy(q);
        return cuda_err(e, "MLP allocation");
    }
    // Glorot-uniform weights over the true fan-in (4 for layer 0), zero biases
    std::vector<float> p(off, 0.0f);
    for (int l = 0; l < NL; ++l) {
        const int fin = l == 0 ? IN : DIM_IN[l];
        const float a = std::sqrt(6.0f / (float)(fin + DIM_OUT[l]));
        std::uniform_real_distribution<float> u(-a, a);
        for (int o = 0; o < DIM_OUT[l]; ++o)
            for (int i = 0; i < fin; ++i) p[q->off_w[l] + (int64_t)o * DIM_IN[l] + i] = u(q->rng);
    }
    int rc = ek_mlp_set_params(q, p.data());
    if (rc != EK_OK) {
        ek_mlp_destroy(q);
        return rc;
    }
    *out = q;
    return EK_OK;
}

int ek_mlp_destroy(ek_mlp *q) {
    if (!q) return ek::ctx_fail(EK_ERR_INVALID, "null MLP");
    if (q->stream) cudaStreamSynchronize(q->stream);
    if (q->side) cudaStreamSynchronize(q->side);
    if (q->graph) cudaGraphExecDestroy(q->graph);
    void *bufs[] = {q->p, q->g, q->m, q->v, q->x, q->xt, q->t, q->y, q->dy, q->dyt, q->step, q->base, q->err,
                    q->xs, q->ts, q->idx, q->loss, q->ey};
    for (void *b : bufs)
        if (b) cudaFree(b);
    for (int l = 0; l < NL; ++l) {
        if (q->wb[l]) cudaFree(q->wb[l]);
        if (q->wt[l]) cudaFree(q->wt[l]);
    }
    for (int l = 0; l < 3; ++l) {
        void *b2[] = {q->z[l], q->h[l], q->ht[l], q->dz[l], q->dzt[l]};
        for (void *b : b2)
            if (b) cudaFree(b);
    }
    for (cudaEvent_t ev : q->ready)
        if (ev) cudaEventDestroy(ev);
    if (q->joined) cudaEventDestroy(q->joined);
    if (q->side) cudaStreamDestroy(q->side);
    if (q->stream) cudaStreamDestroy(q->stream);
    delete q;
    return EK_OK;
}

int ek_mlp_param_count(const ek_mlp *q, int64_t *n) {
    if (!q || !n) return ek::ctx_fail(EK_ERR_INVALID, "null argument");
    *n = q->nparam;
    return EK_OK;
}

int ek_mlp_get_params(ek_mlp *q, float *flat) {
    if (!q || !flat) return ek::ctx_fail(EK_ERR_INVALID, "null argument");
    EK_MCUDA(cudaMemcpyAsync(flat, q->p, q->nparam * 4, cudaMemcpyDeviceToHost, q->stream), "parameters");
    EK_MCUDA(cudaStreamSynchronize(q->stream), "parameters");
    return EK_OK;
}

int ek_mlp_set_params(ek_mlp *q, const float *flat) {
    if (!q || !flat) return ek::ctx_fail(EK_ERR_INVALID, "null argument");
    for (int64_t i = 0; i < q->nparam; ++i)
        if (!std::isfinite(flat[i])) return ek::ctx_fail(EK_ERR_INVALID, "non-finite parameter");
    EK_MCUDA(cudaMemcpyAsync(q->p, flat, q->nparam * 4, cudaMemcpyHostToDevice, q->stream), "parameters");
    EK_MCUDA(cudaMemsetAsync(q->m, 0, q->nparam * 4, q->stream), "Adam state");
    EK_MCUDA(cudaMemsetAsync(q->v, 0, q->nparam * 4, q->stream), "Adam state");
    EK_MCUDA(cudaMemsetAsync(q->step, 0, 8, q->stream), "step");
    q->host_step = 0;
    int rc = cast_all(q, false);
    if (rc != EK_OK) return rc;
    EK_MCUDA(cudaStreamSynchronize(q->stream), "parameters");
    return EK_OK;
}

int ek_mlp_set_data(ek_mlp *q, const float *x, const float *t, int64_t n) {
    if (!q || !x || !t || n < q->B) return ek::ctx_fail(EK_ERR_INVALID, "need at least one batch of rows");
    for (int64_t i = 0; i < n * IN; ++i)
        if (!std::isfinite(x[i])) return ek::ctx_fail(EK_ERR_INVALID, "non-finite input");
    for (int64_t i = 0; i < n * OUT; ++i)
        if (!std::isfinite(t[i])) return ek::ctx_fail(EK_ERR_INVALID, "non-finite target");
    EK_MCUDA(cudaStreamSynchronize(q->stream), "data");
    if (q->graph) cudaGraphExecDestroy(q->graph);  // it holds the old data pointers
    q->graph = nullptr;
    q->perm.clear();
    if (q->xs) cudaFree(q->xs);
    if (q->ts) cudaFree(q->ts);
    q->xs = q->ts = nullptr;
    EK_MCUDA(cudaMalloc(&q->xs, n * IN * 4), "data set");
    EK_MCUDA(cudaMalloc(&q->ts, n * OUT * 4), "data set");
    EK_MCUDA(cudaMemcpyAsync(q->xs, x, n * IN * 4, cudaMemcpyHostToDevice, q->stream), "data set");
    EK_MCUDA(cudaMemcpyAsync(q->ts, t, n * OUT * 4, cudaMemcpyHostToDevice, q->stream), "data set");
    EK_MCUDA(cudaStreamSynchronize(q->stream), "data set");
    q->nrows = n;
    return EK_OK;
}

// `iters` Adam iterations over shuffled batches (a new permutation of the data
// set every epoch, from the MLP's seeded generator); loss_out (optional) gets
// each iteration's mean squared error.
int ek_mlp_train(ek_mlp *q, int32_t iters, float lr, double *loss_out) {
    if (!q || iters < 0 || !(lr > 0.0f)) return ek::ctx_fail(EK_ERR_INVALID, "bad training arguments");
    if (!q->xs) return ek::ctx_fail(EK_ERR_INVALID, "call ek_mlp_set_data first");
    const int64_t per_epoch = q->nrows / q->B;
    constexpr int64_t CHUNK = 1024;  // iterations per index upload
    if (!q->idx) {
        EK_MCUDA(cudaMalloc(&q->idx, CHUNK * q->B * sizeof(int)), "index buffer");
        EK_MCUDA(cudaMalloc(&q->loss, CHUNK * sizeof(double)), "loss buffer");
    }
    if (q->graph && q->graph_lr != lr) {
        cudaGraphExecDestroy(q->graph);
        q->graph = nullptr;
    }
    std::vector<int> idx;
    std::vector<double> losses;
    int64_t done = 0;
    while (done < iters) {
        const int64_t n = std::min<int64_t>(CHUNK, iters - done);
        idx.clear();
        for (int64_t it = 0; it < n; ++it) {
            const int64_t e = (q->host_step + it) % per_epoch;
            if (e == 0 || (int64_t)q->perm.size() != q->nrows) {
                q->perm.resize(q->nrows);
                for (int64_t i = 0; i < q->nrows; ++i) q->perm[i] = (int)i;
                std::shuffle(q->perm.begin(), q->perm.end(), q->rng);
            }
            for (int b = 0; b < q->B; ++b) idx.push_back(q->perm[(size_t)(e * q->B + b)]);
        }
        EK_MCUDA(cudaMemcpyAsync(q->idx, idx.data(), idx.size() * sizeof(int), cudaMemcpyHostToDevice, q->stream),
                 "batch indices");
        EK_MCUDA(cudaMemcpyAsync(q->base, q->step, 8, cudaMemcpyDeviceToDevice, q->stream), "iteration base");
        EK_MCUDA(cudaMemsetAsync(q->loss, 0, n * sizeof(double), q->stream), "loss buffer");
        if (!q->graph) {
            cudaGraph_t g = nullptr;
            const int64_t l0 = q->launches;
            EK_MCUDA(cudaStreamBeginCapture(q->stream, cudaStreamCaptureModeThreadLocal), "graph capture");
            int rc = train_iteration(q, lr);
            cudaError_t e = cudaStreamEndCapture(q->stream, &g);
            q->launches = l0;
            if (rc != EK_OK) {
                if (g) cudaGraphDestroy(g);
                return rc;
            }
            EK_MCUDA(e, "graph capture");
            e = cudaGraphInstantiate(&q->graph, g, 0);
            cudaGraphDestroy(g);
            EK_MCUDA(e, "graph instantiate");
            q->graph_lr = lr;
        }
        for (int64_t it = 0; it < n; ++it) {
            EK_MCUDA(cudaGraphLaunch(q->graph, q->stream), "graph launch");
            q->launches += 16;
        }
        if (loss_out) {
            losses.resize(n);
            EK_MCUDA(cudaMemcpyAsync(losses.data(), q->loss, n * sizeof(double), cudaMemcpyDeviceToHost, q->stream),
                     "losses");
        }
        int rc = check_err(q);
        if (rc != EK_OK) return rc;
        if (loss_out) std::copy(losses.begin(), losses.end(), loss_out + done);
        q->host_step += n;
        done += n;
    }
    return EK_OK;
}

// Gradients (flat, the layout of the parameters) and loss of one batch of B
// rows, without an update.
int ek_mlp_gradients(ek_mlp *q, const float *x, const float *t, float *grads, double *loss) {
    if (!q || !x || !t || !grads) return ek::ctx_fail(EK_ERR_INVALID, "null argument");
    float *xs = nullptr, *ts = nullptr;
    int *idx = nullptr;
    double *l = nullptr;
    std::vector<int> id(q->B);
    for (int i = 0; i < q->B; ++i) id[i] = i;
    auto run = [&]() -> int {
        EK_MCUDA(cudaMalloc(&xs, (size_t)q->B * IN * 4), "staging");
        EK_MCUDA(cudaMalloc(&ts, (size_t)q->B * OUT * 4), "staging");
        EK_MCUDA(cudaMalloc(&idx, (size_t)q->B * 4), "staging");
        EK_MCUDA(cudaMalloc(&l, 8), "staging");
        EK_MCUDA(cudaMemcpyAsync(xs, x, (size_t)q->B * IN * 4, cudaMemcpyHostToDevice, q->stream), "staging");
        EK_MCUDA(cudaMemcpyAsync(ts, t, (size_t)q->B * OUT * 4, cudaMemcpyHostToDevice, q->stream), "staging");
        EK_MCUDA(cudaMemcpyAsync(idx, id.data(), (size_t)q->B * 4, cudaMemcpyHostToDevice, q->stream), "staging");
        EK_MCUDA(cudaMemsetAsync(l, 0, 8, q->stream), "staging");
        gather_batch<<<q->B, 256, 0, q->stream>>>(xs, ts, idx, nullptr, nullptr, q->B, q->x, q->xt, q->t);
        EK_MCUDA(cudaGetLastError(), "batch gather");
        int rc = forward(q);
        if (rc != EK_OK) return rc;
        double *saved = q->loss;
        q->loss = l;
        rc = backward(q, false);
        q->loss = saved;
        if (rc != EK_OK) return rc;
        EK_MCUDA(cudaMemcpyAsync(grads, q->g, q->nparam * 4, cudaMemcpyDeviceToHost, q->stream), "gradients");
        if (loss) EK_MCUDA(cudaMemcpyAsync(loss, l, 8, cudaMemcpyDeviceToHost, q->stream), "loss");
        return check_err(q);
    };
    const int rc = run();
    cudaFree(xs);
    cudaFree(ts);
    cudaFree(idx);
    cudaFree(l);
    return rc;
}

// y (n x 512) = network(x (n x 4)), up to EVAL_ROWS rows in flight at once,
// in a workspace kept with the network: five launches for a call of up to
// EVAL_ROWS rows.  (In batches of the training size with scratch allocated by
// the call, 1000 rows took 1.59 ms on B200.)
int ek_mlp_forward(ek_mlp *q, const float *x, int64_t n, float *y) {
    if (!q || !x || !y || n < 0) return ek::ctx_fail(EK_ERR_INVALID, "bad forward arguments");
    if (n > 0) {
        const int rc = eval_reserve(q, std::min<int64_t>(n, EVAL_ROWS));
        if (rc != EK_OK) return rc;
    }
    for (int64_t r0 = 0; r0 < n; r0 += q->eval_cap) {
        const int64_t cnt = std::min<int64_t>(q->eval_cap, n - r0);
        const int rows = (int)((cnt + TM - 1) / TM * TM);
        EK_MCUDA(cudaMemcpyAsync(q->ex, x + r0 * IN, (size_t)cnt * IN * 4, cudaMemcpyHostToDevice, q->stream), "inputs");
        pad_inputs<<<rows / 128, 128, 0, q->stream>>>((const float4 *)q->ex, (int)cnt, rows, (uint4 *)q->exb);
        EK_MCUDA(cudaGetLastError(), "inputs");
        const bf16 *in = q->exb;
        int ldin = INP;
        for (int l = 0; l < 3; ++l) {
            GemmArgs a;
            EK_MCUDA(gemm_args(a, in, ldin, q->wb[l], DIM_IN[l], rows, HID, DIM_IN[l], q->err, q->wait_cycles), "operand maps");
            a.bias = q->p + q->off_b[l];
            a.h = q->eh[l & 1];
            a.ldh = HID;
            EK_MCUDA(gemm<EPI_FWD_HIDDEN>(a, q->stream), "forward GEMM");
            in = a.h;
            ldin = HID;
        }
        GemmArgs a;
        EK_MCUDA(gemm_args(a, in, HID, q->wb[3], HID, rows, OUT, HID, q->err, q->wait_cycles), "operand maps");
        a.bias = q->p + q->off_b[3];
        a.c = q->ey;
        a.ldc = OUT;
        EK_MCUDA(gemm<EPI_FWD_OUT>(a, q->stream), "output GEMM");
        q->launches += 5;
        EK_MCUDA(cudaMemcpyAsync(y + r0 * OUT, q->ey, (size_t)cnt * OUT * 4, cudaMemcpyDeviceToHost, q->stream), "output");
    }
    return check_err(q);
}

int ek_mlp_launch_count(const ek_mlp *q, int64_t *out) {
    if (!q || !out) return ek::ctx_fail(EK_ERR_INVALID, "null argument");
    *out = q->launches;
    return EK_OK;
}

int ek_mlp_set_wait_cycles(ek_mlp *q, int64_t cycles) {
    if (!q || cycles < 1) return ek::ctx_fail(EK_ERR_INVALID, "need a network and cycles >= 1");
    EK_MCUDA(cudaStreamSynchronize(q->stream), "wait bound");
    if (q->graph) cudaGraphExecDestroy(q->graph);  // it holds the old bound
    q->graph = nullptr;
    q->wait_cycles = cycles;
    return EK_OK;
}

}  // extern "C"

namespace {
// One block of 64 threads: thread 0 waits, at most `cycles`, on an mbarrier
// that expects one arrival; thread 32 (another warp) arrives only if
// `arrive`.  out[0] = 1 if the wait gave up, out[1] = 1 when thread 0 is done.
__global__ void __launch_bounds__(64) wait_selftest(long long cycles, int arrive, int *out) {
    __shared__ __align__(8) uint64_t bar;
    if (threadIdx.x == 0) {
        ek::tc::mbar_init(&bar, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    if (threadIdx.x == 32 && arrive)
        asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(ek::tc::smem_u32(&bar)) : "memory");
    if (threadIdx.x == 0) {
        const bool ok = ek::tc::mbar_wait_bounded(&bar, 0, cycles);
        out[0] = ok ? 0 : 1;
        out[1] = 1;
    }
}
}  // namespace

extern "C" {

int ek_wait_selftest(int64_t cycles, int32_t arrive) {
    if (cycles < 1) return ek::ctx_fail(EK_ERR_INVALID, "need cycles >= 1");
    int *out = nullptr;
    EK_MCUDA(cudaMalloc(&out, 2 * sizeof(int)), "self-test word");
    cudaError_t e = cudaMemset(out, 0, 2 * sizeof(int));
    if (e == cudaSuccess) {
        wait_selftest<<<1, 64>>>((long long)cycles, arrive ? 1 : 0, out);
        e = cudaGetLastError();
    }
    int h[2] = {0, 0};
    if (e == cudaSuccess) e = cudaMemcpy(h, out, sizeof(h), cudaMemcpyDeviceToHost);
    cudaFree(out);
    EK_MCUDA(e, "self-test kernel");
    if (h[1] != 1) return ek::ctx_fail(EK_ERR_CUDA, "self-test kernel did not finish");
    if (h[0]) return ek::ctx_fail(EK_ERR_TIMEOUT, "the bounded wait gave up (as asked: nothing arrived)");
    return EK_OK;
}

// C (m x n, FP32, row stride ldc) = A (m x k) B (n x k)^T on the tensor cores;
// BF16 device operands, m a multiple of 128, n a multiple of 16 (and of 128
// above 128), k a multiple of 16, lda and ldb multiples of 8.
int ek_gemm_bf16(const uint16_t *a, int32_t lda, const uint16_t *b, int32_t ldb, float *c, int32_t ldc, int32_t m,
                 int32_t n, int32_t k, void *stream) {
    if (!a || !b || !c || m <= 0 || n <= 0 || k <= 0) return ek::ctx_fail(EK_ERR_INVALID, "bad GEMM arguments");
    if (m % TM || n % 16 || (n > NT_MAX && n % NT_MAX) || k % 16 || lda % 8 || ldb % 8 || lda < k || ldb < k ||
        ldc < n)
        return ek::ctx_fail(EK_ERR_UNSUPPORTED, "GEMM shape outside the supported tiling");
    if (((uintptr_t)a | (uintptr_t)b) & 15) return ek::ctx_fail(EK_ERR_INVALID, "operands must be 16-byte aligned");
    static int *err = nullptr;
    if (!err) {
        EK_MCUDA(cudaMalloc(&err, 4), "error word");
        EK_MCUDA(cudaMemset(err, 0, 4), "error word");
    }
    EK_MCUDA(gemm_set_attributes(), "GEMM attributes");
    GemmArgs g;
    EK_MCUDA(gemm_args(g, (const bf16 *)a, lda, (const bf16 *)b, ldb, m, n, k, err), "operand maps");
    g.c = c;
    g.ldc = ldc;
    g.c_vec = ldc % 4 == 0 && ((uintptr_t)c & 15) == 0;
    // an ordinary launch: the operands may come from the kernel just before
    mlp_gemm<EPI_F32><<<dim3(m / TM, n / g.nt), GT, g.zoff, (cudaStream_t)stream>>>(g);
    EK_MCUDA(cudaGetLastError(), "GEMM");
    int v = 0;
    EK_MCUDA(cudaMemcpyAsync(&v, err, 4, cudaMemcpyDeviceToHost, (cudaStream_t)stream), "error word");
    EK_MCUDA(cudaStreamSynchronize((cudaStream_t)stream), "GEMM");
    if (v) {
        cudaMemset(err, 0, 4);
        return ek::ctx_fail(EK_ERR_TIMEOUT, "a bounded wait for the tensor cores gave up");
    }
    return EK_OK;
}

}  // extern "C"
