// Learned lambda warm start: per-particle MLP 12 -> 64 -> 64 -> 64 -> 1 (GELU),
// BF16 weights, FP32 accumulation, on the 5th-generation tensor cores (tcgen05,
// accumulators in TMEM). No reference counterpart.
//
// Every tensor-core kernel runs 128 threads per CTA: thread t owns row t of a
// 128-row tile, which is TMEM lane t of the accumulator, so each epilogue
// (bias, GELU, its derivative, the output layer) is per-thread register work
// on one particle after a tcgen05.ld of that thread's lane.
#include <algorithm>

#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "pbf_device.cuh"
#include "pbf_launch.cuh"
#include "pbf_mlp.h"
#include "pbf_packed.cuh"
#include "pbf_tc.cuh"
#include "pbf_mlp_dev.cuh"

namespace pbf {

using namespace tc;

constexpr int TILE = 128;
constexpr int TMEM_COLS = 256;      // tile GEMM, and training (two products at columns 0 and 128; one CTA per SM by smem)
constexpr int TMEM_COLS_FWD = 128;  // forward: layers 1 and 3 share columns [0, 64), so 4 CTAs fit an SM

// ---------------------------------------------------------------------------
// Tile GEMM (exported for tests): D[128 x N] = A[128 x K] * B[N x K]^T.
// ---------------------------------------------------------------------------
constexpr int TC_GEMM_SMEM_MIN = 96 * 1024;

__global__ void __launch_bounds__(128, 1) k_tc_gemm(const __nv_bfloat16* __restrict__ A,
                                                    const __nv_bfloat16* __restrict__ B, float* __restrict__ D,
                                                    int N, int K, int* __restrict__ err) {
    extern __shared__ __align__(1024) uint8_t smem[];
    __shared__ uint64_t mbar;
    __shared__ uint32_t tmem_slot;
    const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
    uint8_t* sA = smem;
    uint8_t* sB = smem + ((128 * K * 2 + 1023) & ~1023);
    if (warp == 0) tmem_alloc(&tmem_slot, TMEM_COLS);
    if (t == 0) mbar_init(&mbar, 1);
    for (int j = 0; j < K / 8; ++j) {
        const uint4 v = *reinterpret_cast<const uint4*>(A + (size_t)t * K + 8 * j);
        *reinterpret_cast<uint4*>(sA + kmajor_offset(t, 8 * j, 128)) = v;
    }
    for (int r = t; r < N; r += 128)
        for (int j = 0; j < K / 8; ++j) {
            const uint4 v = *reinterpret_cast<const uint4*>(B + (size_t)r * K + 8 * j);
            *reinterpret_cast<uint4*>(sB + kmajor_offset(r, 8 * j, N)) = v;
        }
    fence_async_smem();
    fence_before_sync();
    __syncthreads();
    fence_after_sync();
    const uint32_t tbase = tmem_slot;
    if (t == 0) {
        gemm_issue(tbase, sA, sB, N, K, 0);
        commit(&mbar);
    }
    bool ok = mbar_wait(&mbar, 0);
    if (!ok) {
        if (lane == 0) atomicOr(err, DEVERR_MLP_TIMEOUT);
        ok = mbar_wait(&mbar, 0);  // a second bounded wait for MMAs in flight before TMEM is freed
    }
    fence_after_sync();
    if (ok) {
        for (int c = 0; c < N / 16; ++c) {
            float v[16];
            tmem_ld16(tmem_addr(tbase, 32 * warp, 16 * c), v);
            tmem_wait_ld();
#pragma unroll
            for (int i = 0; i < 16; ++i) D[(size_t)t * N + 16 * c + i] = v[i];
        }
    }
    fence_before_sync();
    __syncthreads();
    if (warp == 0) tmem_dealloc(tbase, TMEM_COLS);
}

int tc_gemm_bf16(const void* A, const void* B, float* D, int N, int K, int* err, cudaStream_t st) {
    const int smem = (128 * K * 2 + 1023) / 1024 * 1024 + N * K * 2;
    const int bytes = smem < TC_GEMM_SMEM_MIN ? TC_GEMM_SMEM_MIN : smem;
    cudaError_t e = cudaFuncSetAttribute(k_tc_gemm, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e != cudaSuccess) return -1;
    k_tc_gemm<<<1, 128, bytes, st>>>((const __nv_bfloat16*)A, (const __nv_bfloat16*)B, D, N, K, err);
    return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

// ---------------------------------------------------------------------------
// Inference over 128-row tiles (persistent CTAs).
// ---------------------------------------------------------------------------
struct FwdIO {
    const uint16_t* w;   // bf16 weights
    const float* b;      // biases and constants
    const float* feat;   // raw features [n][12]
    int n;
    float* out;
    float4* q;
    float* lam_acc;
    float clamp;  // trust-region factor around q.w (0: none)
    int floor;    // 1: lambda0 at least as strong as q.w (same sign, magnitude >= |q.w|)
    int* err;
    // failure injection (the bounded-wait test only): no MMA is issued or
    // committed, so every wait on the barrier runs out after wait_limit polls
    int no_commit = 0;
    long long wait_limit = MBAR_WAIT_LIMIT;
};

constexpr int FWD_SW1 = 0;                              // [64 x 16]   2 KB
constexpr int FWD_SW2 = FWD_SW1 + 64 * 16 * 2;          // [64 x 64]   8 KB
constexpr int FWD_SW3 = FWD_SW2 + 64 * 64 * 2;          // [64 x 64]   8 KB
constexpr int FWD_SX = FWD_SW3 + 64 * 64 * 2;           // [128 x 16]  4 KB
constexpr int FWD_SH1 = FWD_SX + 128 * 16 * 2;          // [128 x 64] 16 KB
constexpr int FWD_SH2 = FWD_SH1 + 128 * 64 * 2;         // [128 x 64] 16 KB
constexpr int FWD_SMEM_INFER = FWD_SH2 + 128 * 64 * 2;

__global__ void __launch_bounds__(128, 1) k_mlp_fwd(FwdIO io) {
    extern __shared__ __align__(1024) uint8_t smem[];
    __shared__ uint64_t mbar;
    __shared__ uint32_t tmem_slot;
    __shared__ float sb[MLP_NUM_BIASES];
    __shared__ float sw4[64];
    const int t = threadIdx.x, warp = t >> 5;
    if (warp == 0) tmem_alloc(&tmem_slot, TMEM_COLS_FWD);
    if (t == 0) mbar_init(&mbar, 1);
    stage_weight(smem + FWD_SW1, io.w + W1_OFF, 64, 16);
    stage_weight(smem + FWD_SW2, io.w + W2_OFF, 64, 64);
    stage_weight(smem + FWD_SW3, io.w + W3_OFF, 64, 64);
    for (int i = t; i < MLP_NUM_BIASES; i += 128) sb[i] = io.b[i];
    if (t < 64) sw4[t] = bf16_val(io.w[W4_OFF + t]);
    fence_before_sync();
    __syncthreads();
    fence_after_sync();
    const uint32_t tbase = tmem_slot;
    const uint32_t lane_base = tmem_addr(tbase, 32 * warp, 0);
    uint32_t phase = 0;
    bool alive = true;
    const int ntiles = (io.n + TILE - 1) / TILE;
    for (int tile = blockIdx.x; tile < ntiles && alive; tile += gridDim.x) {
        const int row = tile * TILE + t;
        const bool valid = row < io.n;
        // normalised features -> bf16 A tile [128 x 16]
        {
            float xf[16];
#pragma unroll
            for (int k = 0; k < 16; ++k) xf[k] = 0.0f;
            if (valid) {
#pragma unroll
                for (int k = 0; k < MLP_IN; ++k)
                    xf[k] = (io.feat[(size_t)row * MLP_IN + k] - sb[FMEAN_OFF + k]) * sb[FISTD_OFF + k];
            }
            uint32_t pk[8];
#pragma unroll
            for (int i = 0; i < 8; ++i)
                pk[i] = (uint32_t)bf16_bits(xf[2 * i]) | ((uint32_t)bf16_bits(xf[2 * i + 1]) << 16);
            *reinterpret_cast<uint4*>(smem + FWD_SX + kmajor_offset(t, 0, 128)) = make_uint4(pk[0], pk[1], pk[2], pk[3]);
            *reinterpret_cast<uint4*>(smem + FWD_SX + kmajor_offset(t, 8, 128)) = make_uint4(pk[4], pk[5], pk[6], pk[7]);
        }
        // ---- layer 1: TMEM cols [0, 64)
        sync_for_mma();
        if (t == 0 && !io.no_commit) {
            gemm_issue(tbase, smem + FWD_SX, smem + FWD_SW1, 64, 16, 0);
            commit(&mbar);
        }
        if (!wait_mma(&mbar, phase, io.err, io.wait_limit)) { alive = false; break; }
#pragma unroll 1
        for (int c = 0; c < 4; ++c) {
            float v[16];
            tmem_ld16(lane_base + 16 * c, v);
            tmem_wait_ld();
#pragma unroll
            for (int i = 0; i < 16; i += 2) {
                const float2 z = vadd(make_float2(v[i], v[i + 1]), make_float2(sb[B1_OFF + 16 * c + i], sb[B1_OFF + 16 * c + i + 1]));
                const float2 hh = gelu2(z);
                v[i] = hh.x;
                v[i + 1] = hh.y;
            }
            put_row64(smem + FWD_SH1, t, v, 16 * c);
        }
        // ---- layer 2: TMEM cols [64, 128)
        sync_for_mma();
        if (t == 0 && !io.no_commit) {
            gemm_issue(tbase + 64, smem + FWD_SH1, smem + FWD_SW2, 64, 64, 0);
            commit(&mbar);
        }
        if (!wait_mma(&mbar, phase, io.err, io.wait_limit)) { alive = false; break; }
#pragma unroll 1
        for (int c = 0; c < 4; ++c) {
            float v[16];
            tmem_ld16(lane_base + 64 + 16 * c, v);
            tmem_wait_ld();
#pragma unroll
            for (int i = 0; i < 16; i += 2) {
                const float2 z = vadd(make_float2(v[i], v[i + 1]), make_float2(sb[B2_OFF + 16 * c + i], sb[B2_OFF + 16 * c + i + 1]));
                const float2 hh = gelu2(z);
                v[i] = hh.x;
                v[i + 1] = hh.y;
            }
            put_row64(smem + FWD_SH2, t, v, 16 * c);
        }
        // ---- layer 3: TMEM cols [0, 64) again (layer 1's values were consumed
        // before layer 2 was issued), then the output layer on CUDA cores
        sync_for_mma();
        if (t == 0 && !io.no_commit) {
            gemm_issue(tbase, smem + FWD_SH2, smem + FWD_SW3, 64, 64, 0);
            commit(&mbar);
        }
        if (!wait_mma(&mbar, phase, io.err, io.wait_limit)) { alive = false; break; }
        float y = sb[B4_OFF];
#pragma unroll 1
        for (int c = 0; c < 4; ++c) {
            float v[16];
            tmem_ld16(lane_base + 16 * c, v);
            tmem_wait_ld();
            float hs[16];
#pragma unroll
            for (int i = 0; i < 16; i += 2) {
                const float2 hh = gelu2(vadd(make_float2(v[i], v[i + 1]),
                                             make_float2(sb[B3_OFF + 16 * c + i], sb[B3_OFF + 16 * c + i + 1])));
                hs[i] = hh.x;
                hs[i + 1] = hh.y;
            }
#pragma unroll
            for (int i = 0; i < 16; ++i) y = __fmaf_rn(hs[i], sw4[16 * c + i], y);
        }
        if (valid) {
            float lam0 = y * sb[OSCALE_OFF];
            if (io.q && io.clamp > 0.0f) {
                // trust region around the plain lambda of the same pass (q.w):
                // same sign, at most clamp times its magnitude
                const float lp = reinterpret_cast<const float*>(io.q)[4 * (size_t)row + 3];
                const float a = io.clamp * lp;
                const float f0 = io.floor ? lp : 0.0f;  // the weak end of the interval
                lam0 = fminf(fmaxf(lam0, fminf(a, f0)), fmaxf(a, f0));
            }
            if (io.out) io.out[row] = lam0;
            if (io.q) reinterpret_cast<float*>(io.q)[4 * (size_t)row + 3] = lam0;
            if (io.lam_acc) io.lam_acc[row] = lam0;
        }
    }
    fence_before_sync();
    __syncthreads();
    if (warp == 0) tmem_dealloc(tbase, TMEM_COLS_FWD);
}

// ---------------------------------------------------------------------------
// Training: one kernel evaluates a 128-row tile forward and backward with every
// activation kept in shared memory (the network's state of a tile is 200 KB), and
// one sums the tiles' gradients in a fixed order and applies Adam.
//
// Forward as in inference, keeping H1, H2 (BF16, both as the next product's
// K-major A tile and transposed) and gelu' of each layer (BF16, registers).
// Backward through a hidden layer with Kin inputs:
//   dW[64 x Kin] = dZ^T H and db = column sums of dZ  (one MMA: a ones row is
//                                                      appended to H^T)
//   dH = dZ W, dZ_prev = dH * gelu'(Z_prev)           (second MMA, if any)
// A tile is a chain of six tensor-core round trips with an epilogue each, so its
// latency is what counts: 512 threads share each epilogue, 16 columns of one row
// per thread (warp w reads TMEM lanes 32 (w & 3) and columns 16 (w >> 2), so one
// tcgen05.ld per thread and product). Batch 4,096: 204 us per step with a kernel
// per layer and direction (activations stored 2 bytes at a time, one launch per
// gradient sum), 27.8 with the two (this one 18.2).
// ---------------------------------------------------------------------------
struct TrainIO {
    const uint16_t* w;    // bf16 weights
    const float* b;       // biases and constants
    const float* feat;    // raw features [n][12]
    const float* target;  // [n]
    float* part;          // per tile: PART_TILE floats
    int n;
    float inv_batch;
    int* err;
};
// gradient partials of a tile: dW3 | db3, dW2 | db2, dW1 | db1, then per warp of
// rows loss, db4, dw4[64]
constexpr int PART_L3 = 0, PART_L2 = PART_L3 + 64 * 64 + 64, PART_L1 = PART_L2 + 64 * 64 + 64;
constexpr int PART_OUT = PART_L1 + 64 * 16 + 64, PART_WARP = 66, PART_TILE = PART_OUT + 4 * PART_WARP;

constexpr int TR_THREADS = 512;
constexpr int TR_W1 = 0;                           // [64 x 16]
constexpr int TR_W2 = TR_W1 + 64 * 16 * 2;         // [64 x 64]
constexpr int TR_W3 = TR_W2 + 64 * 64 * 2;
constexpr int TR_W2T = TR_W3 + 64 * 64 * 2;        // W^T, B of dH
constexpr int TR_W3T = TR_W2T + 64 * 64 * 2;
constexpr int TR_X = TR_W3T + 64 * 64 * 2;         // [128 x 16]
constexpr int TR_XT = TR_X + 128 * 16 * 2;         // [32 x 128]: X^T, the ones row, zeros
constexpr int TR_H1 = TR_XT + 32 * 128 * 2;        // [128 x 64]
constexpr int TR_H1T = TR_H1 + 128 * 64 * 2;       // [80 x 128]
constexpr int TR_H2 = TR_H1T + 80 * 128 * 2;
constexpr int TR_H2T = TR_H2 + 128 * 64 * 2;
constexpr int TR_DZ = TR_H2T + 80 * 128 * 2;       // [128 x 64]
constexpr int TR_DZT = TR_DZ + 128 * 64 * 2;       // [128 x 128], rows 64.. zero
constexpr int TR_H3F = TR_DZT + 128 * 128 * 2;     // [128][65] fp32
constexpr int TR_SMEM = TR_H3F + 128 * 65 * 4;

// 16 BF16 values of columns c0.. of row `row` into a K-major [128 x 64] tile
__device__ __forceinline__ void put_bits16(uint8_t* s, int row, int c0, const uint16_t (&h)[16]) {
    uint32_t pk[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) pk[i] = (uint32_t)h[2 * i] | ((uint32_t)h[2 * i + 1] << 16);
    *reinterpret_cast<uint4*>(s + kmajor_offset(row, c0, 128)) = make_uint4(pk[0], pk[1], pk[2], pk[3]);
    *reinterpret_cast<uint4*>(s + kmajor_offset(row, c0 + 8, 128)) = make_uint4(pk[4], pk[5], pk[6], pk[7]);
}
// the same values into column `row` of the transposed tile of R rows
__device__ __forceinline__ void put_bits16_t(uint8_t* s, int R, int row, int c0, const uint16_t (&h)[16]) {
#pragma unroll
    for (int i = 0; i < 16; ++i) *reinterpret_cast<uint16_t*>(s + kmajor_offset(c0 + i, row, R)) = h[i];
}

__global__ void __launch_bounds__(TR_THREADS, 1) k_mlp_train(TrainIO io) {
    extern __shared__ __align__(1024) uint8_t smem[];
    __shared__ uint64_t mbar;
    __shared__ uint32_t tmem_slot;
    __shared__ float sb[MLP_NUM_BIASES];
    __shared__ float sw4[64];
    __shared__ float s_dy[128];
    const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
    const int m = 32 * (warp & 3) + lane;  // this thread's row of the tile
    const int cq = warp >> 2, c0 = 16 * cq;  // and its 16 columns
    if (warp == 0) tmem_alloc(&tmem_slot, TMEM_COLS);
    if (t == 0) mbar_init(&mbar, 1);
    // what stays zero: rows 64.. of dZ^T, the rows after the ones rows
    const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
    for (int i = t; i < 64 * 16; i += TR_THREADS)
        *reinterpret_cast<uint4*>(smem + TR_DZT + kmajor_offset(64 + i / 16, 8 * (i % 16), 128)) = zero;
    for (int i = t; i < 16 * 16; i += TR_THREADS) {
        *reinterpret_cast<uint4*>(smem + TR_H1T + kmajor_offset(64 + i / 16, 8 * (i % 16), 80)) = zero;
        *reinterpret_cast<uint4*>(smem + TR_H2T + kmajor_offset(64 + i / 16, 8 * (i % 16), 80)) = zero;
        *reinterpret_cast<uint4*>(smem + TR_XT + kmajor_offset(16 + i / 16, 8 * (i % 16), 32)) = zero;
    }
    // everything above overlaps the end of the kernel before (the reduction that
    // wrote these weights); nothing below does
    pdl_launch();
    pdl_wait();
    stage_weight(smem + TR_W1, io.w + W1_OFF, 64, 16);
    stage_weight(smem + TR_W2, io.w + W2_OFF, 64, 64);
    stage_weight(smem + TR_W3, io.w + W3_OFF, 64, 64);
    stage_weight_t(smem + TR_W2T, io.w + W2_OFF, 64);
    stage_weight_t(smem + TR_W3T, io.w + W3_OFF, 64);
    for (int i = t; i < MLP_NUM_BIASES; i += TR_THREADS) sb[i] = io.b[i];
    if (t < 64) sw4[t] = bf16_val(io.w[W4_OFF + t]);
    fence_before_sync();
    __syncthreads();
    fence_after_sync();
    const uint32_t tbase = tmem_slot;
    const uint32_t lane_base = tmem_addr(tbase, 32 * (warp & 3), c0);
    float* h3f = reinterpret_cast<float*>(smem + TR_H3F);
    uint32_t phase = 0;
    bool alive = true;
    // one product (two with a second B) and the wait for it; false: the wait expired
    auto product = [&](int a, int bt, int N, int K, int a2, int b2) {
        sync_for_mma();
        if (t == 0) {
            gemm_issue(tbase, smem + a, smem + bt, N, K, 0);
            if (a2 >= 0) gemm_issue(tbase + 128, smem + a2, smem + b2, 64, 64, 0);
            commit(&mbar);
        }
        return wait_mma(&mbar, phase, io.err);
    };
    const int ntiles = (io.n + TILE - 1) / TILE;
    for (int tile = blockIdx.x; tile < ntiles && alive; tile += gridDim.x) {
        const int row = tile * TILE + m;
        const bool valid = row < io.n;
        float* part = io.part + (size_t)tile * PART_TILE;
        // normalised features -> BF16, four per thread
        {
            uint16_t xb[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int k = 4 * cq + i;
                const float xf = valid && k < MLP_IN
                                     ? (io.feat[(size_t)row * MLP_IN + k] - sb[FMEAN_OFF + k]) * sb[FISTD_OFF + k]
                                     : 0.0f;
                xb[i] = bf16_bits(xf);
                *reinterpret_cast<uint16_t*>(smem + TR_XT + kmajor_offset(k, m, 32)) = xb[i];
            }
            *reinterpret_cast<uint2*>(smem + TR_X + kmajor_offset(m, 4 * cq, 128)) =
                make_uint2((uint32_t)xb[0] | ((uint32_t)xb[1] << 16), (uint32_t)xb[2] | ((uint32_t)xb[3] << 16));
            if (cq == 0) {
                const uint16_t one = valid ? 0x3F80 : 0;  // the ones row: db comes out of the dW product
                *reinterpret_cast<uint16_t*>(smem + TR_XT + kmajor_offset(16, m, 32)) = one;
                *reinterpret_cast<uint16_t*>(smem + TR_H1T + kmajor_offset(64, m, 80)) = one;
                *reinterpret_cast<uint16_t*>(smem + TR_H2T + kmajor_offset(64, m, 80)) = one;
            }
        }
        const float tgt = t < TILE && valid ? io.target[row] : 0.0f;
        uint16_t g1[16], g2[16], g3[16];
        // ---- hidden layers 1 and 2
#pragma unroll
        for (int l = 0; l < 2; ++l) {
            alive = l == 0 ? product(TR_X, TR_W1, 64, 16, -1, -1) : product(TR_H1, TR_W2, 64, 64, -1, -1);
            if (!alive) break;
            const float* bias = sb + (l == 0 ? B1_OFF : B2_OFF) + c0;
            uint16_t(&g)[16] = l == 0 ? g1 : g2;
            float v[16];
            tmem_ld16(lane_base, v);
            tmem_wait_ld();
            uint16_t h[16];
#pragma unroll
            for (int i = 0; i < 16; i += 2) {
                const float2 z = vadd(make_float2(v[i], v[i + 1]), make_float2(bias[i], bias[i + 1]));
                g[i] = bf16_bits(gelu_grad(z.x));
                g[i + 1] = bf16_bits(gelu_grad(z.y));
                const float2 hh = gelu2(z);
                h[i] = bf16_bits(hh.x);
                h[i + 1] = bf16_bits(hh.y);
            }
            put_bits16(smem + (l == 0 ? TR_H1 : TR_H2), m, c0, h);
#pragma unroll
            for (int i = 0; i < 16; ++i) h[i] = valid ? h[i] : 0;
            put_bits16_t(smem + (l == 0 ? TR_H1T : TR_H2T), 80, m, c0, h);
        }
        if (!alive) break;
        // ---- layer 3, kept in FP32
        alive = product(TR_H2, TR_W3, 64, 64, -1, -1);
        if (!alive) break;
        {
            float v[16];
            tmem_ld16(lane_base, v);
            tmem_wait_ld();
#pragma unroll
            for (int i = 0; i < 16; i += 2) {
                const float2 hh = gelu2(vadd(make_float2(v[i], v[i + 1]),
                                             make_float2(sb[B3_OFF + c0 + i], sb[B3_OFF + c0 + i + 1])));
                h3f[m * 65 + c0 + i] = hh.x;
                h3f[m * 65 + c0 + i + 1] = hh.y;
            }
#pragma unroll
            for (int i = 0; i < 16; ++i) g3[i] = bf16_bits(gelu_grad(v[i] + sb[B3_OFF + c0 + i]));
        }
        __syncthreads();
        // ---- output layer: loss = mean (y - target/scale)^2 ; dy = 2 (y - t) / B
        if (t < TILE) {  // thread t is row t here: warps 0 .. 3 have m = t
            float y = sb[B4_OFF];
#pragma unroll 16
            for (int i = 0; i < 64; ++i) y = __fmaf_rn(h3f[t * 65 + i], sw4[i], y);
            const float r = valid ? (y - tgt / sb[OSCALE_OFF]) : 0.0f;
            const float dy = 2.0f * r * io.inv_batch;
            s_dy[t] = dy;
            float l = r * r * io.inv_batch, db = dy;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                l += __shfl_xor_sync(0xffffffffu, l, o);
                db += __shfl_xor_sync(0xffffffffu, db, o);
            }
            // this warp's sums go to its own slot; the slots are added in a fixed
            // order, so the gradients do not depend on the blocks' timing
            if (lane == 0) {
                part[PART_OUT + warp * PART_WARP] = l;
                part[PART_OUT + warp * PART_WARP + 1] = db;
            }
        }
        __syncthreads();
        {
            uint16_t dz[16];
            const float dy = s_dy[m];
#pragma unroll
            for (int i = 0; i < 16; ++i) dz[i] = valid ? bf16_bits(dy * sw4[c0 + i] * bf16_val(g3[i])) : 0;
            put_bits16(smem + TR_DZ, m, c0, dz);
            put_bits16_t(smem + TR_DZT, 128, m, c0, dz);
        }
        if (t >= 256) {  // dw4: column nn of 32 rows, added as a butterfly over 32 lanes would
            const int wr = (t - 256) >> 6, nn = t & 63;
            float a[32];
#pragma unroll
            for (int i = 0; i < 32; ++i) a[i] = s_dy[32 * wr + i] * h3f[(32 * wr + i) * 65 + nn];
#pragma unroll
            for (int o = 16; o > 0; o >>= 1)
#pragma unroll
                for (int i = 0; i < o; ++i) a[i] = a[i] + a[i + o];
            part[PART_OUT + wr * PART_WARP + 2 + nn] = a[0];
        }
        // ---- backward through layers 3, 2 and 1
#pragma unroll
        for (int l = 3; l >= 1; --l) {
            alive = l == 3   ? product(TR_DZT, TR_H2T, 80, 128, TR_DZ, TR_W3T)
                    : l == 2 ? product(TR_DZT, TR_H1T, 80, 128, TR_DZ, TR_W2T)
                             : product(TR_DZT, TR_XT, 32, 128, -1, -1);
            if (!alive) break;
            const int kin = l == 1 ? 16 : 64;
            float* dst = part + (l == 3 ? PART_L3 : l == 2 ? PART_L2 : PART_L1);
            if ((warp & 3) < 2) {  // rows 0 .. 63 of the dW product: output unit m
                if (c0 < kin) {
                    float v[16];
                    tmem_ld16(lane_base, v);
                    tmem_wait_ld();
#pragma unroll
                    for (int i = 0; i < 16; i += 4)
                        *reinterpret_cast<float4*>(dst + m * kin + c0 + i) =
                            make_float4(v[i], v[i + 1], v[i + 2], v[i + 3]);
                }
                if (cq == 1) {  // the column of the ones row
                    float v[16];
                    tmem_ld16(tmem_addr(tbase, 32 * (warp & 3), kin), v);
                    tmem_wait_ld();
                    dst[64 * kin + m] = v[0];
                }
            }
            if (l > 1) {
                const uint16_t(&g)[16] = l == 3 ? g2 : g1;
                float v[16];
                tmem_ld16(lane_base + 128, v);
                tmem_wait_ld();
                uint16_t dz[16];
#pragma unroll
                for (int i = 0; i < 16; ++i) dz[i] = valid ? bf16_bits(v[i] * bf16_val(g[i])) : 0;
                put_bits16(smem + TR_DZ, m, c0, dz);
                put_bits16_t(smem + TR_DZT, 128, m, c0, dz);
            }
        }
    }
    fence_before_sync();
    __syncthreads();
    if (warp == 0) tmem_dealloc(tbase, TMEM_COLS);
}

struct AdamIO {
    float *pw, *pb, *mw, *mb, *vw, *vb;  // parameters and moments of weights and biases
    uint16_t* w16;
    float lr, b1, b2, eps, c1, c2;
};

// Gradients of all parameters (one thread each) and the loss: the tiles' partials
// in tile order, p = 0, 1, ... (deterministic: the same bits on every run), and
// with ADAM the parameter's Adam step on the FP32 masters, refreshing the BF16
// weights. Bound by the latency of its loads, so they are issued 32 at a time.
constexpr int REDUCE_UNROLL = 32;
template <bool ADAM>
__global__ void __launch_bounds__(64) k_mlp_reduce(const float* __restrict__ part, int tiles, float* __restrict__ gw,
                                                   float* __restrict__ gb, float* __restrict__ loss, AdamIO a) {
    const int i = blockIdx.x * 64 + threadIdx.x;
    const int j = i - MLP_NUM_WEIGHTS;  // >= 0: bias j, then the loss
    if (j > MLP_NUM_TRAINED_BIASES) return;
    // where the parameter lies in a slot; output-layer slots are one per warp of rows
    int at;
    bool out = false;
    if (j < 0) {
        if (i < W2_OFF) at = PART_L1 + (i - W1_OFF);
        else if (i < W3_OFF) at = PART_L2 + (i - W2_OFF);
        else if (i < W4_OFF) at = PART_L3 + (i - W3_OFF);
        else { at = PART_OUT + 2 + (i - W4_OFF); out = true; }
    } else if (j < B2_OFF) at = PART_L1 + 64 * 16 + (j - B1_OFF);
    else if (j < B3_OFF) at = PART_L2 + 64 * 64 + (j - B2_OFF);
    else if (j < B4_OFF) at = PART_L3 + 64 * 64 + (j - B3_OFF);
    else { at = PART_OUT + (j == B4_OFF ? 1 : 0); out = true; }
    pdl_wait();  // the partials of the training kernel before this one
    float s = 0.0f;
    const int slots = out ? 4 * tiles : tiles;
    for (int q0 = 0; q0 < slots; q0 += REDUCE_UNROLL) {
        float v[REDUCE_UNROLL];
#pragma unroll
        for (int u = 0; u < REDUCE_UNROLL; ++u) {
            const int q = q0 + u;
            const size_t o = out ? (size_t)(q >> 2) * PART_TILE + (q & 3) * PART_WARP : (size_t)q * PART_TILE;
            v[u] = q < slots ? part[o + at] : 0.0f;
        }
#pragma unroll
        for (int u = 0; u < REDUCE_UNROLL; ++u)
            if (q0 + u < slots) s += v[u];
    }
    if (j == MLP_NUM_TRAINED_BIASES) {
        *loss = s;
        return;
    }
    if (j < 0) gw[i] = s;
    else gb[j] = s;
    if (ADAM) {
        const int k = j < 0 ? i : j;
        float *p = j < 0 ? a.pw : a.pb, *mo = j < 0 ? a.mw : a.mb, *ve = j < 0 ? a.vw : a.vb;
        const float mi = a.b1 * mo[k] + (1.0f - a.b1) * s;
        const float vi = a.b2 * ve[k] + (1.0f - a.b2) * s * s;
        mo[k] = mi;
        ve[k] = vi;
        const float upd = a.lr * (mi / a.c1) / (sqrtf(vi / a.c2) + a.eps);
        const float pi = p[k] - upd;
        p[k] = pi;
        if (j < 0) a.w16[k] = bf16_bits(pi);
    }
}

__global__ void k_to_bf16(const float* p, uint16_t* q, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) q[i] = bf16_bits(p[i]);
}

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------
static int sm_count() {
    static int n = 0;
    if (!n) {
        int dev = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
        if (n <= 0) n = 148;
    }
    return n;
}

int mlp_infer(const uint16_t* w_bf16, const float* b, const float* feat, int n, float* out, float4* q, float* lam_acc,
              float clamp, int floor, int* err, cudaStream_t st) {
    if (n <= 0) return 0;
    static bool attr = false;
    if (!attr) {
        if (cudaFuncSetAttribute(k_mlp_fwd, cudaFuncAttributeMaxDynamicSharedMemorySize, FWD_SMEM_INFER) !=
            cudaSuccess)
            return -1;
        attr = true;
    }
    FwdIO io{};
    io.w = w_bf16;
    io.b = b;
    io.feat = feat;
    io.n = n;
    io.out = out;
    io.q = q;
    io.lam_acc = lam_acc;
    io.clamp = clamp;
    io.floor = floor;
    io.err = err;
    // four CTAs per SM (54 KB of shared memory and 128 TMEM columns each) overlap
    // one another's tensor-core waits
    const int tiles = (n + TILE - 1) / TILE;
    const int grid = tiles < 4 * sm_count() ? tiles : 4 * sm_count();
    k_mlp_fwd<<<grid, 128, FWD_SMEM_INFER, st>>>(io);
    return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

int mlp_infer_uncommitted(const uint16_t* w_bf16, const float* b, const float* feat, int n, float* out,
                          long long wait_limit, int* err, cudaStream_t st) {
    if (n <= 0) return 0;
    if (cudaFuncSetAttribute(k_mlp_fwd, cudaFuncAttributeMaxDynamicSharedMemorySize, FWD_SMEM_INFER) !=
        cudaSuccess)
        return -1;
    FwdIO io{};
    io.w = w_bf16;
    io.b = b;
    io.feat = feat;
    io.n = n;
    io.out = out;
    io.err = err;
    io.no_commit = 1;
    io.wait_limit = wait_limit;
    const int tiles = (n + TILE - 1) / TILE;
    k_mlp_fwd<<<tiles, 128, FWD_SMEM_INFER, st>>>(io);
    return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

struct MlpTrainer {
    int cap = 0;
    float *w32 = nullptr, *b32 = nullptr, *mw = nullptr, *vw = nullptr, *mb = nullptr, *vb = nullptr;
    float *gw = nullptr, *gb = nullptr, *loss = nullptr;
    float* part = nullptr;  // gradient partials per tile, summed in a fixed order
    int* err = nullptr;
    uint16_t* w16 = nullptr;
    int step = 0;
};

MlpTrainer* mlp_trainer_create(int max_batch, const float* w32, const float* b32) {
    MlpTrainer* t = new MlpTrainer();
    t->cap = max_batch;
    bool ok = true;
    auto A = [&](void** p, size_t bytes) {
        if (ok && cudaMalloc(p, bytes) != cudaSuccess) ok = false;
        if (ok) cudaMemset(*p, 0, bytes);
    };
    A((void**)&t->w32, sizeof(float) * MLP_NUM_WEIGHTS);
    A((void**)&t->b32, sizeof(float) * MLP_NUM_BIASES);
    A((void**)&t->mw, sizeof(float) * MLP_NUM_WEIGHTS);
    A((void**)&t->vw, sizeof(float) * MLP_NUM_WEIGHTS);
    A((void**)&t->mb, sizeof(float) * MLP_NUM_BIASES);
    A((void**)&t->vb, sizeof(float) * MLP_NUM_BIASES);
    A((void**)&t->gw, sizeof(float) * MLP_NUM_WEIGHTS);
    A((void**)&t->gb, sizeof(float) * MLP_NUM_BIASES);
    A((void**)&t->loss, sizeof(float));
    A((void**)&t->err, sizeof(int));
    A((void**)&t->w16, sizeof(uint16_t) * MLP_NUM_WEIGHTS);
    const size_t tiles = ((size_t)max_batch + TILE - 1) / TILE;
    A((void**)&t->part, sizeof(float) * tiles * PART_TILE);
    if (!ok) {
        mlp_trainer_destroy(t);
        return nullptr;
    }
    cudaMemcpy(t->w32, w32, sizeof(float) * MLP_NUM_WEIGHTS, cudaMemcpyHostToDevice);
    cudaMemcpy(t->b32, b32, sizeof(float) * MLP_NUM_BIASES, cudaMemcpyHostToDevice);
    k_to_bf16<<<(MLP_NUM_WEIGHTS + 255) / 256, 256>>>(t->w32, t->w16, MLP_NUM_WEIGHTS);
    if (cudaDeviceSynchronize() != cudaSuccess) {
        mlp_trainer_destroy(t);
        return nullptr;
    }
    return t;
}

void mlp_trainer_destroy(MlpTrainer* t) {
    if (!t) return;
    void* ps[] = {t->w32, t->b32, t->mw, t->vw, t->mb, t->vb, t->gw, t->gb, t->loss, t->err, t->w16,
                  t->part};
    for (void* p : ps)
        if (p) cudaFree(p);
    delete t;
}

// The tiles' gradient partials of a batch; the caller sums them.
static int launch_train(MlpTrainer* t, const float* feat, const float* target, int B, cudaStream_t st) {
    if (B <= 0 || B > t->cap) return -1;
    // (per call: the attribute belongs to the current device)
    if (cudaFuncSetAttribute(k_mlp_train, cudaFuncAttributeMaxDynamicSharedMemorySize, TR_SMEM) != cudaSuccess)
        return -1;
    const int tiles = (B + TILE - 1) / TILE;
    const int grid = tiles < sm_count() ? tiles : sm_count();
    const TrainIO io{t->w16, t->b32, feat, target, t->part, B, 1.0f / (float)B, t->err};
    return launch(true, k_mlp_train, grid, TR_THREADS, TR_SMEM, st, io);
}

constexpr int REDUCE_BLOCKS = (MLP_NUM_WEIGHTS + MLP_NUM_TRAINED_BIASES + 1 + 63) / 64;

int mlp_gradients(MlpTrainer* t, const float* feat, const float* target, int B, cudaStream_t st) {
    if (launch_train(t, feat, target, B, st)) return -1;
    return launch(true, k_mlp_reduce<false>, REDUCE_BLOCKS, 64, 0, st, t->part, (B + TILE - 1) / TILE, t->gw, t->gb,
                      t->loss, AdamIO{});
}

int mlp_train_step(MlpTrainer* t, const float* feat, const float* target, int B, float lr, float beta1, float beta2,
                   float eps, cudaStream_t st) {
    if (launch_train(t, feat, target, B, st)) return -1;
    t->step += 1;
    const AdamIO a{t->w32, t->b32, t->mw, t->mb, t->vw, t->vb, t->w16, lr, beta1, beta2, eps,
                   1.0f - powf(beta1, (float)t->step), 1.0f - powf(beta2, (float)t->step)};
    return launch(true, k_mlp_reduce<true>, REDUCE_BLOCKS, 64, 0, st, t->part, (B + TILE - 1) / TILE, t->gw, t->gb,
                      t->loss, a);
}

int mlp_read(MlpTrainer* t, float* w32, float* b32, float* gw, float* gb, float* loss, int* err) {
    cudaDeviceSynchronize();
    if (w32) cudaMemcpy(w32, t->w32, sizeof(float) * MLP_NUM_WEIGHTS, cudaMemcpyDeviceToHost);
    if (b32) cudaMemcpy(b32, t->b32, sizeof(float) * MLP_NUM_BIASES, cudaMemcpyDeviceToHost);
    if (gw) cudaMemcpy(gw, t->gw, sizeof(float) * MLP_NUM_WEIGHTS, cudaMemcpyDeviceToHost);
    if (gb) cudaMemcpy(gb, t->gb, sizeof(float) * MLP_NUM_BIASES, cudaMemcpyDeviceToHost);
    if (loss) cudaMemcpy(loss, t->loss, sizeof(float), cudaMemcpyDeviceToHost);
    if (err) cudaMemcpy(err, t->err, sizeof(int), cudaMemcpyDeviceToHost);
    return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

const uint16_t* mlp_weights_bf16(MlpTrainer* t) { return t->w16; }
const float* mlp_biases(MlpTrainer* t) { return t->b32; }

}  // namespace pbf
