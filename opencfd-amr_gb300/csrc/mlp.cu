// Chemistry surrogate network on the 5th-generation tensor cores: BF16 weights
// and activations, FP32 accumulation in tensor memory (tcgen05.mma, TMEM),
// operands staged in shared memory (tcgen05.cuh for the layouts).
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <string>
#include <vector>

#include "level.h"
#include "mlp_kernel.cuh"

namespace ocfd {

using namespace tc;

// C[128 x N] = A[128 x K] * B[N x K]^T for row-major BF16 A, B (K contiguous) and
// row-major FP32 C: one CTA of 128 threads, the whole K staged in shared memory.
__global__ void __launch_bounds__(128) k_tc_gemm(const uint16_t* __restrict__ A, const uint16_t* __restrict__ B,
                                                 float* __restrict__ C, int N, int K, unsigned* err) {
    extern __shared__ __align__(1024) unsigned char sm[];
    unsigned char* sA = sm;
    unsigned char* sB = sm + 128 * K * 2;
    uint64_t* bar = reinterpret_cast<uint64_t*>(sB + N * K * 2);
    uint32_t* tslot = reinterpret_cast<uint32_t*>(bar + 1);
    const int tid = threadIdx.x, warp = tid >> 5;
    const uint32_t ncols = tmem_cols(N);
    for (int e = tid; e < 128 * K; e += 128)
        *reinterpret_cast<uint16_t*>(sA + kmajor_offset(e / K, e % K, 128)) = A[e];
    for (int e = tid; e < N * K; e += 128)
        *reinterpret_cast<uint16_t*>(sB + kmajor_offset(e / K, e % K, N)) = B[e];
    if (tid == 0) mbar_init(bar, 1);
    if (warp == 0) {
        tmem_alloc(tslot, ncols);
        tmem_relinquish();
    }
    fence_async_smem();
    fence_before_sync();
    __syncthreads();
    fence_after_sync();
    const uint32_t tbase = *tslot;
    if (tid == 0) {
        const uint32_t idesc = idesc_bf16_f32(128, N);
        for (int ks = 0; ks < K / 16; ++ks)
            mma_bf16(tbase, smem_desc(smem_u32(sA + ks * 128 * 32)), smem_desc(smem_u32(sB + ks * N * 32)), idesc,
                     ks > 0 ? 1u : 0u);
        mma_commit(bar);
    }
    const bool ok = mbar_wait_all(bar, 0, 0, 128);
    fence_after_sync();
    if (!ok) {
        if (tid == 0) atomicOr(err, 1u);
    } else {
        for (int c0 = 0; c0 < N; c0 += 16) {
            float v[16];
            tmem_ld16(tbase + ((uint32_t)(warp * 32) << 16) + (uint32_t)c0, v);
#pragma unroll
            for (int i = 0; i < 16; ++i) C[(long long)tid * N + c0 + i] = v[i];
        }
    }
    fence_before_sync();
    __syncthreads();
    if (warp == 0) tmem_dealloc(tbase, ncols);
}

// Training forward: X [M x 16] BF16 normalised inputs (row-major) -> Y [M x 16]
// FP32, stashing Z_l, H_l (l = 1..4) as [4][M/128][128 x 128] blocks; NG tiles in
// flight per CTA, 4 / NG warpgroups per tile (the first stages the inputs and
// writes Y).
template <int NG>
__global__ void __launch_bounds__(MLP_THREADS) k_mlp_forward(MlpNet net, const uint16_t* __restrict__ X, float* Y,
                                                             float* Z, uint16_t* H, int ntile, unsigned* err) {
    extern __shared__ __align__(1024) unsigned char sm[];
    constexpr int G = 4 / NG, GT = 128 * G;
    const int tid = threadIdx.x, warp = tid >> 5, group = tid / GT, gt = tid % GT;
    uint64_t* bar = reinterpret_cast<uint64_t*>(sm + S_BAR) + group;
    uint32_t* tslot = reinterpret_cast<uint32_t*>(sm + S_TSLOT);
    unsigned char* a0 = sm + s_a0(group);
    mlp_stage_weights(net, sm);
    if (gt == 0) mbar_init(bar, 1);
    if (warp == 0) {
        tmem_alloc(tslot, 128 * NG);
        tmem_relinquish();
    }
    fence_before_sync();
    __syncthreads();
    fence_after_sync();
    const uint32_t tbase = *tslot;
    uint32_t phase = 0;
    bool ok = true;
    for (int t = blockIdx.x + gridDim.x * group; t < ntile && ok; t += gridDim.x * NG) {
        const long long row = (long long)t * 128 + gt;
        if (gt < 128) {
            // one row of 16 BF16 inputs: two 16-byte core-matrix rows
            const uint4* xr = reinterpret_cast<const uint4*>(X + row * 16);
            *reinterpret_cast<uint4*>(a0 + kmajor_offset(gt, 0, 128)) = xr[0];
            *reinterpret_cast<uint4*>(a0 + kmajor_offset(gt, 8, 128)) = xr[1];
        }
        float out[16];
        // stash layout: block t of layer l at ((l * ntile + t) * 128 + row) * 128
        ok = mlp_tile<G>(net.late, sm, a0, group, gt, tbase + 128 * group, bar, phase, out,
                         Z ? Z + (long long)t * 128 * 128 : nullptr, H ? H + (long long)t * 128 * 128 : nullptr,
                         (long long)ntile * 128);
        if (ok && gt < 128)
#pragma unroll
            for (int i = 0; i < 16; i += 4)
                *reinterpret_cast<float4*>(Y + row * 16 + i) = make_float4(out[i], out[i + 1], out[i + 2], out[i + 3]);
    }
    if (!ok && gt == 0) atomicOr(err, 1u);
    fence_before_sync();
    __syncthreads();
    if (warp == 0) tmem_dealloc(tbase, 128 * NG);
}

__device__ __forceinline__ float gelu_grad(float z) {
    return 0.5f * (1.0f + erff(z * 0.70710678118654752f)) + z * 0.39894228040143268f * expf(-0.5f * z * z);
}

// pack normalised FP32 features [M x 12] into the BF16 input operand rows [M x 16]
__global__ void k_mlp_pack(const float* __restrict__ X, uint16_t* Xb, long long M) {
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < M * 16;
         e += (long long)gridDim.x * blockDim.x) {
        const long long m = e >> 4;
        const int k = (int)(e & 15);
        Xb[e] = k < MLP_IN ? bf16_bits(X[m * MLP_IN + k]) : (uint16_t)0;
    }
}

// Backward pass of the activations, one 128-row tile through all layers (the tile
// routine's mirror image): the output gradient dZ_4 = dloss / dY of loss = mean over
// rows and the 10 outputs of (Y - T)^2, then for l = 4..1 the product dZ_l W_l on the
// tensor cores (A = dZ_l 128 x N_l, B(j, n) = W_l[n][j]) times gelu'(Z_{l-1}) in the
// epilogue, which stores dZ_{l-1} in FP32 in place of Z_{l-1} (nothing reads that any
// more) for the weight gradients and, as BF16, as the next product's A operand.  The
// transposed weights of all four layers (100 KB) are staged once per CTA; four
// warpgroups share a tile's epilogue by columns, which bounds it (erf, exp).  A training step's batch of 8192 rows: four launches of one
// warpgroup per tile, each staging its weights element by element, 164 us, this one
// 36 us.
// lossp[block] = the block's share of the sum of squares.
constexpr int SD_W = 0;                                 // W_1^T .. W_3^T, then W_4^T (128 x 16)
constexpr int SD_A = 3 * 128 * 128 * 2 + 128 * 16 * 2;  // dZ_l, BF16
constexpr int SD_BAR = SD_A + 128 * 128 * 2, SD_RED = SD_BAR + 16, SD_TOT = SD_RED + 4 * 4;
__host__ __device__ constexpr int sd_w(int l) { return SD_W + (l - 1) * 128 * 128 * 2; }

__global__ void __launch_bounds__(MLP_THREADS) k_mlp_bwd(int late, const uint16_t* __restrict__ Wt,
                                                         const float* __restrict__ Y, const float* __restrict__ T,
                                                         float* Z, float* dZ4, float* lossp, int ntile, unsigned* err) {
    extern __shared__ __align__(1024) unsigned char sm[];
    uint64_t* bar = reinterpret_cast<uint64_t*>(sm + SD_BAR);
    uint32_t* tslot = reinterpret_cast<uint32_t*>(sm + SD_BAR + 8);
    float* red = reinterpret_cast<float*>(sm + SD_RED);
    const int tid = threadIdx.x, warp = tid >> 5, lrow = tid & 127, cg = tid >> 7;
    for (int l = 1; l < 5; ++l) {
        const int N = LN(l);  // K extent of the product (this layer's outputs)
        const uint16_t* src = Wt + WOFF(l);
        for (int q = tid; q < 128 * N / 8; q += MLP_THREADS) {
            const int j = q / (N / 8), n = (q % (N / 8)) * 8;
            *reinterpret_cast<uint4*>(sm + sd_w(l) + kmajor_offset(j, n, 128)) =
                __ldg(reinterpret_cast<const uint4*>(src + (long long)j * N + n));
        }
    }
    if (tid == 0) mbar_init(bar, 1);
    if (warp == 0) {
        tmem_alloc(tslot, 128);
        tmem_relinquish();
    }
    fence_before_sync();
    __syncthreads();
    fence_after_sync();
    const uint32_t tbase = *tslot;
    const uint32_t trow = tbase + ((uint32_t)((warp & 3) * 32) << 16);
    const long long M = (long long)ntile * 128;
    const float scale = 2.0f / (float)(M * MLP_OUT);
    uint32_t phase = 0;
    bool ok = true;
    float acc = 0.0f;
    for (int t = blockIdx.x; t < ntile && ok; t += gridDim.x) {
        const long long row = (long long)t * 128 + lrow;
        if (tid < 128) {
            float g[16];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const float4 y = *reinterpret_cast<const float4*>(Y + row * 16 + 4 * q);
                g[4 * q] = y.x;
                g[4 * q + 1] = y.y;
                g[4 * q + 2] = y.z;
                g[4 * q + 3] = y.w;
            }
#pragma unroll
            for (int j = 0; j < 16; ++j) {
                if (j < MLP_OUT) {
                    const float d = g[j] - T[row * MLP_OUT + j];
                    acc += d * d;
                    g[j] = scale * d;
                } else {
                    g[j] = 0.0f;
                }
            }
#pragma unroll
            for (int q = 0; q < 4; ++q)
                *reinterpret_cast<float4*>(dZ4 + row * 16 + 4 * q) =
                    make_float4(g[4 * q], g[4 * q + 1], g[4 * q + 2], g[4 * q + 3]);
#pragma unroll
            for (int q = 0; q < 16; q += 8)
                *reinterpret_cast<uint4*>(sm + SD_A + kmajor_offset(lrow, q, 128)) =
                    make_uint4(bf16x2_bits(g[q], g[q + 1]), bf16x2_bits(g[q + 2], g[q + 3]),
                               bf16x2_bits(g[q + 4], g[q + 5]), bf16x2_bits(g[q + 6], g[q + 7]));
        }
        for (int l = 4; l >= 1; --l) {
            fence_async_smem();
            fence_before_sync();
            __syncthreads();
            fence_after_sync();
            if (tid == 0) {
                const uint32_t idesc = idesc_bf16_f32(128, 128);
                for (int ks = 0; ks < LN(l) / 16; ++ks)
                    mma_bf16(tbase, smem_desc(smem_u32(sm + SD_A + ks * 128 * 32)),
                             smem_desc(smem_u32(sm + sd_w(l) + ks * 128 * 32)), idesc, ks > 0 ? 1u : 0u);
                mma_commit(bar);
            }
            ok = mbar_wait_all(bar, phase, 0, MLP_THREADS, mlp_wait_limit(late));
            phase ^= 1u;
            fence_after_sync();
            if (!ok) break;
            const long long q0 = (long long)(l - 1) * M * 128 + row * 128 + cg * 32;
            float z[32], v[32];  // all of the row's Z before its first store
#pragma unroll
            for (int c = 0; c < 32; c += 4) {
                const float4 q = *reinterpret_cast<const float4*>(Z + q0 + c);
                z[c] = q.x;
                z[c + 1] = q.y;
                z[c + 2] = q.z;
                z[c + 3] = q.w;
            }
            tmem_ld32(trow + (uint32_t)(cg * 32), v);
#pragma unroll
            for (int c = 0; c < 32; c += 8) {
#pragma unroll
                for (int i = 0; i < 8; ++i) v[c + i] *= gelu_grad(z[c + i]);
                *reinterpret_cast<float4*>(Z + q0 + c) = make_float4(v[c], v[c + 1], v[c + 2], v[c + 3]);
                *reinterpret_cast<float4*>(Z + q0 + c + 4) = make_float4(v[c + 4], v[c + 5], v[c + 6], v[c + 7]);
                if (l > 1)
                    *reinterpret_cast<uint4*>(sm + SD_A + kmajor_offset(lrow, cg * 32 + c, 128)) =
                        make_uint4(bf16x2_bits(v[c], v[c + 1]), bf16x2_bits(v[c + 2], v[c + 3]),
                                   bf16x2_bits(v[c + 4], v[c + 5]), bf16x2_bits(v[c + 6], v[c + 7]));
            }
        }
        fence_before_sync();
        __syncthreads();
    }
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if (tid < 128 && (tid & 31) == 0) red[warp] = acc;
    if (!ok && tid == 0) atomicOr(err, 1u);
    fence_before_sync();
    __syncthreads();
    if (tid == 0) lossp[blockIdx.x] = red[0] + red[1] + red[2] + red[3];
    if (warp == 0) tmem_dealloc(tbase, 128);
}

// Weight and bias gradients of layer blockIdx.y over one chunk of 128 rows (block x):
// dW_l[n][k] = sum_m dZ_l[m][n] A_l[m][k], db_l[n] = sum_m dZ_l[m][n], as
// partials partW[c][.], partb[c][.].  The tensor-core M dimension (128 rows)
// is n for l < 4 and k for l = 4 (whose N_l = 16); the MMA K dimension is the
// chunk's rows, so both operands are the transposes of row-major arrays: a thread
// gathers two columns of eight rows (coalesced across the warp's columns) into two
// 16-byte core-matrix rows.  64 KB of operands, three CTAs per SM; all five layers
// in one launch (8192 rows: 320 CTAs, 20 us; five launches of 32 CTAs gathering
// element by element took 231 us).
constexpr int CHUNK = 128;       // rows per weight-gradient block
constexpr int BATCH_ROWS = 256;  // training batches are multiples of this
constexpr int WG_THREADS = 256;
constexpr int SW_A = 0, SW_B = 128 * CHUNK * 2, SW_RED = 2 * 128 * CHUNK * 2, SW_BAR = SW_RED + 4 * 128 * 4,
              SW_TOT = SW_BAR + 16;

// columns of src [rows m0.. x ld] as a K-major operand of `ncol` rows; FP32 sources
// also leave the sums of their columns over the chunk in red[4][ncol]
__device__ __forceinline__ void stage_columns(unsigned char* dst, const float* __restrict__ src, int ncol, float* red) {
    const int np = ncol / 2;
    for (int it = threadIdx.x; it < np * 4; it += WG_THREADS) {
        const int p = it % np, g = it / np;  // column pair, quarter of the rows
        float s0 = 0.0f, s1 = 0.0f;
#pragma unroll
        for (int o = 0; o < CHUNK / 32; ++o) {
            const int mm = (g * (CHUNK / 32) + o) * 8;
            float2 v[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) v[i] = *reinterpret_cast<const float2*>(src + (long long)(mm + i) * ncol + 2 * p);
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                s0 += v[i].x;
                s1 += v[i].y;
            }
            *reinterpret_cast<uint4*>(dst + kmajor_offset(2 * p, mm, ncol)) =
                make_uint4(bf16x2_bits(v[0].x, v[1].x), bf16x2_bits(v[2].x, v[3].x), bf16x2_bits(v[4].x, v[5].x),
                           bf16x2_bits(v[6].x, v[7].x));
            *reinterpret_cast<uint4*>(dst + kmajor_offset(2 * p + 1, mm, ncol)) =
                make_uint4(bf16x2_bits(v[0].y, v[1].y), bf16x2_bits(v[2].y, v[3].y), bf16x2_bits(v[4].y, v[5].y),
                           bf16x2_bits(v[6].y, v[7].y));
        }
        red[g * ncol + 2 * p] = s0;
        red[g * ncol + 2 * p + 1] = s1;
    }
}
__device__ __forceinline__ void stage_columns(unsigned char* dst, const uint16_t* __restrict__ src, int ncol) {
    const int np = ncol / 2;
    for (int it = threadIdx.x; it < np * (CHUNK / 8); it += WG_THREADS) {
        const int p = it % np, mm = it / np * 8;
        uint32_t v[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) v[i] = *reinterpret_cast<const uint32_t*>(src + (long long)(mm + i) * ncol + 2 * p);
        uint4 lo, hi;
        lo.x = __byte_perm(v[0], v[1], 0x5410);
        lo.y = __byte_perm(v[2], v[3], 0x5410);
        lo.z = __byte_perm(v[4], v[5], 0x5410);
        lo.w = __byte_perm(v[6], v[7], 0x5410);
        hi.x = __byte_perm(v[0], v[1], 0x7632);
        hi.y = __byte_perm(v[2], v[3], 0x7632);
        hi.z = __byte_perm(v[4], v[5], 0x7632);
        hi.w = __byte_perm(v[6], v[7], 0x7632);
        *reinterpret_cast<uint4*>(dst + kmajor_offset(2 * p, mm, ncol)) = lo;
        *reinterpret_cast<uint4*>(dst + kmajor_offset(2 * p + 1, mm, ncol)) = hi;
    }
}

__global__ void __launch_bounds__(WG_THREADS) k_mlp_bwd_weight(int late, const float* __restrict__ dZ4,
                                                               const float* __restrict__ dZ,
                                                               const uint16_t* __restrict__ Xb,
                                                               const uint16_t* __restrict__ H, long long M, float* partW,
                                                               float* partb, unsigned* err) {
    extern __shared__ __align__(1024) unsigned char sm[];
    uint64_t* bar = reinterpret_cast<uint64_t*>(sm + SW_BAR);
    uint32_t* tslot = reinterpret_cast<uint32_t*>(sm + SW_BAR + 8);
    float* red = reinterpret_cast<float*>(sm + SW_RED);
    const int tid = threadIdx.x, warp = tid >> 5, l = blockIdx.y;
    const int N = LN(l), K = LK(l);
    const long long m0 = (long long)blockIdx.x * CHUNK;
    const bool swap = (l == 4);
    const int ncol = swap ? N : K;  // columns of D
    const float* dz = (l == 4 ? dZ4 : dZ + (long long)l * M * 128) + m0 * N;
    const uint16_t* in = (l == 0 ? Xb : H + (long long)(l - 1) * M * 128) + m0 * K;
    stage_columns(sm + (swap ? SW_B : SW_A), dz, N, red);
    stage_columns(sm + (swap ? SW_A : SW_B), in, K);
    if (tid == 0) mbar_init(bar, 1);
    if (warp == 0) {
        tmem_alloc(tslot, 128);
        tmem_relinquish();
    }
    fence_async_smem();
    fence_before_sync();
    __syncthreads();
    fence_after_sync();
    const uint32_t tbase = *tslot;
    if (tid == 0) {
        const uint32_t idesc = idesc_bf16_f32(128, ncol);
        for (int ks = 0; ks < CHUNK / 16; ++ks)
            mma_bf16(tbase, smem_desc(smem_u32(sm + SW_A + ks * 128 * 32)),
                     smem_desc(smem_u32(sm + SW_B + ks * ncol * 32)), idesc, ks > 0 ? 1u : 0u);
        mma_commit(bar);
    }
    if (tid < N)
        partb[(long long)blockIdx.x * BTOT + BOFF(l) + tid] =
            (red[tid] + red[N + tid]) + (red[2 * N + tid] + red[3 * N + tid]);
    const bool ok = mbar_wait_all(bar, 0, 0, WG_THREADS, mlp_wait_limit(late));
    fence_after_sync();
    if (!ok) {
        if (tid == 0) atomicOr(err, 1u);
    } else {
        float* pw = partW + (long long)blockIdx.x * WTOT + WOFF(l);
        const int r = (warp & 3) * 32 + (tid & 31);
        for (int c0 = (warp >> 2) * 16; c0 < ncol; c0 += 32) {
            float v[16];
            tmem_ld16(tbase + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)c0, v);
            // row r, columns c0.. of D
            if (swap) {
#pragma unroll
                for (int i = 0; i < 16; ++i) pw[(c0 + i) * K + r] = v[i];  // D[k][n] -> W[n][k]
            } else {
#pragma unroll
                for (int i = 0; i < 16; i += 4)  // D[n][k]
                    *reinterpret_cast<float4*>(pw + r * K + c0 + i) = make_float4(v[i], v[i + 1], v[i + 2], v[i + 3]);
            }
        }
    }
    fence_before_sync();
    __syncthreads();
    if (warp == 0) tmem_dealloc(tbase, 128);
}

// element of W_1^T .. W_4^T (each N_l contiguous per input) of weight element q
__device__ __forceinline__ int transposed_index(int q) {
    const int l = q < WOFF(2) ? 1 : (q < WOFF(3) ? 2 : (q < WOFF(4) ? 3 : 4));
    const int r = q - WOFF(l), N = LN(l);
    return WOFF(l) + (r % 128) * N + r / 128;
}

// gradients = sum of the chunk partials in chunk order; Adam step on the FP32
// master parameters (bias-corrected, Kingma & Ba 2015); BF16 copy of the weights
__global__ void k_mlp_reduce_adam(const float* __restrict__ partW, const float* __restrict__ partb, int nchunk,
                                  float* W32, float* b32, float* mW, float* vW, float* mb, float* vb, uint16_t* Wb, uint16_t* Wt,
                                  float* gW, float* gb, float lr, float c1, float c2, int update) {
    const float beta1 = 0.9f, beta2 = 0.999f, eps = 1e-8f;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < WTOT + BTOT; i += gridDim.x * blockDim.x) {
        const bool isw = i < WTOT;
        const int q = isw ? i : i - WTOT;
        const float* part = isw ? partW : partb;
        const int stride = isw ? WTOT : BTOT;
        float g = 0.0f;
#pragma unroll 8
        for (int c = 0; c < nchunk; ++c) g += part[(long long)c * stride + q];
        if (gW && isw) gW[q] = g;
        if (gb && !isw) gb[q] = g;
        if (!update) continue;
        float* p = isw ? W32 + q : b32 + q;
        float* m = isw ? mW + q : mb + q;
        float* v = isw ? vW + q : vb + q;
        *m = beta1 * *m + (1.0f - beta1) * g;
        *v = beta2 * *v + (1.0f - beta2) * g * g;
        *p -= lr * (*m * c1) / (sqrtf(*v * c2) + eps);
        if (isw) {
            Wb[q] = bf16_bits(*p);
            if (q >= WOFF(1)) Wt[transposed_index(q)] = Wb[q];
        }
    }
}

__global__ void k_mlp_to_bf16(const float* W32, uint16_t* Wb, uint16_t* Wt) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < WTOT; i += gridDim.x * blockDim.x) {
        Wb[i] = bf16_bits(W32[i]);
        if (i >= WOFF(1)) Wt[transposed_index(i)] = Wb[i];
    }
}

}  // namespace ocfd

// ------------------------------------------------------------------ the object
struct ocfd_mlp {
    ocfd_context* ctx = nullptr;
    int max_batch = 0;
    float *W32 = nullptr, *b32 = nullptr, *mW = nullptr, *vW = nullptr, *mb = nullptr, *vb = nullptr;
    uint16_t* Wb = nullptr;
    uint16_t* Wt = nullptr;  // W_1 .. W_4 transposed, at the offsets of Wb
    float norm[2 * ocfd::MLP_IN + 3 * ocfd::MLP_OUT] = {};
    long long steps = 0;
    int late = -1;  // MlpNet::late
    // training scratch (max_batch rows)
    uint16_t* Xb = nullptr;
    float* Y = nullptr;
    float* Z = nullptr;      // 4 x M x 128: pre-activations, then their gradients
    uint16_t* H = nullptr;   // 4 x M x 128
    float* dZ4 = nullptr;    // M x 16
    float* partW = nullptr;  // nchunk x WTOT
    float* partb = nullptr;  // nchunk x BTOT
    float* lossp = nullptr;
    float* gW = nullptr;
    float* gb = nullptr;
    // pinned host copies of a step's results: loss partials, error word, gradients
    float* host = nullptr;
};
constexpr int HOST_LOSS = 1024, HOST_ERR = HOST_LOSS, HOST_GW = HOST_LOSS + 16, HOST_GB = HOST_GW + ocfd::WTOT,
              HOST_TOT = HOST_GB + ocfd::BTOT;

namespace ocfd {

MlpNet mlp_net(const ocfd_mlp* n);
static MlpNet net_of(const ocfd_mlp* n) { return mlp_net(n); }
MlpNet mlp_net(const ocfd_mlp* n) {
    MlpNet d{};
    d.late = n->late;
    d.W = n->Wb;
    d.b = n->b32;
    for (int i = 0; i < MLP_IN; ++i) {
        d.in_mu[i] = n->norm[i];
        d.in_isd[i] = n->norm[MLP_IN + i];
    }
    for (int i = 0; i < MLP_OUT; ++i) {
        d.out_mu[i] = n->norm[2 * MLP_IN + i];
        d.out_sd[i] = n->norm[2 * MLP_IN + MLP_OUT + i];
        d.out_scale[i] = n->norm[2 * MLP_IN + 2 * MLP_OUT + i];
    }
    return d;
}

static ocfd_status mlp_configure() {
    static bool done = false;
    if (done) return OCFD_OK;
    if (cudaFuncSetAttribute(k_mlp_forward<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, s_tot(1)) != cudaSuccess ||
        cudaFuncSetAttribute(k_mlp_forward<2>, cudaFuncAttributeMaxDynamicSharedMemorySize, s_tot(2)) != cudaSuccess ||
        cudaFuncSetAttribute(k_mlp_bwd, cudaFuncAttributeMaxDynamicSharedMemorySize, SD_TOT) != cudaSuccess ||
        cudaFuncSetAttribute(k_mlp_bwd_weight, cudaFuncAttributeMaxDynamicSharedMemorySize, SW_TOT) != cudaSuccess)
        return check_launch("MLP kernel attributes");
    done = true;
    return OCFD_OK;
}

// forward (+ stash) over M rows of normalised FP32 features
static ocfd_status mlp_forward(ocfd_mlp* n, const float* X, long long M, cudaStream_t st) {
    const int sms = n->ctx->num_sms;
    k_mlp_pack<<<grid_for(M * 16, 256, sms), 256, 0, st>>>(X, n->Xb, M);
    const int ntile = (int)(M / 128);
    if (mlp_groups(ntile, sms) == 2)
        k_mlp_forward<2><<<sms, MLP_THREADS, s_tot(2), st>>>(net_of(n), n->Xb, n->Y, n->Z, n->H, ntile, n->ctx->d_error);
    else
        k_mlp_forward<1><<<ntile, MLP_THREADS, s_tot(1), st>>>(net_of(n), n->Xb, n->Y, n->Z, n->H, ntile,
                                                               n->ctx->d_error);
    return check_launch("MLP forward");
}

// `nblk` receives the number of partial sums in lossp
static ocfd_status mlp_backward(ocfd_mlp* n, const float* T, long long M, cudaStream_t st, int& nblk) {
    const int ntile = (int)(M / 128);
    nblk = std::min(ntile, n->ctx->num_sms);
    k_mlp_bwd<<<nblk, MLP_THREADS, SD_TOT, st>>>(n->late, n->Wt, n->Y, T, n->Z, n->dZ4, n->lossp, ntile,
                                                 n->ctx->d_error);
    k_mlp_bwd_weight<<<dim3((unsigned)(M / CHUNK), 5), WG_THREADS, SW_TOT, st>>>(n->late, n->dZ4, n->Z, n->Xb, n->H, M,
                                                                              n->partW, n->partb, n->ctx->d_error);
    return check_launch("MLP backward");
}

}  // namespace ocfd

using namespace ocfd;

extern "C" {

ocfd_status ocfd_mlp_create(ocfd_context* ctx, int32_t max_batch, uint64_t seed, ocfd_mlp** out) {
    if (!ctx || !out || max_batch < BATCH_ROWS || max_batch % BATCH_ROWS)
        return fail(OCFD_BAD_ARG, "ocfd_mlp_create: max_batch must be a positive multiple of 256");
    *out = nullptr;
    ocfd_status s = mlp_configure();
    if (s != OCFD_OK) return s;
    ocfd_mlp* n = new ocfd_mlp();
    n->ctx = ctx;
    n->max_batch = max_batch;
    const long long M = max_batch, nchunk = M / CHUNK;
    bool ok = true;
    auto al = [&](void** p, size_t bytes) {
        if (cudaMalloc(p, bytes) != cudaSuccess) ok = false;
        else cudaMemset(*p, 0, bytes);
    };
    al((void**)&n->W32, 4 * WTOT);
    al((void**)&n->b32, 4 * BTOT);
    al((void**)&n->mW, 4 * WTOT);
    al((void**)&n->vW, 4 * WTOT);
    al((void**)&n->mb, 4 * BTOT);
    al((void**)&n->vb, 4 * BTOT);
    al((void**)&n->Wb, 2 * WTOT);
    al((void**)&n->Wt, 2 * WTOT);
    al((void**)&n->Xb, 2 * M * 16);
    al((void**)&n->Y, 4 * M * 16);
    al((void**)&n->Z, 4 * 4 * M * 128);
    al((void**)&n->H, 2 * 4 * M * 128);
    al((void**)&n->dZ4, 4 * M * 16);
    al((void**)&n->partW, 4 * nchunk * WTOT);
    al((void**)&n->partb, 4 * nchunk * BTOT);
    al((void**)&n->lossp, 4 * 1024);
    al((void**)&n->gW, 4 * WTOT);
    al((void**)&n->gb, 4 * BTOT);
    if (cudaHostAlloc((void**)&n->host, sizeof(float) * HOST_TOT, cudaHostAllocDefault) != cudaSuccess) ok = false;
    if (!ok) {
        cudaGetLastError();
        ocfd_mlp_destroy(n);
        return fail(OCFD_OUT_OF_MEMORY, "ocfd_mlp_create");
    }
    // He-normal initial weights (Box-Muller on a 64-bit LCG), zero biases and padding
    std::vector<float> W(WTOT, 0.0f);
    uint64_t x = seed * 6364136223846793005ull + 1442695040888963407ull;
    auto uni = [&]() {
        x = x * 6364136223846793005ull + 1442695040888963407ull;
        return ((x >> 11) + 0.5) * (1.0 / 9007199254740992.0);
    };
    for (int l = 0; l < 5; ++l) {
        const int N = LN(l), K = LK(l);
        const int kin = (l == 0) ? MLP_IN : K, nout = (l == 4) ? MLP_OUT : N;
        const double sd = std::sqrt(2.0 / kin);
        for (int i = 0; i < nout; ++i)
            for (int j = 0; j < kin; ++j) {
                const double u1 = uni(), u2 = uni();
                W[WOFF(l) + i * K + j] = (float)(sd * std::sqrt(-2.0 * std::log(u1)) * std::cos(6.283185307179586 * u2));
            }
    }
    for (int i = 0; i < MLP_IN; ++i) n->norm[MLP_IN + i] = 1.0f;
    for (int i = 0; i < MLP_OUT; ++i) n->norm[2 * MLP_IN + MLP_OUT + i] = 1.0f;
    cudaMemcpy(n->W32, W.data(), 4 * WTOT, cudaMemcpyHostToDevice);
    k_mlp_to_bf16<<<64, 256>>>(n->W32, n->Wb, n->Wt);
    s = check_launch("ocfd_mlp_create");
    if (s == OCFD_OK && cudaDeviceSynchronize() != cudaSuccess) s = check_launch("ocfd_mlp_create");
    if (s != OCFD_OK) {
        ocfd_mlp_destroy(n);
        return s;
    }
    *out = n;
    return OCFD_OK;
}

ocfd_status ocfd_mlp_destroy(ocfd_mlp* n) {
    if (!n) return OCFD_OK;
    void* ps[] = {n->W32, n->b32, n->mW, n->vW, n->mb, n->vb, n->Wb, n->Wt, n->Xb, n->Y, n->Z, n->H, n->dZ4,
                  n->partW, n->partb, n->lossp, n->gW, n->gb};
    for (void* p : ps) cudaFree(p);
    if (n->host) cudaFreeHost(n->host);
    delete n;
    return OCFD_OK;
}

ocfd_status ocfd_mlp_set_norm(ocfd_mlp* n, const float* in_mu, const float* in_isd, const float* out_mu,
                              const float* out_sd) {
    if (!n || !in_mu || !in_isd || !out_mu || !out_sd) return fail(OCFD_BAD_ARG, "ocfd_mlp_set_norm");
    for (int i = 0; i < MLP_IN; ++i) {
        n->norm[i] = in_mu[i];
        n->norm[MLP_IN + i] = in_isd[i];
    }
    for (int i = 0; i < MLP_OUT; ++i) {
        n->norm[2 * MLP_IN + i] = out_mu[i];
        n->norm[2 * MLP_IN + MLP_OUT + i] = out_sd[i];
    }
    return OCFD_OK;
}

ocfd_status ocfd_mlp_set_target_scale(ocfd_mlp* n, const float* scale) {
    if (!n || !scale) return fail(OCFD_BAD_ARG, "ocfd_mlp_set_target_scale");
    for (int i = 0; i < MLP_OUT; ++i) n->norm[2 * MLP_IN + 2 * MLP_OUT + i] = scale[i];
    return OCFD_OK;
}

ocfd_status ocfd_mlp_get_params(ocfd_mlp* n, float* W, float* b) {
    if (!n) return fail(OCFD_BAD_ARG, "ocfd_mlp_get_params");
    if ((W && cudaMemcpy(W, n->W32, 4 * WTOT, cudaMemcpyDeviceToHost) != cudaSuccess) ||
        (b && cudaMemcpy(b, n->b32, 4 * BTOT, cudaMemcpyDeviceToHost) != cudaSuccess))
        return check_launch("ocfd_mlp_get_params");
    return OCFD_OK;
}

ocfd_status ocfd_mlp_set_params(ocfd_mlp* n, const float* W, const float* b) {
    if (!n) return fail(OCFD_BAD_ARG, "ocfd_mlp_set_params");
    if ((W && cudaMemcpy(n->W32, W, 4 * WTOT, cudaMemcpyHostToDevice) != cudaSuccess) ||
        (b && cudaMemcpy(n->b32, b, 4 * BTOT, cudaMemcpyHostToDevice) != cudaSuccess))
        return check_launch("ocfd_mlp_set_params");
    k_mlp_to_bf16<<<64, 256>>>(n->W32, n->Wb, n->Wt);
    return check_launch("ocfd_mlp_set_params");
}

static ocfd_status mlp_check_error(ocfd_mlp* n, cudaStream_t st, const char* who) {
    uint32_t e = 0;
    if (cudaMemcpyAsync(&e, n->ctx->d_error, sizeof(e), cudaMemcpyDeviceToHost, st) != cudaSuccess ||
        cudaStreamSynchronize(st) != cudaSuccess)
        return check_launch(who);
    if (e) {
        cudaMemsetAsync(n->ctx->d_error, 0, sizeof(uint32_t), st);
        return fail(OCFD_TIMEOUT, std::string(who) + ": a tensor-core completion wait ran out");
    }
    return OCFD_OK;
}

ocfd_status ocfd_check_mlp_late_thread(ocfd_mlp* n, int32_t thread) {
    if (!n || thread < -1 || thread >= MLP_THREADS) return fail(OCFD_BAD_ARG, "ocfd_check_mlp_late_thread");
    n->late = thread;
    return OCFD_OK;
}

// Y [M x 10] = network(X [M x 12]) in normalised units (device arrays)
ocfd_status ocfd_mlp_forward(ocfd_mlp* n, const float* X, float* Y, int64_t M, void* stream) {
    if (!n || !X || !Y || M <= 0 || M % 128 || M > n->max_batch) return fail(OCFD_BAD_ARG, "ocfd_mlp_forward: M");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    ocfd_status s = mlp_forward(n, X, M, st);
    if (s != OCFD_OK) return s;
    if (cudaMemcpy2DAsync(Y, sizeof(float) * MLP_OUT, n->Y, sizeof(float) * 16, sizeof(float) * MLP_OUT, (size_t)M,
                          cudaMemcpyDeviceToDevice, st) != cudaSuccess)
        return check_launch("ocfd_mlp_forward");
    return mlp_check_error(n, st, "ocfd_mlp_forward");
}

// One training step on (X [M x 12], T [M x 10]) normalised device arrays:
// forward, MSE loss, backward, Adam (lr).  update = 0 computes the gradients
// only (gW [WTOT], gb [BTOT] on the host when given).  loss: host scalar.
ocfd_status ocfd_mlp_train_step(ocfd_mlp* n, const float* X, const float* T, int64_t M, float lr, int32_t update,
                                float* loss, float* gW, float* gb, void* stream) {
    if (!n || !X || !T || M <= 0 || M % BATCH_ROWS || M > n->max_batch)
        return fail(OCFD_BAD_ARG, "ocfd_mlp_train_step: M must be a multiple of 256 up to max_batch");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    ocfd_status s = mlp_forward(n, X, M, st);
    if (s != OCFD_OK) return s;
    int nblk = 0;
    s = mlp_backward(n, T, M, st, nblk);
    if (s != OCFD_OK) return s;
    if (update) ++n->steps;
    const float c1 = update ? (float)(1.0 / (1.0 - std::pow(0.9, (double)n->steps))) : 1.0f;
    const float c2 = update ? (float)(1.0 / (1.0 - std::pow(0.999, (double)n->steps))) : 1.0f;
    k_mlp_reduce_adam<<<grid_for(WTOT + BTOT, 256, n->ctx->num_sms), 256, 0, st>>>(
        n->partW, n->partb, (int)(M / CHUNK), n->W32, n->b32, n->mW, n->vW, n->mb, n->vb, n->Wb, n->Wt, n->gW, n->gb, lr, c1,
        c2, update);
    s = check_launch("ocfd_mlp_train_step");
    if (s != OCFD_OK) return s;
    // one wait for everything the host gets, through pinned memory (three waits and
    // pageable copies took 40 us of a step of 8192 rows)
    const auto fetch = [&](int at, const void* src, size_t words) {
        return cudaMemcpyAsync(n->host + at, src, 4 * words, cudaMemcpyDeviceToHost, st) == cudaSuccess;
    };
    if ((loss && !fetch(0, n->lossp, nblk)) || (gW && !fetch(HOST_GW, n->gW, WTOT)) ||
        (gb && !fetch(HOST_GB, n->gb, BTOT)) || !fetch(HOST_ERR, n->ctx->d_error, 1) ||
        cudaStreamSynchronize(st) != cudaSuccess)
        return check_launch("ocfd_mlp_train_step");
    uint32_t e;
    std::memcpy(&e, n->host + HOST_ERR, 4);
    if (e) {
        cudaMemsetAsync(n->ctx->d_error, 0, sizeof(uint32_t), st);
        return fail(OCFD_TIMEOUT, "ocfd_mlp_train_step: a tensor-core completion wait ran out");
    }
    if (loss) {
        double acc = 0;
        for (int i = 0; i < nblk; ++i) acc += n->host[i];
        *loss = (float)(acc / ((double)M * MLP_OUT));
    }
    if (gW) std::memcpy(gW, n->host + HOST_GW, 4 * WTOT);
    if (gb) std::memcpy(gb, n->host + HOST_GB, 4 * BTOT);
    return OCFD_OK;
}

}  // extern "C"

extern "C" ocfd_status ocfd_tc_gemm_bf16(ocfd_context* ctx, const uint16_t* A, const uint16_t* B, float* C, int N,
                                         int K, void* stream) {
    if (!ctx || !A || !B || !C || N < 16 || N > 256 || N % 16 || K < 16 || K > 256 || K % 16)
        return fail(OCFD_BAD_ARG, "ocfd_tc_gemm_bf16: N in [16, 256] and K in [16, 256], multiples of 16");
    const size_t smem = (size_t)(128 + N) * K * 2 + 16;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (cudaFuncSetAttribute(k_tc_gemm, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)
        return check_launch("ocfd_tc_gemm_bf16 attribute");
    cudaMemsetAsync(ctx->d_error, 0, sizeof(uint32_t), st);
    k_tc_gemm<<<1, 128, smem, st>>>(A, B, C, N, K, ctx->d_error);
    ocfd_status s = check_launch("ocfd_tc_gemm_bf16");
    if (s != OCFD_OK) return s;
    uint32_t e = 0;
    if (cudaMemcpyAsync(&e, ctx->d_error, sizeof(e), cudaMemcpyDeviceToHost, st) != cudaSuccess ||
        cudaStreamSynchronize(st) != cudaSuccess)
        return check_launch("ocfd_tc_gemm_bf16");
    if (e) return fail(OCFD_TIMEOUT, "ocfd_tc_gemm_bf16: the MMA completion wait ran out");
    return OCFD_OK;
}
