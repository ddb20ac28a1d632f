// The chemistry surrogate network's fused tile routine (5 layers on the tensor
// cores for 128 rows), shared by the training kernels (mlp.cu) and the solver's
// surrogate chemistry substep (chem.cu).
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

#include "ocfd/ocfd.h"
#include "tcgen05.cuh"

namespace ocfd {

using namespace tc;

__device__ __forceinline__ uint16_t bf16_bits(float x) {  // round to nearest even
    const uint32_t u = __float_as_uint(x);
    if ((u & 0x7f800000u) == 0x7f800000u) return (uint16_t)((u >> 16) | ((u & 0xffffu) ? 0x40u : 0u));
    return (uint16_t)((u + 0x7fffu + ((u >> 16) & 1u)) >> 16);
}

__host__ __device__ __forceinline__ uint32_t tmem_cols(int n) {
    uint32_t c = 32;
    while ((int)c < n) c <<= 1;
    return c;
}

// ============================================================ the network
// 12 inputs (T, p, 9 Y, log10 dt), 4 hidden layers of 128 with GELU, 10 outputs
// (increments of T and of the 9 Y).  Layer l has W_l [N_l x K_l] (out x in,
// row-major BF16) and b_l [N_l] (FP32); the input is padded to K_1 = 16 and the
// output to N_5 = 16 with zero weights.
constexpr int MLP_IN = 12, MLP_OUT = 10, MLP_H = 128;
__host__ __device__ constexpr int LN(int l) { return l == 4 ? 16 : 128; }                  // outputs of layer l
__host__ __device__ constexpr int LK(int l) { return l == 0 ? 16 : 128; }                  // inputs of layer l
__host__ __device__ constexpr int WOFF(int l) { return l == 0 ? 0 : 2048 + (l - 1) * 16384; }  // element offset of W_l
constexpr int WTOT = 53248;
__host__ __device__ constexpr int BOFF(int l) { return 128 * l; }
constexpr int BTOT = 528;
// shared memory of the fused kernel with NG tiles in flight (bytes): the weights
// and biases once, each tile's operands and completion barrier
constexpr int S_W = 0;             // the five B operands, K-major, as WOFF * 2
constexpr int S_B = WTOT * 2;      // biases, FP32
constexpr int S_BAR = S_B + BTOT * 4;  // two barriers, then the TMEM base
constexpr int S_TSLOT = S_BAR + 16;
constexpr int S_OP = (S_TSLOT + 16 + 127) / 128 * 128;
constexpr int S_A0_BYTES = 128 * 16 * 2, S_H_BYTES = 128 * 128 * 2;  // input and hidden operand of a tile
__host__ __device__ constexpr int s_a0(int g) { return S_OP + g * (S_A0_BYTES + S_H_BYTES); }
__host__ __device__ constexpr int s_tot(int ng) { return s_a0(ng); }

struct MlpNet {
    const uint16_t* W;  // BF16 weights, WTOT elements
    const float* b;     // FP32 biases, BTOT
    float in_mu[MLP_IN], in_isd[MLP_IN];     // feature normalisation: (x - mu) * isd
    float out_mu[MLP_OUT], out_sd[MLP_OUT];  // target scaling: y * sd + mu
    float out_scale[MLP_OUT];                // > 0: y is sign(r) log1p(|r| / scale) of the rate r
    int late = -1;                           // thread of every CTA that gives up its waits at once (test hook), or -1
};
// polls of this thread's completion waits
__device__ __forceinline__ uint32_t mlp_wait_limit(int late) {
    return (int)threadIdx.x == late ? 0u : tc::kWaitLimit;
}

__device__ __forceinline__ float gelu(float z) { return 0.5f * z * (1.0f + erff(z * 0.70710678118654752f)); }

// stage the weights (K-major B operands) and biases of the network
__device__ __forceinline__ void mlp_stage_weights(const MlpNet& net, unsigned char* sm) {
    for (int l = 0; l < 5; ++l) {
        const int N = LN(l), K = LK(l);
        unsigned char* dst = sm + S_W + WOFF(l) * 2;
        const uint16_t* src = net.W + WOFF(l);
        // 8 consecutive k of a row are one 16-byte core-matrix row in both layouts
        // (W and every WOFF(l) * 2 are 16-byte aligned)
        for (int q = threadIdx.x; q < N * K / 8; q += blockDim.x) {
            const int n = q / (K / 8), k = (q % (K / 8)) * 8;
            *reinterpret_cast<uint4*>(dst + kmajor_offset(n, k, N)) =
                __ldg(reinterpret_cast<const uint4*>(src + (long long)n * K + k));
        }
    }
    float* sb = reinterpret_cast<float*>(sm + S_B);
    for (int e = threadIdx.x; e < BTOT; e += blockDim.x) sb[e] = net.b[e];
}

// Threads of a CTA: 512, as NG groups of G warpgroups (128 threads each).  A group
// takes one 128-row tile through the network; the bias + GELU epilogue of a hidden
// layer (erf and BF16 packing per element) takes far longer than the layer's MMAs,
// so it is split over the group's G warpgroups by columns.  With NG = 2 the two
// tiles' waits (MMA completion, barriers, the 128-thread prologue and tail)
// overlap the other tile's epilogue; with fewer tiles than SMs one tile per CTA on
// all four warpgroups has the shorter latency.  mlp_groups() draws the line.
// Measured with one tile -> two tiles in flight and the packed BF16 conversion,
// same bits: one surrogate substep of 2^20 cells, a quarter of them falling back
// to FP64, 4.55 -> 3.63 ms (this and the cell lists no longer made for
// contiguous cells); a training step of 8192 rows (64 tiles) 528 -> 508 us, by the
// conversion (148 us with the backward pass of mlp.cu).  The training forward of
// 2^19 rows takes 1.00 ms, 54 TFLOP/s.
constexpr int MLP_THREADS = 512;
inline int mlp_groups(long long ntile, int sms) { return ntile > sms ? 2 : 1; }

// two floats to packed BF16, round to nearest even (lo in the low half)
__device__ __forceinline__ uint32_t bf16x2_bits(float lo, float hi) {
    uint32_t r;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
    return r;
}

// barrier of one group of a CTA (whole warps; id 0 is __syncthreads')
__device__ __forceinline__ void group_sync(int group, int threads) {
    asm volatile("bar.sync %0, %1;" ::"r"(group + 1), "r"(threads) : "memory");
}

// one 128-row tile through the five layers; the input operand (a0, followed by the
// hidden operand) is staged.  Called by a group's 128 G threads: thread gt serves
// row gt % 128 (warp w reads TMEM lanes 32 (w % 4) .. 32 (w % 4) + 31) and columns
// [(gt / 128) 128 / G, (gt / 128 + 1) 128 / G) of every hidden layer; the output
// layer's 16 columns go to the first warpgroup (out[]).  Hidden activations go to
// `zs` / `hs` (FP32 pre-activations, BF16 activations; may be null).  Returns
// false - to all threads of the group - when an MMA completion wait ran out.
template <int G>
__device__ __forceinline__ bool mlp_tile(int late, unsigned char* sm, unsigned char* a0, int group, int gt,
                                         uint32_t tbase, uint64_t* bar, uint32_t& phase, float* out, float* zs, uint16_t* hs,
                                         long long ld) {
    static_assert(G == 2 || G == 4, "warpgroups per tile");
    constexpr int CW = MLP_H / G;
    const int row = gt & 127, cg = gt >> 7;
    const float* sb = reinterpret_cast<const float*>(sm + S_B);
    unsigned char* h = a0 + S_A0_BYTES;
    const uint32_t trow = tbase + ((uint32_t)(((gt >> 5) & 3) * 32) << 16);
    for (int l = 0; l < 5; ++l) {
        fence_async_smem();
        fence_before_sync();
        group_sync(group, 128 * G);
        fence_after_sync();
        if (gt == 0) {
            const uint32_t idesc = idesc_bf16_f32(128, LN(l));
            const unsigned char* A = l == 0 ? a0 : h;
            const unsigned char* B = sm + S_W + WOFF(l) * 2;
            for (int ks = 0; ks < LK(l) / 16; ++ks)
                mma_bf16(tbase, smem_desc(smem_u32(A + ks * 128 * 32)), smem_desc(smem_u32(B + ks * LN(l) * 32)),
                         idesc, ks > 0 ? 1u : 0u);
            mma_commit(bar);
        }
        const bool ok = mbar_wait_all(bar, phase, group + 1, 128 * G, mlp_wait_limit(late));
        phase ^= 1u;
        fence_after_sync();
        if (!ok) return false;
        if (l < 4) {
            // bias + GELU, BF16 into the hidden operand: 8 consecutive columns of a
            // row are one 16-byte core-matrix row, stored at once
            for (int c0 = cg * CW; c0 < (cg + 1) * CW; c0 += 32) {
                float v[32];
                tmem_ld32(trow + (uint32_t)c0, v);
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    uint32_t pk[4];
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        const int i = q * 8 + e * 4;
                        const float4 b = *reinterpret_cast<const float4*>(sb + BOFF(l) + c0 + i);
                        const float4 z = make_float4(v[i] + b.x, v[i + 1] + b.y, v[i + 2] + b.z, v[i + 3] + b.w);
                        pk[2 * e] = bf16x2_bits(gelu(z.x), gelu(z.y));
                        pk[2 * e + 1] = bf16x2_bits(gelu(z.z), gelu(z.w));
                        if (zs)
                            *reinterpret_cast<float4*>(zs + (long long)l * 128 * ld + (long long)row * 128 + c0 + i) = z;
                    }
                    const uint4 w = make_uint4(pk[0], pk[1], pk[2], pk[3]);
                    *reinterpret_cast<uint4*>(h + kmajor_offset(row, c0 + q * 8, 128)) = w;
                    if (hs)
                        *reinterpret_cast<uint4*>(hs + (long long)l * 128 * ld + (long long)row * 128 + c0 + q * 8) = w;
                }
            }
        } else if (cg == 0) {
            float v[16];
            tmem_ld16(trow, v);
#pragma unroll
            for (int i = 0; i < 16; ++i) out[i] = v[i] + sb[BOFF(4) + i];
        }
    }
    return true;
}

// the device view of a network object (mlp.cu)
MlpNet mlp_net(const ocfd_mlp* n);

}  // namespace ocfd
