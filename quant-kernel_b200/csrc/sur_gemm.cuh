// sur_gemm.cuh -- BF16 tensor-core GEMM for the surrogate MLP (sm_100a).
//
//   C[M x N] = A[M x K] . B[N x K]^T      A, B bf16 row-major (K contiguous)
//
// One CTA computes a 128 x BN tile over a K range (split-K over blockIdx.z):
//   * warp 0 / lane 0 loads 128x64 A and BNx64 B tiles with TMA
//     (cp.async.bulk.tensor, 128-byte swizzle) into a 4-stage ring, each stage
//     guarded by "full" and "empty" mbarriers;
//   * warp 1 / lane 0 issues tcgen05.mma (kind::f16, BF16 x BF16 -> FP32,
//     M = 128, N = BN, K = 16 per instruction) from shared-memory descriptors
//     into a TMEM accumulator, and frees a stage with tcgen05.commit;
//   * all eight warps then read the accumulator with tcgen05.ld (warp w reads
//     TMEM lanes 32 (w % 4) .. + 31 = tile rows, column half w / 4) and run the
//     fused epilogue.
// Every mbarrier wait is bounded: on timeout the kernel records an error code
// in *err, drains what it issued (again bounded), frees its TMEM and returns.
#pragma once

#include <cstdint>
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include "device_once.h"

namespace qkb {

enum : int {
    kEpiF32 = 0,    // C fp32 (split-K partial slab per blockIdx.z)
    kEpiFwd = 1,    // h = silu(acc + bias): write H (bf16)
    kEpiLast = 2,   // layer 3 + head: y = silu(acc + b3) . w4 + b4
};

struct GemmArgs {
    int M, N, K;             // problem size (K range split over gridDim.z)
    int k_per_split;         // multiple of 64
    // epilogue operands
    float* c_f32;            // kEpiF32: [gridDim.z][M][N]
    const float* bias;       // [N]
    __nv_bfloat16* h_out;    // [M][N]
    const float* w4;         // head weights [N]
    const float* b4;         // head bias [1]
    float* y_out;            // [M]
    const float* base;       // [M] added to y_out, or null
    int* err;                // error word (0 = ok)
};

// Fused MLP inference: y[i] = w4 . silu(W3 silu(W2 silu(W1 x_i + b1) + b2) + b3) + b4
// (+ base[i] when base is not null) for normalised bf16 rows x [n][64] (see
// sur_gemm.cu, mlp_infer_kernel).
struct InferArgs {
    int64_t n;               // rows
    const float* b1;         // [256]
    const float* b2;
    const float* b3;
    const float* w4;
    const float* b4;         // [1]
    const float* base;       // [n] added to the network's output, or null
    float* y;                // [n]
    int* err;                // error word (0 = ok)
};
// Lets `kernel` use `bytes` of dynamic shared memory on the current device.
template <typename... P>
cudaError_t allow_shared(DeviceOnce& once, void (*kernel)(P...), size_t bytes) {
    int dev = 0;
    const cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    return once.run(dev, [&] {
        return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    static_cast<int>(bytes));
    });
}

// Launches a kernel that may start while the previous one of the stream still
// runs: it calls griddepcontrol.wait before it touches what that one writes.
// A training step is two short kernels; with the set-up of each under the tail
// of the other, an epoch of 182 steps of 384 rows takes 8.63 ms instead of
// 9.25, one of 32 steps of 8192 rows 2.65 instead of 2.71.
template <typename... P, typename... A>
cudaError_t launch_dependent(void (*kernel)(P...), int grid, int threads, size_t smem, cudaStream_t st,
                             const A&... args) {
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(static_cast<unsigned>(grid));
    cfg.blockDim = dim3(static_cast<unsigned>(threads));
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, args...);
}

// tx: x [n][64] and tw1: W1 [256][64] read through their first 16 columns
// (make_tmap_bf16_k16: the 9 features and their zero padding; boxes 16 x 128
// and 16 x 256, 32-byte swizzle); tw2, tw3: [256][256] (boxes 64 x 256).
// ctas: persistent grid size (one CTA per SM).
cudaError_t launch_mlp_infer(const CUtensorMap& tx, const CUtensorMap& tw1, const CUtensorMap& tw2,
                             const CUtensorMap& tw3, const InferArgs& a, int ctas, cudaStream_t st);

// Fused training pass over one minibatch (mlp_train_kernel in sur_gemm.cu):
// rows perm[(step % steps_per_epoch) batch + i] of xall, forward, head, loss
// gradient, backward, and one slab of each weight gradient per 128 rows.
struct TrainMaps {
    CUtensorMap w1;            // W1 [256][64], first 16 columns, box 16 x 256
    CUtensorMap w2, w3;        // [256][256], boxes 64 x 256
    CUtensorMap w3t, w2t;      // their transposes
};
struct TrainArgs {
    const __nv_bfloat16* xall;  // rows of x_stride bf16, first 16 read
    int x_stride;
    const float* tall;
    const int32_t* perm;
    const int* step;
    const int* steps_per_epoch;
    int batch;                  // multiple of 128
    float loss_scale;           // dL/dy = loss_scale (y - target)
    const float *b1, *b2, *b3, *w4, *b4;
    // bf16 [batch / 128 tiles][32 chunks of 8 columns][128 rows]
    uint4 *z1, *z2, *h1;        // this pass's scratch
    uint4 *h3, *dz3, *dz2, *dz1;
    float *y_out, *dy_out, *target_out;  // [batch]
    // slabs [tile][2 halves of 128 rows][chunks of 4 columns][128 rows]: 4
    // chunks (the first 16 columns of W1), 64, 64
    float4 *dw1, *dw2, *dw3;
    int* err;                   // error word (0 = ok)
};
cudaError_t launch_mlp_train(const TrainMaps& maps, const TrainArgs& a, cudaStream_t st);

// Host side: tensor maps over bf16 row-major [rows][cols] (cols contiguous).
bool make_tmap_bf16(CUtensorMap* map, const void* base, uint64_t rows, uint64_t cols,
                    uint32_t box_rows);
// The same over columns 0..15 only (a 16 x box_rows box, 32-byte swizzle).
bool make_tmap_bf16_k16(CUtensorMap* map, const void* base, uint64_t rows, uint64_t cols,
                        uint32_t box_rows);
cudaError_t launch_umma_gemm(int epi, int bn, const CUtensorMap& ta, const CUtensorMap& tb,
                             const GemmArgs& a, int splits, cudaStream_t st);

}  // namespace qkb
