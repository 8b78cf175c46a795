// mlp_layout.h -- sizes, parameter layout and device buffers of the surrogate
// network, shared by the host API (mlp.cu) and its kernels (mlp_fused.cu).
#pragma once
#include <cuda_runtime.h>

#include <cstddef>
#include <cstdint>

#include "pticm_engine.h"

namespace pticm {

constexpr int MLP_IN = 7;         // features + normalised energy
constexpr int MLP_K0 = 64;        // input width padded for the tensor cores
constexpr int MLP_H = 256;        // hidden width
constexpr int MLP_LAYERS = 4;     // hidden layers
constexpr int MLP_TILE = 128;     // rows of a tile

// flat parameter layout: W1 [H x K0], b1, W2 [H x H], b2, W3, b3, W4, b4, w5 [H], b5
constexpr size_t kW1 = 0, kB1 = kW1 + (size_t)MLP_H * MLP_K0;
constexpr size_t kW2 = kB1 + MLP_H, kB2 = kW2 + (size_t)MLP_H * MLP_H;
constexpr size_t kW3 = kB2 + MLP_H, kB3 = kW3 + (size_t)MLP_H * MLP_H;
constexpr size_t kW4 = kB3 + MLP_H, kB4 = kW4 + (size_t)MLP_H * MLP_H;
constexpr size_t kW5 = kB4 + MLP_H, kB5 = kW5 + MLP_H;
constexpr size_t kParams = kB5 + 1;

// Matrices that the tensor cores read are kept as the images that shared
// memory holds: chunks of 64 K-columns, a chunk a row of 128 bytes per matrix
// row, its 16-byte units permuted by the 128-byte swizzle (unit u of row r at
// u ^ (r & 7)).  A tile's chunk is one contiguous bulk copy.
constexpr uint32_t kChunkRow = 128;                          // bytes of a row in a chunk
constexpr uint32_t kChunkH = MLP_H * kChunkRow;              // a chunk of a 256-row matrix: 32 KB

// Byte of element (row r, column k) in an image of `rows` rows.
__host__ __device__ constexpr size_t image_at(int r, long long k, int rows) {
    return (size_t)(k >> 6) * ((size_t)rows * kChunkRow) + (size_t)r * kChunkRow +
           (size_t)((((int)(k & 63) >> 3) ^ (r & 7)) << 4) + (size_t)(k & 7) * 2;
}

// Device buffers of a network and of one call (see mlp_fused.cu).  B is the
// batch (a multiple of 128); tiled arrays [c / 4][b] (float4) or [c / 8][b]
// (eight bf16) keep a row's columns apart so that a warp of rows is one
// contiguous access.
struct MlpArgs {
    const float* X;            // dataset rows [.. x 7]
    const float* Y;            // targets (training)
    const uint32_t* idx;       // ring of batches of n_valid rows (null: rows in order)
    long long* ctr;            // [0] iteration of the call, [1] Adam steps taken (null: gradients only)
    int ring;                  // batches in the ring
    int B;
    long long n_valid;         // rows of a batch (training) or of the call (prediction)
    float* P;                  // parameters, gradients, Adam moments
    float* G;
    float* Mm;
    float* Vm;
    uint8_t* Wi[MLP_LAYERS];   // images of W_l [256 x K_l] and, but for the first layer, of W_l^T [K_l x 256] (bf16)
    uint8_t* WTi[MLP_LAYERS];
    float4* Z[MLP_LAYERS];     // pre-activations, tiled
    float4* dZf[MLP_LAYERS];   // their gradients, tiled
    uint8_t* dZT[MLP_LAYERS];  // images of dZ_l^T [256 x B]
    uint8_t* HT[MLP_LAYERS];   // images of the layer inputs' transposes [K_l x B]
    uint4* H4;                 // last activations, tiled (bf16)
    float* dy;
    float* y;
    float* loss_tile;          // sum of squared errors of each tile
    float* losses;             // mean loss per iteration (training), or one value
    float lr;
    DevStatus* status;
    int* abort_flag;
};

cudaError_t mlp_images(const float* P, uint8_t* const* Wi, uint8_t* const* WTi, cudaStream_t st);
cudaError_t mlp_div(const float* a, const float* b, float* q, long long count, cudaStream_t st);
cudaError_t mlp_predict_rows(const MlpArgs& a, cudaStream_t st);
cudaError_t mlp_train_step(const MlpArgs& a, cudaStream_t st);

}  // namespace pticm
