// Bit-exact integer GEMM for prompts, batched steps and operator products (gemm_mma.cu): weight copies and launch wrappers.
#pragma once
#include "kernels.cuh"

namespace wick {

// A second copy of a quantised matrix in the order in which the lanes of a warp take it as mma.sync operands: chunks of 16 rows x
// one block, block after block, MMA_CHUNK bytes each: 32 x 16 bytes of quants (lane (g, c) = 4g + c: for each NEON lane group one
// word with elements 2c and 2c + 1 of its eight, row g in the low half, row g + 8 in the high one) and the scales as 8 x 2 floats
// (rows g and g + 8).  Q4_0 quants are e5m2 bytes of the value (exact: -8 .. 7), Q8_0 quants the value + 128.  Rows are padded to a
// multiple of 16 and blocks to one of MMA_STAGE_BLOCKS, with zero quants and zero scales.
constexpr int MMA_ROWS = 16, MMA_CHUNK = 32 * 16 + MMA_ROWS * 4, MMA_STAGE_BLOCKS = 8;
struct MmaWeight {
    uint8_t* p = nullptr;
    int m = 0, k = 0, dtype = 0;
    int row_tiles() const { return (m + MMA_ROWS - 1) / MMA_ROWS; }
    int stages() const { return (k / QK + MMA_STAGE_BLOCKS - 1) / MMA_STAGE_BLOCKS; }
    size_t bytes() const { return (size_t)row_tiles() * stages() * MMA_STAGE_BLOCKS * MMA_CHUNK; }
};

// Up to three matrices with the same k that share one set of quantised activations (gate + up, or Q + K + V): their tiles are
// scheduled as one grid so that narrow matrices do not leave SMs idle.
struct MmaJob {
    const uint8_t* w[3];
    float* out[3];      // [n][m[i]] each
    int m[3];
    int tile_start[4];  // first linear tile of each matrix; [count..3] = total
    const uint8_t* x;   // the activations in operand order (MmaInput::p, MmaWeight::stages() stages of blocks), or null and
    const int8_t* xq;   // quantised activations [n][k]
    const float* xs;    // [n][k / 32]
    int n, k;
};

// True when the shapes meet the kernel's requirements (k a multiple of 128).
bool mma_gemm_supported(int m, int k);

// Fills the copy at `p` (MmaWeight::bytes() of device memory) from the grouped layout of `w`.
cudaError_t mma_weight_fill(cudaStream_t st, const DevWeight& w, uint8_t* p);

// out[i][j][r] for matrix i < count (<= 3, equal k), token j < n, row r < m_i (token-major, like launch_gemm), with the arithmetic of
// gemm_q*_q8_0_neon (simd.rs:696-1019) in its order, for any f32 scales.  xq: 4-byte aligned.  err: word (device or mapped host
// memory) that receives a non-zero code if a bounded wait expired.  tile (tests): a shape to take, or -1 for the rule's; receives what ran.
struct MmaTileShape {
    int index = -1, rows = 0, tokens = 0;
};
cudaError_t launch_gemm_mma(cudaStream_t st, const MmaWeight* const* w, float* const* out, int count, const uint8_t* x, const int8_t* xq, const float* xs,
                            int n, uint32_t* err, MmaTileShape* tile = nullptr);
constexpr int MMA_SHAPES = 7;

}  // namespace wick
