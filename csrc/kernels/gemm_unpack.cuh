// GEMM of up to 256 activation rows with super-block GGUF weights that stay packed in HBM (gemm_unpack.cu).
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace oxb {

struct GemmUnpackParams {
  int M, N, K;        // K a multiple of 256
  int m_pad;          // M rounded up to 16: rows of the activation box
  float* out;         // [M, N] fp32, added to
  long long ldo;
  int* status;
  uint32_t spin_limit;
  int x_stages, x_boxes, w_stages;  // set by the launcher: ring sizes, boxes of 64 values per activation stage
};

// Bytes of one box row of the weight map for a block type, 0 for types that this kernel does not take. The map is two-dimensional, in
// 16-bit elements: [N rows][row bytes / 2], boxes of 128 rows; rows have to be a multiple of 16 bytes apart.
int gemm_unpack_box(int q_type);
// tmX: activations [M, K] bf16, boxes of m_pad rows x 64 values, 128-byte swizzle.
void launch_gemm_unpack(const CUtensorMap& tmW, const CUtensorMap& tmX, const GemmUnpackParams& p, int q_type, cudaStream_t stream);

}  // namespace oxb
