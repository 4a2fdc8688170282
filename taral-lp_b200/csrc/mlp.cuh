// Elementwise steps of the warm-start MLP that more than one kernel takes (mlp.cu, mlp_tc.cu).
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>

namespace taral {
namespace mlp {

using bf16 = __nv_bfloat16;

__device__ __forceinline__ float gelu(float z) { return 0.5f * z * (1.f + erff(z * 0.70710678118654752f)); }
__device__ __forceinline__ float gelu_grad(float z) {
    const float cdf = 0.5f * (1.f + erff(z * 0.70710678118654752f));
    const float pdf = 0.39894228040143268f * expf(-0.5f * z * z);
    return cdf + z * pdf;
}

// One Adam step's constants: learning rate, decay rates, epsilon and the bias corrections 1 - b^t.
struct AdamStep {
    float lr, b1, b2, eps, c1, c2;
};
// Adam on one FP32 master weight w with moments m, v and gradient g. The roundings are spelled out, so that every kernel
// takes the same step to the last bit.
__device__ __forceinline__ void adam_step(const AdamStep& s, float g, float& w, float& m, float& v) {
    m = fmaf(1.f - s.b1, g, __fmul_rn(s.b1, m));
    v = fmaf(__fmul_rn(1.f - s.b2, g), g, __fmul_rn(s.b2, v));
    w = __fsub_rn(w, __fdiv_rn(__fmul_rn(s.lr, __fdiv_rn(m, s.c1)), __fadd_rn(__fsqrt_rn(__fdiv_rn(v, s.c2)), s.eps)));
}

// Layout of the FP32 masters and moments of a weight matrix whose Adam step runs in the epilogue of its gradient's GEMM
// (mlp_tc.cu): blocks of 128 rows x 16 columns, in a block the 32-row quadrants, in a quadrant the 16-byte groups of 4
// columns, in a group the rows. A warp that holds 32 rows x 16 columns of the gradient in registers, a row per lane, so
// reads and writes 2 KB in a row of each array, and a CTA's tile is one contiguous range. `groups`: column groups of 16.
__host__ __device__ __forceinline__ size_t blocked_at(int r, int c, int groups) {
    return (size_t(r >> 7) * groups + (c >> 4)) * 2048 + size_t(((r >> 5) & 3) * 512 + ((c >> 2) & 3) * 128 + (r & 31) * 4 + (c & 3));
}
inline int blocked_groups(int cols) { return (cols + 15) / 16; }
inline size_t blocked_size(int rows, int cols) { return size_t((rows + 127) / 128) * blocked_groups(cols) * 2048; }

}  // namespace mlp
}  // namespace taral
