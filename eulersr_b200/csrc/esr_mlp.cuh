// esr_mlp.cuh -- input rows of the warm-start MLP, shared by the kernels that
// build them.
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>

namespace esr {

constexpr int kFeatureRows = 128;   // rows (and threads) per block

// The 13 features of one row and the 3 zeros that pad them to 16:
// [x, y, wall distance, wall normal x, y (static), IDW primitives normalised,
// asinh(IDW dp/dx / s_p), asinh(dp/dy / s_p), M_n, alpha_n]; q receives the
// normalised primitives (the prediction that the MLP corrects).
__device__ __forceinline__ void feature_row(const float* __restrict__ stat5, const float prim[4], const float gradp[2],
                                            float mach_n, float aoa_n, const float* __restrict__ mu,
                                            const float* __restrict__ sig, __nv_bfloat16 x[16], float q[4]) {
#pragma unroll
  for (int j = 0; j < 5; ++j) x[j] = __float2bfloat16(stat5[j]);
#pragma unroll
  for (int v = 0; v < 4; ++v) {
    q[v] = (prim[v] - mu[v]) / sig[v];
    x[5 + v] = __float2bfloat16(q[v]);
  }
  const float sp = sig[3] + 1e-8f;
  x[9] = __float2bfloat16(asinhf(gradp[0] / sp));
  x[10] = __float2bfloat16(asinhf(gradp[1] / sp));
  x[11] = __float2bfloat16(mach_n);
  x[12] = __float2bfloat16(aoa_n);
#pragma unroll
  for (int j = 13; j < 16; ++j) x[j] = __float2bfloat16(0.f);
}

// The block's rows from shared memory into X, zero padded to ld columns.
// vec: ld a multiple of 8 and X 16-byte aligned, so that neighbouring threads
// write neighbouring 16-byte chunks (25,968 rows x 128: 5 us; 42 us with each
// thread writing its own row 2 bytes at a time).
__device__ __forceinline__ void store_features(const __nv_bfloat16 (*sh)[16], int row0, int rows, int ld,
                                               __nv_bfloat16* __restrict__ X, bool vec) {
  const int n = min(kFeatureRows, rows - row0);
  if (vec) {
    const int chunks = ld / 8;
    for (int i = threadIdx.x; i < n * chunks; i += blockDim.x) {
      const int r = i / chunks, c = i - r * chunks;
      const uint4 v = c < 2 ? reinterpret_cast<const uint4*>(sh[r])[c] : make_uint4(0, 0, 0, 0);
      reinterpret_cast<uint4*>(X + (size_t)(row0 + r) * ld)[c] = v;
    }
  } else {
    for (int i = threadIdx.x; i < n * ld; i += blockDim.x) {
      const int r = i / ld, c = i - r * ld;
      X[(size_t)(row0 + r) * ld + c] = c < 16 ? sh[r][c] : __float2bfloat16(0.f);
    }
  }
}

}  // namespace esr
