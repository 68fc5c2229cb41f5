// esr_warm.cuh -- IDW interpolation and the warm start's input rows.
#pragma once
#include "esr_device.cuh"
#include "esr_mlp.cuh"

namespace esr {

// eval/core.py:135-142 with utils/metrics.py:9-14: weights from float64
// distances, float32 weighted sum over the k neighbours in order. A
// neighbour index outside [0, n_src) is never read: the row becomes NaN and
// *bad is set (the host reads it with esr_idw_status).
__device__ int g_idw_bad = 0;

constexpr int kMaxNeighbours = 16;

// neighbours and float32 weights of row i; false when an index is out of range
template <int K>
__device__ __forceinline__ bool idw_weights(const int* __restrict__ idx, const float* __restrict__ dist, int i, int k,
                                            int n_src, int q[K], float wf[K]) {
  double w[K], wsum = 0.0;
  bool in_range = true;
#pragma unroll
  for (int j = 0; j < K; ++j) {
    if (j >= k) break;
    q[j] = idx[(size_t)i * k + j];
    in_range = in_range && q[j] >= 0 && q[j] < n_src;
    const double d = (double)dist[(size_t)i * k + j];
    w[j] = 1.0 / (d * d + 1e-12);
    wsum += w[j];
  }
#pragma unroll
  for (int j = 0; j < K; ++j)
    if (j < k) wf[j] = (float)(w[j] / wsum);
  return in_range;
}

static __global__ void k_idw(const float* __restrict__ src, int n_src, int n_vars, const int* __restrict__ idx,
                             const float* __restrict__ dist, int n_dst, int k, float* __restrict__ out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n_dst) return;
  int q[kMaxNeighbours];
  float wf[kMaxNeighbours];
  if (!idw_weights<kMaxNeighbours>(idx, dist, i, k, n_src, q, wf)) {
    atomicExch(&g_idw_bad, 1);
    for (int v = 0; v < n_vars; ++v) out[(size_t)i * n_vars + v] = __int_as_float(0x7fc00000);
    return;
  }
  for (int v = 0; v < n_vars; ++v) {
    float acc = 0.0f;
#pragma unroll
    for (int j = 0; j < kMaxNeighbours; ++j)
      if (j < k) acc += wf[j] * src[(size_t)q[j] * n_vars + v];
    out[(size_t)i * n_vars + v] = acc;
  }
}

// One case's input rows straight from the coarse solution: IDW (6 neighbours)
// of the primitives and the pressure gradient, then the feature row, without
// the interpolated fields passing through memory; rows .. rows_out are zero.
// One launch for four, bound by its latency (25,968 rows: IDW 8.7 + 6.2 us,
// fills 6.7 us and features 5.2 us before).
static __global__ void __launch_bounds__(kFeatureRows) k_warm_inputs(
    const float* __restrict__ src_prim, const float* __restrict__ src_gradp, int n_src, const int* __restrict__ idx,
    const float* __restrict__ dist, const float* __restrict__ stat5, int rows, int rows_out, float mach_n, float aoa_n,
    const float* __restrict__ mu, const float* __restrict__ sig, int ld, __nv_bfloat16* __restrict__ X,
    float* __restrict__ base, bool vec) {
  constexpr int K = 6;
  __shared__ __align__(16) __nv_bfloat16 sh[kFeatureRows][16];
  const int r = blockIdx.x * kFeatureRows + threadIdx.x;
  float y[4] = {0.f, 0.f, 0.f, 0.f};
  if (r < rows) {
    int q[K];
    float wf[K], prim[4] = {0.f, 0.f, 0.f, 0.f}, gradp[2] = {0.f, 0.f};
    if (idw_weights<K>(idx, dist, r, K, n_src, q, wf)) {
#pragma unroll
      for (int j = 0; j < K; ++j) {
#pragma unroll
        for (int v = 0; v < 4; ++v) prim[v] += wf[j] * src_prim[(size_t)q[j] * 4 + v];
        gradp[0] += wf[j] * src_gradp[(size_t)q[j] * 2];
        gradp[1] += wf[j] * src_gradp[(size_t)q[j] * 2 + 1];
      }
    } else {
      atomicExch(&g_idw_bad, 1);
      const float nan = __int_as_float(0x7fc00000);
      prim[0] = prim[1] = prim[2] = prim[3] = gradp[0] = gradp[1] = nan;
    }
    feature_row(stat5 + (size_t)r * 5, prim, gradp, mach_n, aoa_n, mu, sig, sh[threadIdx.x], y);
  } else {
#pragma unroll
    for (int j = 0; j < 16; ++j) sh[threadIdx.x][j] = __float2bfloat16(0.f);
  }
  if (r < rows_out)
#pragma unroll
    for (int v = 0; v < 4; ++v) base[(size_t)r * 4 + v] = y[v];
  __syncthreads();
  store_features(sh, blockIdx.x * kFeatureRows, rows_out, ld, X, vec);
}

}  // namespace esr
