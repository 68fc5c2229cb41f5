// esr_mlp.cu -- BF16 training and inference kernels of the warm-start MLP.
//
// The network corrects an IDW interpolation of the coarse solution cell by
// cell: 32 input features (13 used) -> 256 -> 3 residual blocks of 256 ->
// 4 outputs. Its 256-wide layers are GEMMs of rows (cells) x 256 x 256 run
// on the tensor cores by one kernel template:
//   C[M x N] = A[M x K] * B[K x N], BF16 operands, FP32 accumulation
//   (mma.sync m16n8k16), 128 x 128 x 32 CTA tiles, 8 warps of 64 x 32,
//   3-stage cp.async pipeline, ldmatrix (.trans for the transposed operands)
// with fused epilogues:
//   EPI_F32   store the FP32 tile (split-K partials of the weight gradients)
//   EPI_FWD   z = acc + bias; out = residual + relu(z)   (z kept for backward)
//   EPI_BWD   dh = acc + dh_next; dz_prev = dh * (z_prev > 0)
// The 4-wide head, the loss, AdamW and the fixed-order reductions are plain
// SIMT kernels, bound by reading their operands once. Every reduction is deterministic (no atomics).
#include <cuda_bf16.h>
#include <cuda.h>
#include <cuda_runtime.h>
#include <cudaTypedefs.h>
#include <stdint.h>

#include <algorithm>
#include <string>

#include "esr_internal.h"
#include "esr_mlp.cuh"
#include "esr_per_device.h"

namespace {

using bf16 = __nv_bfloat16;
using namespace esr;

constexpr int BM = 128, BN = 128, BK = 32, STAGES = 3, THREADS = 256;
constexpr int PAD = 8;
constexpr int LD_K = BK + PAD;     // row stride of K-contiguous tiles (elements)
constexpr int LD_MN = BM + PAD;    // row stride of M/N-contiguous tiles

enum { EPI_F32 = 0, EPI_FWD = 1, EPI_BWD = 2 };

// Eight consecutive BF16 values, as one 16-byte access (VEC) or one by one
// where a caller's buffer is not aligned for it.
template <bool VEC>
__device__ __forceinline__ void load8(const bf16* p, float v[8]) {
  if (VEC) {
    const uint4 u = *reinterpret_cast<const uint4*>(p);
    const unsigned w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      v[2 * i] = __uint_as_float(w[i] << 16);
      v[2 * i + 1] = __uint_as_float(w[i] & 0xFFFF0000u);
    }
  } else {
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = __bfloat162float(p[i]);
  }
}
template <bool VEC>
__device__ __forceinline__ void store8(bf16* p, const float v[8]) {
  if (VEC) {
    unsigned w[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const __nv_bfloat162 b = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
      w[i] = *reinterpret_cast<const unsigned*>(&b);
    }
    *reinterpret_cast<uint4*>(p) = make_uint4(w[0], w[1], w[2], w[3]);
  } else {
#pragma unroll
    for (int i = 0; i < 8; ++i) p[i] = __float2bfloat16(v[i]);
  }
}
inline bool aligned16(const void* p) { return ((uintptr_t)p & 15) == 0; }

struct Epi {
  const float* bias;     // FWD: per-column bias
  const bf16* res;       // FWD: residual input; BWD: dh of the next layer
  const bf16* aux;       // BWD: z of the previous layer (relu mask)
  void* out0;            // F32: float partials; FWD: activation out; BWD: dh
  bf16* out1;            // FWD: z; BWD: dz_prev
  int ldo;               // leading dimension of res/aux/out0/out1
  long long split_stride;// F32: elements between split-K partial tiles
  bool vec;              // every pointer and row of this epilogue is 16-byte aligned
};

__device__ __forceinline__ void cp_async16(void* smem, const void* gmem) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gmem));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N)); }

__device__ __forceinline__ void ldsm_x4(unsigned r[4], const void* p) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(p);
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(s));
}
__device__ __forceinline__ void ldsm_x4_t(unsigned r[4], const void* p) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(p);
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(s));
}
__device__ __forceinline__ void mma_bf16(float c[4], const unsigned a[4], unsigned b0, unsigned b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%0,%1,%2,%3};\n"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// A(m,k): A_T ? A[k*lda + m] : A[m*lda + k];  B(k,n): B_T ? B[k*ldb + n] : B[n*ldb + k]
template <bool A_T, bool B_T, int EPI>
__global__ void __launch_bounds__(THREADS) k_gemm(int M, int N, int K_split, const bf16* __restrict__ A, int lda,
                                                  const bf16* __restrict__ B, int ldb, Epi e) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  constexpr int A_ELEMS = A_T ? BK * LD_MN : BM * LD_K;
  constexpr int B_ELEMS = B_T ? BK * LD_MN : BN * LD_K;
  bf16* sA = reinterpret_cast<bf16*>(smem_raw);
  bf16* sB = sA + STAGES * A_ELEMS;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int wm = warp >> 2, wn = warp & 3;
  const int m_blk = blockIdx.y * BM, n_blk = blockIdx.x * BN;
  const int k_begin = blockIdx.z * K_split;
  const int KT = K_split / BK;

  auto load_tile = [&](int stage, int kt) {
    const int k0 = k_begin + kt * BK;
    bf16* a = sA + stage * A_ELEMS;
    bf16* b = sB + stage * B_ELEMS;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int c = tid + i * THREADS;   // 512 chunks of 8 elements per operand tile
      if (!A_T) {
        const int r = c >> 2, kc = (c & 3) * 8;
        cp_async16(a + r * LD_K + kc, A + (size_t)(m_blk + r) * lda + k0 + kc);
      } else {
        const int r = c >> 4, mc = (c & 15) * 8;
        cp_async16(a + r * LD_MN + mc, A + (size_t)(k0 + r) * lda + m_blk + mc);
      }
      if (!B_T) {
        const int r = c >> 2, kc = (c & 3) * 8;
        cp_async16(b + r * LD_K + kc, B + (size_t)(n_blk + r) * ldb + k0 + kc);
      } else {
        const int r = c >> 4, nc = (c & 15) * 8;
        cp_async16(b + r * LD_MN + nc, B + (size_t)(k0 + r) * ldb + n_blk + nc);
      }
    }
  };

  float acc[4][4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int q = 0; q < 4; ++q) acc[i][j][q] = 0.f;

#pragma unroll
  for (int s = 0; s < STAGES - 1; ++s) {
    if (s < KT) load_tile(s, s);
    cp_async_commit();
  }
  for (int kt = 0; kt < KT; ++kt) {
    cp_async_wait<STAGES - 2>();
    __syncthreads();
    const int pf = kt + STAGES - 1;
    if (pf < KT) load_tile(pf % STAGES, pf);
    cp_async_commit();
    const bf16* a = sA + (kt % STAGES) * A_ELEMS;
    const bf16* b = sB + (kt % STAGES) * B_ELEMS;
#pragma unroll
    for (int kk = 0; kk < BK; kk += 16) {
      unsigned af[4][4], bfr[2][4];
#pragma unroll
      for (int mi = 0; mi < 4; ++mi) {
        const int m0 = wm * 64 + mi * 16;
        if (!A_T) ldsm_x4(af[mi], a + (m0 + (lane & 15)) * LD_K + kk + (lane >> 4) * 8);
        else ldsm_x4_t(af[mi], a + (kk + (lane & 7) + (lane >> 4) * 8) * LD_MN + m0 + ((lane >> 3) & 1) * 8);
      }
#pragma unroll
      for (int nj = 0; nj < 2; ++nj) {
        const int n0 = wn * 32 + nj * 16;
        if (!B_T) ldsm_x4(bfr[nj], b + (n0 + (lane & 7) + (lane >> 4) * 8) * LD_K + kk + ((lane >> 3) & 1) * 8);
        else ldsm_x4_t(bfr[nj], b + (kk + (lane & 7) + ((lane >> 3) & 1) * 8) * LD_MN + n0 + (lane >> 4) * 8);
      }
#pragma unroll
      for (int mi = 0; mi < 4; ++mi)
#pragma unroll
        for (int ni = 0; ni < 4; ++ni)
          mma_bf16(acc[mi][ni], af[mi], bfr[ni >> 1][(ni & 1) * 2], bfr[ni >> 1][(ni & 1) * 2 + 1]);
    }
  }
  cp_async_wait<0>();

  const int g = lane >> 2, tig = lane & 3;
#pragma unroll
  for (int mi = 0; mi < 4; ++mi)
#pragma unroll
    for (int ni = 0; ni < 4; ++ni)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int m = m_blk + wm * 64 + mi * 16 + g + h * 8;
        const int n = n_blk + wn * 32 + ni * 8 + tig * 2;
        const float v0 = acc[mi][ni][2 * h], v1 = acc[mi][ni][2 * h + 1];
        const size_t o = (size_t)m * e.ldo + n;
        if (EPI == EPI_F32) {
          float* out = static_cast<float*>(e.out0) + (size_t)blockIdx.z * e.split_stride;
          *reinterpret_cast<float2*>(out + o) = make_float2(v0, v1);
        } else if (EPI == EPI_FWD) {
          const float z0 = v0 + e.bias[n], z1 = v1 + e.bias[n + 1];
          float r0 = 0.f, r1 = 0.f;
          if (e.res) {
            const __nv_bfloat162 r = *reinterpret_cast<const __nv_bfloat162*>(e.res + o);
            r0 = __bfloat162float(r.x);
            r1 = __bfloat162float(r.y);
          }
          *reinterpret_cast<__nv_bfloat162*>(e.out1 + o) = __floats2bfloat162_rn(z0, z1);
          *reinterpret_cast<__nv_bfloat162*>(static_cast<bf16*>(e.out0) + o) =
              __floats2bfloat162_rn(r0 + fmaxf(z0, 0.f), r1 + fmaxf(z1, 0.f));
        } else {
          float d0 = v0, d1 = v1;
          if (e.res) {
            const __nv_bfloat162 r = *reinterpret_cast<const __nv_bfloat162*>(e.res + o);
            d0 += __bfloat162float(r.x);
            d1 += __bfloat162float(r.y);
          }
          *reinterpret_cast<__nv_bfloat162*>(static_cast<bf16*>(e.out0) + o) = __floats2bfloat162_rn(d0, d1);
          if (e.aux) {
            const __nv_bfloat162 z = *reinterpret_cast<const __nv_bfloat162*>(e.aux + o);
            *reinterpret_cast<__nv_bfloat162*>(e.out1 + o) = __floats2bfloat162_rn(
                __bfloat162float(z.x) > 0.f ? d0 : 0.f, __bfloat162float(z.y) > 0.f ? d1 : 0.f);
          }
        }
      }
}

// ------------------------------------------------------------- SIMT kernels
// y[r][j] = sum_k H[r][k] W[j][k] + b[j], 4 outputs, FP32 accumulation
__global__ void k_head_fwd(const bf16* __restrict__ H, int rows, int K, const float* __restrict__ W,
                           const float* __restrict__ b, const float* __restrict__ base, float* __restrict__ y) {
  const int r = blockIdx.x * (blockDim.x / 32) + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (r >= rows) return;
  float s[4] = {0.f, 0.f, 0.f, 0.f};
  for (int k = lane; k < K; k += 32) {
    const float h = __bfloat162float(H[(size_t)r * K + k]);
#pragma unroll
    for (int j = 0; j < 4; ++j) s[j] += h * W[j * K + k];
  }
#pragma unroll
  for (int j = 0; j < 4; ++j)
    for (int o = 16; o > 0; o >>= 1) s[j] += __shfl_xor_sync(0xffffffffu, s[j], o);
  if (lane < 4) y[(size_t)r * 4 + lane] = s[lane] + b[lane] + (base ? base[(size_t)r * 4 + lane] : 0.f);
}

// The same sums in the same order for 256 columns: a lane keeps its columns
// (lane + 32 i) of W in registers, a warp walks groups of 4 rows and requests
// the next group before it sums the current one. Bound by reading H once:
// 32,768 rows take 13 us, 17 us row by row.
__global__ void __launch_bounds__(256, 2) k_head_fwd256(const bf16* __restrict__ H, int rows,
                                                        const float* __restrict__ W, const float* __restrict__ b,
                                                        const float* __restrict__ base, float* __restrict__ y) {
  constexpr int R = 4;
  const int lane = threadIdx.x & 31, step = R * gridDim.x * (blockDim.x >> 5);
  int r0 = R * (blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5));
  bf16 h[R][8], hn[R][8];
  auto fetch = [&](int r, bf16 v[R][8]) {
#pragma unroll
    for (int q = 0; q < R; ++q)
#pragma unroll
      for (int i = 0; i < 8; ++i) v[q][i] = H[(size_t)min(r + q, rows - 1) * 256 + lane + 32 * i];
  };
  fetch(r0, h);
  float w[4][8];
#pragma unroll
  for (int j = 0; j < 4; ++j)
#pragma unroll
    for (int i = 0; i < 8; ++i) w[j][i] = W[j * 256 + lane + 32 * i];
  const float bias = b[lane & 3];
  for (; r0 < rows; r0 += step) {
    fetch(r0 + step, hn);
#pragma unroll
    for (int q = 0; q < R; ++q) {
      float s[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const float v = __bfloat162float(h[q][i]);
#pragma unroll
        for (int j = 0; j < 4; ++j) s[j] += v * w[j][i];
      }
#pragma unroll
      for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s[j] += __shfl_xor_sync(0xffffffffu, s[j], o);
      if (lane < 4 && r0 + q < rows) {
        const float v = lane == 0 ? s[0] : lane == 1 ? s[1] : lane == 2 ? s[2] : s[3];
        y[(size_t)(r0 + q) * 4 + lane] = v + bias + (base ? base[(size_t)(r0 + q) * 4 + lane] : 0.f);
      }
    }
#pragma unroll
    for (int q = 0; q < R; ++q)
#pragma unroll
      for (int i = 0; i < 8; ++i) h[q][i] = hn[q][i];
  }
}

// Two consecutive BF16 values, as one 4-byte access (VEC) or one by one.
template <bool VEC>
__device__ __forceinline__ __nv_bfloat162 load2(const bf16* p) {
  if (VEC) return *reinterpret_cast<const __nv_bfloat162*>(p);
  __nv_bfloat162 v;
  v.x = p[0];
  v.y = p[1];
  return v;
}
template <bool VEC>
__device__ __forceinline__ void store2(bf16* p, float a, float b) {
  const __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
  if (VEC) {
    *reinterpret_cast<__nv_bfloat162*>(p) = v;
  } else {
    p[0] = v.x;
    p[1] = v.y;
  }
}

// The head's backward over 256 columns, one block per `rows_per_block` rows:
// dH[r][k] = sum_j dY[r][j] W[j][k] and dZ = dH * (z > 0) as BF16, and the
// block's partials of dW[j][k] = sum_r dY[r][j] H[r][k] and db[j] = sum_r
// dY[r][j], summed row by row. One group of 128 threads sums (two columns a
// thread), three write dH and dZ of a third of the rows each; dY waits in
// shared memory and the next rows of H or Z are requested before the current
// ones are used, since it is the memory that must be kept busy, not the chains
// over rows. 32,768 rows take 23 us; 26 us with one group for both, 102 us as a
// thread per element and a second kernel that waits for each row.
constexpr int kHeadSlab = 256, kHeadGroups = 4;
template <bool VEC>
__global__ void __launch_bounds__(128 * kHeadGroups) k_head_bwd(
    const float* __restrict__ dY, const bf16* __restrict__ H, const bf16* __restrict__ Z, int rows,
    const float* __restrict__ W, bf16* __restrict__ dH, bf16* __restrict__ dZ, int rows_per_block,
    float* __restrict__ part) {
  constexpr int K = 256;
  __shared__ float4 sd[kHeadSlab];
  const int grp = threadIdx.x >> 7, col = (threadIdx.x & 127) * 2;
  const int r0 = blockIdx.x * rows_per_block, r1 = min(rows, r0 + rows_per_block);
  float w[4][2], g[4][2], gb[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    w[j][0] = W[j * K + col];
    w[j][1] = W[j * K + col + 1];
    g[j][0] = g[j][1] = gb[j] = 0.f;
  }
  // N rows of X from r on, none past `stop`
  auto fetch = [&](const bf16* X, int r, int stop, auto& v) {
    constexpr int N = sizeof(v) / sizeof(v[0]);
#pragma unroll
    for (int q = 0; q < N; ++q) v[q] = load2<VEC>(X + (size_t)min(r + q, stop - 1) * K + col);
  };
  for (int slab = r0; slab < r1; slab += kHeadSlab) {
    const int n = min(kHeadSlab, r1 - slab);
    __syncthreads();
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
      const float* p = dY + (size_t)(slab + i) * 4;
      sd[i] = make_float4(p[0], p[1], p[2], p[3]);
    }
    __syncthreads();
    if (grp == 0) {
      constexpr int N = 16;
      __nv_bfloat162 h[N], hn[N];
      fetch(H, slab, slab + n, h);
      for (int i = 0; i < n; i += N) {
        fetch(H, slab + i + N, slab + n, hn);
#pragma unroll
        for (int q = 0; q < N; ++q) {
          if (i + q < n) {
            const float4 dv = sd[i + q];
            const float d[4] = {dv.x, dv.y, dv.z, dv.w};
            const float h0 = __bfloat162float(h[q].x), h1 = __bfloat162float(h[q].y);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              g[j][0] += d[j] * h0;
              g[j][1] += d[j] * h1;
              gb[j] += d[j];
            }
          }
        }
#pragma unroll
        for (int q = 0; q < N; ++q) h[q] = hn[q];
      }
    } else {
      constexpr int N = 12;
      const int third = (n + 2) / 3, i0 = (grp - 1) * third, i1 = min(n, i0 + third);
      __nv_bfloat162 z[N], zn[N];
      if (i0 < i1) fetch(Z, slab + i0, slab + i1, z);
      for (int i = i0; i < i1; i += N) {
        fetch(Z, slab + i + N, slab + i1, zn);
#pragma unroll
        for (int q = 0; q < N; ++q) {
          if (i + q < i1) {
            const float4 dv = sd[i + q];
            const float d[4] = {dv.x, dv.y, dv.z, dv.w};
            float s0 = 0.f, s1 = 0.f;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              s0 += d[j] * w[j][0];
              s1 += d[j] * w[j][1];
            }
            const size_t o = (size_t)(slab + i + q) * K + col;
            store2<VEC>(dH + o, s0, s1);
            store2<VEC>(dZ + o, __bfloat162float(z[q].x) > 0.f ? s0 : 0.f, __bfloat162float(z[q].y) > 0.f ? s1 : 0.f);
          }
        }
#pragma unroll
        for (int q = 0; q < N; ++q) z[q] = zn[q];
      }
    }
  }
  if (grp > 0) return;
  float* p = part + (size_t)blockIdx.x * (4 * K + 4);
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    p[j * K + col] = g[j][0];
    p[j * K + col + 1] = g[j][1];
  }
  if (threadIdx.x == 0)
    for (int j = 0; j < 4; ++j) p[4 * K + j] = gb[j];
}

// Per-cell inputs of one case (BF16 rows of `ld` columns, zero padded):
// [x, y, wall distance, wall normal x, y (5 static), IDW primitives
// normalised (4), asinh(IDW dp/dx / s_p), asinh(dp/dy / s_p) (2), M_n, alpha_n]
__global__ void k_features(const float* __restrict__ stat5, const float* __restrict__ idw_prim,
                           const float* __restrict__ idw_gradp, int rows, float mach_n, float aoa_n,
                           const float* __restrict__ mu, const float* __restrict__ sig, int ld, bf16* __restrict__ X,
                           float* __restrict__ base, bool vec) {
  __shared__ __align__(16) bf16 sh[kFeatureRows][16];
  const int r = blockIdx.x * kFeatureRows + threadIdx.x;
  if (r < rows) {
    float prim[4], gradp[2], q[4];
#pragma unroll
    for (int v = 0; v < 4; ++v) prim[v] = idw_prim[(size_t)r * 4 + v];
    gradp[0] = idw_gradp[(size_t)r * 2];
    gradp[1] = idw_gradp[(size_t)r * 2 + 1];
    feature_row(stat5 + (size_t)r * 5, prim, gradp, mach_n, aoa_n, mu, sig, sh[threadIdx.x], q);
    if (base)   // the IDW prediction the MLP corrects
#pragma unroll
      for (int v = 0; v < 4; ++v) base[(size_t)r * 4 + v] = q[v];
  }
  __syncthreads();
  store_features(sh, blockIdx.x * kFeatureRows, rows, ld, X, vec);
}

// normalised primitive prediction -> conserved state (float64 rows), with
// density and pressure kept above `floor_frac` of their freestream values
__global__ void k_decode(const float* __restrict__ pred_n, int rows, const float* __restrict__ mu,
                         const float* __restrict__ sig, float gamma, float rho_floor, float p_floor,
                         double* __restrict__ W) {
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= rows) return;
  const float rho = fmaxf(pred_n[(size_t)r * 4] * sig[0] + mu[0], rho_floor);
  const float u = pred_n[(size_t)r * 4 + 1] * sig[1] + mu[1];
  const float v = pred_n[(size_t)r * 4 + 2] * sig[2] + mu[2];
  const float p = fmaxf(pred_n[(size_t)r * 4 + 3] * sig[3] + mu[3], p_floor);
  W[(size_t)r * 4] = rho;
  W[(size_t)r * 4 + 1] = (double)rho * u;
  W[(size_t)r * 4 + 2] = (double)rho * v;
  W[(size_t)r * 4 + 3] = (double)p / (gamma - 1.0) + 0.5 * (double)rho * ((double)u * u + (double)v * v);
}

// out[i] = sum_s part[s * stride + i] in split order, for several sets of
// partials in one launch (a block per 256 outputs of one set). The loads of 16
// splits are in flight at once: 256 outputs of 128 partials take 3 us, 11 us
// load by load.
struct Reduction {
  const float* part;
  float* out;
  long long stride, n;
  int splits, blocks;    // blocks before this set's
};
constexpr int kMaxReductions = 16;
struct Reductions {
  Reduction r[kMaxReductions];
  int n;
};
__global__ void __launch_bounds__(256) k_reduce_splits(const __grid_constant__ Reductions q) {
  int k = 0;
  while (k + 1 < q.n && (int)blockIdx.x >= q.r[k + 1].blocks) ++k;
  const Reduction& r = q.r[k];
  const long long i = (long long)((int)blockIdx.x - r.blocks) * 256 + threadIdx.x;
  if (i >= r.n) return;
  const float* p = r.part + i;
  float s = 0.f;
  int z = 0;
  for (; z + 16 <= r.splits; z += 16) {
    float v[16];
#pragma unroll
    for (int u = 0; u < 16; ++u) v[u] = p[(size_t)(z + u) * r.stride];
#pragma unroll
    for (int u = 0; u < 16; ++u) s += v[u];
  }
  for (; z < r.splits; ++z) s += p[(size_t)z * r.stride];
  r.out[i] = s;
}

// column sums of a BF16 [rows x C] matrix in fixed row blocks, row by row
// (bias gradients), 32 rows in flight. A thread owns two columns in 4-byte
// loads (VEC), one where C is odd or X not aligned for them: 32,768 x 256 (16.8
// MB) takes 5 us (as a quarter of one launch), 22 us load by load; 32,768 x 7
// 6 us, 16 us with two columns a thread.
template <bool VEC>
__global__ void __launch_bounds__(128) k_colsum_part(const bf16* __restrict__ X, int rows, int C, int rows_per_block,
                                                     float* __restrict__ part) {
  constexpr int U = 32;
  const int c = (VEC ? 2 : 1) * (blockIdx.y * blockDim.x + threadIdx.x);
  if (c >= C) return;
  const int r0 = blockIdx.x * rows_per_block, r1 = min(rows, r0 + rows_per_block);
  float s0 = 0.f, s1 = 0.f;
  int r = r0;
  if constexpr (VEC) {
    for (; r + U <= r1; r += U) {
      __nv_bfloat162 v[U];
#pragma unroll
      for (int u = 0; u < U; ++u) v[u] = load2<true>(X + (size_t)(r + u) * C + c);
#pragma unroll
      for (int u = 0; u < U; ++u) { s0 += __bfloat162float(v[u].x); s1 += __bfloat162float(v[u].y); }
    }
    for (; r < r1; ++r) {
      const __nv_bfloat162 v = load2<true>(X + (size_t)r * C + c);
      s0 += __bfloat162float(v.x);
      s1 += __bfloat162float(v.y);
    }
    part[(size_t)blockIdx.x * C + c + 1] = s1;
  } else {
    for (; r + U <= r1; r += U) {
      bf16 v[U];
#pragma unroll
      for (int u = 0; u < U; ++u) v[u] = X[(size_t)(r + u) * C + c];
#pragma unroll
      for (int u = 0; u < U; ++u) s0 += __bfloat162float(v[u]);
    }
    for (; r < r1; ++r) s0 += __bfloat162float(X[(size_t)r * C + c]);
  }
  part[(size_t)blockIdx.x * C + c] = s0;
}

// shock-weighted relative MSE (loss.py:20-23) on pred = base + head:
// L = mean_v [ sum_r w_r (p - t)^2 / R / (mean_r t^2 + 1e-8) ]; dpred written;
// per-block partial sums of the loss numerators
__global__ void k_loss(const float* __restrict__ pred, const float* __restrict__ tgt, const float* __restrict__ w,
                       int rows, const float* __restrict__ inv_den, float* __restrict__ dpred,
                       float* __restrict__ part) {
  __shared__ float sh[256];
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  float l = 0.f;
  if (r < rows) {
    const float wr = w ? w[r] : 1.f;
#pragma unroll
    for (int v = 0; v < 4; ++v) {
      const float d = pred[(size_t)r * 4 + v] - tgt[(size_t)r * 4 + v];
      l += wr * d * d * inv_den[v];
      dpred[(size_t)r * 4 + v] = 2.f * wr * d * inv_den[v] / (4.f * rows);
    }
  }
  sh[threadIdx.x] = l;
  __syncthreads();
  for (int s = blockDim.x / 2; s > 0; s >>= 1) {
    if (threadIdx.x < s) sh[threadIdx.x] += sh[threadIdx.x + s];
    __syncthreads();
  }
  if (threadIdx.x == 0) part[blockIdx.x] = sh[0] / (4.f * rows);
}

// AdamW on FP32 master weights with a BF16 (or FP32) working copy
__global__ void k_adamw(float* __restrict__ p, const float* __restrict__ g, float* __restrict__ m,
                        float* __restrict__ v, long long n, float lr, float b1, float b2, float eps, float wd,
                        float bc1, float bc2, bf16* __restrict__ p_bf16) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float gi = g[i];
  const float mi = b1 * m[i] + (1.f - b1) * gi;
  const float vi = b2 * v[i] + (1.f - b2) * gi * gi;
  m[i] = mi;
  v[i] = vi;
  const float mh = mi / bc1, vh = vi / bc2;
  const float pi = p[i] * (1.f - lr * wd) - lr * mh / (sqrtf(vh) + eps);
  p[i] = pi;
  if (p_bf16) p_bf16[i] = __float2bfloat16(pi);
}

// ------------------------------------------------------ tcgen05 GEMM path
// The same C = A B with the fifth-generation tensor cores: TMA boxes bring
// the operands into shared memory in the 128-byte swizzled canonical layouts
// the UMMA descriptors describe, one thread issues the loads and
// tcgen05.mma (128 x N x 16, BF16 in, FP32 accumulators in tensor memory),
// mbarriers track each stage (tiles landed / MMAs done reading), and the
// epilogue reads the accumulators back with tcgen05.ld, stages them in shared
// memory and applies the epilogue in row-contiguous order.
namespace tc {

constexpr int BM = 128, BK = 64, THREADS = 256;
constexpr int A_BYTES = BM * BK * 2;                    // 16 KB of A per stage
constexpr int SLD = 128 + 4;                            // row stride (floats) of a staged 128-column accumulator half
constexpr long long kSpinLimit = 1LL << 20;             // bounded mbarrier polls

// Tile width 128 (3 stages) or 256 (2 stages): a 256-wide tile reads each
// 128-row block of A once for the whole 256-column output; both use 96 KB of
// pipeline buffers, so two CTAs fit on an SM.
template <int TBN>
struct Cfg {
  static constexpr int BN = TBN;
  static constexpr int STAGES = TBN == 256 ? 2 : 3;
  static constexpr int B_BYTES = TBN * BK * 2;
  static constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
  static constexpr int SMEM = 1024 + STAGES * STAGE_BYTES + (2 * STAGES + 1) * 8 + 16;
  static_assert(BM * SLD * 4 <= STAGES * STAGE_BYTES, "accumulator staging must fit the pipeline buffers");
};

__device__ int g_tc_error = 0;                          // set when a wait gave up

__device__ __forceinline__ uint32_t saddr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(bar), "r"(count));
}
// true once the barrier's phase with this parity has completed; false after the spin limit
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity) {
  for (long long i = 0; i < kSpinLimit; ++i) {
    uint32_t done;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(done) : "r"(bar), "r"(parity) : "memory");
    if (done) return true;
  }
  atomicExch(&g_tc_error, 1);
  return false;
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory"); }

// Shared-memory matrix descriptor, 128-byte swizzle. K-major: rows of 64
// elements (128 B), 8-row groups 1024 B apart (SBO), LBO unused (1).
// MN-major: 64-element MN groups `lbo` bytes apart, 8-row K groups 1024 B apart.
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr, uint32_t lbo_bytes, uint32_t sbo_bytes) {
  uint64_t d = 0;
  d |= (uint64_t)((addr >> 4) & 0x3FFF);
  d |= (uint64_t)((lbo_bytes >> 4) & 0x3FFF) << 16;
  d |= (uint64_t)((sbo_bytes >> 4) & 0x3FFF) << 32;
  d |= (uint64_t)1 << 46;                // descriptor version of sm_100
  d |= (uint64_t)2 << 61;                // SWIZZLE_128B
  return d;
}

// kind::f16 instruction descriptor: FP32 accumulate, BF16 A and B, majors, N, M
template <bool A_MN, bool B_MN, int N>
__host__ __device__ constexpr uint32_t instr_desc() {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((A_MN ? 1u : 0u) << 15) | ((B_MN ? 1u : 0u) << 16) |
         ((uint32_t)(N >> 3) << 17) | ((uint32_t)(BM >> 4) << 24);
}

__device__ __forceinline__ void umma(uint32_t tmem, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n"
      ::"r"(tmem), "l"(a), "l"(b), "r"(idesc), "r"(acc));
}
__device__ __forceinline__ void umma_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(bar) : "memory");
}
// TMA: one 2-D box of a tensor map into shared memory, completion counted in
// bytes on an mbarrier (no multicast)
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* map, int x, int y, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];\n"
      ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(bar) : "memory");
}

__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t v[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
        "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
}

// 32 columns, to be waited for with tmem_wait
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t v[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,"
      "%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];\n"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
        "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]),
        "=r"(v[16]), "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]),
        "=r"(v[24]), "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
      : "r"(taddr));
}
__device__ __forceinline__ void tmem_wait(uint32_t v[32]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
#pragma unroll
  for (int i = 0; i < 32; ++i) asm volatile("" : "+r"(v[i]));   // no use of v before the wait
}

// Shared-memory tile layouts (what the TMA boxes with the 128-byte swizzle
// produce and the UMMA descriptors describe). K-major tile (rows x 64 K):
// row r at r * 128 B, its 16-byte chunk c at ((c ^ (r & 7)) * 16). MN-major
// tile (64 K-rows x MN): groups of 64 MN elements 8 KB apart, K-row k of a
// group at (k >> 3) * 1024 + (k & 7) * 128 B, chunk c at ((c ^ (k & 7)) * 16).

template <bool A_T, bool B_T, int EPI, int TBN>
__global__ void __launch_bounds__(THREADS) k_gemm_tc(int M, int N, int K_split, const __grid_constant__ CUtensorMap tmA,
                                                     const __grid_constant__ CUtensorMap tmB, Epi e) {
  using C = Cfg<TBN>;
  constexpr int BN = C::BN, STAGES = C::STAGES, STAGE_BYTES = C::STAGE_BYTES;
  extern __shared__ unsigned char smem_raw[];
  const uint32_t raw = saddr(smem_raw);
  const uint32_t tiles = (raw + 1023u) & ~1023u;                   // swizzle atoms need 1 KB alignment
  unsigned char* gtiles = smem_raw + (tiles - raw);
  const uint32_t empty = tiles + STAGES * STAGE_BYTES;             // per stage: MMAs done reading it
  const uint32_t full = empty + STAGES * 8;                        // per stage: its tiles have landed
  const uint32_t done = full + STAGES * 8;                         // all MMAs of the tile are done
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(gtiles + STAGES * STAGE_BYTES + (2 * STAGES + 1) * 8);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int m_blk = blockIdx.y * BM, n_blk = blockIdx.x * BN;
  const int k_begin = blockIdx.z * K_split;
  const int KT = K_split / BK;

  __shared__ int s_abort;   // set when a pipeline wait gave up: the tile is not written
  if (tid == 0) {
    s_abort = 0;
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(empty + 8 * s, 1);
      mbar_init(full + 8 * s, 1);
    }
    mbar_init(done, 1);
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  if (warp == 0) {   // BN TMEM columns: the 128 x BN FP32 accumulator
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(saddr(tmem_slot)), "n"(BN));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;

  // One thread is both the TMA producer and the MMA issuer; the other warps
  // wait for the last MMA and then run the epilogue.
  if (warp == 0) {
    if (lane == 0) {
      // the tiles of K-block kt into stage s: K-major boxes are 64 K x rows,
      // MN-major boxes 64 MN x 64 K, one per 64-element MN group (8 KB apart)
      auto produce = [&](int kt, int s) {
        const int k0 = k_begin + kt * BK;
        const uint32_t a = tiles + s * STAGE_BYTES, b = a + A_BYTES, bar = full + 8 * s;
        mbar_expect_tx(bar, STAGE_BYTES);
        if (!A_T) tma_load_2d(a, &tmA, k0, m_blk, bar);
        else for (int g = 0; g < BM / 64; ++g) tma_load_2d(a + g * 8192, &tmA, m_blk + 64 * g, k0, bar);
        if (!B_T) tma_load_2d(b, &tmB, k0, n_blk, bar);
        else for (int g = 0; g < BN / 64; ++g) tma_load_2d(b + g * 8192, &tmB, n_blk + 64 * g, k0, bar);
      };
      constexpr uint32_t idesc = instr_desc<A_T, B_T, BN>();
      int issued = 0;      // K-blocks whose loads have been issued
      int landed = 0;      // K-blocks whose loads are known to have landed
      bool ok = true;
      for (int p = 0; p < STAGES && p < KT; ++p) { produce(p, p); issued = p + 1; }
      for (int kt = 0; kt < KT && ok; ++kt) {
        const int s = kt % STAGES;
        if (!mbar_wait(full + 8 * s, (kt / STAGES) & 1)) { ok = false; break; }
        landed = kt + 1;
        tc_fence_after();
        const uint32_t a = tiles + s * STAGE_BYTES, b = a + A_BYTES;
#pragma unroll
        for (int j = 0; j < BK / 16; ++j) {   // K = 16 per instruction
          const uint64_t ad = A_T ? smem_desc(a + j * 2048, 8192, 1024) : smem_desc(a + j * 32, 16, 1024);
          const uint64_t bd = B_T ? smem_desc(b + j * 2048, 8192, 1024) : smem_desc(b + j * 32, 16, 1024);
          umma(tmem, ad, bd, idesc, (kt | j) != 0);
        }
        umma_commit(empty + 8 * s);   // arrives when these MMAs (and all earlier ones) are done
        // refill the stage the MMAs of the previous K-block read, once they are done
        const int nxt = kt - 1 + STAGES;
        if (kt >= 1 && nxt < KT) {
          const int ps = (kt - 1) % STAGES;
          if (!mbar_wait(empty + 8 * ps, ((kt - 1) / STAGES) & 1)) { ok = false; break; }
          produce(nxt, ps);
          issued = nxt + 1;
        }
      }
      if (!ok) {
        // A wait gave up: nothing more is issued. Loads already issued may
        // still be landing in shared memory; give each a bounded wait before
        // the block can exit (each stage has at most one load outstanding).
        for (int j = landed; j < issued; ++j) mbar_wait(full + 8 * (j % STAGES), (j / STAGES) & 1);
        s_abort = 1;
      }
      umma_commit(done);   // its one phase completes when every MMA issued so far has
    }
    __syncwarp();
  }
  // The other warps reach this wait while the mainloop is still running. A
  // stage barrier cannot serve here: waiting on parity 1 of a barrier still in
  // its first phase returns at once. `done` completes exactly once.
  const bool done_ok = mbar_wait(done, 0);
  if (!done_ok) atomicOr(&s_abort, 1);
  __syncthreads();
  if (s_abort) {
    // The tile is not complete: write nothing. The accumulator is released
    // once the MMAs issued have finished (one more bounded wait), so the
    // block holds no tensor memory when it returns; the host sees the flag.
    if (warp == 0) {
      if (!done_ok) mbar_wait(done, 0);
      __syncwarp();
      tc_fence_after();
      asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "n"(BN));
    }
    return;
  }
  tc_fence_after();

  // Accumulators -> shared memory (the pipeline buffers are free now), 128
  // columns at a time: warp w reads TMEM lanes 32 (w % 4) .. +31 (rows) and
  // columns 64 (w / 4) .. +63 of the half.
  float* stile = reinterpret_cast<float*>(gtiles);
#pragma unroll 1
  for (int h = 0; h < BN / 128; ++h) {
    if (h > 0) __syncthreads();   // the previous half has been stored
    {
      const int wq = warp & 3, col0 = (warp >> 2) * 64;
      const int r = wq * 32 + lane;
#pragma unroll
      for (int cc = 0; cc < 64; cc += 16) {
        uint32_t v[16];
        tmem_ld16(tmem + ((uint32_t)(wq * 32) << 16) + (uint32_t)(h * 128 + col0 + cc), v);
        float4* dst = reinterpret_cast<float4*>(stile + r * SLD + col0 + cc);
#pragma unroll
        for (int q = 0; q < 4; ++q)
          dst[q] = make_float4(__uint_as_float(v[4 * q]), __uint_as_float(v[4 * q + 1]), __uint_as_float(v[4 * q + 2]),
                               __uint_as_float(v[4 * q + 3]));
      }
    }
    tc_fence_before();
    __syncthreads();
    if (h == BN / 128 - 1 && warp == 0) {   // every tcgen05.ld has completed: release the accumulator
      tc_fence_after();
      asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "n"(BN));
    }
    if (EPI != EPI_F32 && e.vec) {
      // epilogue in row-contiguous order, 8 columns per thread: every global
      // access is 16 bytes, and the loads of 4 row groups are in flight
      // before the first is used (32,768 x 256 x 256 with bias, residual and two
      // BF16 outputs 22.6 -> 16.5 us). FP32 partials, which read nothing, go out
      // by the pairs below: eight columns a thread are two half-used 32-byte
      // sectors per store there (14.4 us against 16.6)
      constexpr int IT = (BM * 128 / 8) / THREADS, GROUP = 4;
#pragma unroll 1
      for (int it0 = 0; it0 < IT; it0 += GROUP) {
        float res[GROUP][8], aux[GROUP][8];
#pragma unroll
        for (int u = 0; u < GROUP; ++u) {
          const int q = (it0 + u) * THREADS + tid;
          const size_t o = (size_t)(m_blk + q / 16) * e.ldo + n_blk + h * 128 + (q % 16) * 8;
          if (e.res) load8<true>(e.res + o, res[u]);
          if (EPI == EPI_BWD && e.aux) load8<true>(e.aux + o, aux[u]);
        }
#pragma unroll
        for (int u = 0; u < GROUP; ++u) {
          const int q = (it0 + u) * THREADS + tid, r = q / 16, c = (q % 16) * 8;
          const int n = n_blk + h * 128 + c;
          const size_t o = (size_t)(m_blk + r) * e.ldo + n;
          const float4 a0 = *reinterpret_cast<const float4*>(stile + r * SLD + c);
          const float4 a1 = *reinterpret_cast<const float4*>(stile + r * SLD + c + 4);
          float v[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
          if (EPI == EPI_FWD) {
            const float4 b0 = *reinterpret_cast<const float4*>(e.bias + n);
            const float4 b1 = *reinterpret_cast<const float4*>(e.bias + n + 4);
            const float b[8] = {b0.x, b0.y, b0.z, b0.w, b1.x, b1.y, b1.z, b1.w};
            float hv[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) {
              v[i] += b[i];
              hv[i] = (e.res ? res[u][i] : 0.f) + fmaxf(v[i], 0.f);
            }
            store8<true>(e.out1 + o, v);
            store8<true>(static_cast<bf16*>(e.out0) + o, hv);
          } else {
            if (e.res)
#pragma unroll
              for (int i = 0; i < 8; ++i) v[i] += res[u][i];
            if (e.out0) store8<true>(static_cast<bf16*>(e.out0) + o, v);
            if (e.aux) {
#pragma unroll
              for (int i = 0; i < 8; ++i) v[i] = aux[u][i] > 0.f ? v[i] : 0.f;
              store8<true>(e.out1 + o, v);
            }
          }
        }
      }
      continue;
    }
    // FP32 partials, and buffers that are not 16-byte aligned: a warp covers 32 column pairs of one row
#pragma unroll 4
    for (int it = 0; it < (BM * 128 / 2) / THREADS; ++it) {
      const int q = it * THREADS + tid;
      const int r = q / 64, cp = q % 64;
      const int m = m_blk + r, n = n_blk + h * 128 + 2 * cp;
      const float2 acc = *reinterpret_cast<const float2*>(stile + r * SLD + 2 * cp);
      const float v0 = acc.x, v1 = acc.y;
      const size_t o = (size_t)m * e.ldo + n;
      if (EPI == EPI_F32) {
        float* out = static_cast<float*>(e.out0) + (size_t)blockIdx.z * e.split_stride;
        *reinterpret_cast<float2*>(out + o) = make_float2(v0, v1);
      } else if (EPI == EPI_FWD) {
        const float z0 = v0 + e.bias[n], z1 = v1 + e.bias[n + 1];
        float r0 = 0.f, r1 = 0.f;
        if (e.res) {
          const __nv_bfloat162 rr = *reinterpret_cast<const __nv_bfloat162*>(e.res + o);
          r0 = __bfloat162float(rr.x);
          r1 = __bfloat162float(rr.y);
        }
        *reinterpret_cast<__nv_bfloat162*>(e.out1 + o) = __floats2bfloat162_rn(z0, z1);
        *reinterpret_cast<__nv_bfloat162*>(static_cast<bf16*>(e.out0) + o) =
            __floats2bfloat162_rn(r0 + fmaxf(z0, 0.f), r1 + fmaxf(z1, 0.f));
      } else {
        float d0 = v0, d1 = v1;
        if (e.res) {
          const __nv_bfloat162 rr = *reinterpret_cast<const __nv_bfloat162*>(e.res + o);
          d0 += __bfloat162float(rr.x);
          d1 += __bfloat162float(rr.y);
        }
        if (e.out0)
          *reinterpret_cast<__nv_bfloat162*>(static_cast<bf16*>(e.out0) + o) = __floats2bfloat162_rn(d0, d1);
        if (e.aux) {
          const __nv_bfloat162 zz = *reinterpret_cast<const __nv_bfloat162*>(e.aux + o);
          *reinterpret_cast<__nv_bfloat162*>(e.out1 + o) = __floats2bfloat162_rn(
              __bfloat162float(zz.x) > 0.f ? d0 : 0.f, __bfloat162float(zz.y) > 0.f ? d1 : 0.f);
        }
      }
    }
  }
}

// ---- the whole network forward in one kernel: a CTA owns TILES x 128 rows and
// keeps their activations in shared memory from layer to layer.
//   A   per tile 128 x 256 BF16 activations, K-major with the 128-byte swizzle
//       (64 KB); layer l's MMAs read h_{l-1} there and its epilogue replaces
//       it by h_l
//   W   a ring of 64-wide K-blocks of the weights (32 KB each, by TMA), streamed
//       through for every layer of every tile
// One warp loads, one issues tcgen05.mma, 8 warps per tile read the
// accumulators back (warp w of a tile: rows 32 (w % 4) .., columns 128 (w / 4)
// ..), add bias and residual and round as the layer-by-layer GEMM does; the
// head ends in the summation order of k_head_fwd. Inference moves 272 B per
// row instead of 4.4 KB and is one launch instead of five; a training forward
// also writes h and z. Two tiles take turns: one's MMAs (2,400 cycles a layer)
// run while the other's epilogue (6,000; 15,000 with h and z on their way to
// memory) does. Inference of 25,984 rows takes 33 us and a training
// forward of 32,768 rows 55; 40 and 63 with both tiles in step and a head of
// 160 shuffles per 8 rows (14,400 of 61,000 cycles), 98 and 84 layer by layer.
struct MlpMaps { CUtensorMap x, w[4]; };
struct MlpNet {
  const float* b[4];
  const float *w4, *b4, *base;
  float* y;
  bf16 *h[4], *z[4];       // null: not kept
  int rows;
};
template <bool KEEP, int TILES>
struct Fwd {
  static constexpr int STAGES = TILES == 1 ? 4 : KEEP ? 2 : 3;
  static constexpr int W = TILES * 65536;                  // after the activations
  static constexpr int BARS = W + STAGES * 32768;          // X, done and ready per tile, full and empty per stage, TMEM address
  static constexpr int TURN = BARS + 128;                  // kept forward: 2 KB per warp to turn z's rows around
  static constexpr int SMEM = 1024 + TURN + (KEEP ? TILES * 8 * 2048 : 0);
  static constexpr int THREADS = TILES * 256 + 64;         // epilogues, MMA issuer, loader
  static_assert(SMEM <= 227 * 1024, "one CTA per SM");
};

// byte offset of (row, 8-column chunk c8) in a tile's swizzled activations
__device__ __forceinline__ uint32_t act_chunk(int row, int c8) {
  return (uint32_t)((c8 >> 3) * 16384 + row * 128 + (((c8 & 7) ^ (row & 7)) << 4));
}

template <bool KEEP, int TILES>
__global__ void __launch_bounds__((Fwd<KEEP, TILES>::THREADS)) k_mlp_fwd(const __grid_constant__ MlpMaps maps,
                                                                         const __grid_constant__ MlpNet net) {
  using C = Fwd<KEEP, TILES>;
  constexpr int S = C::STAGES;
  extern __shared__ unsigned char smem_raw[];
  const uint32_t raw = saddr(smem_raw), A = (raw + 1023u) & ~1023u, Wt = A + C::W;
  unsigned char* g = smem_raw + (A - raw);
  const uint32_t xfull = A + C::BARS, done = xfull + 8, ready = done + 8 * TILES, full = ready + 8 * TILES;
  const uint32_t empty = full + 8 * S;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(g + C::BARS + 112);
  __shared__ int s_abort;   // set when a wait gave up
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, m0 = blockIdx.x * (TILES * 128);
  if (tid == 0) {
    s_abort = 0;
    mbar_init(xfull, 1);
    for (int t = 0; t < TILES; ++t) {
      mbar_init(done + 8 * t, 1);
      mbar_init(ready + 8 * t, 8);
    }
    for (int k = 0; k < S; ++k) {
      mbar_init(full + 8 * k, 1);
      mbar_init(empty + 8 * k, 1);
    }
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(saddr(tmem_slot)),
                 "n"(TILES * 256));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  int issued = 0;   // K-blocks whose loads have been issued (loader)
  auto gave_up = [&]() { return *(volatile int*)&s_abort != 0; };
  if (warp == TILES * 8 + 1) {   // loader: X, then the K-blocks of every layer, tile by tile
    if (lane == 0) {
      mbar_expect_tx(xfull, TILES * 32768);
      for (int t = 0; t < TILES; ++t)
        for (int kb = 0; kb < 2; ++kb) tma_load_2d(A + t * 65536 + kb * 16384, &maps.x, kb * 64, m0 + t * 128, xfull);
      bool ok = true;
      for (int l = 0; l < 4 && ok; ++l)
        for (int i = 0; i < TILES * (l ? 4 : 2); ++i) {
          const int st = issued % S;
          if (issued >= S && (!mbar_wait(empty + 8 * st, (uint32_t)((issued / S - 1) & 1)) || gave_up())) {
            atomicOr(&s_abort, 1);
            ok = false;
            break;
          }
          mbar_expect_tx(full + 8 * st, 32768);
          tma_load_2d(Wt + st * 32768, &maps.w[l], (i & (l ? 3 : 1)) * 64, 0, full + 8 * st);
          ++issued;
        }
    }
    __syncwarp();
  } else if (warp == TILES * 8) {   // MMA issuer
    if (lane == 0) {
      constexpr uint32_t idesc = instr_desc<false, false, 256>();
      bool ok = mbar_wait(xfull, 0);
      int i = 0;
      for (int l = 0; l < 4; ++l)
        for (int t = 0; t < TILES; ++t) {
          // h_{l-1} is in place and the accumulator has been read
          if (ok && l > 0) ok = mbar_wait(ready + 8 * t, (uint32_t)((l - 1) & 1)) && !gave_up();
          tc_fence_after();
          for (int kb = 0; kb < (l ? 4 : 2) && ok; ++kb, ++i) {
            const int st = i % S;
            ok = mbar_wait(full + 8 * st, (uint32_t)((i / S) & 1));
            if (!ok) break;
            tc_fence_after();
#pragma unroll
            for (int j = 0; j < 4; ++j)
              umma(tmem + t * 256, smem_desc(A + t * 65536 + kb * 16384 + j * 32, 16, 1024),
                   smem_desc(Wt + st * 32768 + j * 32, 16, 1024), idesc, (kb | j) != 0);
            umma_commit(empty + 8 * st);
          }
          if (!ok) {
            atomicOr(&s_abort, 1);
            __threadfence_block();
          }
          umma_commit(done + 8 * t);   // completes once every MMA issued so far has
        }
    }
    __syncwarp();
  } else {
    const int t = warp >> 3;
#pragma unroll 1
    for (int l = 0; l < 4; ++l) {
      if (!mbar_wait(done + 8 * t, (uint32_t)(l & 1))) atomicOr(&s_abort, 1);
      if (__any_sync(0xffffffffu, gave_up())) break;
      tc_fence_after();
      const int row = (warp & 3) * 32 + lane, col0 = ((warp >> 2) & 1) * 128;
      const uint32_t acc = tmem + (uint32_t)(t * 256) + ((uint32_t)((warp & 3) * 32) << 16);
      unsigned char* act = g + t * 65536;
      unsigned char* turn = g + C::TURN + warp * 2048;
      const float* bias = net.b[l];
      const bool stored = KEEP && m0 + t * 128 < net.rows;
#pragma unroll 1
      for (int c32 = col0; c32 < col0 + 128; c32 += 32) {
        // everything the chunk needs is requested before the one wait (36 -> 33 us, 58 -> 55)
        uint32_t v[32];
        tmem_ld32(acc + (uint32_t)c32, v);
        uint4 res[4];
        float4 bv[8];
#pragma unroll
        for (int p = 0; p < 4; ++p) {
          if (l > 0) res[p] = *reinterpret_cast<const uint4*>(act + act_chunk(row, (c32 >> 3) + p));
          bv[2 * p] = __ldg(reinterpret_cast<const float4*>(bias + c32) + 2 * p);
          bv[2 * p + 1] = __ldg(reinterpret_cast<const float4*>(bias + c32) + 2 * p + 1);
        }
        tmem_wait(v);
#pragma unroll
        for (int p = 0; p < 4; ++p) {
          const int c = c32 + 8 * p;
          bf16* a = reinterpret_cast<bf16*>(act + act_chunk(row, c >> 3));
          const float4 b0 = bv[2 * p], b1 = bv[2 * p + 1];
          const float b[8] = {b0.x, b0.y, b0.z, b0.w, b1.x, b1.y, b1.z, b1.w};
          float zv[8], hv[8];
          if (l > 0) load8<true>(reinterpret_cast<const bf16*>(&res[p]), hv);
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            zv[i] = __uint_as_float(v[8 * p + i]) + b[i];
            hv[i] = (l > 0 ? hv[i] : 0.f) + fmaxf(zv[i], 0.f);
          }
          store8<true>(a, hv);
          if (KEEP) store8<true>(reinterpret_cast<bf16*>(turn + lane * 64 + ((p ^ ((lane >> 1) & 3)) << 4)), zv);
        }
        if (KEEP) {
          // 32 rows x 32 columns of this warp, eight rows (64 B each) per store:
          // a lane writing its own row would touch 32 lines at a time
          __syncwarp();
          if (stored) {
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              const int r = q * 8 + (lane >> 2), ch = lane & 3, gr = (warp & 3) * 32 + r;
              const size_t o = (size_t)(m0 + t * 128 + gr) * 256 + c32 + ch * 8;
              *reinterpret_cast<uint4*>(net.z[l] + o) =
                  *reinterpret_cast<const uint4*>(turn + r * 64 + ((ch ^ ((r >> 1) & 3)) << 4));
              *reinterpret_cast<uint4*>(net.h[l] + o) =
                  *reinterpret_cast<const uint4*>(act + act_chunk(gr, (c32 >> 3) + ch));
            }
          }
          __syncwarp();
        }
      }
      tc_fence_before();
      asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");   // h_l before the next layer's MMAs read it
      __syncwarp();
      if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(ready + 8 * t) : "memory");
    }
    // h_3 of the tile is in place once its 8 warps are here
    asm volatile("bar.sync %0, 256;\n" ::"r"(1 + t) : "memory");
    // head: a warp sums 16 rows, 8 at a time; a lane the columns lane + 32 i in
    // order. The 32 sums over lanes of a pass (8 rows x 4 outputs) halve their
    // number at each step of the butterfly (31 shuffles instead of 160; the
    // pairs added are those of k_head_fwd), so that each lane ends with one.
    if (!__any_sync(0xffffffffu, gave_up())) {
      float2 w01[8], w23[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int c = lane + 32 * i;
        w01[i] = make_float2(net.w4[c], net.w4[256 + c]);
        w23[i] = make_float2(net.w4[512 + c], net.w4[768 + c]);
      }
      const float bias = net.b4[lane & 3];
      const unsigned char* act = g + t * 65536;
#pragma unroll 1
      for (int q = 0; q < 16; q += 8) {
        float s[32];   // row q + (k >> 2), output k & 3
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          const int r = (warp & 7) * 16 + q + k;
          float2 a = make_float2(0.f, 0.f), b = a;
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const int c = lane + 32 * i;
            const float v = __bfloat162float(reinterpret_cast<const bf16*>(act + act_chunk(r, c >> 3))[c & 7]);
            a = __ffma2_rn(make_float2(v, v), w01[i], a);
            b = __ffma2_rn(make_float2(v, v), w23[i], b);
          }
          s[4 * k] = a.x; s[4 * k + 1] = a.y; s[4 * k + 2] = b.x; s[4 * k + 3] = b.y;
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
          const bool up = (lane & o) != 0;   // keeps the upper half of the sums
#pragma unroll
          for (int k = 0; k < o; ++k) {
            const float keep = up ? s[k + o] : s[k], send = up ? s[k] : s[k + o];
            s[k] = keep + __shfl_xor_sync(0xffffffffu, send, o);
          }
        }
        const long long row = m0 + t * 128 + (warp & 7) * 16 + q + (lane >> 2);
        if (row < net.rows)
          net.y[row * 4 + (lane & 3)] = s[0] + bias + (net.base ? net.base[row * 4 + (lane & 3)] : 0.f);
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (s_abort) {
    // A wait gave up: the outputs are not complete and the host sees the flag.
    // Loads still landing in shared memory and the MMAs issued get a bounded
    // wait each, the accumulators are released.
    if (warp == TILES * 8 + 1 && lane == 0) {
      mbar_wait(xfull, 0);
      for (int j = max(0, issued - S); j < issued; ++j) mbar_wait(full + 8 * (j % S), (uint32_t)((j / S) & 1));
    }
    if (warp == 0)
      for (int t = 0; t < TILES; ++t) mbar_wait(done + 8 * t, 1);   // the last layer's commit
    __syncthreads();
  }
  if (warp == 0) {   // every tcgen05.ld has completed
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "n"(TILES * 256));
  }
}

// ---- the weight and bias gradients of the four layers in one launch:
// dW_l = dz_l^T src_l (src_0 = X, src_l = h_{l-1}) as `splits` partials, each
// one accumulator over an equal range of rows, and db_l = sum of dz_l's rows
// as partials of 256 rows, row by row: the sums and their order are those of
// one split-K GEMM and one column sum per layer, bit for bit. A CTA owns one
// 128 x 128 tile of one layer's dW (14 tiles) and up to four ranges, each with
// an accumulator of its own, so that a launch's start is paid once and one
// range's partial goes out while the next one's MMAs run. Warp 1 loads, warp 0
// issues the MMAs, warps 2-3 of the tiles with n = 0 add up dz's columns from
// the same shared-memory tiles (no pass of their own over dz), warps 4-7 write
// the partials. Bound by the operands' way through L2 (134 MB,
// twice) and the partials (33 MB) at 32,768 rows: 43 us, against four GEMMs of
// 16 us and 19 us of column sums.
constexpr int WG_TILES = 14, WG_STAGES = 4, WG_ACC = 4;
struct WgradMaps { CUtensorMap dz[4], src[4]; };
struct WgradOut { float *dw[4], *db; };   // dw[l]: splits x 256 x (l ? 256 : 128); db: 4 x blocks of 256 rows x 256, or null
struct Wg {
  static constexpr int STAGE_BYTES = 32768;
  static constexpr int TILE = WG_STAGES * STAGE_BYTES;    // 4 x 32 rows of a partial on their way out
  static constexpr int BARS = TILE + BM * SLD * 4;        // full and empty per stage, done per accumulator, TMEM address
  static constexpr int SMEM = 1024 + BARS + 128;
  static_assert(SMEM <= 227 * 1024 && 2 * SMEM > 227 * 1024, "one CTA per SM: it takes all of TMEM");
};

__global__ void __launch_bounds__(THREADS) k_mlp_wgrad(const __grid_constant__ WgradMaps maps, const WgradOut out,
                                                       int rows, int splits, int per_cta) {
  extern __shared__ unsigned char smem_raw[];
  const uint32_t raw = saddr(smem_raw), tiles = (raw + 1023u) & ~1023u;
  unsigned char* g = smem_raw + (tiles - raw);
  const uint32_t full = tiles + Wg::BARS, empty = full + 8 * WG_STAGES, done = empty + 8 * WG_STAGES;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(g + Wg::BARS + 112);
  __shared__ int s_abort;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int t = blockIdx.x, l = t < 12 ? 1 + (t >> 2) : 0;
  const int m_blk = (t < 12 ? (t >> 1) & 1 : t - 12) * BM, n_blk = t < 12 ? (t & 1) * 128 : 0, kin = l ? 256 : 128;
  const int c0 = blockIdx.y * per_cta, nc = min(per_cta, splits - c0);   // this CTA's ranges
  const int KC = rows / splits / BK, kb0 = c0 * KC, KT = nc * KC;
  const bool bias = n_blk == 0 && out.db != nullptr;
  if (tid == 0) {
    s_abort = 0;
    for (int s = 0; s < WG_STAGES; ++s) {
      mbar_init(full + 8 * s, 1);
      mbar_init(empty + 8 * s, bias ? 3 : 1);   // the MMAs, and the two summing warps
    }
    for (int q = 0; q < WG_ACC; ++q) mbar_init(done + 8 * q, 1);
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(saddr(tmem_slot)),
                 "n"(WG_ACC * 128));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;

  int issued = 0;   // K-blocks whose loads have been issued (warp 1)
  if (warp == 1) {
    if (lane == 0) {
      for (; issued < KT; ++issued) {
        const int s = issued % WG_STAGES, k0 = (kb0 + issued) * BK;
        if (issued >= WG_STAGES && !mbar_wait(empty + 8 * s, (uint32_t)((issued / WG_STAGES - 1) & 1))) {
          atomicOr(&s_abort, 1);
          break;
        }
        const uint32_t a = tiles + s * Wg::STAGE_BYTES, bar = full + 8 * s;
        mbar_expect_tx(bar, Wg::STAGE_BYTES);
        for (int q = 0; q < 2; ++q) {
          tma_load_2d(a + q * 8192, &maps.dz[l], m_blk + 64 * q, k0, bar);
          tma_load_2d(a + 16384 + q * 8192, &maps.src[l], n_blk + 64 * q, k0, bar);
        }
      }
    }
    __syncwarp();
  } else if (warp == 0) {
    if (lane == 0) {
      constexpr uint32_t idesc = instr_desc<true, true, 128>();
      int kt = 0;
      bool ok = true;
      for (int q = 0; q < nc; ++q) {
        for (int k = 0; k < KC && ok; ++k, ++kt) {
          const int s = kt % WG_STAGES;
          if (!mbar_wait(full + 8 * s, (uint32_t)((kt / WG_STAGES) & 1))) {
            atomicOr(&s_abort, 1);
            __threadfence_block();
            ok = false;
            break;
          }
          tc_fence_after();
          const uint32_t a = tiles + s * Wg::STAGE_BYTES, b = a + 16384;
#pragma unroll
          for (int j = 0; j < BK / 16; ++j)
            umma(tmem + (uint32_t)(q * 128), smem_desc(a + j * 2048, 8192, 1024), smem_desc(b + j * 2048, 8192, 1024),
                 idesc, (k | j) != 0);
          umma_commit(empty + 8 * s);
        }
        umma_commit(done + 8 * q);   // its one phase completes when every MMA issued so far has
      }
    }
    __syncwarp();
  } else if (warp < 4) {
    if (bias) {
      // a thread adds two columns row by row; a warp reads the 128 bytes of one row
      const int u = tid - 64, nblk = (rows + 255) / 256;
      const unsigned char* col = g + (u >> 5) * 8192 + (u & 3) * 4;
      float s0 = 0.f, s1 = 0.f;
      for (int kt = 0; kt < KT; ++kt) {
        const int s = kt % WG_STAGES;
        if (!mbar_wait(full + 8 * s, (uint32_t)((kt / WG_STAGES) & 1))) { atomicOr(&s_abort, 1); break; }
        const unsigned char* p = col + s * Wg::STAGE_BYTES;
        uint32_t v[BK];   // all on their way before the chain of additions
#pragma unroll
        for (int k = 0; k < BK; ++k)
          v[k] = *reinterpret_cast<const uint32_t*>(p + (k >> 3) * 1024 + (k & 7) * 128 + ((((u >> 2) & 7) ^ (k & 7)) << 4));
        __syncwarp();
        if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(empty + 8 * s) : "memory");
#pragma unroll
        for (int k = 0; k < BK; ++k) {
          s0 += __uint_as_float(v[k] << 16);
          s1 += __uint_as_float(v[k] & 0xFFFF0000u);
        }
        const int kb = kb0 + kt;
        if ((kb & 3) == 3 || kb == rows / BK - 1) {
          *reinterpret_cast<float2*>(out.db + ((size_t)l * nblk + (kb >> 2)) * 256 + m_blk + 2 * u) = make_float2(s0, s1);
          s0 = s1 = 0.f;
        }
      }
    }
  } else {
    const int wq = warp & 3;
    float* stile = reinterpret_cast<float*>(g + Wg::TILE) + wq * 32 * SLD;
    for (int q = 0; q < nc; ++q) {
      if (!mbar_wait(done + 8 * q, 0)) atomicOr(&s_abort, 1);
      if (__any_sync(0xffffffffu, *(volatile int*)&s_abort)) break;
      tc_fence_after();
#pragma unroll 2
      for (int cc = 0; cc < 128; cc += 16) {
        uint32_t v[16];
        tmem_ld16(tmem + ((uint32_t)(wq * 32) << 16) + (uint32_t)(q * 128 + cc), v);
        uint4* dst = reinterpret_cast<uint4*>(stile + lane * SLD + cc);
#pragma unroll
        for (int i = 0; i < 4; ++i) dst[i] = make_uint4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
      }
      __syncwarp();
      float* dw = out.dw[l] + ((size_t)(c0 + q) * 256 + m_blk + wq * 32) * kin + n_blk + lane * 4;
#pragma unroll 8
      for (int r = 0; r < 32; ++r)
        *reinterpret_cast<float4*>(dw + (size_t)r * kin) = *reinterpret_cast<const float4*>(stile + r * SLD + lane * 4);
      __syncwarp();
    }
    tc_fence_before();
  }
  __syncthreads();
  // A wait gave up: loads that may still be landing and the MMAs issued get a
  // bounded wait each; the partials are not complete and the host sees the flag.
  if (s_abort) {
    if (warp == 1 && lane == 0)
      for (int j = max(0, issued - WG_STAGES); j < issued; ++j)
        mbar_wait(full + 8 * (j % WG_STAGES), (uint32_t)((j / WG_STAGES) & 1));
    if (warp == 0) mbar_wait(done + 8 * (nc - 1), 0);
    __syncthreads();
  }
  if (warp == 0) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "n"(WG_ACC * 128));
  }
}

}  // namespace tc

int mfail(int code, const std::string& msg) { return esr::report_error(code, msg); }

// Raises KERNEL's dynamic shared-memory limit on the current device
template <auto KERNEL>
cudaError_t allow_smem(int bytes) {
  static PerDevice set;
  int device = 0;
  const cudaError_t err = cudaGetDevice(&device);
  if (err != cudaSuccess) return err;
  return (cudaError_t)set.once(device, [&](int) {
    return (int)cudaFuncSetAttribute(KERNEL, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  });
}

template <bool AT, bool BT, int EPI>
int launch_gemm(int M, int N, int K, int splits, const bf16* A, int lda, const bf16* B, int ldb, const Epi& e,
                cudaStream_t st) {
  constexpr int A_ELEMS = AT ? BK * LD_MN : BM * LD_K;
  constexpr int B_ELEMS = BT ? BK * LD_MN : BN * LD_K;
  const int smem = STAGES * (A_ELEMS + B_ELEMS) * (int)sizeof(bf16);
  const cudaError_t err = allow_smem<&k_gemm<AT, BT, EPI>>(smem);
  if (err != cudaSuccess) return mfail(ESR_ERR_CUDA, std::string("gemm: ") + cudaGetErrorString(err));
  dim3 grid(N / BN, M / BM, splits);
  k_gemm<AT, BT, EPI><<<grid, THREADS, smem, st>>>(M, N, K / splits, A, lda, B, ldb, e);
  return ESR_OK;
}

// 2-D BF16 tensor map: `inner` contiguous elements per row, `outer` rows,
// rows `ld` elements apart; boxes of box_in x box_out with the 128-byte swizzle
// the UMMA descriptors expect
int make_map(CUtensorMap* map, const bf16* base, uint64_t inner, uint64_t outer, uint64_t ld, uint32_t box_in,
             uint32_t box_out) {
  static PFN_cuTensorMapEncodeTiled_v12000 encode = nullptr;
  if (!encode) {
    cudaDriverEntryPointQueryResult q{};
    void* fn = nullptr;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess || !fn)
      return mfail(ESR_ERR_CUDA, "gemm: cuTensorMapEncodeTiled is not available");
    encode = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(fn);
  }
  const cuuint64_t dims[2] = {inner, outer};
  const cuuint64_t strides[1] = {ld * sizeof(bf16)};
  const cuuint32_t box[2] = {box_in, box_out};
  const cuuint32_t estr[2] = {1, 1};
  const CUresult r = encode(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<bf16*>(base), dims, strides, box, estr,
                            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                            CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return mfail(ESR_ERR_ARG, "gemm: tensor map rejected (error " + std::to_string((int)r) + ")");
  return ESR_OK;
}

template <bool AT, bool BT, int EPI>
int launch_gemm_tc(int M, int N, int K, int splits, const bf16* A, int lda, const bf16* B, int ldb, const Epi& e,
                   cudaStream_t st) {
  // 256-wide tiles (A read once per row block) when there are still enough
  // of them to give every SM one; otherwise 128-wide tiles for parallelism
  const int tbn = (N % 256 == 0 && (long long)(M / tc::BM) * (N / 256) * splits >= 148) ? 256 : 128;
  CUtensorMap ma, mb;
  int rc = AT ? make_map(&ma, A, M, K, lda, 64, 64) : make_map(&ma, A, K, M, lda, 64, tc::BM);
  if (rc != ESR_OK) return rc;
  rc = BT ? make_map(&mb, B, N, K, ldb, 64, 64) : make_map(&mb, B, K, N, ldb, 64, tbn);
  if (rc != ESR_OK) return rc;
  const cudaError_t err = tbn == 256 ? allow_smem<&tc::k_gemm_tc<AT, BT, EPI, 256>>(tc::Cfg<256>::SMEM)
                                     : allow_smem<&tc::k_gemm_tc<AT, BT, EPI, 128>>(tc::Cfg<128>::SMEM);
  if (err != cudaSuccess) return mfail(ESR_ERR_CUDA, std::string("gemm: ") + cudaGetErrorString(err));
  if (tbn == 256) {
    dim3 grid(N / 256, M / tc::BM, splits);
    tc::k_gemm_tc<AT, BT, EPI, 256><<<grid, tc::THREADS, tc::Cfg<256>::SMEM, st>>>(M, N, K / splits, ma, mb, e);
  } else {
    dim3 grid(N / 128, M / tc::BM, splits);
    tc::k_gemm_tc<AT, BT, EPI, 128><<<grid, tc::THREADS, tc::Cfg<128>::SMEM, st>>>(M, N, K / splits, ma, mb, e);
  }
  return ESR_OK;
}

template <bool KEEP, int TILES>
int launch_fwd(const tc::MlpMaps& maps, const tc::MlpNet& n, void* stream) {
  using C = tc::Fwd<KEEP, TILES>;
  const cudaError_t attr = allow_smem<&tc::k_mlp_fwd<KEEP, TILES>>(C::SMEM);
  if (attr != cudaSuccess) return mfail(ESR_ERR_CUDA, std::string("mlp_forward: ") + cudaGetErrorString(attr));
  tc::k_mlp_fwd<KEEP, TILES><<<(n.rows / 128 + TILES - 1) / TILES, C::THREADS, C::SMEM, (cudaStream_t)stream>>>(maps, n);
  return ESR_OK;
}

}  // namespace

extern "C" {

// C = A * B with the epilogue `epi` (0 F32 split-K partials, 1 forward, 2 backward).
// trans_a: A stored [K][M] (lda >= M); else [M][K] (lda >= K).
// trans_b: B stored [K][N] (ldb >= N); else [N][K] (ldb >= K).
// M, N multiples of 128; K a multiple of 32 * splits; rows 16-byte aligned.
namespace {
// argument checks shared by both GEMM paths; bk = K granularity of the kernel
int gemm_check(int32_t trans_a, int32_t trans_b, int32_t M, int32_t N, int32_t K, const void* A, int32_t lda,
               const void* B, int32_t ldb, int32_t epi, const float* bias, const void* aux, void* out0, void* out1,
               int32_t ldo, int32_t splits, int bk) {
  if (!A || !B || !out0) return mfail(ESR_ERR_ARG, "gemm: null operand");
  if (M <= 0 || N <= 0 || K <= 0 || M % BM || N % BN) return mfail(ESR_ERR_ARG, "gemm: M and N must be multiples of 128");
  if (splits < 1 || K % (bk * splits))
    return mfail(ESR_ERR_ARG, "gemm: K must be a multiple of " + std::to_string(bk) + " x splits");
  if (lda % 8 || ldb % 8 || ldo % 2) return mfail(ESR_ERR_ARG, "gemm: leading dimensions must keep 16-byte rows");
  if ((trans_a ? lda < M : lda < K) || (trans_b ? ldb < N : ldb < K) || ldo < N)
    return mfail(ESR_ERR_ARG, "gemm: leading dimension too small");
  if (((uintptr_t)A | (uintptr_t)B) & 15) return mfail(ESR_ERR_ARG, "gemm: operands must be 16-byte aligned");
  if (epi == EPI_FWD && (!bias || !out1)) return mfail(ESR_ERR_ARG, "gemm: forward epilogue needs bias and z output");
  if (epi == EPI_BWD && aux && !out1) return mfail(ESR_ERR_ARG, "gemm: backward epilogue with z needs dz output");
  if (epi != EPI_F32 && splits != 1) return mfail(ESR_ERR_ARG, "gemm: split-K only with the F32 epilogue");
  return ESR_OK;
}
}  // namespace

int esr_gemm_bf16(int32_t trans_a, int32_t trans_b, int32_t M, int32_t N, int32_t K, const void* A, int32_t lda,
                  const void* B, int32_t ldb, int32_t epi, const float* bias, const void* res, const void* aux,
                  void* out0, void* out1, int32_t ldo, int32_t splits, void* stream) {
  int rc = gemm_check(trans_a, trans_b, M, N, K, A, lda, B, ldb, epi, bias, aux, out0, out1, ldo, splits, tc::BK);
  if (rc != ESR_OK) return rc;
  // rows and buffers aligned for the 16-byte epilogue (a null one is not touched)
  const bool vec = ldo % 8 == 0 && aligned16(bias) && aligned16(res) && aligned16(aux) && aligned16(out0) && aligned16(out1);
  Epi e{bias, (const bf16*)res, (const bf16*)aux, out0, (bf16*)out1, ldo, (long long)M * ldo, vec};
  cudaStream_t st = (cudaStream_t)stream;
  const bf16* a = (const bf16*)A;
  const bf16* b = (const bf16*)B;
#define ESR_GEMM_CASE(TA, TB, E) \
  if (!!trans_a == TA && !!trans_b == TB && epi == E) rc = launch_gemm_tc<TA, TB, E>(M, N, K, splits, a, lda, b, ldb, e, st); else
  ESR_GEMM_CASE(false, false, EPI_FWD)
  ESR_GEMM_CASE(false, true, EPI_BWD)
  ESR_GEMM_CASE(true, true, EPI_F32)
  ESR_GEMM_CASE(false, false, EPI_F32)
  ESR_GEMM_CASE(false, true, EPI_F32)
  ESR_GEMM_CASE(false, false, EPI_BWD)
  return mfail(ESR_ERR_ARG, "gemm: unsupported layout/epilogue combination");
#undef ESR_GEMM_CASE
  if (rc != ESR_OK) return rc;
  cudaError_t err = cudaGetLastError();
  return err == cudaSuccess ? ESR_OK : mfail(ESR_ERR_CUDA, std::string("gemm: ") + cudaGetErrorString(err));
}

int esr_mlp_forward(const esr_mlp_net* net, const void* X, int32_t rows, const float* base, float* y,
                    void* const* h, void* const* z, void* stream) {
  if (!net || !X || !y || rows <= 0 || rows % 128) return mfail(ESR_ERR_ARG, "mlp_forward: rows must be a multiple of 128");
  if ((h == nullptr) != (z == nullptr)) return mfail(ESR_ERR_ARG, "mlp_forward: h and z are kept together");
  for (int l = 0; l < 4; ++l) {
    if (!net->W[l] || !net->b[l] || (h && (!h[l] || !z[l]))) return mfail(ESR_ERR_ARG, "mlp_forward: null operand");
    if (!aligned16(net->W[l]) || !aligned16(net->b[l]) || (h && (!aligned16(h[l]) || !aligned16(z[l]))))
      return mfail(ESR_ERR_ARG, "mlp_forward: operands must be 16-byte aligned");
  }
  if (!net->W4 || !net->b4 || !aligned16(X)) return mfail(ESR_ERR_ARG, "mlp_forward: bad operand");
  tc::MlpMaps maps;
  int rc = make_map(&maps.x, (const bf16*)X, 128, rows, 128, 64, 128);
  for (int l = 0; l < 4 && rc == ESR_OK; ++l) {
    const uint64_t k = l == 0 ? 128 : 256;
    rc = make_map(&maps.w[l], (const bf16*)net->W[l], k, 256, k, 64, 256);
  }
  if (rc != ESR_OK) return rc;
  tc::MlpNet n{};
  for (int l = 0; l < 4; ++l) {
    n.b[l] = net->b[l];
    n.h[l] = h ? (bf16*)h[l] : nullptr;
    n.z[l] = z ? (bf16*)z[l] : nullptr;
  }
  n.w4 = net->W4;
  n.b4 = net->b4;
  n.base = base;
  n.y = y;
  n.rows = rows;
  // One tile per CTA while every tile gets an SM of its own; beyond that two
  // tiles per CTA, which take turns (a second round of CTAs would start over).
  const bool two = rows / 128 > 148;
  if (h) rc = two ? launch_fwd<true, 2>(maps, n, stream) : launch_fwd<true, 1>(maps, n, stream);
  else rc = two ? launch_fwd<false, 2>(maps, n, stream) : launch_fwd<false, 1>(maps, n, stream);
  if (rc != ESR_OK) return rc;
  cudaError_t err = cudaGetLastError();
  return err == cudaSuccess ? ESR_OK : mfail(ESR_ERR_CUDA, std::string("mlp_forward: ") + cudaGetErrorString(err));
}

int esr_mlp_wgrad(const void* const* dz, const void* const* src, int32_t rows, int32_t splits, float* const* dw, float* db,
                  void* stream) {
  if (!dz || !src || !dw || rows <= 0 || rows % 128)
    return mfail(ESR_ERR_ARG, "mlp_wgrad: rows must be a multiple of 128");
  if (splits < 1 || splits > 65535 || rows % (tc::BK * (int64_t)splits))
    return mfail(ESR_ERR_ARG, "mlp_wgrad: rows must be a multiple of 64 x splits");
  if (db && (splits > 1 && rows / splits % 256 || !aligned16(db)))
    return mfail(ESR_ERR_ARG, "mlp_wgrad: column sums need splits of whole 256-row blocks");
  tc::WgradMaps maps;
  tc::WgradOut out{};
  out.db = db;
  for (int l = 0; l < 4; ++l) {
    if (!dz[l] || !src[l] || !dw[l]) return mfail(ESR_ERR_ARG, "mlp_wgrad: null operand");
    if (!aligned16(dz[l]) || !aligned16(src[l]) || !aligned16(dw[l]))
      return mfail(ESR_ERR_ARG, "mlp_wgrad: operands must be 16-byte aligned");
    const uint64_t kin = l == 0 ? 128 : 256;
    int rc = make_map(&maps.dz[l], (const bf16*)dz[l], 256, rows, 256, 64, 64);
    if (rc == ESR_OK) rc = make_map(&maps.src[l], (const bf16*)src[l], kin, rows, kin, 64, 64);
    if (rc != ESR_OK) return rc;
    out.dw[l] = dw[l];
  }
  const cudaError_t attr = allow_smem<&tc::k_mlp_wgrad>(tc::Wg::SMEM);
  if (attr != cudaSuccess) return mfail(ESR_ERR_CUDA, std::string("mlp_wgrad: ") + cudaGetErrorString(attr));
  // as many ranges per CTA as keep the launch to one CTA per SM, at most one per accumulator
  const int per = std::min(tc::WG_ACC, (splits + 148 / tc::WG_TILES - 1) / (148 / tc::WG_TILES));
  tc::k_mlp_wgrad<<<dim3(tc::WG_TILES, (splits + per - 1) / per), tc::THREADS, tc::Wg::SMEM, (cudaStream_t)stream>>>(
      maps, out, rows, splits, per);
  cudaError_t err = cudaGetLastError();
  return err == cudaSuccess ? ESR_OK : mfail(ESR_ERR_CUDA, std::string("mlp_wgrad: ") + cudaGetErrorString(err));
}

int esr_gemm_bf16_mma_sync(int32_t trans_a, int32_t trans_b, int32_t M, int32_t N, int32_t K, const void* A,
                           int32_t lda, const void* B, int32_t ldb, int32_t epi, const float* bias, const void* res,
                           const void* aux, void* out0, void* out1, int32_t ldo, int32_t splits, void* stream) {
  int rc = gemm_check(trans_a, trans_b, M, N, K, A, lda, B, ldb, epi, bias, aux, out0, out1, ldo, splits, BK);
  if (rc != ESR_OK) return rc;
  Epi e{bias, (const bf16*)res, (const bf16*)aux, out0, (bf16*)out1, ldo, (long long)M * ldo, false};
  cudaStream_t st = (cudaStream_t)stream;
  const bf16* a = (const bf16*)A;
  const bf16* b = (const bf16*)B;
#define ESR_GEMM_CASE(TA, TB, E) \
  if (!!trans_a == TA && !!trans_b == TB && epi == E) rc = launch_gemm<TA, TB, E>(M, N, K, splits, a, lda, b, ldb, e, st); else
  ESR_GEMM_CASE(false, false, EPI_FWD)
  ESR_GEMM_CASE(false, true, EPI_BWD)
  ESR_GEMM_CASE(true, true, EPI_F32)
  ESR_GEMM_CASE(false, false, EPI_F32)
  ESR_GEMM_CASE(false, true, EPI_F32)
  ESR_GEMM_CASE(false, false, EPI_BWD)
  return mfail(ESR_ERR_ARG, "gemm: unsupported layout/epilogue combination");
#undef ESR_GEMM_CASE
  if (rc != ESR_OK) return rc;
  cudaError_t err = cudaGetLastError();
  return err == cudaSuccess ? ESR_OK : mfail(ESR_ERR_CUDA, std::string("gemm: ") + cudaGetErrorString(err));
}

int esr_gemm_tc_status(int32_t* gave_up) {
  if (!gave_up) return mfail(ESR_ERR_ARG, "gemm_tc_status: null output");
  int v = 0;
  const int zero = 0;
  cudaError_t err = cudaMemcpyFromSymbol(&v, tc::g_tc_error, sizeof(int));
  if (err == cudaSuccess) err = cudaMemcpyToSymbol(tc::g_tc_error, &zero, sizeof(int));
  if (err != cudaSuccess) return mfail(ESR_ERR_CUDA, std::string("gemm_tc_status: ") + cudaGetErrorString(err));
  *gave_up = v;
  return ESR_OK;
}

// 4-wide head: y = H W^T + b (+ base); H [rows x K] BF16, W [4 x K] FP32
int esr_mlp_head_fwd(const void* H, int32_t rows, int32_t K, const float* W, const float* b, const float* base,
                     float* y, void* stream) {
  if (!H || !W || !b || !y || rows <= 0 || K <= 0) return mfail(ESR_ERR_ARG, "head_fwd: bad argument");
  const int wpb = 8;
  if (K == 256)   // four rows per warp and pass, two resident blocks per SM
    k_head_fwd256<<<std::min((rows + 4 * wpb - 1) / (4 * wpb), 148 * 2), wpb * 32, 0, (cudaStream_t)stream>>>(
        (const bf16*)H, rows, W, b, base, y);
  else
    k_head_fwd<<<(rows + wpb - 1) / wpb, wpb * 32, 0, (cudaStream_t)stream>>>((const bf16*)H, rows, K, W, b, base, y);
  cudaError_t err = cudaGetLastError();
  return err == cudaSuccess ? ESR_OK : mfail(ESR_ERR_CUDA, cudaGetErrorString(err));
}

// head backward: dH = dY W and dZ = dH * (z > 0) (BF16), dW/db partials per
// block of `rpb` rows (4*K + 4 floats per block)
int esr_mlp_head_bwd(const float* dY, const void* H, const void* Z, int32_t rows, int32_t K, const float* W, void* dH,
                     void* dZ, float* part, int32_t rpb, void* stream) {
  if (!dY || !H || !Z || !W || !dH || !dZ || !part || rows <= 0 || K != 256 || rpb <= 0)
    return mfail(ESR_ERR_ARG, "head_bwd: bad argument");
  cudaStream_t st = (cudaStream_t)stream;
  auto* k = (((uintptr_t)H | (uintptr_t)Z | (uintptr_t)dH | (uintptr_t)dZ) & 3) == 0 ? k_head_bwd<true> : k_head_bwd<false>;
  k<<<(rows + rpb - 1) / rpb, 128 * kHeadGroups, 0, st>>>(dY, (const bf16*)H, (const bf16*)Z, rows, W, (bf16*)dH, (bf16*)dZ, rpb, part);
  cudaError_t err = cudaGetLastError();
  return err == cudaSuccess ? ESR_OK : mfail(ESR_ERR_CUDA, cudaGetErrorString(err));
}

int esr_mlp_features(const float* stat5, const float* idw_prim, const float* idw_gradp, int32_t rows, float mach_n,
                     float aoa_n, const float* mu, const float* sig, int32_t ld, void* X, float* base, void* stream) {
  if (!stat5 || !idw_prim || !idw_gradp || !mu || !sig || !X || rows <= 0 || ld < 13)
    return mfail(ESR_ERR_ARG, "features: bad argument");
  k_features<<<(rows + kFeatureRows - 1) / kFeatureRows, kFeatureRows, 0, (cudaStream_t)stream>>>(
      stat5, idw_prim, idw_gradp, rows, mach_n, aoa_n, mu, sig, ld, (bf16*)X, base, ld % 8 == 0 && aligned16(X));
  cudaError_t err = cudaGetLastError();
  return err == cudaSuccess ? ESR_OK : mfail(ESR_ERR_CUDA, cudaGetErrorString(err));
}

int esr_mlp_decode(const float* pred_n, int32_t rows, const float* mu, const float* sig, float gamma, float rho_floor,
                   float p_floor, double* W, void* stream) {
  if (!pred_n || !mu || !sig || !W || rows <= 0) return mfail(ESR_ERR_ARG, "decode: bad argument");
  k_decode<<<(rows + 127) / 128, 128, 0, (cudaStream_t)stream>>>(pred_n, rows, mu, sig, gamma, rho_floor, p_floor, W);
  cudaError_t err = cudaGetLastError();
  return err == cudaSuccess ? ESR_OK : mfail(ESR_ERR_CUDA, cudaGetErrorString(err));
}

int esr_reduce_splits(const float* part, int32_t splits, int64_t stride, int64_t n, float* out, void* stream) {
  const esr_reduction r{part, out, stride, n, splits, 0};
  return esr_reduce_many(&r, 1, stream);
}

int esr_reduce_many(const esr_reduction* sets, int32_t n_sets, void* stream) {
  if (n_sets < 0 || n_sets > kMaxReductions || (n_sets > 0 && !sets))
    return mfail(ESR_ERR_ARG, "reduce_splits: between 0 and " + std::to_string(kMaxReductions) + " sets");
  Reductions q{};
  long long blocks = 0;
  for (int i = 0; i < n_sets; ++i) {
    const esr_reduction& r = sets[i];
    if (!r.part || !r.out || r.splits <= 0 || r.n <= 0 || r.stride < r.n)
      return mfail(ESR_ERR_ARG, "reduce_splits: bad argument");
    q.r[q.n++] = Reduction{r.part, r.out, r.stride, r.n, r.splits, (int)blocks};
    blocks += (r.n + 255) / 256;
    if (blocks > INT32_MAX) return mfail(ESR_ERR_ARG, "reduce_splits: too many outputs");
  }
  if (blocks == 0) return ESR_OK;
  k_reduce_splits<<<(unsigned)blocks, 256, 0, (cudaStream_t)stream>>>(q);
  cudaError_t err = cudaGetLastError();
  return err == cudaSuccess ? ESR_OK : mfail(ESR_ERR_CUDA, cudaGetErrorString(err));
}

// Workspace of esr_mlp_backward, each part on 256 bytes
struct BackwardWork {
  static constexpr int RPB = 256;   // rows per partial of the head's gradients and of the bias gradients
  int splits = 1, head_blocks;
  bool sums_with_wgrad;             // a range is whole 256-row blocks
  size_t dz[4], dh, dw[4], db, head, bytes;
  explicit BackwardWork(int rows) {
    // ranges of at least 1,024 rows
    while (splits < 64 && rows % (tc::BK * splits * 2) == 0 && rows / (splits * 2) >= 1024) splits *= 2;
    sums_with_wgrad = splits == 1 || rows / splits % RPB == 0;
    head_blocks = (rows + RPB - 1) / RPB;
    size_t at = 0;
    auto take = [&](size_t n) { const size_t o = at; at += (n + 255) / 256 * 256; return o; };
    for (auto& o : dz) o = take((size_t)rows * 256 * sizeof(bf16));
    dh = take((size_t)rows * 256 * sizeof(bf16));
    for (int l = 0; l < 4; ++l) dw[l] = take((size_t)splits * 256 * (l ? 256 : 128) * sizeof(float));
    db = take((size_t)4 * head_blocks * 256 * sizeof(float));
    head = take((size_t)head_blocks * (4 * 256 + 4) * sizeof(float));
    bytes = at;
  }
};

int64_t esr_mlp_backward_workspace(int32_t rows) {
  return rows > 0 && rows % 128 == 0 ? (int64_t)BackwardWork(rows).bytes : -1;
}

int esr_mlp_backward(const esr_mlp_net* net, const void* X, int32_t rows, const float* dY, const void* const* h,
                     const void* const* z, void* work, const esr_mlp_grads* out, void* stream) {
  if (!net || !X || !dY || !h || !z || !work || !out || !net->W4 || !out->W4 || !out->b4)
    return mfail(ESR_ERR_ARG, "mlp_backward: null operand");
  if (rows <= 0 || rows % 128) return mfail(ESR_ERR_ARG, "mlp_backward: rows must be a multiple of 128");
  for (int l = 0; l < 4; ++l) {
    if (!h[l] || !z[l] || !out->W[l] || !out->b[l] || (l && !net->W[l])) return mfail(ESR_ERR_ARG, "mlp_backward: null operand");
    if (!aligned16(h[l]) || !aligned16(z[l]) || (l && !aligned16(net->W[l])))
      return mfail(ESR_ERR_ARG, "mlp_backward: operands must be 16-byte aligned");
  }
  if (!aligned16(work)) return mfail(ESR_ERR_ARG, "mlp_backward: the workspace must be 16-byte aligned");
  const BackwardWork at(rows);
  char* base = static_cast<char*>(work);
  auto f32 = [&](size_t o) { return reinterpret_cast<float*>(base + o); };
  void* dz[4];
  for (int l = 0; l < 4; ++l) dz[l] = base + at.dz[l];
  bf16* dh = reinterpret_cast<bf16*>(base + at.dh);
  int rc = esr_mlp_head_bwd(dY, h[3], z[3], rows, 256, net->W4, dh, dz[3], f32(at.head), BackwardWork::RPB, stream);
  // dh_{l-1} = dh_l + dz_l W_l, in place: an element is read and written by one
  // thread. dh_0 has no reader, only its dz_0 is written.
  for (int l = 3; l > 0 && rc == ESR_OK; --l) {
    const Epi e{nullptr, dh, (const bf16*)z[l - 1], l > 1 ? dh : nullptr, (bf16*)dz[l - 1], 256, (long long)rows * 256, true};
    rc = launch_gemm_tc<false, true, EPI_BWD>(rows, 256, 256, 1, (const bf16*)dz[l], 256, (const bf16*)net->W[l], 256, e,
                                              (cudaStream_t)stream);
  }
  if (rc != ESR_OK) return rc;
  const void* src[4] = {X, h[0], h[1], h[2]};
  float* dw[4];
  for (int l = 0; l < 4; ++l) dw[l] = f32(at.dw[l]);
  rc = esr_mlp_wgrad(dz, src, rows, at.splits, dw, at.sums_with_wgrad ? f32(at.db) : nullptr, stream);
  const size_t db_layer = (size_t)at.head_blocks * 256;
  if (!at.sums_with_wgrad)
    for (int l = 0; l < 4 && rc == ESR_OK; ++l)
      rc = esr_colsum_bf16(dz[l], rows, 256, BackwardWork::RPB, f32(at.db) + l * db_layer, stream);
  if (rc != ESR_OK) return rc;
  esr_reduction sums[10];
  int n = 0;
  const int64_t hs = 4 * 256 + 4;
  sums[n++] = {f32(at.head), out->W4, hs, 4 * 256, at.head_blocks, 0};
  sums[n++] = {f32(at.head) + 4 * 256, out->b4, hs, 4, at.head_blocks, 0};
  for (int l = 0; l < 4; ++l) {
    const int64_t m = 256 * (l ? 256 : 128);
    sums[n++] = {dw[l], out->W[l], m, m, at.splits, 0};
    sums[n++] = {f32(at.db) + l * db_layer, out->b[l], 256, 256, at.head_blocks, 0};
  }
  return esr_reduce_many(sums, n, stream);
}

int esr_colsum_bf16(const void* X, int32_t rows, int32_t C, int32_t rpb, float* part, void* stream) {
  if (!X || !part || rows <= 0 || C <= 0 || rpb <= 0) return mfail(ESR_ERR_ARG, "colsum: bad argument");
  const bool vec = C % 2 == 0 && ((uintptr_t)X & 3) == 0;
  dim3 grid((rows + rpb - 1) / rpb, vec ? (C + 255) / 256 : (C + 127) / 128);
  auto* k = vec ? k_colsum_part<true> : k_colsum_part<false>;
  k<<<grid, 128, 0, (cudaStream_t)stream>>>((const bf16*)X, rows, C, rpb, part);
  cudaError_t err = cudaGetLastError();
  return err == cudaSuccess ? ESR_OK : mfail(ESR_ERR_CUDA, cudaGetErrorString(err));
}

int esr_mlp_loss(const float* pred, const float* tgt, const float* w, int32_t rows, const float* inv_den,
                 float* dpred, float* part, void* stream) {
  if (!pred || !tgt || !inv_den || !dpred || !part || rows <= 0) return mfail(ESR_ERR_ARG, "loss: bad argument");
  k_loss<<<(rows + 255) / 256, 256, 0, (cudaStream_t)stream>>>(pred, tgt, w, rows, inv_den, dpred, part);
  cudaError_t err = cudaGetLastError();
  return err == cudaSuccess ? ESR_OK : mfail(ESR_ERR_CUDA, cudaGetErrorString(err));
}

int esr_adamw(float* p, const float* g, float* m, float* v, int64_t n, float lr, float b1, float b2, float eps,
              float wd, int32_t step, void* p_bf16, void* stream) {
  if (!p || !g || !m || !v || n <= 0 || step < 1) return mfail(ESR_ERR_ARG, "adamw: bad argument");
  const float bc1 = 1.f - powf(b1, (float)step), bc2 = 1.f - powf(b2, (float)step);
  k_adamw<<<(unsigned)((n + 255) / 256), 256, 0, (cudaStream_t)stream>>>(p, g, m, v, n, lr, b1, b2, eps, wd, bc1, bc2,
                                                                         (bf16*)p_bf16);
  cudaError_t err = cudaGetLastError();
  return err == cudaSuccess ? ESR_OK : mfail(ESR_ERR_CUDA, cudaGetErrorString(err));
}

}  // extern "C"
