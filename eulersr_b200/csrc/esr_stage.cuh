// esr_stage.cuh -- one Runge-Kutta stage of a MUSCL solve in one kernel.
//
// A block advances one tile of the mesh (a compact group of cells, TileHead)
// for 1 << slot_shift case slots. From the state alone it
//   A  loads the states of the tile, of the ring of cells around it and of the
//      ring around that, and keeps their primitives (and the boundary ghosts'
//      of the first two) in shared memory,
//   B  forms the limited face states of the tile and its first ring (the
//      ring's are recomputed by every tile that touches it: no face state
//      leaves the block),
//   C  evaluates the face fluxes of the tile's cells,
//   D  sums them per cell in edge order, applies the sponge and the stage update.
// What bounds it: instruction issue in large batches (57-60 % of issue slots,
// 660-677 thread instructions per cell and slot, of which 324 are phase B's; 19
// B of DRAM traffic per cell and slot in a first stage, 35 in a second), the
// latency of one launch and its four dependent phases in single solves. The
// separate K1 / K2 pass 96 B of face states per item and stage through memory
// and pay two launches; here a stage moves the state alone, for about a third
// more reconstructions. Measured 400 steps from freestream, us per SRK2 step,
// the separate kernels of this build at their best shape -> fused: 1 slot x
// 1,450 cells 15.1 -> 7.1, 1 x 25,968 16.8 -> 8.7, 32 x 1,810 15.6 -> 11.9, 32 x
// 25,968 64.4 -> 58.8, 256 x 25,049 460 -> 388. Where this build has no separate
// form, against the earlier one: float64 1 x 19,384 37.1 -> 13.7, 24 x 25,968
// 224 -> 129; reference fidelity 1 x 19,384 34.2 -> 26.7.
//
// CANON (fast fidelity): each face of the tile once, from its owner (the
// lower cell), the flux stored over the two face states it came from, negated
// for the other cell. Otherwise (reference fidelity): every
// side of every cell from its own perspective, as the reference evaluates
// them, into a buffer of its own.
#pragma once
#include <limits.h>

#include <type_traits>

#include "esr_device.cuh"

namespace esr {

// Launches of k_stage overlap (programmatic dependent launch): a block may start
// while the previous launch still runs, reads the tile tables, which never
// change, and waits here until that launch has finished and its results are
// visible. Everything a launch writes (states, control words, local steps) is
// read after this, by loads that bypass the read-only cache. Worth 1.5 us per
// step of a single solve (8.9 -> 7.4 at 1,450 cells, 10.6 -> 9.1 at 25,968).
// k_stage_pair runs without it: its launches are long or its blocks' own
// chains of dependent work dominate (32 x 1,810 cells 12.4 us either way).
__device__ __forceinline__ void stage_begin() {
  asm volatile("griddepcontrol.wait;\n" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
}
__device__ __forceinline__ float4 fresh(const float4* p) {
  float4 v;
  asm volatile("ld.global.cg.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p));
  return v;
}
__device__ __forceinline__ double4 fresh(const double4* p) {
  double4 v;
  asm volatile("ld.global.cg.v2.f64 {%0,%1}, [%2];" : "=d"(v.x), "=d"(v.y) : "l"(p));
  asm volatile("ld.global.cg.v2.f64 {%0,%1}, [%2+16];" : "=d"(v.z), "=d"(v.w) : "l"(p));
  return v;
}
__device__ __forceinline__ float fresh(const float* p) {
  float v;
  asm volatile("ld.global.cg.f32 %0, [%1];" : "=f"(v) : "l"(p));
  return v;
}
__device__ __forceinline__ double fresh(const double* p) {
  double v;
  asm volatile("ld.global.cg.f64 %0, [%1];" : "=d"(v) : "l"(p));
  return v;
}
__device__ __forceinline__ int fresh(const int* p) {
  int v;
  asm volatile("ld.global.cg.s32 %0, [%1];" : "=r"(v) : "l"(p));
  return v;
}

template <typename T>
struct StageMap {
  const Seg<T>* segs;
  const int4* blk;    // (mesh segment, tile, first slot) per block; unused for one mesh
  Seg<T> seg0;
  int groups;         // one mesh: slot groups per tile, else 0
};

// Exponent word of the largest of four primitives and `top`. From 2^200
// (kFarWord) a block's limiter divides three times (xr::limited_faces): its
// cross products, of the order of the fourth power, overflow at 2^256. Looked
// at here, in integers and once a block, it costs 0.7 % of a float64 stage (32 x
// 25,968 cells 164.7 -> 166.1 us per step); a branch in the limiter 4 %.
constexpr int kFarWord = (1023 + 200) << 20;
__device__ __forceinline__ int top_word(const double q[4], int top) {
#pragma unroll
  for (int v = 0; v < 4; ++v) top = max(top, __double2hiint(q[v]) & 0x7fffffff);
  return top;
}

// Phase B of a block with such values, out of line: the loop that every other
// block runs keeps its size and its registers.
static __device__ __noinline__ void far_faces(const V4<double>* P, V4<double>* FV, const StageCell<double>* cells,
                                              int n1, int sh, int slot, double venk_eps, double eps_lim) {
  Consts<double> kc;
  kc.venk_eps = venk_eps;
  kc.eps_lim = eps_lim;
  for (int i = threadIdx.x; i < n1 << sh; i += blockDim.x) {
    const StageCell<double> r = cells[i >> sh];
    double Pk[3][4], q[3][4];
    const V4<double> pc = P[i];
    const double Pc[4] = {pc.x, pc.y, pc.z, pc.w};
    for (int k = 0; k < 3; ++k) {
      const V4<double> p = P[((int)r.nbr[k] << sh) + slot];
      Pk[k][0] = p.x; Pk[k][1] = p.y; Pk[k][2] = p.z; Pk[k][3] = p.w;
    }
    xr::limited_faces<double, 4, true>(Pc, Pk, r.gc, kc, q);
    for (int k = 0; k < 3; ++k) {
      if (r.slot[k] == kNoSlot) continue;
      const bool inner = slot_kind((int)r.kinds, k) == K_INTERIOR;
      FV[((int)r.slot[k] << sh) + slot] = inner ? mk4<double>(q[k][0], q[k][1], q[k][2], q[k][3]) : pc;
    }
  }
}

// value of face state `q`'s flux through the unit normal n, in the run's rounding
template <typename T, bool FAST, int FLUX>
__device__ __forceinline__ void stage_flux(T qL[4], T qR[4], T nx, T ny, const Consts<T>& kc, T F[4]) {
  if constexpr (kXr<T, FAST> && FLUX == 0) {
    xr::hllc<T>(qL, qR, nx, ny, kc, F);
  } else if constexpr (kFastPath<T, FAST>) {
    xr::rusanov<T>(qL, qR, nx, ny, kc, F);
  } else {
    const V4<T> WL = cons<T, FAST>(qL, kc.gm1, kc.inv_gm1, kc.half), WR = cons<T, FAST>(qR, kc.gm1, kc.inv_gm1, kc.half);
    if constexpr (!kXr<T, FAST>) {   // the reference's conserved round trip
      prim<T, FAST>(WL, kc.gm1, kc.half, qL);
      prim<T, FAST>(WR, kc.gm1, kc.half, qR);
    }
    if (FLUX == 0) hllc<T, FAST>(WL, qL, WR, qR, nx, ny, kc, F);
    else rusanov<T, FAST>(WL, qL, WR, qR, nx, ny, kc, F);
  }
}

// residual acc / area - sponge (euler_solver.py:602-628, helper.py:262-295)
// and the stage update (euler_solver.py:630-653)
template <typename T, bool FAST, int STAGE>
__device__ __forceinline__ V4<T> stage_update(const T acc[4], T area, T sig, const V4<T>& inlet, const V4<T>& Wc,
                                              const V4<T>& W0, T dt, const Consts<T>& kc, T* R0_out) {
  if constexpr (kXr<T, FAST>) {
    return xr::cell_update4<STAGE, T>(acc, area, sig, inlet, Wc, W0, dt, kc.half, R0_out);
  } else {
    const T R0 = acc[0] / area - sig * (inlet.x - Wc.x);
    const T R1 = acc[1] / area - sig * (inlet.y - Wc.y);
    const T R2 = acc[2] / area - sig * (inlet.z - Wc.z);
    const T R3 = acc[3] / area - sig * (inlet.w - Wc.w);
    *R0_out = R0;
    if (STAGE == ST_FIRST) return mk4<T>(Wc.x - dt * R0, Wc.y - dt * R1, Wc.z - dt * R2, Wc.w - dt * R3);
    if (STAGE == ST_SRK2_SECOND)
      return mk4<T>(kc.half * (W0.x + Wc.x - dt * R0), kc.half * (W0.y + Wc.y - dt * R1),
                    kc.half * (W0.z + Wc.z - dt * R2), kc.half * (W0.w + Wc.w - dt * R3));
    return mk4<T>(kc.half * (W0.x - dt * R0 + Wc.x), kc.half * (W0.y - dt * R1 + Wc.y),
                  kc.half * (W0.z - dt * R2 + Wc.z), kc.half * (W0.w - dt * R3 + Wc.w));
  }
}

// A second stage runs in place (Wbase = Wout = the state): both kernels read a
// cell's Wbase before they write it, in the thread that writes it, and declare
// neither pointer __restrict__.
// threads of a block (most) and resident blocks per SM a kernel is compiled for
#ifndef ESR_STAGE_MINB
#define ESR_STAGE_MINB 3
#endif
#ifndef ESR_STAGE_MINB_F64
#define ESR_STAGE_MINB_F64 4
#endif
#ifndef ESR_STAGE_THREADS_F64
#define ESR_STAGE_THREADS_F64 128
#endif
template <typename T>
constexpr int kStageThreads = sizeof(T) == 8 ? ESR_STAGE_THREADS_F64 : 256;
template <typename T>
constexpr int kStageBlocks = sizeof(T) == 8 ? ESR_STAGE_MINB_F64 : ESR_STAGE_MINB;

template <typename T, bool FAST, int FLUX, int STAGE, bool LOCALDT>
__global__ void __launch_bounds__(kStageThreads<T>, kStageBlocks<T>) k_stage(
    const StageMap<T> sm, const V4<T>* __restrict__ Win, const V4<T>* Wbase, V4<T>* Wout,
    Cases<T> cs, Consts<T> kc, int pos, T* __restrict__ dt_local, T* __restrict__ res_out, int p_rows, int fv_rows) {
  using V = V4<T>;
  constexpr bool CANON = FAST;
  extern __shared__ __align__(16) unsigned char stage_smem[];
  V* P = reinterpret_cast<V*>(stage_smem);      // primitives
  V* FV = P + p_rows;                           // face states; then, when CANON, the fluxes
  V* FX = FV + fv_rows;                         // the fluxes when not CANON
  Seg<T> s;
  int tile, b0;
  if (sm.groups) {
    s = sm.seg0;
    tile = (int)(blockIdx.x / (unsigned)sm.groups);
    b0 = (int)(blockIdx.x - (unsigned)tile * (unsigned)sm.groups) << s.slot_shift;
  } else {
    const int4 e = sm.blk[blockIdx.x];
    s = sm.segs[e.x];
    tile = e.y;
    b0 = e.z;
  }
  const int sh = s.slot_shift, nt = blockDim.x;
  const TileHead h = s.tile_head[tile];
  // each thread always works on the same slot (nt is a multiple of 1 << sh)
  const int slot = threadIdx.x & ((1 << sh) - 1), b = b0 + slot;
  const bool in_seg = b < s.B;
  const int g = s.case0 + (in_seg ? b : 0);
  const int* list = s.tile_list + h.list;
  const StageCell<T>* cells = s.tile_cells + h.cells;
  StageCell<T> r = cells[min((int)threadIdx.x >> sh, h.n1 - 1)];
  const int c0 = list[min((int)threadIdx.x >> sh, h.n2 - 1)];
  stage_begin();
  const int act = fresh(cs.active + g), done = fresh(cs.step + g), cap = fresh(cs.nmax + g);
  const V inlet = fresh(cs.inlet + g);
  const bool live = in_seg && act && done + pos < cap;
  if (!__syncthreads_or(live)) return;          // every slot of the group idle
  const V* win = Win + s.off + (in_seg ? b : 0);
  // A: primitives of the tile, its two rings and its ghosts
  static_assert(FAST || sizeof(T) == 4, "float64 in the reference's sequence runs the separate kernels");
  constexpr bool SCALED = sizeof(T) == 8;   // the limiter's products have a range (limited_faces)
  int top = 0;                                              // largest exponent word of the primitives
  for (int i = threadIdx.x, c = c0; i < h.n2 << sh; i += nt) {
    T q[4];
    const V w = fresh(win + (long long)c * s.B);
    if (i + nt < h.n2 << sh) c = list[(i + nt) >> sh];
    cell_prim<T, FAST>(w, kc, q);
    if constexpr (SCALED) if (live) top = top_word(q, top);
    P[i] = mk4<T>(q[0], q[1], q[2], q[3]);
  }
  for (int i = threadIdx.x; i < h.n_ghosts << sh; i += nt) {
    const StageGhost<T> w = s.tile_ghosts[h.ghosts + (i >> sh)];
    T q[4];
    ghost_prim<T, FAST>(w.kind, fresh(win + (long long)w.cell * s.B), w.nx, w.ny, inlet, kc, q);
    if constexpr (SCALED) if (live) top = top_word(q, top);
    P[(h.n2 << sh) + i] = mk4<T>(q[0], q[1], q[2], q[3]);
  }
  // B: limited face states of the tile and its first ring. The first record
  // of each phase is on its way before the barrier.
  bool far = false;
  if constexpr (SCALED) far = __syncthreads_or(top >= kFarWord);
  else __syncthreads();
  for (int i = (SCALED && far) ? INT_MAX : (int)threadIdx.x; i < h.n1 << sh; i += nt) {
    const int lc = i >> sh;
    StageCell<T> rn = r;
    if (kFastPath<T, FAST> && i + nt < h.n1 << sh) rn = cells[(i + nt) >> sh];   // the next one meanwhile
    T Pk[3][4], q[3][4];
    const V pc = P[i];
    const T Pc[4] = {pc.x, pc.y, pc.z, pc.w};
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      const V p = P[((int)r.nbr[k] << sh) + slot];
      Pk[k][0] = p.x; Pk[k][1] = p.y; Pk[k][2] = p.z; Pk[k][3] = p.w;
    }
    limited_faces<T, FAST>(Pc, Pk, r.gc, s.lsq, (!FAST && sizeof(T) == 4) ? list[lc] : 0, kc, q);
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      if (r.slot[k] == kNoSlot) continue;
      const bool inner = slot_kind((int)r.kinds, k) == K_INTERIOR;
      FV[((int)r.slot[k] << sh) + slot] = inner ? mk4<T>(q[k][0], q[k][1], q[k][2], q[k][3]) : pc;
    }
    if (!kFastPath<T, FAST> && i + nt < h.n1 << sh) rn = cells[(i + nt) >> sh];
    r = rn;
  }
  if constexpr (SCALED) if (far) far_faces(P, FV, cells, h.n1, sh, slot, kc.venk_eps, kc.eps_lim);
  const StageFace<T>* faces = s.tile_faces + h.faces;
  StageFace<T> f = faces[min((int)threadIdx.x >> sh, h.n_faces - 1)];
  __syncthreads();
  // C: face fluxes. Each face-state slot belongs to one face, so in the
  // CANON form the flux replaces the states it was formed from (a ring
  // cell's copy is never read).
  for (int i = threadIdx.x; i < h.n_faces << sh; i += nt) {
    const int iL = ((int)(f.slots & 0xFFFF) << sh) + slot, iR = ((int)(f.slots >> 16) << sh) + slot;
    const V fl = FV[iL], fr = f.kind == K_INTERIOR ? FV[iR] : P[iR];
    T qL[4] = {fl.x, fl.y, fl.z, fl.w}, qR[4] = {fr.x, fr.y, fr.z, fr.w}, F[4];
    stage_flux<T, FAST, FLUX>(qL, qR, f.nx, f.ny, kc, F);
    if (CANON) {
      FV[iL] = mk4<T>(F[0], F[1], F[2], F[3]);
      if (f.kind == K_INTERIOR) FV[iR] = mk4<T>(-F[0], -F[1], -F[2], -F[3]);
    } else {
      FX[iL] = mk4<T>(F[0], F[1], F[2], F[3]);
    }
    if (i + nt < h.n_faces << sh) f = faces[(i + nt) >> sh];
  }
  // D: residual, sponge and stage update of the tile's own cells
  const V* G = CANON ? FV : FX;
  const T strength = fresh(cs.strength + g);
  const T case_dt = fresh(cs.dt + g);
  const StageOwn<T>* own = s.tile_own + h.own;
  StageOwn<T> o = own[min((int)threadIdx.x >> sh, h.n_own - 1)];
  const long long base = s.off + (in_seg ? b : 0);
  V Wc = fresh(Win + base + (long long)o.cell * s.B), W0 = Wc;
  if (STAGE != ST_FIRST) W0 = fresh(Wbase + base + (long long)o.cell * s.B);
  __syncthreads();
  if (!live) return;
  for (int i = threadIdx.x; i < h.n_own << sh; i += nt) {
    const int lc = i >> sh;
    if (i >= nt) {   // not the first
      o = own[lc];
      Wc = fresh(Win + base + (long long)o.cell * s.B);
      W0 = STAGE == ST_FIRST ? Wc : fresh(Wbase + base + (long long)o.cell * s.B);
    }
    const long long gi = base + (long long)o.cell * s.B;
    T acc[4], dt = case_dt;
    if (LOCALDT) {   // dt holds the case's CFL number
      if (STAGE == ST_FIRST) {
        T q[4];
        cell_prim<T, FAST>(Wc, kc, q);
        dt = local_dt<T, FAST>(q, o.n, o.s, o.area, kc) * case_dt;
        dt_local[gi] = dt;
      } else {
        dt = fresh(dt_local + gi);
      }
    }
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      const V f = G[((3 * lc + k) << sh) + slot];
      const T F[4] = {f.x, f.y, f.z, f.w}, sk = o.s[k];
      if constexpr (kXr<T, FAST>) {
        xr::accumulate<T>(k, sk, F, acc);
      } else if (k == 0) {
        acc[0] = sk * F[0]; acc[1] = sk * F[1]; acc[2] = sk * F[2]; acc[3] = sk * F[3];
      } else {
        acc[0] = acc[0] + sk * F[0]; acc[1] = acc[1] + sk * F[1];
        acc[2] = acc[2] + sk * F[2]; acc[3] = acc[3] + sk * F[3];
      }
    }
    T sig, R0;
    if constexpr (kXr<T, FAST>) sig = xr::mul(strength, o.blend3);
    else sig = strength * o.blend3;
    const V w = stage_update<T, FAST, STAGE>(acc, o.area, sig, inlet, Wc, W0, dt, kc, &R0);
    // density residual of the state the step starts from (density-L2 stop rule)
    if (STAGE == ST_FIRST && res_out != nullptr) res_out[gi] = R0;
    Wout[gi] = w;
  }
}

// the states of two slots dB apart; wide: they are neighbours on a 32-byte
// boundary, one access (as two 16-byte ones every sector is fetched twice).
// For Win alone, which no launch writes: the read-only path.
__device__ __forceinline__ void state_pair(const float4* p, int dB, bool wide, float4& a, float4& b) {
  if (wide) {
    asm("ld.global.nc.v8.f32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
        : "=f"(a.x), "=f"(a.y), "=f"(a.z), "=f"(a.w), "=f"(b.x), "=f"(b.y), "=f"(b.z), "=f"(b.w) : "l"(p));
  } else {
    a = p[0];
    b = p[dB];
  }
}
// the same for Wbase, which a second stage overwrites in place (Wbase = Wout):
// the ordinary path, and never moved past a store
__device__ __forceinline__ void base_pair(const float4* p, int dB, bool wide, float4& a, float4& b) {
  if (wide) {
    asm volatile("ld.global.v8.f32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=f"(a.x), "=f"(a.y), "=f"(a.z), "=f"(a.w), "=f"(b.x), "=f"(b.y), "=f"(b.z), "=f"(b.w)
                 : "l"(p) : "memory");
  } else {
    a = p[0];
    b = p[dB];
  }
}

// The same stage for batches of the fast float32 solve, two case slots
// per thread: every multiply and add of the pair is one packed instruction,
// and the geometry, the neighbour records and the addresses are fetched once
// for both. 1 << SH pairs of slots per block. The roundings are k_stage's.
#ifndef ESR_PAIR_MINB
#define ESR_PAIR_MINB 5
#endif
#ifndef ESR_PAIR_THREADS
#define ESR_PAIR_THREADS 128
#endif
// 128 threads and 5 blocks per SM (94 registers, 45 KB of shared memory at 64
// cells x 8 slots), swept on an earlier build (with IEEE square roots; 388 us now):
// 404 us per step of 256 x 25,049 against 448 at 4 blocks, 413 at 80 cells x
// 160 threads x 4, 419 at 96 x 192 x 3, 429-455 at 48 cells
constexpr int kPairThreads = ESR_PAIR_THREADS;
constexpr int kLoads = 4;            // state rows a thread has in flight
constexpr uint32_t kAnyBoundary = 7u | 7u << 6 | 7u << 12;   // kind bits of the packed slot word

__device__ __forceinline__ void load_pair(const float4* lo, const float4* hi, int i, float2 q[4]) {
  const float4 a = lo[i], b = hi[i];
  q[0] = make_float2(a.x, a.y); q[1] = make_float2(a.z, a.w);
  q[2] = make_float2(b.x, b.y); q[3] = make_float2(b.z, b.w);
}
__device__ __forceinline__ void store_pair(float4* lo, float4* hi, int i, const float2 q[4]) {
  lo[i] = make_float4(q[0].x, q[0].y, q[1].x, q[1].y);
  hi[i] = make_float4(q[2].x, q[2].y, q[3].x, q[3].y);
}
__device__ __forceinline__ void pair_of(const float4& a, const float4& b, float2 q[4]) {
  q[0] = make_float2(a.x, b.x); q[1] = make_float2(a.y, b.y);
  q[2] = make_float2(a.z, b.z); q[3] = make_float2(a.w, b.w);
}

template <int FLUX, int STAGE, bool LOCALDT, int SH>
__global__ void __launch_bounds__(kPairThreads, ESR_PAIR_MINB) k_stage_pair(
    const StageMap<float> sm, const float4* __restrict__ Win, const float4* Wbase, float4* Wout, Cases<float> cs,
    Consts<float> kc, int pos, float* __restrict__ dt_local, float* __restrict__ res_out, int p_rows, int fv_rows) {
  constexpr int NP = 1 << SH;
  extern __shared__ __align__(16) unsigned char stage_smem[];
  float4* P0 = reinterpret_cast<float4*>(stage_smem);   // primitives: (rho, u) and (v, p) of both slots
  float4* P1 = P0 + p_rows;
  float4* F0 = P1 + p_rows;                             // face states, then the fluxes
  float4* F1 = F0 + fv_rows;
  Seg<float> s;
  int tile, b0;
  if (sm.groups) {
    s = sm.seg0;
    tile = (int)(blockIdx.x / (unsigned)sm.groups);
    b0 = (int)(blockIdx.x - (unsigned)tile * (unsigned)sm.groups) * (2 * NP);
  } else {
    const int4 e = sm.blk[blockIdx.x];
    s = sm.segs[e.x];
    tile = e.y;
    b0 = e.z;
  }
  const TileHead h = s.tile_head[tile];
  const int pr = threadIdx.x & (NP - 1);
  // slots b and b + 1; one past the segment repeats the last slot and is not stored
  const int bA = min(b0 + 2 * pr, s.B - 1), bB = min(b0 + 2 * pr + 1, s.B - 1);
  const int gA = s.case0 + bA, gB = s.case0 + bB;
  const int* list = s.tile_list + h.list;
  const int n2 = h.n2 << SH;
  int c[kLoads];
#pragma unroll
  for (int u = 0; u < kLoads; ++u) c[u] = list[min((int)threadIdx.x + u * kPairThreads, n2 - 1) >> SH];
  const int actA = cs.active[gA], actB = cs.active[gB];
  const int doneA = cs.step[gA], doneB = cs.step[gB];
  const int capA = cs.nmax[gA], capB = cs.nmax[gB];
  const bool liveA = b0 + 2 * pr < s.B && actA && doneA + pos < capA;
  const bool liveB = b0 + 2 * pr + 1 < s.B && actB && doneB + pos < capB;
  if (!__syncthreads_or(liveA || liveB)) return;   // every slot of the group idle
  const float4* winA = Win + s.off + bA;
  const int dB = bB - bA;
  // both slots in one 32-byte access: every row of the state starts on 32 bytes
  const bool wide = dB == 1 && ((s.off | s.B) & 1) == 0;
  // A: primitives of the tile, its two rings and its ghosts; the states of
  // kLoads rows are requested before the first is used
  for (int i0 = threadIdx.x; i0 < n2; i0 += kLoads * kPairThreads) {
    float4 a[kLoads], b[kLoads];
#pragma unroll
    for (int u = 0; u < kLoads; ++u) state_pair(winA + (long long)c[u] * s.B, dB, wide, a[u], b[u]);
    if (i0 + kLoads * kPairThreads < n2)
#pragma unroll
      for (int u = 0; u < kLoads; ++u) c[u] = list[min(i0 + (kLoads + u) * kPairThreads, n2 - 1) >> SH];
#pragma unroll
    for (int u = 0; u < kLoads; ++u) {
      const int i = i0 + u * kPairThreads;
      float2 W[4], q[4];
      pair_of(a[u], b[u], W);
      xr::prim<float2>(W, kc.gm1, kc.half, q);
      if (i < n2) store_pair(P0, P1, i, q);
    }
  }
  for (int i = threadIdx.x; i < h.n_ghosts << SH; i += kPairThreads) {
    const StageGhost<float> w = s.tile_ghosts[h.ghosts + (i >> SH)];
    const long long at = (long long)w.cell * s.B;
    float a[4], b[4];
    xr::ghost_prim<float>(w.kind, winA[at], w.nx, w.ny, cs.inlet[gA], kc, a);
    xr::ghost_prim<float>(w.kind, winA[at + dB], w.nx, w.ny, cs.inlet[gB], kc, b);
    float2 q[4];
#pragma unroll
    for (int v = 0; v < 4; ++v) q[v] = make_float2(a[v], b[v]);
    store_pair(P0, P1, n2 + i, q);
  }
  // B: limited face states of the tile and its first ring, two variables at a
  // time. The first record of each phase is on its way before the barrier,
  // the next one while the current is used.
  const StageCell<float>* cells = s.tile_cells + h.cells;
  StageCell<float> r = cells[min((int)threadIdx.x >> SH, h.n1 - 1)];
  __syncthreads();
  for (int i = threadIdx.x; i < h.n1 << SH; i += kPairThreads) {
    const StageCell<float> rn = cells[min((i + kPairThreads) >> SH, h.n1 - 1)];
    const bool own = i < h.n_own << SH;
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      const float4* P = half ? P1 : P0;
      float4* FV = half ? F1 : F0;
      float2 Pc[2], Pk[3][2], q[3][2];
      const float4 pc = P[i];
      Pc[0] = make_float2(pc.x, pc.y);
      Pc[1] = make_float2(pc.z, pc.w);
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        const float4 p = P[((int)r.nbr[k] << SH) + pr];
        Pk[k][0] = make_float2(p.x, p.y);
        Pk[k][1] = make_float2(p.z, p.w);
      }
      xr::limited_faces<float2, 2>(Pc, Pk, r.gc, kc, q);
      if (r.kinds & kAnyBoundary) {   // a boundary face keeps the cell's own state
#pragma unroll
        for (int k = 0; k < 3; ++k)
          if (slot_kind((int)r.kinds, k) != K_INTERIOR) { q[k][0] = Pc[0]; q[k][1] = Pc[1]; }
      }
#pragma unroll
      for (int k = 0; k < 3; ++k)
        if (own || r.slot[k] != kNoSlot)
          FV[((int)r.slot[k] << SH) + pr] = make_float4(q[k][0].x, q[k][0].y, q[k][1].x, q[k][1].y);
    }
    r = rn;
  }
  // C: each face of the tile's cells once, the flux over the two states it
  // came from (a ring cell's copy is never read)
  const StageFace<float>* faces = s.tile_faces + h.faces;
  StageFace<float> f = faces[min((int)threadIdx.x >> SH, h.n_faces - 1)];
  __syncthreads();
  for (int i = threadIdx.x; i < h.n_faces << SH; i += kPairThreads) {
    const StageFace<float> fn = faces[min((i + kPairThreads) >> SH, h.n_faces - 1)];
    const int iL = ((int)(f.slots & 0xFFFF) << SH) + pr, iR = ((int)(f.slots >> 16) << SH) + pr;
    const bool inner = f.kind == K_INTERIOR;
    float2 qL[4], qR[4], F[4];
    load_pair(F0, F1, iL, qL);
    load_pair(inner ? F0 : P0, inner ? F1 : P1, iR, qR);
    if constexpr (FLUX == 0) xr::hllc<float2>(qL, qR, f.nx, f.ny, kc, F);
    else xr::rusanov<float2>(qL, qR, f.nx, f.ny, kc, F);
    store_pair(F0, F1, iL, F);
    if (inner) {
#pragma unroll
      for (int v = 0; v < 4; ++v) F[v] = xr::neg(F[v]);
      store_pair(F0, F1, iR, F);
    }
    f = fn;
  }
  // D: residual, sponge and stage update of the tile's own cells
  const StageOwn<float>* owns = s.tile_own + h.own;
  StageOwn<float> o = owns[min((int)threadIdx.x >> SH, h.n_own - 1)];
  float4 wa, wb;
  state_pair(winA + (long long)o.cell * s.B, dB, wide, wa, wb);
  const float2 strength = make_float2(cs.strength[gA], cs.strength[gB]);
  const float2 case_dt = make_float2(cs.dt[gA], cs.dt[gB]);
  float2 inlet[4];
  pair_of(cs.inlet[gA], cs.inlet[gB], inlet);
  __syncthreads();
  if (!liveA && !liveB) return;
  for (int i = threadIdx.x; i < h.n_own << SH; i += kPairThreads) {
    const int lc = i >> SH;
    const long long gi = s.off + (long long)o.cell * s.B + bA;
    float2 Wc[4], W0[4], acc[4], w[4], R0;
    pair_of(wa, wb, Wc);
    if (STAGE != ST_FIRST) {
      float4 a, b;
      base_pair(Wbase + gi, dB, wide, a, b);
      pair_of(a, b, W0);
    }
    float2 dt = case_dt;
    if (LOCALDT) {   // dt holds the case's CFL number
      if (STAGE == ST_FIRST) {
        float2 q[4];
        xr::prim<float2>(Wc, kc.gm1, kc.half, q);
        dt = xr::mul(xr::local_dt<float2>(q, o.n, o.s, o.area, kc), case_dt);
        if (liveA) dt_local[gi] = dt.x;
        if (liveB) dt_local[gi + dB] = dt.y;
      } else {
        dt = make_float2(dt_local[gi], dt_local[gi + dB]);
      }
    }
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      float2 F[4];
      load_pair(F0, F1, ((3 * lc + k) << SH) + pr, F);
      xr::accumulate<float2>(k, o.s[k], F, acc);
    }
    const float2 sig = xr::mul(strength, make_float2(o.blend3, o.blend3));
    xr::cell_update<STAGE, float2>(acc, o.area, sig, inlet, Wc, W0, dt, kc.half, &R0, w);
    if (i + kPairThreads < h.n_own << SH) {
      o = owns[(i + kPairThreads) >> SH];
      state_pair(winA + (long long)o.cell * s.B, dB, wide, wa, wb);
    }
    // density residual of the state the step starts from (density-L2 stop rule)
    if (STAGE == ST_FIRST && res_out != nullptr) {
      if (liveA) res_out[gi] = R0.x;
      if (liveB) res_out[gi + dB] = R0.y;
    }
    const float4 wA = make_float4(w[0].x, w[1].x, w[2].x, w[3].x), wB = make_float4(w[0].y, w[1].y, w[2].y, w[3].y);
    if (wide && liveA && liveB) {
      asm volatile("st.global.v8.f32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(Wout + gi), "f"(wA.x), "f"(wA.y),
                   "f"(wA.z), "f"(wA.w), "f"(wB.x), "f"(wB.y), "f"(wB.z), "f"(wB.w) : "memory");
    } else {
      if (liveA) Wout[gi] = wA;
      if (liveB) Wout[gi + dB] = wB;
    }
  }
}

// One stage launch of a solver: the block map, the grid and the shared-memory
// layout its tiles need (in 4-value vectors)
template <typename T>
struct StageLaunch {
  StageMap<T> map;
  int blocks, threads, smem;
  int p_rows, fv_rows;
  int pairs;          // >= 0: k_stage_pair with 1 << pairs pairs of slots per block
};

// FAST = false in float32 is instantiated in esr_faithful.cu alone.
// every (flux, stage, local step) form: fn(FLUX, STAGE, LOCALDT) as integral constants
template <typename F>
void stage_form(bool rusanov, int stage, bool local, F&& fn) {
  auto with_local = [&](auto f, auto s) {
    if (local) fn(f, s, std::integral_constant<bool, true>{});
    else fn(f, s, std::integral_constant<bool, false>{});
  };
  auto with_stage = [&](auto f) {
    if (stage == ST_FIRST) with_local(f, std::integral_constant<int, ST_FIRST>{});
    else if (stage == ST_SRK2_SECOND) with_local(f, std::integral_constant<int, ST_SRK2_SECOND>{});
    else with_local(f, std::integral_constant<int, ST_RK2_SECOND>{});
  };
  if (rusanov) with_stage(std::integral_constant<int, 1>{});
  else with_stage(std::integral_constant<int, 0>{});
}
template <int FLUX, int STAGE, bool LOCALDT>
auto pair_kernel(int sh) {
  return sh == 0 ? k_stage_pair<FLUX, STAGE, LOCALDT, 0>
       : sh == 1 ? k_stage_pair<FLUX, STAGE, LOCALDT, 1> : k_stage_pair<FLUX, STAGE, LOCALDT, 2>;
}
template <typename T, bool FAST>
cudaError_t launch_stage(const StageLaunch<T>& L, bool rusanov, int stage, bool local, const V4<T>* win,
                         const V4<T>* wbase, V4<T>* wout, const Cases<T>& cs, const Consts<T>& kc, int pos, T* dt_local,
                         T* res, cudaStream_t st) {
  cudaLaunchAttribute overlap{};
  overlap.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  overlap.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)L.blocks);
  cfg.blockDim = dim3((unsigned)L.threads);
  cfg.dynamicSmemBytes = (size_t)L.smem;
  cfg.stream = st;
  cfg.attrs = &overlap;
  cfg.numAttrs = L.pairs >= 0 ? 0 : 1;   // k_stage_pair does not wait for the previous launch by itself
  cudaError_t e = cudaSuccess;
  stage_form(rusanov, stage, local, [&](auto f, auto s, auto l) {
    auto* k = &k_stage<T, FAST, f(), s(), l()>;
    if constexpr (kFastPath<T, FAST>)
      if (L.pairs >= 0) k = pair_kernel<f(), s(), l()>(L.pairs);
    e = cudaLaunchKernelEx(&cfg, k, L.map, win, wbase, wout, cs, kc, pos, dt_local, res, L.p_rows, L.fv_rows);
  });
  return e;
}
// blocks of a k_stage of this layout that an SM holds at once
template <typename T, bool FAST>
cudaError_t stage_residents(const StageLaunch<T>& L, bool rusanov, bool local, int* blocks) {
  cudaError_t e = cudaSuccess;
  stage_form(rusanov, ST_FIRST, local, [&](auto f, auto s, auto l) {
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks, k_stage<T, FAST, f(), s(), l()>, L.threads, L.smem);
  });
  return e;
}
// Raises the dynamic shared-memory limit of every form a solver of this flux
// and time step launches, to what a block may hold at most: the limit is the
// function's, shared by every solver of the process.
constexpr int kStageSmemMax = 227 * 1024;
template <typename T, bool FAST>
cudaError_t allow_stage(bool rusanov, bool local) {
  cudaError_t e = cudaSuccess;
  for (int stage : {ST_FIRST, ST_SRK2_SECOND, ST_RK2_SECOND})
    stage_form(rusanov, stage, local, [&](auto f, auto s, auto l) {
      const cudaError_t r = cudaFuncSetAttribute(k_stage<T, FAST, f(), s(), l()>,
                                                 cudaFuncAttributeMaxDynamicSharedMemorySize, kStageSmemMax);
      if (e == cudaSuccess) e = r;
      if constexpr (kFastPath<T, FAST>)
        for (int sh = 0; sh <= 2 && e == cudaSuccess; ++sh)
          e = cudaFuncSetAttribute(pair_kernel<f(), s(), l()>(sh), cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   kStageSmemMax);
    });
  return e;
}

}  // namespace esr
