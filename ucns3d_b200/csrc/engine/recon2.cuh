// Reconstruction for WENO / CWENO / high-order MUSCL.
//
// LEAST_SQUARES (src/gradients.f90:253-497), stencil polynomials G[ll][d][v]:
//   k_lsq_ring  cells that read their own tables, streamed from DRAM through
//               shared memory (interleaved over groups of 32 cells)
//   k_lsq_set   cells that share a matrix set, tiled (and k_lsq_low, the
//               CWENO directional stencils of those cells)
//   k_lsq_lane  IORDER 1 on large meshes, one lane per cell
// CP_RECONSTRUCTION (src/reconstruct_p.f90:920-1250), CHECKSOL, MUSCL
// fall-back, CHECKSOLX (3126-3406):
//   k_wface     conserved variables, one warp per variable: IORDER 4 with the
//               indicators of k_wis / k_wis_set, below with its own where
//               that is faster (wface_own)
//   k_char_forms, k_char_face  characteristic variables
//   k_wpost     one lane per cell: the MUSCL fall-back of the cells that the
//               above flag; alone where k_wface is not taken and for high-order
//               MUSCL
#pragma once

#include "device.cuh"

namespace ucg {

// rows of G that one warp holds in registers per pass (DH x 5 values of T)
template <int P, typename T>
struct LsqRows {
  static constexpr int ID = Deg<P>::ideg;
  static constexpr int value = P == 4 ? (sizeof(T) == 4 ? 34 : 17) : P == 3 ? (sizeof(T) == 4 ? 19 : 10) : ID;
};

// Gathers of a producer warp for the 32 cells of its consumer.  The lanes
// share a member's 32 records of 40 bytes element by element, lane l taking
// the elements l, l + 32, ... of the 160, so that a load touches the lines of
// six or seven records instead of 32 (a lane per record reads five values of
// 32 distant records, five times over: with scattered members the L1 tag
// lookups alone bound the kernel).  The differences go to shared memory as
// they come, [cell][variable], which the consumer reads without bank
// conflicts (row stride 5).
struct GatherShare {
  int r[NV], v[NV];
  __device__ __forceinline__ explicit GatherShare(int lane) {
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      r[i] = (lane + 32 * i) / NV;
      v[i] = lane + 32 * i - r[i] * NV;
    }
  }
  // the lane's elements of the records of cells y (lane = cell)
  __device__ __forceinline__ void load(const double* __restrict__ U, int y, double (&u)[NV]) const {
#pragma unroll
    for (int i = 0; i < NV; ++i) u[i] = U[(int64_t)__shfl_sync(0xffffffffu, y, r[i]) * NV + v[i]];
  }
};

// polls of one stage wait (about 20 ms; a stage normally lands in microseconds)
constexpr long LSQ_WAIT = 1L << 16;
inline long lsq_wait(const Problem& p) { return p.lsq_wait < 0 ? LSQ_WAIT : p.lsq_wait; }

// mbar_wait of a warp that also gives up when another warp of the block has
__device__ __forceinline__ bool ring_wait(uint64_t* bar, unsigned parity, long limit, const volatile int* stop) {
  bool ok = false;
  for (long it = 0; it < limit; ++it) {
    ok = mbar_try_wait(bar, parity);
    if (ok || *stop) break;
    if (it > 64) __nanosleep(256);
  }
  return __all_sync(0xffffffffu, ok);
}
// The same with the bound in shared memory, read only when a poll has failed
// (k_lsq_set: a limit that the loops carry took 102 registers instead of 96 and
// with them the second block per SM, 2.13 -> 3.37 ms); a warp that gives up sets
// it to -1 for the others.
__device__ __forceinline__ bool set_wait(uint64_t* bar, unsigned parity, const volatile int* limit) {
  bool ok = false;
  for (long it = 0; it < LSQ_WAIT; ++it) {
    ok = mbar_try_wait(bar, parity);
    if (ok || it >= *limit) break;
    if (it > 64) __nanosleep(256);
  }
  return __all_sync(0xffffffffu, ok);
}

template <int N>
struct IntC {
  static constexpr int value = N;
};

// acc[row] += r[row] du of one 16-byte vector of rows.  FP32 in packed pairs
// of rows (FFMA2: two IEEE multiply-adds, the same values): one scalar FFMA a
// cycle is half of the FP32 rate.
template <typename T>
struct RowAcc;
template <>
struct RowAcc<float> {
  float2 a[2][NV];
  __device__ __forceinline__ void zero() {
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
      for (int v = 0; v < NV; ++v) a[h][v] = make_float2(0.0f, 0.0f);
  }
  __device__ __forceinline__ void add(const float* m, const float (&du)[NV]) {
    const float4 r = *(const float4*)m;
    const float2 r0 = make_float2(r.x, r.y), r1 = make_float2(r.z, r.w);
#pragma unroll
    for (int v = 0; v < NV; ++v) a[0][v] = __ffma2_rn(r0, make_float2(du[v], du[v]), a[0][v]);
#pragma unroll
    for (int v = 0; v < NV; ++v) a[1][v] = __ffma2_rn(r1, make_float2(du[v], du[v]), a[1][v]);
  }
  __device__ __forceinline__ float get(int i, int v) const { return i & 1 ? a[i >> 1][v].y : a[i >> 1][v].x; }
};
template <>
struct RowAcc<double> {
  double a[2][NV];
  __device__ __forceinline__ void zero() {
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
      for (int v = 0; v < NV; ++v) a[h][v] = 0.0;
  }
  __device__ __forceinline__ void add(const double* m, const double (&du)[NV]) {
    const double2 r = *(const double2*)m;
#pragma unroll
    for (int v = 0; v < NV; ++v) a[0][v] += r.x * du[v];
#pragma unroll
    for (int v = 0; v < NV; ++v) a[1][v] += r.y * du[v];
  }
  __device__ __forceinline__ double get(int i, int v) const { return a[i][v]; }
};

// LEAST_SQUARES of the cells that share a matrix set (table_id of ucg_recon:
// cells of the same local geometry).  Streaming every cell's own copy of the
// pseudo-inverses from DRAM (100 KB a cell for WENO5 in FP32) bounds
// k_lsq_ring; here a block takes 64 cells of one set and one stencil, keeps
// the stencil's rows in shared memory and reads them as 16-byte broadcasts,
// each row feeding five multiply-adds of a cell, so the kernel is bound by the
// multiply-adds.  Per 32 cells NPR producer warps take turns to gather the
// differences of MS members (all in flight, their indices loaded a turn ahead)
// into a ring of NSTG stages, and NSL consumer warps multiply, each a slice of
// the rows: with all 34 rows in one warp (170 accumulators) a scheduler has
// one warp to run, whose shared-memory latencies nothing hides (64^3 WENO5,
// mixed: 3.95 ms; and 4.36 ms with the gathers in the same warp).  The members
// are added in their order per row and variable, so that G does not depend on
// the kernel that forms it, bit for bit.
// One lane per cell reading its own tables took 5.48 ms (64^3 WENO5, mixed),
// 1.43 ms (27,000 cells, FP64) and 0.97 ms (271,872-cell CWENO4, mixed); this
// kernel 2.13, 0.51 and, with k_lsq_low and the 48 groups left to k_lsq_ring,
// 0.43.  Its shared-memory loads (34 words a row of five multiply-adds, 70
// cycles a member and 32 cells in FP32) stand before the multiply-adds (43).
// A wait that gives up (`wait` polls) sets HEALTH_TIMEOUT and ends the waits of
// the block's other warps, and its polynomials are not stored.
template <typename T, int ND>
struct SetRing {
  static constexpr int VEC = Vec<T>::N, NVEC = (ND + VEC - 1) / VEC;  // vectors of rows
  static constexpr int NSL = (NVEC + (VEC == 4 ? 2 : 4)) / (VEC == 4 ? 3 : 5);
  static constexpr int MAXV = (NVEC + NSL - 1) / NSL;  // of a slice
  // producers of 32 cells: two keep up with three or more slices (64,000 cells,
  // WENO5 mixed: 0.711 ms with one, 0.534 with two; 27,000, FP64: 0.533, 0.506)
  // and with two in FP32 (271,872 cells, CWENO4: 0.494, 0.436); elsewhere the
  // second only takes registers (32,768-cell CWENO4 FP64: 0.236, 0.253)
  static constexpr int NPR = NSL > (VEC == 4 ? 1 : 2) ? 2 : 1;
  static constexpr int WARPS = 2 * (NSL + NPR);
  static constexpr int MS = 4, NSTG = 4;  // members of a stage, stages (a multiple of NPR)
  static constexpr int elems = MS * 32 * NV;  // of a stage
  static_assert(2 * NSTG * elems == SET_RING, "plan_sets asks whether the rings fit");
};
template <int P, typename T, int ND>
__global__ void __launch_bounds__(32 * SetRing<T, ND>::WARPS)
    k_lsq_set(Problem p, const double* __restrict__ U, int wait) {
  constexpr int ID = Deg<P>::ideg;
  constexpr int RS = set_stride<T>(ND);
  using R = SetRing<T, ND>;
  constexpr int VEC = R::VEC, MS = R::MS, NSTG = R::NSTG;
  constexpr int TH = 32 * R::WARPS;
  extern __shared__ __align__(16) unsigned char ls_smem[];
  __shared__ __align__(8) uint64_t s_full[2][NSTG], s_empty[2][NSTG];
  __shared__ int s_limit;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, half = warp & 1, role = warp >> 1;
  const int64_t tile = blockIdx.x >> 1;
  const int ll = blockIdx.y;
  const int nk = p.imax, A = p.admis_max, W = p.imax + 1;
  const int32_t* tc = p.tcell + tile * SET_TILE + (blockIdx.x & 1) * 64;
  if (tc[0] < 0) return;  // the tile's second half may hold no cell
  T* s = (T*)ls_smem;
  T* ring = s + nk * RS + half * NSTG * R::elems;
  uint64_t *full = s_full[half], *empty = s_empty[half];
  if (threadIdx.x == 0) {
    s_limit = wait;
    for (int w = 0; w < 2; ++w)
      for (int i = 0; i < NSTG; ++i) {
        mbar_init(&s_full[w][i], wait ? 1 : 2);  // limit 0: no stage is ever full
        mbar_init(&s_empty[w][i], R::NSL);
      }
    mbar_fence_init();
  }
  {
    const float4* src = (const float4*)((const T*)p.setmat + p.tset[tile] * p.sstride + p.sso[ll]);
    for (int i = threadIdx.x; i < nk * RS / VEC; i += TH) ((float4*)s)[i] = src[i];
  }
  const int mine = tc[half * 32 + lane];
  const bool live = mine >= 0;
  const int c = live ? mine : tc[0];
  const bool act = live && ll < p.admis[c];
  const bool any = __any_sync(0xffffffffu, act);
  __syncthreads();
  int slot = 0;
  unsigned ph = 0;  // phase of the ring's current round
  bool ok = true;
  if (role >= R::NSL) {
    slot = role - R::NSL;  // this producer's first stage
    if (any) {
      const GatherShare sh(lane);
      const int32_t* S = p.sten + (int64_t)(c >> 5) * (A * W) * 32 + (c & 31) + (ll * W + 1) * 32;
      auto member = [&](int k) -> int { return act ? S[(k < nk ? k : nk - 1) * 32] : c; };
      double u0[NV];
      sh.load(U, c, u0);
      int y[MS];
#pragma unroll
      for (int j = 0; j < MS; ++j) y[j] = member(slot * MS + j);
      for (int k = slot * MS; k < nk; k += R::NPR * MS) {
        double u[MS][NV];
#pragma unroll
        for (int j = 0; j < MS; ++j) sh.load(U, y[j], u[j]);
#pragma unroll
        for (int j = 0; j < MS; ++j) y[j] = member(k + R::NPR * MS + j);
        if (!(ok = set_wait(&empty[slot], ph ^ 1u, &s_limit))) break;  // the first round finds them empty
        T* du = ring + slot * R::elems + lane;
#pragma unroll
        for (int j = 0; j < MS; ++j)
#pragma unroll
          for (int i = 0; i < NV; ++i) du[(j * NV + i) * 32] = T(u[j][i] - u0[i]);
        __syncwarp();
        if (lane == 0) mbar_arrive(&full[slot]);
        if ((slot += R::NPR) >= NSTG) slot -= NSTG, ph ^= 1u;
      }
    }
  } else {
    // this warp's vectors of rows [q0, q0 + NQ), NQ = MAXV or one less
    const int q0 = role * R::NVEC / R::NSL, nq = (role + 1) * R::NVEC / R::NSL - q0;
    auto multiply = [&](auto nqc) {
      constexpr int NQ = decltype(nqc)::value;
      RowAcc<T> acc[NQ];
#pragma unroll
      for (int q = 0; q < NQ; ++q) acc[q].zero();
      auto add = [&](const T* m, const T* d) {
        T du[NV];
#pragma unroll
        for (int v = 0; v < NV; ++v) du[v] = d[v];
#pragma unroll
        for (int q = 0; q < NQ; ++q) acc[q].add(m + q * VEC, du);
      };
      if (any)
        for (int k = 0; k < nk; k += MS) {
          if (!(ok = set_wait(&full[slot], ph, &s_limit))) break;
          const T* d = ring + slot * R::elems + lane * NV;
          const T* m = s + k * RS + q0 * VEC;
          if (k + MS <= nk) {
#pragma unroll
            for (int j = 0; j < MS; ++j) add(m + j * RS, d + j * 32 * NV);
          } else {
            for (int j = 0; j < nk - k; ++j) add(m + j * RS, d + j * 32 * NV);
          }
          __syncwarp();
          if (lane == 0) mbar_arrive(&empty[slot]);
          if (++slot == NSTG) slot = 0, ph ^= 1u;
        }
      T* Gi = (T*)p.gbuf + (int64_t)(c >> 5) * (A * ID * NV) * 32 + (int64_t)(ll * ID + q0 * VEC) * NV * 32 + (c & 31);
      if (ok && live)
#pragma unroll
        for (int q = 0; q < NQ; ++q)
#pragma unroll
          for (int i = 0; i < VEC; ++i)
            if ((q0 + q) * VEC + i < ND)
#pragma unroll
              for (int v = 0; v < NV; ++v) Gi[(int64_t)((q * VEC + i) * NV + v) * 32] = act ? acc[q].get(i, v) : T(0);
    };
    if (R::NVEC % R::NSL == 0 || nq == R::MAXV) multiply(IntC<R::MAXV>());
    else multiply(IntC<(R::MAXV > 1 ? R::MAXV - 1 : 1)>());
  }
  if (!ok && lane == 0) {
    atomicOr(p.health, HEALTH_TIMEOUT);
    *(volatile int*)&s_limit = -1;
  }
}

// The CWENO directional stencils (ND = IDEGFREE2 rows of a few members) of the
// tiled cells: a tile and a stencil per block, one lane per cell; a warp
// gathers four members at a time through its own shared-memory buffer.
template <int P, typename T, int ND>
__global__ void __launch_bounds__(SET_TILE) k_lsq_low(Problem p, const double* __restrict__ U) {
  constexpr int ID = Deg<P>::ideg;
  constexpr int RS = set_stride<T>(ND);
  constexpr int VEC = Vec<T>::N;
  constexpr int GRP = 4;
  extern __shared__ __align__(16) unsigned char lw_smem[];
  __shared__ T s_du[SET_TILE / 32][GRP][32 * NV];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t tile = blockIdx.x;
  const int ll = blockIdx.y + 1;
  const int nk = p.imax2, A = p.admis_max, W = p.imax + 1;
  T* s = (T*)lw_smem;
  {
    const float4* src = (const float4*)((const T*)p.setmat + p.tset[tile] * p.sstride + p.sso[ll]);
    for (int i = threadIdx.x; i < nk * RS / VEC; i += SET_TILE) ((float4*)s)[i] = src[i];
  }
  const int mine = p.tcell[tile * SET_TILE + threadIdx.x];
  const bool live = mine >= 0;
  const int c = live ? mine : p.tcell[tile * SET_TILE];
  const bool act = live && ll < p.admis[c];
  const int32_t* S = p.sten + (int64_t)(c >> 5) * (A * W) * 32 + (c & 31) + (ll * W + 1) * 32;
  const GatherShare sh(lane);
  double u0[NV];
  sh.load(U, c, u0);
  T acc[ND][NV];
#pragma unroll
  for (int j = 0; j < ND; ++j)
#pragma unroll
    for (int v = 0; v < NV; ++v) acc[j][v] = T(0);
  __syncthreads();
  for (int k = 0; k < nk; k += GRP) {
    double u[GRP][NV];
#pragma unroll
    for (int j = 0; j < GRP; ++j) sh.load(U, act ? S[(k + j < nk ? k + j : nk - 1) * 32] : c, u[j]);
    __syncwarp();  // the last group's differences have been read
#pragma unroll
    for (int j = 0; j < GRP; ++j)
#pragma unroll
      for (int i = 0; i < NV; ++i) s_du[warp][j][lane + 32 * i] = T(u[j][i] - u0[i]);
    __syncwarp();
#pragma unroll
    for (int j = 0; j < GRP; ++j)
      if (k + j < nk) {
        T du[NV];
#pragma unroll
        for (int v = 0; v < NV; ++v) du[v] = s_du[warp][j][lane * NV + v];
#pragma unroll
        for (int q = 0; q < RS / VEC; ++q) {
          T r[VEC];
          ldv(s + (k + j) * RS + q * VEC, r);
#pragma unroll
          for (int i = 0; i < VEC; ++i)
            if (q * VEC + i < ND)
#pragma unroll
              for (int v = 0; v < NV; ++v) acc[q * VEC + i][v] += r[i] * du[v];
        }
      }
  }
  if (!live) return;
  T* Gi = (T*)p.gbuf + (int64_t)(c >> 5) * (A * ID * NV) * 32 + (int64_t)(ll * ID) * NV * 32 + (c & 31);
#pragma unroll
  for (int j = 0; j < ND; ++j)
#pragma unroll
    for (int v = 0; v < NV; ++v) Gi[(int64_t)(j * NV + v) * 32] = act ? acc[j][v] : T(0);
}

// Smoothness indicators of the tiled cells: a tile and a stencil per block,
// the set's triangle in shared memory as 16-byte broadcasts, two variables of
// the cell's polynomial in registers per pass (one would leave the kernel
// bound by the shared-memory loads).  k_wis, whose warps read each cell's own
// copy of the triangle, takes the other cells.
template <int P, typename T>
__global__ void __launch_bounds__(SET_TILE) k_wis_set(Problem p) {
  constexpr int ID = Deg<P>::ideg;
  constexpr int VEC = Vec<T>::N;
  constexpr int VI = 2;
  extern __shared__ __align__(16) unsigned char wi_smem[];
  T* s = (T*)wi_smem;
  const int64_t tile = blockIdx.x;
  const int ll = blockIdx.y, A = p.admis_max;
  {
    const float4* tri = (const float4*)((const T*)p.setind + p.tset[tile] * p.istride);
    for (int i = threadIdx.x; i < p.i2off / VEC; i += SET_TILE) ((float4*)s)[i] = tri[i];
  }
  __syncthreads();
  const int64_t c = p.tcell[tile * SET_TILE + threadIdx.x];
  if (c < 0 || (!p.mprev && !p.full[c]) || ll >= p.admis[c]) return;
  const T* Gc = (const T*)p.gbuf + (c >> 5) * (int64_t)(A * ID * NV) * 32 + (int64_t)(ll * ID) * NV * 32 + (c & 31);
  double* o = p.isb + (((c >> 5) * A + ll) * (int64_t)NV) * 32 + (c & 31);
#pragma unroll 1
  for (int v0 = 0; v0 < NV; v0 += VI) {
    T g[ID][VI], is[VI];
#pragma unroll
    for (int d = 0; d < ID; ++d)
#pragma unroll
      for (int k = 0; k < VI; ++k) g[d][k] = v0 + k < NV ? Gc[(int64_t)(d * NV + v0 + k) * 32] : T(0);
#pragma unroll
    for (int k = 0; k < VI; ++k) is[k] = T(0);
    int rs = 0;
#pragma unroll
    for (int d = 0; d < ID; ++d) {
      T t[VI];
#pragma unroll
      for (int k = 0; k < VI; ++k) t[k] = T(0);
#pragma unroll
      for (int q = 0; q < (ID - d + VEC - 1) / VEC; ++q) {
        T x[VEC];
        ldv(s + (rs + q) * VEC, x);
#pragma unroll
        for (int i = 0; i < VEC; ++i)
          if (d + q * VEC + i < ID)
#pragma unroll
            for (int k = 0; k < VI; ++k) t[k] += x[i] * g[d + q * VEC + i][k];
      }
      rs += (ID - d + VEC - 1) / VEC;
#pragma unroll
      for (int k = 0; k < VI; ++k) is[k] += g[d][k] * t[k];
      asm volatile("" ::: "memory");  // as in quad_form
    }
#pragma unroll
    for (int k = 0; k < VI; ++k)
      if (v0 + k < NV) o[(v0 + k) * 32] = (double)is[k];
  }
}

// LEAST_SQUARES of the cells that read their own tables: the pseudo-inverse
// rows and the gathered differences come through shared memory.  One or two
// blocks per SM, four pairs of warps: a producer gathers the members'
// differences (as in k_lsq_set) into a stage of its pair's ring and issues the
// bulk copies (cp.async.bulk) of the members' rows [d0, d0 + DH) of the 32
// cells, which are contiguous in the interleaved layout; the consumer
// multiplies.  The full barrier of a stage completes on the producer's arrival
// and the copied bytes, the empty barrier on the consumer's arrival.  The
// kernel is bound by the table bytes from DRAM.  One lane per cell holding the
// accumulators and the loads in flight was bound by the bytes that its
// registers left room for and by the chain index -> state -> product of each
// member; here the copies run NSTG stages ahead.  The work is the list of
// (group, stencil) items, an equal share of consecutive items per pair, so
// that a mesh of any size fills the SMs (one lane per cell: 16,464 cells were
// 129 blocks).  With tiles (p.ntile) the groups are those with cells that are
// not tiled (p.ugrp).  Against one lane per cell: 16,464 tetrahedra, WENO5
// mixed, 0.500 -> 0.257 ms (1.63 GB, 6.3 TB/s); 82,944, WENO3, FP64 0.312 ->
// 0.201 (6.4 TB/s), mixed 0.205 -> 0.190; 24,576, CWENO4, FP64 0.160 -> 0.107,
// mixed 0.237 -> 0.067; two blocks per SM at IORDER 2 and 3 against one: 0.267
// -> 0.201 (WENO3 FP64), 0.121 -> 0.067 (CWENO4 mixed).
//
// Every wait is bounded (`wait` polls).  A wait that gives up sets
// HEALTH_TIMEOUT and s_stop; the other warps see it in their own waits, and a
// producer leaves only after its copies in flight have landed (each wait
// bounded by LSQ_WAIT, whatever `wait` is).
template <int P, typename T>
struct Ring {
  static constexpr int DH = LsqRows<P, T>::value;
  static constexpr int TAB = DH * 32 * sizeof(T), DU = NV * 32 * sizeof(T);  // of a member
  static constexpr int MS = 2;                                               // members of a stage
  static constexpr int STAGE = MS * (TAB + DU);
  // blocks per SM: two where the accumulators leave room (128 registers)
  static constexpr int BPS = DH * NV * sizeof(T) <= 400 ? 2 : 1;
  static constexpr int NSTG = 56000 / BPS / STAGE < 8 ? 56000 / BPS / STAGE : 8;
  static constexpr int GRP = 4;  // members that a producer gathers together
  static constexpr size_t smem = (size_t)4 * NSTG * STAGE;
};
template <int P, typename T>
__global__ void __launch_bounds__(256, Ring<P, T>::BPS) k_lsq_ring(Problem p, const double* __restrict__ U, int64_t items, long wait) {
  using R = Ring<P, T>;
  constexpr int ID = Deg<P>::ideg, DH = R::DH, NSTG = R::NSTG, GRP = R::GRP, MS = R::MS;
  extern __shared__ __align__(128) unsigned char rg_smem[];
  __shared__ __align__(8) uint64_t s_full[4][NSTG], s_empty[4][NSTG];
  __shared__ int s_stop;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, pair = warp & 3;
  const bool producer = warp >= 4;
  unsigned char* ring = rg_smem + (size_t)pair * NSTG * R::STAGE;
  uint64_t *full = s_full[pair], *empty = s_empty[pair];
  if (threadIdx.x == 0) {
    s_stop = 0;
    for (int w = 0; w < 4; ++w)
      for (int s = 0; s < NSTG; ++s) {
        mbar_init(&s_full[w][s], 1);
        mbar_init(&s_empty[w][s], 1);
      }
    mbar_fence_init();
  }
  __syncthreads();
  const int A = p.admis_max, W = p.imax + 1;
  const bool cw = p.ees == 5;
  const int64_t pairs = (int64_t)gridDim.x * 4, me = (int64_t)blockIdx.x * 4 + pair;
  const int64_t i0 = items * me / pairs, i1 = items * (me + 1) / pairs;
  const GatherShare sh(lane);
  int slot = 0;
  unsigned ph = 0;  // phase of the ring's current round
  int issued = 0;   // producer: stages filled, for the drain
  bool ok = true;
  for (int64_t it = i0; it < i1 && ok; ++it) {
    const int64_t g = it / A;
    const int ll = (int)(it - g * A);
    const int64_t grp = p.ntile ? p.ugrp[g] : g, c = grp * 32 + lane;
    const bool low = cw && ll > 0, live = c < p.n && !(p.ntile && p.tiled[c]);
    const int nk = low ? p.imax2 : p.imax, nd = low ? p.ideg2 : ID;
    const bool act = live && ll < p.admis[c];
    const bool any = __any_sync(0xffffffffu, act);
    if (producer) {
      if (!any) continue;
      const int32_t* S = p.sten + (grp * (int64_t)(A * W) + ll * W + 1) * 32 + lane;
      const int own = (int)(c < p.n ? c : grp * 32);
      auto member = [&](int k) -> int { return act ? S[(k < nk ? k : nk - 1) * 32] : own; };
      double u0[NV];
      sh.load(U, own, u0);
      const T* M = (const T*)p.invmat + (grp * p.tstride + p.soff[ll]) * 32;
      for (int d0 = 0; d0 < nd && ok; d0 += DH) {
        const unsigned bytes = (unsigned)((nd - d0 < DH ? nd - d0 : DH) * 32 * sizeof(T));
        int y[GRP];
#pragma unroll
        for (int j = 0; j < GRP; ++j) y[j] = member(j);
        for (int k = 0; k < nk && ok; k += GRP) {
          double u[GRP][NV];
#pragma unroll
          for (int j = 0; j < GRP; ++j) sh.load(U, y[j], u[j]);
#pragma unroll
          for (int j = 0; j < GRP; ++j) y[j] = member(k + GRP + j);
#pragma unroll
          for (int j0 = 0; j0 < GRP; j0 += MS) {
            if (k + j0 >= nk) break;
            if (!(ok = ring_wait(&empty[slot], ph ^ 1u, wait, &s_stop))) break;  // the first round finds them empty
            unsigned char* st = ring + slot * R::STAGE;
            T* du = (T*)(st + MS * R::TAB) + lane;
#pragma unroll
            for (int j = 0; j < MS; ++j)
#pragma unroll
              for (int i = 0; i < NV; ++i) du[(j * NV + i) * 32] = T(u[j0 + j][i] - u0[i]);
            __syncwarp();
            if (lane == 0) {
              const int km = nk - k - j0 < MS ? nk - k - j0 : MS;
              fence_proxy_async();
              mbar_expect_tx(&full[slot], bytes * km);
              for (int j = 0; j < km; ++j)
                bulk_g2s(st + j * R::TAB, M + ((int64_t)(k + j0 + j) * nd + d0) * 32, bytes, &full[slot]);
            }
            ++issued;
            if (++slot == NSTG) slot = 0, ph ^= 1u;
          }
        }
      }
    } else {
      T* Gi = (T*)p.gbuf + grp * (int64_t)(A * ID * NV) * 32 + (int64_t)(ll * ID) * NV * 32 + lane;
      for (int d0 = 0; d0 < nd && ok; d0 += DH) {
        T acc[DH][NV];
#pragma unroll
        for (int j = 0; j < DH; ++j)
#pragma unroll
          for (int v = 0; v < NV; ++v) acc[j][v] = T(0);
        if (any)
          for (int k = 0; k < nk; k += MS) {
            if (!(ok = ring_wait(&full[slot], ph, wait, &s_stop))) break;
            const unsigned char* st = ring + slot * R::STAGE;
            const T* m = (const T*)st + lane;
            const T* d = (const T*)(st + MS * R::TAB) + lane * NV;
            const int km = nk - k < MS ? nk - k : MS;
#pragma unroll 1
            for (int q = 0; q < km; ++q, m += R::TAB / sizeof(T), d += 32 * NV) {
              T du[NV];
#pragma unroll
              for (int v = 0; v < NV; ++v) du[v] = d[v];
#pragma unroll
              for (int j = 0; j < DH; ++j)
                if (d0 + j < nd) {
                  const T r = m[j * 32];
#pragma unroll
                  for (int v = 0; v < NV; ++v) acc[j][v] += r * du[v];
                }
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(&empty[slot]);
            if (++slot == NSTG) slot = 0, ph ^= 1u;
          }
        if (ok && live)
#pragma unroll
          for (int j = 0; j < DH; ++j)
            if (d0 + j < nd)
#pragma unroll
              for (int v = 0; v < NV; ++v) Gi[(int64_t)((d0 + j) * NV + v) * 32] = act ? acc[j][v] : T(0);
      }
    }
  }
  if (!ok && lane == 0) {
    atomicOr(p.health, HEALTH_TIMEOUT);
    *(volatile int*)&s_stop = 1;
  }
  if (producer) {  // no copy may be in flight into a block that has ended
    const int nout = issued < NSTG ? issued : NSTG;
    for (int j = 0; j < nout; ++j) {
      if (--slot < 0) slot = NSTG - 1, ph ^= 1u;
      mbar_wait(&full[slot], ph, LSQ_WAIT);
    }
  }
}

// LEAST_SQUARES at IORDER 1, one lane per cell: three rows a stencil are so
// little that the accumulators leave room for the loads, and what a block of
// k_lsq_ring or k_lsq_set sets up before its first product does not pay.  From 128
// cells per SM on (below, one wave of lanes waits for its own loads: 512 cells 15
// us, the ring 11; 8,000 17, 15).  In FP64 and FP32: 114,048 mixed cells WENO 64 and
// 57 us, the ring 96 and 92, tiles 109 and 80, CWENO 66 and 56, 89 and 83, 109 and
// 91; 33,408 cells 33 and 22, 36 and 31, 41 and 34.
template <int P, typename T>
__global__ void __launch_bounds__(128, 1) k_lsq_lane(Problem p, const double* __restrict__ U) {
  constexpr int ID = Deg<P>::ideg;
  const int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int A = p.admis_max, W = p.imax + 1;
  const int64_t grp = c >> 5;
  const int lane = (int)(c & 31);
  const bool live = c < p.n;
  const int adm = live ? p.admis[c] : 0;
  double u0[NV];
#pragma unroll
  for (int v = 0; v < NV; ++v) u0[v] = live ? U[c * NV + v] : 0.0;
  const T* Mi = (const T*)p.invmat + grp * p.tstride * 32 + lane;
  const int32_t* Si = p.sten + grp * (int64_t)(A * W) * 32 + lane;
  T* Gi = (T*)p.gbuf + grp * (int64_t)(A * ID * NV) * 32 + lane;
  for (int ll = 0; ll < A; ++ll) {
    const bool low = p.ees == 5 && ll > 0;
    const int nk = low ? p.imax2 : p.imax, nd = low ? p.ideg2 : ID;
    T acc[ID][NV];
#pragma unroll
    for (int d = 0; d < ID; ++d)
#pragma unroll
      for (int v = 0; v < NV; ++v) acc[d][v] = T(0);
    if (ll < adm) {
      const T* M = Mi + (int64_t)p.soff[ll] * 32;
      const int32_t* S = Si + (ll * W + 1) * 32;
#pragma unroll 2
      for (int k = 0; k < nk; ++k) {
        const double* uy = U + (int64_t)S[k * 32] * NV;
        T du[NV];
#pragma unroll
        for (int v = 0; v < NV; ++v) du[v] = T(uy[v] - u0[v]);
        const T* Mk = M + (int64_t)k * nd * 32;
#pragma unroll
        for (int d = 0; d < ID; ++d)
          if (d < nd) {
            const T m = Mk[d * 32];
#pragma unroll
            for (int v = 0; v < NV; ++v) acc[d][v] += m * du[v];
          }
      }
    }
    if (live)
#pragma unroll
      for (int d = 0; d < ID; ++d)
        if (d < nd)
#pragma unroll
          for (int v = 0; v < NV; ++v) Gi[(int64_t)((ll * ID + d) * NV + v) * 32] = acc[d][v];
  }
}

// the cells' own tables: all groups, or those with cells that are not tiled
template <int P, typename T>
cudaError_t launch_lsq_ring(const Problem& p, const double* U, cudaStream_t st) {
  using R = Ring<P, T>;
  const cudaError_t e = smem_limit(k_lsq_ring<P, T>, R::smem);
  if (e != cudaSuccess) return e;
  const int64_t items = (p.ntile ? p.nugrp : (p.n + 31) / 32) * p.admis_max, nb = (items + 3) / 4;
  k_lsq_ring<P, T><<<(unsigned)(nb < p.nsm * R::BPS ? nb : p.nsm * R::BPS), 256, R::smem, st>>>(p, U, items, lsq_wait(p));
  return cudaGetLastError();
}

// the least squares of the tiled cells, and of the others through k_lsq_ring
template <int P, typename T, int ND>
cudaError_t launch_lsq_set_t(const Problem& p, const double* U, unsigned nst, cudaStream_t st) {
  using R = SetRing<T, ND>;
  const size_t smem = ((size_t)p.imax * set_stride<T>(ND) + SET_RING) * sizeof(T);
  const cudaError_t e = smem_limit(k_lsq_set<P, T, ND>, SET_SMEM);
  if (e != cudaSuccess) return e;
  k_lsq_set<P, T, ND><<<dim3((unsigned)p.ntile * 2, nst), 32 * R::WARPS, smem, st>>>(p, U, (int)(lsq_wait(p) < LSQ_WAIT ? lsq_wait(p) : LSQ_WAIT));
  return cudaGetLastError();
}
template <int P, typename T, int ND>
cudaError_t launch_lsq_low(const Problem& p, const double* U, cudaStream_t st) {
  const size_t smem = (size_t)p.imax2 * set_stride<T>(ND) * sizeof(T);
  const cudaError_t e = smem_limit(k_lsq_low<P, T, ND>, LOW_SMEM);
  if (e != cudaSuccess) return e;
  k_lsq_low<P, T, ND><<<dim3((unsigned)p.ntile, (unsigned)p.admis_max - 1), SET_TILE, smem, st>>>(p, U);
  return cudaGetLastError();
}
// The tiled cells' indicators come from k_wis_set: IORDER 4 (the only order
// with indicators of their own kernel) without CWENO, whose central polynomial
// (the central stencil less the directional ones) only k_wis forms.
template <int P>
bool sets_give_is(const Problem& p) {
  return P == 4 && p.ntile && p.isb && p.scheme == 3 && p.ees != 5;
}
template <int P, typename T>
cudaError_t launch_lsq_set(const Problem& p, const double* U, cudaStream_t st, int64_t* launches) {
  constexpr int ID = Deg<P>::ideg;
  const bool cw = p.ees == 5 && p.admis_max > 1;
  cudaError_t e = launch_lsq_set_t<P, T, ID>(p, U, cw ? 1 : (unsigned)p.admis_max, st);
  if (e == cudaSuccess && cw) {
    if constexpr (P > 1) {
      if (p.ideg2 == 9) e = launch_lsq_low<P, T, 9>(p, U, st);
    }
    if (p.ideg2 == 3) e = launch_lsq_low<P, T, 3>(p, U, st);
    ++*launches;
  }
  if (e == cudaSuccess && p.nugrp) {
    e = launch_lsq_ring<P, T>(p, U, st);
    ++*launches;
  }
  return e;
}

// the stencil polynomials of every cell into p.gbuf, from the state U
template <int P, typename T>
cudaError_t launch_lsq(const Problem& p, const double* U, cudaStream_t st, int64_t* launches) {
  ++*launches;
  if constexpr (P == 1) {
    if (!p.lsq_bulk && !p.ntile && p.n >= (int64_t)p.nsm * 128) {
      k_lsq_lane<P, T><<<(unsigned)((p.n + 127) / 128), 128, 0, st>>>(p, U);
      return cudaGetLastError();
    }
  }
  return p.ntile ? launch_lsq_set<P, T>(p, U, st, launches) : launch_lsq_ring<P, T>(p, U, st);
}

// ------------------------------------------------------------- k_wpost
// Smoothness matrices are packed upper triangles, interleaved over 32-cell
// groups like the pseudo-inverses: entry (d, e >= d) of cell c is element
// tri(d, e) = d*nd - d*(d-1)/2 + (e - d) of the cell's block, and an
// off-diagonal entry holds S_de + S_ed, so that
//   g^T S g = sum_d g_d * sum_{e >= d} P_de g_e
// is the full quadratic form of INDICATORMATRIX (src/prestore.f90:1529-1673)
// with half the loads and multiplies.

// variables per register pass of each phase: indicators (IS), combined
// polynomial + face values (FACE), MUSCL fall-back (FALL); the polynomial
// of a pass ([ID] x variables) stays in registers.  Measured on the 64^3
// WENO5 stage (B200): FP32 FACE 5 takes 1.95 ms against 2.75 ms for 3 and
// 3.17 ms for 2 (one read of the polynomials, CHECKSOL in registers); FP64
// IS 3 / FACE 3 takes 6.50 ms against 6.95 ms for 2 / 2, 8.11 ms for IS 1
// and 7.46 ms for FACE 5 (spills).
#ifndef UCG_WV_IS_F
#define UCG_WV_IS_F 5
#endif
#ifndef UCG_WV_FACE_F
#define UCG_WV_FACE_F 5
#endif
#ifndef UCG_WV_FALL_F
#define UCG_WV_FALL_F 1
#endif
#ifndef UCG_WV_IS_D
#define UCG_WV_IS_D 3
#endif
#ifndef UCG_WV_FACE_D
#define UCG_WV_FACE_D 3
#endif
#ifndef UCG_WV_FALL_D
#define UCG_WV_FALL_D 1
#endif
template <typename T>
struct WVars {
  static constexpr int is = sizeof(T) == 4 ? UCG_WV_IS_F : UCG_WV_IS_D;
  static constexpr int face = sizeof(T) == 4 ? UCG_WV_FACE_F : UCG_WV_FACE_D;
  static constexpr int fall = sizeof(T) == 4 ? UCG_WV_FALL_F : UCG_WV_FALL_D;
};

// is[k] += sum_d g[d][k] * sum_{e>=d} P_de g[e][k] over d, e < nd <= NMAX.
// P: the cell's packed triangle, vector-interleaved (rows padded to VEC);
// entries past nd in a row's last vector are zero, and so is g[e] for e >= nd.
template <int NMAX, int VG, typename T>
__device__ __forceinline__ void quad_form(const T* __restrict__ P, const T (&g)[NMAX][VG], int nd, T (&is)[VG]) {
  constexpr int VEC = Vec<T>::N;
  int rs = 0;  // first vector of row d
#pragma unroll
  for (int d = 0; d < NMAX; ++d) {
    if (d < nd) {
      T t[VG];
#pragma unroll
      for (int k = 0; k < VG; ++k) t[k] = T(0);
#pragma unroll
      for (int q = 0; q < (NMAX - d + VEC - 1) / VEC; ++q)
        if (d + q * VEC < nd) {
          T s[VEC];
          ldv(P + (int64_t)(rs + q) * 32 * VEC, s);
#pragma unroll
          for (int i = 0; i < VEC; ++i)
            if (d + q * VEC + i < NMAX)
#pragma unroll
              for (int k = 0; k < VG; ++k) t[k] += s[i] * g[d + q * VEC + i][k];
        }
      rs += (nd - d + VEC - 1) / VEC;
#pragma unroll
      for (int k = 0; k < VG; ++k) is[k] += g[d][k] * t[k];
      // keep the loads of one row together: without this fence the
      // compiler hoists the whole triangle and spills it
      asm volatile("" ::: "memory");
    }
  }
}

// Smoothness indicators IS[ll][v] = g^T S g of every stencil polynomial,
// one block per 32-cell group with one warp per stencil: lane i of warp ll
// takes stencil ll of cell i of the group.  The warps of a block read the
// same packed triangles (the cells' INDICATOR, prestore.f90:1529-1673) at
// about the same time, so each triangle comes from DRAM once and is reused
// from L1/L2 by the other stencils, instead of once per stencil as when one
// lane runs all the stencils of its cell.  Output: p.isb, FP64, interleaved
// over 32-cell groups ((group * A + ll) * NV + v) * 32 + lane; cells that
// take the MUSCL fall-back outright (not FULL) are skipped, except under
// MOOD, where every cell is reconstructed.  MASK: not the cells of p.tiled.
template <int P, typename T, bool MASK = false>
__global__ void __launch_bounds__(224) k_wis(Problem p) {
  constexpr int ID = Deg<P>::ideg;
  constexpr int VEC = Vec<T>::N;
  constexpr int L2 = ID < 9 ? ID : 9;
  constexpr int VI = WVars<T>::is;
  const int lane = threadIdx.x & 31, ll = threadIdx.x >> 5;
  const int64_t grp = blockIdx.x, c = grp * 32 + lane;
  if (c >= p.n || (!p.mprev && !p.full[c])) return;
  if (MASK && p.tiled[c]) return;
  const int adm = p.admis[c];
  if (ll >= adm) return;
  const int A = p.admis_max, ID2 = p.ideg2;
  const bool cw = p.ees == 5, low = cw && ll > 0;
  const T* Gc = (const T*)p.gbuf + grp * (int64_t)(A * ID * NV) * 32 + lane;
  auto G = [&](int l, int d, int v) -> T { return Gc[(int64_t)((l * ID + d) * NV + v) * 32]; };
  const double lc1 = 1.0 - 1.0 / p.lwci;
  const double lk = adm > 1 ? (1.0 - lc1) / (adm - 1) : 0.0;
  const T* Pc = (const T*)p.ind + grp * p.istride * 32 + lane * VEC;
  double* out = p.isb + (grp * A + ll) * (int64_t)NV * 32 + lane;
  for (int v0 = 0; v0 < NV; v0 += VI) {
    T is[VI];
#pragma unroll
    for (int k = 0; k < VI; ++k) is[k] = T(0);
    if (low) {
      T g[L2][VI];
#pragma unroll
      for (int d = 0; d < L2; ++d)
#pragma unroll
        for (int k = 0; k < VI; ++k) g[d][k] = (v0 + k < NV && d < ID2) ? G(ll, d, v0 + k) : T(0);
      quad_form<L2, VI>(Pc + (int64_t)(p.i2off / VEC) * 32 * VEC, g, ID2, is);
    } else {
      T g[ID][VI];
#pragma unroll
      for (int d = 0; d < ID; ++d)
#pragma unroll
        for (int k = 0; k < VI; ++k) g[d][k] = (v0 + k < NV) ? G(ll, d, v0 + k) : T(0);
      if (ll == 0 && cw) {  // the CWENO central polynomial with the lower-order stencils removed
        T g3[L2][VI];
#pragma unroll
        for (int d = 0; d < L2; ++d)
#pragma unroll
          for (int k = 0; k < VI; ++k) g3[d][k] = T(0);
        for (int l2 = 1; l2 < adm; ++l2)
#pragma unroll
          for (int d = 0; d < L2; ++d)
#pragma unroll
            for (int k = 0; k < VI; ++k)
              if (v0 + k < NV && d < ID2) g3[d][k] = g3[d][k] + T(lk) * G(l2, d, v0 + k);
#pragma unroll
        for (int d = 0; d < ID; ++d)
#pragma unroll
          for (int k = 0; k < VI; ++k)
            if (v0 + k < NV) g[d][k] = T(1.0 / lc1) * (g[d][k] - (d < L2 ? g3[d][k] : T(0)));
      }
      quad_form<ID, VI>(Pc, g, ID, is);
    }
#pragma unroll
    for (int k = 0; k < VI; ++k)
      if (v0 + k < NV) out[(int64_t)(v0 + k) * 32] = (double)is[k];
  }
}

// k_wface (conserved-variable WENO; IORDER 4: indicators from k_wis): the
// nonlinear weights, the combined polynomial and its face values, one block
// per 32-cell group with one warp per conserved variable (lane i: cell i of
// the group).  A thread holds one variable's combined polynomial (ID
// coefficients) instead of all five, so the block runs at several times
// k_wpost's occupancy.  The group's face points are staged in shared memory
// once (the five warps evaluate at the same points); the values of one face
// go through shared memory, [cell][point][variable] with an odd row stride
// (no bank conflicts), from where the block tests CHECKSOL (0.85) and stores
// them as one contiguous run per cell.  Cells that fail CHECKSOL, or are not
// FULL, are marked in p.wflag for k_wpost<..., FB> (the MUSCL fall-back).
// Weights, combination and face values take k_wpost's operations in
// k_wpost's order.  Under MOOD the cells that are not FULL are reconstructed
// too (over their admissible stencils) and marked.
// OWN (IORDER 1-3, where wface_own says so): each warp forms its variable's
// indicators itself, g^T S g of one polynomial at a time from the cells'
// triangles, which the five warps read from L1.
template <typename T>
__host__ __device__ constexpr size_t wface_smem(int QS) {
  return ((size_t)MF * QS * 3 + ((QS * NV) | 1)) * 32 * sizeof(T);
}
template <int P, typename T, bool OWN = false>
__global__ void __launch_bounds__(32 * NV) k_wface(Problem p, const double* __restrict__ U) {
  constexpr int ID = Deg<P>::ideg;
  constexpr int L2 = ID < 9 ? ID : 9;
  constexpr int MA = 7;  // stencils per cell at most
  extern __shared__ __align__(16) unsigned char wf_smem[];
  __shared__ int s_flag[32];
  const int QS = p.nq_quad > p.nq_tri ? p.nq_quad : p.nq_tri;
  const int FQ = MF * QS;
  const int RS = (QS * NV) | 1;  // row stride of a cell in s_o
  T* s_x = (T*)wf_smem;          // [FQ * 3][32]: the group's face points, as in p.qpts
  T* s_o = s_x + FQ * 3 * 32;    // [32][RS]: the values of one face
  const int tid = threadIdx.x, lane = tid & 31, v = tid >> 5;
  const int64_t grp = blockIdx.x, c = grp * 32 + lane;
  {
    const T* xg = (const T*)p.qpts + grp * (int64_t)FQ * 3 * 32;
    for (int i = tid; i < FQ * 3 * 32; i += 32 * NV) s_x[i] = __ldcs(xg + i);
  }
  const bool cell = c < p.n;
  const bool full = cell && p.full[c];
  const bool live = cell && (full || p.mprev);
  const int A = p.admis_max;
  const int adm = live ? p.admis[c] : 0;
  const bool cw = p.ees == 5;
  const int ID2 = p.ideg2;
  const double lc1 = 1.0 - 1.0 / p.lwci;
  const double lk = adm > 1 ? (1.0 - lc1) / (adm - 1) : 0.0;
  if (tid < 32) s_flag[tid] = full ? 0 : 1;
  const T* Gc = (const T*)p.gbuf + grp * (int64_t)(A * ID * NV) * 32 + v * 32 + lane;
  auto G = [&](int l, int d) -> T { return Gc[(int64_t)((l * ID + d) * NV) * 32]; };
  // the central polynomial (CWENO: the central stencil with the lower-order
  // ones removed, reconstruct_p.f90:956-965)
  auto central = [&](T (&g)[ID]) {
#pragma unroll
    for (int d = 0; d < ID; ++d) g[d] = live ? G(0, d) : T(0);
    if (live && cw) {
      T g3[L2];
#pragma unroll
      for (int d = 0; d < L2; ++d) g3[d] = T(0);
      for (int l2 = 1; l2 < adm; ++l2)
#pragma unroll
        for (int d = 0; d < L2; ++d)
          if (d < ID2) g3[d] = g3[d] + T(lk) * G(l2, d);
#pragma unroll
      for (int d = 0; d < ID; ++d) g[d] = T(1.0 / lc1) * (g[d] - (d < L2 ? g3[d] : T(0)));
    }
  };
  // ---- weights of variable v (WENOWEIGHTS, FP64)
  double w[MA];
  {
    const double* isg = OWN ? nullptr : p.isb + grp * (int64_t)A * NV * 32 + lane + v * 32;
    double is[MA];
    if constexpr (OWN) {
      constexpr int VEC = Vec<T>::N;
      const T* Pc = (const T*)p.ind + grp * p.istride * 32 + lane * VEC;
#pragma unroll
      for (int l = 0; l < MA; ++l) {
        is[l] = 0.0;
        if (l < adm) {
          T q[1] = {T(0)};
          if (cw && l > 0) {
            T g[L2][1];
#pragma unroll
            for (int d = 0; d < L2; ++d) g[d][0] = d < ID2 ? G(l, d) : T(0);
            quad_form<L2, 1>(Pc + (int64_t)(p.i2off / VEC) * 32 * VEC, g, ID2, q);
          } else {
            T c0[ID], g[ID][1];
            if (l == 0) central(c0);
#pragma unroll
            for (int d = 0; d < ID; ++d) g[d][0] = l == 0 ? c0[d] : G(l, d);
            quad_form<ID, 1>(Pc, g, ID, q);
          }
          is[l] = (double)q[0];
        }
      }
    } else {
#pragma unroll
      for (int l = 0; l < MA; ++l) is[l] = l < adm ? isg[(int64_t)l * NV * 32] : 0.0;
    }
    const double lam0 = cw ? lc1 : p.lwci, lamk = cw ? lk : 1.0;
    double tau = 0.0, sum = 0.0;
    if (cw && p.wenoz) {
#pragma unroll
      for (int l = 0; l < MA; ++l)
        if (l < adm) tau += fabs(is[0] - is[l]);
      tau = tau / (adm - 1);
    }
#pragma unroll
    for (int l = 0; l < MA; ++l) {
      w[l] = 0.0;
      if (l < adm) {
        const double e = p.weno_eps + is[l];
        const double lam = l == 0 ? lam0 : lamk;
        double wt;
        if (cw && p.wenoz) {
          double q = tau / e;
          q = q * q;
          wt = lam * (1.0 + q * q);
        } else {
          const double e2 = e * e;
          wt = lam / (e2 * e2);
        }
        w[l] = wt;
        sum += wt;
      }
    }
#pragma unroll
    for (int l = 0; l < MA; ++l) w[l] = w[l] / sum;
  }
  // ---- combined polynomial of variable v
  T gh[ID];
  central(gh);
  if (live) {
    const T w0 = T(w[0]);
#pragma unroll
    for (int d = 0; d < ID; ++d) gh[d] = w0 * gh[d];
    // every stencil row of the table is in the buffer (l < A), so the loads
    // need no guard on adm and can all be in flight; rows past adm add 0 * 0
#pragma unroll
    for (int l = 1; l < MA; ++l)
      if (l < A) {
        const bool on = l < adm;
        const T wl = on ? T(w[l]) : T(0);
#pragma unroll
        for (int d = 0; d < ID; ++d)
          if (!cw || d < ID2) {
            const T gv = G(l, d);
            gh[d] += wl * (on ? gv : T(0));
          }
      }
  }
  T cb = T(0);
  {
    const T* bmv = (const T*)p.bmean + grp * (int64_t)ID * 32 + lane;
#pragma unroll
    for (int d = 0; d < ID; ++d) cb += bmv[d * 32] * gh[d];
  }
  // ---- face values, CHECKSOL and the stores, face by face
  __syncthreads();  // s_x
  const T* xq = s_x + lane;
  const int nf = cell ? p.nfaces[c] : 0;
  double u0[NV], pm[NV];
#pragma unroll
  for (int k = 0; k < NV; ++k) u0[k] = cell ? U[c * NV + k] : 1.0;
  cons2prim(p.gamma, u0, pm);
  bool flag = false;
  T* out = (T*)p.dul + grp * 32 * (int64_t)FQ * NV;
  const int ncl = p.n - grp * 32 < 32 ? (int)(p.n - grp * 32) : 32;  // cells of this group
  for (int f = 0; f < MF; ++f) {
    T* so = s_o;
    if (f) __syncthreads();  // the stores of face f - 1 have read s_o
    const int nq = live && f < nf ? face_nq(p, p.ftype[c * MF + f]) : 0;
    for (int q = 0; q < QS; ++q) {
      T r = T(0);
      if (q < nq) {
        const T* xi = xq + (int64_t)(f * QS + q) * 3 * 32;
        T m[ID];
        monomials<P, T>(xi[0], xi[32], xi[64], m);
#pragma unroll
        for (int d = 0; d < ID; ++d) r += m[d] * gh[d];
        r = r - cb;
      }
      so[lane * RS + q * NV + v] = r;
    }
    __syncthreads();
    // CHECKSOL: warp v takes the points v, v + NV, ... of its lane's cell
    for (int q = v; q < nq; q += NV) {
      double uf[NV];
#pragma unroll
      for (int k = 0; k < NV; ++k) uf[k] = u0[k] + (double)so[lane * RS + q * NV + k];
      flag = flag || jump_bad(p.gamma, pm, uf, 0.85);
    }
    // the group's values of face f: one run of QS * NV per cell, warp v
    // storing the cells v, v + NV, ...
    for (int cl = v; cl < ncl; cl += NV)
      for (int r = lane; r < QS * NV; r += 32) out[(int64_t)cl * FQ * NV + f * QS * NV + r] = so[cl * RS + r];
  }
  if (flag) atomicOr(&s_flag[lane], 1);
  __syncthreads();
  if (tid < ncl) p.wflag[grp * 32 + tid] = (int8_t)s_flag[tid];
}

// Whether k_wface takes the face values below IORDER 4, rather than k_wpost's one
// lane per cell with all five variables.  k_wpost is bound by load latency at 12
// warps per SM and wins where its work per cell is small and its blocks fill the
// SMs: then five warps that read the triangles and form the monomials again cost
// more than they hide.  Times k_wpost -> k_wface in us:
//   IORDER 2 FP64, always: 8,000 hexahedra 70 -> 32, 262,144 679 -> 398, 48,000
//     tetrahedra 104 -> 94, 82,944 190 -> 131, 271,872 mixed cells (CWENO) 571 -> 526
//     (mixed meshes of 20,000 to 80,000 cells, whose cells without full stencils
//     then wait for the fall-back's launch, lose up to 13 %: 33,408 150 -> 172)
//   IORDER 2 FP32, below 192 cells per SM (28,416): 8,000 39 -> 30, 24,389 49 -> 44,
//     tetrahedra 24,576 43 -> 41; but 29,478 43 -> 57, 29,791 hexahedra 51 -> 60, 83,968
//     mixed cells 152 -> 181, 271,872 302 -> 411; 64,000 hexahedra alone 117 -> 95
//   IORDER 1 FP64, below 192 cells per SM: hexahedra 8,000 30 -> 24, 24,389 34 -> 30,
//     29,791 36 -> 42; CWENO 24,389 54 -> 33, 64,000 65 -> 73; tetrahedra 16,464
//     25 -> 25, 29,478 30 -> 42
//   IORDER 1 FP32, never: 512 to 20,000 cells 21 -> 24, 262,144 117 -> 200
//   IORDER 3, below 128 cells per SM (18,944): CWENO, 9,728 cells FP64 156 -> 89,
//     FP32 75 -> 44; 16,464 tetrahedra 114 -> 99, 61 -> 52; WENO, 17,576 hexahedra
//     189 -> 127, 93 -> 67; 24,576 cells FP64 133 -> 139, 271,872 FP32 564 -> 626
template <int P, typename T>
bool wface_own(const Problem& p) {
  constexpr bool f32 = sizeof(T) == 4;
  if (!p.wface || p.scheme != 3 || (P == 1 && f32)) return false;
  return (P == 2 && !f32) || p.n < (int64_t)p.nsm * (P == 3 ? 128 : 192);
}

// k_wpost: one lane per cell, no block barriers.  Indicators and weights of
// CP_RECONSTRUCTION (src/reconstruct_p.f90:920-1250), the combined
// polynomial, its face values and CHECKSOL; flagged cells (and every cell of
// high-order MUSCL) take the central stencil polynomial limited by
// Venkatakrishnan, then CHECKSOLX (3126-3406).  Output: dul [n][F][QS][5],
// face value minus cell mean, 0 in unused slots.  A face value is
// sum_d m_d(x) g_d - sum_d mean(m_d) g_d: the second sum is formed once per
// polynomial instead of subtracting the basis means at every face point.
// ISB: the indicators come from k_wis (p.isb) instead of being formed here.
// FB: only the cells that k_wface or k_char_face marked in p.wflag, straight to
// the MUSCL fall-back (the others return at once).  MU (with FB): the first MOOD
// cascade, MUSCL on the cells of p.mmus without CHECKSOLX (MUSCL of
// MOOD_OPERATOR_2, mood.f90:353).
// Under MOOD (p.mprev) every cell is reconstructed; a reduced cell (CHECKSOL,
// or not FULL) takes the MUSCL fall-back only if the last MOOD pass
// recomputed it (RECALC, reconstruct_p.f90:2306-2315), else it keeps its
// WENO values and only CHECKSOLX; the reduced flags go to p.wflag.
// Three blocks of 128 per SM where that measured faster than the two that
// the kernel's registers otherwise allow: IORDER 3 in FP32 (2.1 M-cell CWENO4
// Navier-Stokes step 52.7 -> 51.2 ms; in FP64 the bound made the 647 k-cell
// step 31.8 -> 33.8 ms, so FP64 keeps two; 271,872 cells in FP32: 0.557 ms with
// three, 0.577 with two, 0.619 with four), and IORDER 2 (82,944 WENO3 tets: 1.109
// -> 1.083 ms per step mixed, 1.585 -> 1.540 FP64, which k_wface has taken since).
template <int P, typename T, bool ISB = false, bool FB = false, bool MU = false>
__global__ void __launch_bounds__(128, P == 2 || (P == 3 && sizeof(T) == 4) ? 3 : 1)
    k_wpost(Problem p, const double* __restrict__ U) {
  constexpr int ID = Deg<P>::ideg;
  constexpr int VEC = Vec<T>::N;
  constexpr int L2 = ID < 9 ? ID : 9;  // CWENO lower order: IDEGFREE2 3 or 9 (grid_p.f90:6145-6160)
  constexpr int VI = WVars<T>::is, VH = WVars<T>::face, VF = WVars<T>::fall;
  constexpr int BT = 128;              // threads per block
  __shared__ double s_w[7 * NV * BT];  // per thread, [ll][v]: indicators, then weights
  const int tid = threadIdx.x;
  const int64_t c = (int64_t)blockIdx.x * blockDim.x + tid;
  if (c >= p.n) return;
  const int A = p.admis_max;
  const int QS = p.nq_quad > p.nq_tri ? p.nq_quad : p.nq_tri;
  const int FQ = MF * QS;
  const bool cw = p.ees == 5, weno = p.scheme == 3;
  const int ID2 = p.ideg2;
  const int adm = p.admis[c];
  const int nf = p.nfaces[c];
  const int64_t grp = c >> 5;
  const int lane = (int)(c & 31);
  // stencil polynomials G[ll][d][v], interleaved like the tables
  const T* Gc = (const T*)p.gbuf + grp * (int64_t)(A * ID * NV) * 32 + lane;
  auto G = [&](int ll, int d, int v) -> T { return Gc[(int64_t)((ll * ID + d) * NV + v) * 32]; };
  double u0[NV], pm[NV];
#pragma unroll
  for (int v = 0; v < NV; ++v) u0[v] = U[c * NV + v];
  cons2prim(p.gamma, u0, pm);
  const T* xq = (const T*)p.qpts + grp * (int64_t)FQ * 3 * 32 + lane;  // interleaved
  const T* bmv = (const T*)p.bmean + grp * (int64_t)ID * 32 + lane;    // interleaved
  T* out = (T*)p.dul + c * FQ * NV;
  double* sw = s_w + tid;  // sw[(ll * NV + v) * BT]
  const double lc1 = 1.0 - 1.0 / p.lwci;
  const double lk = adm > 1 ? (1.0 - lc1) / (adm - 1) : 0.0;
  auto nq_of = [&](int f) { return f < nf ? face_nq(p, p.ftype[c * MF + f]) : 0; };
  // monomials at face point (f, q)
  auto mono = [&](int f, int q, T (&m)[ID]) {
    const T* xi = xq + (int64_t)(f * QS + q) * 3 * 32;
    monomials<P, T>(__ldcs(xi), __ldcs(xi + 32), __ldcs(xi + 64), m);
  };
  // g[d][k] = G(ll, d, v0 + k) for d < ndl, else 0
  auto load_poly = [&](int ll, int v0, auto& g, int ndl) {
    constexpr int ND = sizeof(g) / sizeof(g[0]);
    constexpr int VV = sizeof(g[0]) / sizeof(T);
#pragma unroll
    for (int d = 0; d < ND; ++d)
#pragma unroll
      for (int k = 0; k < VV; ++k) g[d][k] = (v0 + k < NV && d < ndl) ? G(ll, d, v0 + k) : T(0);
  };
  // central stencil polynomial for variables v0, v0+1, ... (as many as g
  // holds); with `rem`, the CWENO form with the low-order stencils removed
  // (reconstruct_p.f90:956-965)
  auto load_g0 = [&](int v0, auto& g, bool rem) {
    constexpr int VV = sizeof(g[0]) / sizeof(T);
    load_poly(0, v0, g, ID);
    if (rem) {
      T g3[L2][VV];
#pragma unroll
      for (int d = 0; d < L2; ++d)
#pragma unroll
        for (int k = 0; k < VV; ++k) g3[d][k] = T(0);
      for (int l2 = 1; l2 < adm; ++l2)
#pragma unroll
        for (int d = 0; d < L2; ++d)
#pragma unroll
          for (int k = 0; k < VV; ++k)
            if (v0 + k < NV && d < ID2) g3[d][k] = g3[d][k] + T(lk) * G(l2, d, v0 + k);
#pragma unroll
      for (int d = 0; d < ID; ++d)
#pragma unroll
        for (int k = 0; k < VV; ++k)
          if (v0 + k < NV) g[d][k] = T(1.0 / lc1) * (g[d][k] - (d < L2 ? g3[d][k] : T(0)));
    }
  };
  // sum_d mean(m_d) g[d][k]
  auto mean_term = [&](const auto& g, auto& cb) {
    constexpr int VV = sizeof(g[0]) / sizeof(T);
#pragma unroll
    for (int k = 0; k < VV; ++k) cb[k] = T(0);
#pragma unroll
    for (int d = 0; d < ID; ++d) {
      const T b = bmv[d * 32];
#pragma unroll
      for (int k = 0; k < VV; ++k) cb[k] += b * g[d][k];
    }
  };

  // nonlinear weights in FP64 ((10E-12)^4 underflows FP32): sw holds the
  // indicators [ll][v] on entry and the weights on exit
  auto weights = [&]() {
    for (int v = 0; v < NV; ++v) {
      const double lam0 = cw ? lc1 : p.lwci, lamk = cw ? lk : 1.0;
      double tau = 0.0, sum = 0.0;
      if (cw && p.wenoz) {
        for (int ll = 0; ll < adm; ++ll) tau += fabs(sw[v * BT] - sw[(ll * NV + v) * BT]);
        tau = tau / (adm - 1);
      }
      for (int ll = 0; ll < adm; ++ll) {
        const double e = p.weno_eps + sw[(ll * NV + v) * BT];
        const double lam = ll == 0 ? lam0 : lamk;
        double wt;
        if (cw && p.wenoz) {
          double q = tau / e;
          q = q * q;
          wt = lam * (1.0 + q * q);
        } else {
          const double e2 = e * e;
          wt = lam / (e2 * e2);
        }
        sw[(ll * NV + v) * BT] = wt;
        sum += wt;
      }
      for (int ll = 0; ll < adm; ++ll) sw[(ll * NV + v) * BT] = sw[(ll * NV + v) * BT] / sum;
    }
  };
  const bool md = p.mprev != nullptr;
  if (FB && !(MU ? p.mmus[c] : p.wflag[c])) return;
  bool fall = FB || !weno || (!md && !p.full[c]);  // CHECKSOL: FULL = 0 -> REDUCE
  if (!fall && ISB) {
    // ---- smoothness indicators from k_wis
    const double* is = p.isb + grp * (int64_t)A * NV * 32 + lane;
    for (int ll = 0; ll < adm; ++ll)
#pragma unroll
      for (int v = 0; v < NV; ++v) sw[(ll * NV + v) * BT] = is[(int64_t)(ll * NV + v) * 32];
  } else if (!ISB && !fall) {
    // ---- smoothness indicators g^T S g per stencil and variable
    const T* Pc = (const T*)p.ind + grp * p.istride * 32 + lane * VEC;
    for (int ll = 0; ll < adm; ++ll) {
      const bool low = cw && ll > 0;
      for (int v0 = 0; v0 < NV; v0 += VI) {
        T is[VI];
#pragma unroll
        for (int k = 0; k < VI; ++k) is[k] = T(0);
        if (low) {
          T g[L2][VI];
          load_poly(ll, v0, g, ID2);
          quad_form<L2, VI>(Pc + (int64_t)(p.i2off / VEC) * 32 * VEC, g, ID2, is);
        } else {
          T g[ID][VI];
          if (ll == 0) load_g0(v0, g, cw);
          else load_poly(ll, v0, g, ID);
          quad_form<ID, VI>(Pc, g, ID, is);
        }
#pragma unroll
        for (int k = 0; k < VI; ++k)
          if (v0 + k < NV) sw[(ll * NV + v0 + k) * BT] = (double)is[k];
      }
    }
  }
  if (!fall) {
    weights();
    // ---- combined polynomial, face values, CHECKSOL (threshold 0.85)
    bool flag = false;
    for (int v0 = 0; v0 < NV; v0 += VH) {
      T gh[ID][VH];
      load_g0(v0, gh, cw);
#pragma unroll
      for (int k = 0; k < VH; ++k) {
        const T w0 = v0 + k < NV ? T(sw[(v0 + k) * BT]) : T(0);
#pragma unroll
        for (int d = 0; d < ID; ++d) gh[d][k] = w0 * gh[d][k];
      }
      for (int ll = 1; ll < adm; ++ll) {
        T wl[VH];
#pragma unroll
        for (int k = 0; k < VH; ++k) wl[k] = v0 + k < NV ? T(sw[(ll * NV + v0 + k) * BT]) : T(0);
#pragma unroll
        for (int d = 0; d < ID; ++d)
          if (!cw || d < ID2)
#pragma unroll
            for (int k = 0; k < VH; ++k)
              if (v0 + k < NV) gh[d][k] += wl[k] * G(ll, d, v0 + k);
      }
      T cb[VH];
      mean_term(gh, cb);
      for (int f = 0; f < MF; ++f) {
        const int nq = nq_of(f);
        for (int q = 0; q < QS; ++q) {
          T* o = out + (f * QS + q) * NV;
          if (q >= nq) {
#pragma unroll
            for (int k = 0; k < VH; ++k)
              if (v0 + k < NV) o[v0 + k] = T(0);
            continue;
          }
          T m[ID];
          mono(f, q, m);
          T res[VH];
#pragma unroll
          for (int k = 0; k < VH; ++k) {
            T r = T(0);
#pragma unroll
            for (int d = 0; d < ID; ++d) r += m[d] * gh[d][k];
            res[k] = r - cb[k];
            if (v0 + k < NV) o[v0 + k] = res[k];
          }
          if (VH == NV) {
            double uf[NV];
#pragma unroll
            for (int v = 0; v < NV; ++v) uf[v] = u0[v] + (double)res[v % VH];
            flag = flag || jump_bad(p.gamma, pm, uf, 0.85);
          }
        }
      }
    }
    if (VH < NV) {  // CHECKSOL on the stored face values
      for (int f = 0; f < nf; ++f) {
        const int nq = nq_of(f);
        for (int q = 0; q < nq; ++q) {
          const T* o = out + (f * QS + q) * NV;
          double uf[NV];
#pragma unroll
          for (int v = 0; v < NV; ++v) uf[v] = u0[v] + (double)o[v];
          flag = flag || jump_bad(p.gamma, pm, uf, 0.85);
        }
      }
    }
    fall = flag;
  }
  // CHECKSOLX (threshold 0.95) cannot fire where the 0.85 test passed on the
  // same face values
  bool mus = fall, chkx = fall;
  if (md && !FB && weno) {  // MOOD: the fall-back only where RECALC
    const bool reduce = fall || !p.full[c];
    p.wflag[c] = reduce ? 1 : 0;
    mus = reduce && p.mprev[c];
    chkx = reduce;
  } else if (md && FB && !MU) {
    mus = p.mprev[c];
  }
  if (MU) chkx = false;
  if (!mus && !chkx) return;

  if (mus) {
    // ---- MUSCL with the central stencil polynomial (FIND_BOUNDS + Venkatakrishnan)
    double lo[NV], hi[NV];
#pragma unroll
    for (int v = 0; v < NV; ++v) lo[v] = hi[v] = u0[v];
    for (int f = 0; f < nf; ++f) {
      const int64_t nb = p.neigh[c * MF + f];
      if (nb < 0) continue;
#pragma unroll
      for (int v = 0; v < NV; ++v) {
        const double un = U[nb * NV + v];
        lo[v] = fmin(lo[v], un);
        hi[v] = fmax(hi[v], un);
      }
    }
#pragma unroll
    for (int v = 0; v < NV; ++v) {
      lo[v] -= u0[v];
      hi[v] -= u0[v];
    }
    const double e3 = p.kappa_ven * p.minedge[c];
    const double epsi2 = e3 * e3 * e3;
    for (int v0 = 0; v0 < NV; v0 += VF) {
      T g0[ID][VF];
      load_poly(0, v0, g0, ID);
      T cb[VF];
      mean_term(g0, cb);
      double slope[VF];
#pragma unroll
      for (int k = 0; k < VF; ++k) slope[k] = TOLBIG;
      for (int pass = 0; pass < 2; ++pass) {
        for (int f = 0; f < MF; ++f) {
          const int nq = nq_of(f);
          for (int q = 0; q < QS; ++q) {
            T* o = out + (f * QS + q) * NV;
            if (q >= nq) {
              if (pass == 1)
#pragma unroll
                for (int k = 0; k < VF; ++k)
                  if (v0 + k < NV) o[v0 + k] = T(0);
              continue;
            }
            T m[ID];
            mono(f, q, m);
#pragma unroll
            for (int k = 0; k < VF; ++k) {
              const int v = v0 + k;
              if (v >= NV) continue;
              T r = T(0);
#pragma unroll
              for (int d = 0; d < ID; ++d) r += m[d] * g0[d][k];
              r = r - cb[k];
              const double dd = (u0[v] + (double)r) - u0[v];
              if (pass == 0) slope[k] = fmin(slope[k], slope_limiter(p.limiter, dd, lo[v], hi[v], epsi2));
              else o[v] = T((double)T(dd) * slope[k]);
            }
          }
        }
      }
    }
  }
  if (!chkx) return;
  // ---- CHECKSOLX: first order where a face value jumps by 95 %
  bool bad = false;
  for (int f = 0; f < nf; ++f) {
    const int nq = nq_of(f);
    for (int q = 0; q < nq; ++q) {
      const T* o = out + (f * QS + q) * NV;
      double uf[NV];
#pragma unroll
      for (int v = 0; v < NV; ++v) uf[v] = u0[v] + (double)o[v];
      bad = bad || jump_bad(p.gamma, pm, uf, 0.95);
    }
  }
  if (bad)
    for (int i = 0; i < FQ * NV; ++i) out[i] = T(0);
}

// ======================================================================
// Viscous gradients for WENO/CWENO + Navier-Stokes: LSQ on (T,u,v,w) with
// stencil 1 (gradients.f90:502-706), then face gradients (SOLUTIONTRIAV2).
// ======================================================================
// One lane per cell: each stencil member's primitive state is formed once
// and its differences (T, u, v, w) are accumulated for VP variables per pass
// (all four when the FP64 accumulators fit), reading the interleaved table
// rows of stencil 1 with coalesced loads.  Same products and order per
// (row, variable) as one thread per variable.
// T = p / (rho R), u, v, w of every cell, formed once per stage: the viscous
// least squares then gathers 32-byte records (two 16-byte loads, no
// division) instead of forming them from the conserved state per member.
template <int P, typename T>
__global__ void k_visc_prim(Problem p, const double* __restrict__ U) {
  const int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= p.n) return;
  double pm[NV];
  cons2prim(p.gamma, U + c * NV, pm);
  double2* o = (double2*)(p.prim + c * 4);
  o[0] = make_double2(pm[4] / (pm[0] * p.r_gas), pm[1]);
  o[1] = make_double2(pm[2], pm[3]);
}

// Accumulated in the table precision T: FP64 in the FP64 form; in the mixed
// form FP32 on the differences of (T, u, v, w) from the cell's own, like
// the stencil least squares of the conserved variables (all four variables
// in one pass there).
// SET: a block takes a tile of cells that share a matrix set (plan_sets) and
// reads stencil 1's rows from shared memory as 16-byte broadcasts instead of
// streaming every cell's copy from DRAM, with the records of VG members in
// flight; the same sums in the same order.  The first blocks take the groups
// that the tiles leave (p.ugrp), whose few lanes' chain of loads runs beside
// the tiles.  271,872 cells, CWENO4 mixed form: 0.270 -> 0.149 ms (0.167 at three
// blocks per SM, 0.229 at five with two members in flight; the groups left in
// a launch of their own 0.056 more); WENO5 FP64, 8,000 cells, whose 63 blocks
// waited for one chain of loads, all after the least squares 3.23 -> 0.24.
// Blocks of that launch with left-over groups (four each), and the cell of a
// thread of a block, -1 for none: a tiled cell of a left-over group has its
// block among the tiles', so that every cell has one writer.
__host__ __device__ inline int64_t visc_lsq_own(const Problem& p) { return (p.nugrp + 3) / 4; }
template <bool SET>
__host__ __device__ inline int64_t visc_lsq_cell(const Problem& p, int64_t block, int thread) {
  const int64_t own = SET ? visc_lsq_own(p) : 0;
  if (SET && block >= own) return p.tcell[(block - own) * SET_TILE + thread];
  int64_t c = block * 128 + thread;
  if (SET) {
    if ((c >> 5) >= p.nugrp) return -1;
    c = (int64_t)p.ugrp[c >> 5] * 32 + (c & 31);
  }
  return c < p.n && !(SET && p.tiled[c]) ? c : -1;
}
template <int P, typename T, bool SET = false>
__global__ void __launch_bounds__(128, sizeof(T) == 4 && P <= 3 ? 4 : 1) k_visc_lsq(Problem p, const double* __restrict__ U) {
  constexpr int ID = Deg<P>::ideg;
  constexpr int VP = sizeof(T) == 4 || ID * 4 <= 80 ? 4 : 2;  // variables per pass
  constexpr int RS = set_stride<T>(ID), VEC = Vec<T>::N, VG = 4;
  extern __shared__ __align__(16) unsigned char vl_smem[];
  const T* s = (const T*)vl_smem;
  const int IM = p.imax, W = IM + 1;
  const bool tiled = SET && blockIdx.x >= visc_lsq_own(p);
  if (tiled) {
    const int64_t tile = blockIdx.x - visc_lsq_own(p);
    const float4* src = (const float4*)((const T*)p.setmat + p.tset[tile] * p.sstride + p.sso[0]);
    for (int i = threadIdx.x; i < IM * RS / VEC; i += SET_TILE) ((float4*)vl_smem)[i] = src[i];
    __syncthreads();
  }
  const int64_t c = visc_lsq_cell<SET>(p, blockIdx.x, threadIdx.x);
  if (c < 0) return;
  double pm[NV];
  cons2prim(p.gamma, U + c * NV, pm);
  const double s0[4] = {pm[4] / (pm[0] * p.r_gas), pm[1], pm[2], pm[3]};
  const int64_t grp = c >> 5;
  const int lane = (int)(c & 31);
  const int32_t* st = p.sten + grp * (int64_t)p.admis_max * W * 32 + lane;
  const T* M = (const T*)p.invmat + (grp * p.tstride + p.soff[0]) * 32 + lane;
  T* gv = (T*)p.gv;
#pragma unroll 1
  for (int v0 = 0; v0 < 4; v0 += VP) {
    T acc[ID][VP];
#pragma unroll
    for (int d = 0; d < ID; ++d)
#pragma unroll
      for (int j = 0; j < VP; ++j) acc[d][j] = T(0);
    if (tiled) {
      for (int k0 = 0; k0 < IM; k0 += VG) {
        double2 qa[VG], qb[VG];
#pragma unroll
        for (int i = 0; i < VG; ++i) {
          const int k = k0 + i < IM ? k0 + i : IM - 1;
          const double2* q = (const double2*)(p.prim + (int64_t)st[(k + 1) * 32] * 4);
          qa[i] = q[0], qb[i] = q[1];
        }
#pragma unroll
        for (int i = 0; i < VG; ++i)
          if (k0 + i < IM) {
            const double sy[4] = {qa[i].x, qa[i].y, qb[i].x, qb[i].y};
            T ds[VP];
#pragma unroll
            for (int j = 0; j < VP; ++j) ds[j] = T(sy[v0 + j] - s0[v0 + j]);
#pragma unroll
            for (int q = 0; q < RS / VEC; ++q) {
              T m[VEC];
              ldv(s + (k0 + i) * RS + q * VEC, m);
#pragma unroll
              for (int r = 0; r < VEC; ++r)
                if (q * VEC + r < ID)
#pragma unroll
                  for (int j = 0; j < VP; ++j) acc[q * VEC + r][j] += m[r] * ds[j];
            }
          }
      }
    } else {
      for (int k = 0; k < IM; ++k) {
        const double2* q = (const double2*)(p.prim + (int64_t)st[(k + 1) * 32] * 4);
        const double2 qa = q[0], qb = q[1];
        const double sy[4] = {qa.x, qa.y, qb.x, qb.y};
        T ds[VP];
#pragma unroll
        for (int j = 0; j < VP; ++j) ds[j] = T(sy[v0 + j] - s0[v0 + j]);
#pragma unroll
        for (int d = 0; d < ID; ++d) {
          const T m = M[(k * ID + d) * 32];
#pragma unroll
          for (int j = 0; j < VP; ++j) acc[d][j] += m * ds[j];
        }
      }
    }
    // 16-byte stores: a row's four FP32 values, or FP64 pairs (VP even;
    // rows are 16- and 32-byte aligned)
#pragma unroll
    for (int d = 0; d < ID; ++d) {
      if constexpr (sizeof(T) == 4) {
        *(float4*)(gv + (c * ID + d) * 4) = make_float4(acc[d][0], acc[d][1], acc[d][2], acc[d][3]);
      } else {
#pragma unroll
        for (int j = 0; j < VP; j += 2)
          *(double2*)(gv + (c * ID + d) * 4 + v0 + j) = make_double2(acc[d][j], acc[d][j + 1]);
      }
    }
  }
}

// Face-point gradients of T, u, v, w for the viscous flux, one thread per
// (owned face, point): SOLUTIONTRIAV2 (reconstruct_p.f90:2358) on
// both sides of the face at the paired points, and their average, the only
// form CALCULATE_FLUXESHI_DIFFUSIVE uses (flux_p.f90:1614-1779), written
// once per face point to p.fgrad [nown][QS][12] (half the bytes of one
// record per cell face and point, read back once instead of twice).
// evaluated in T (FP32 in the mixed form, from the FP32 coefficients and
// reference-frame points)
template <int P, typename T>
__device__ __forceinline__ void visc_point_grad(const Problem& p, int64_t c, int f, int q, int QS, T* out) {
  constexpr int ID = Deg<P>::ideg;
  const T* xi = (const T*)p.qpts + ((c >> 5) * MF * QS * 3 + (f * QS + q) * 3) * 32 + (c & 31);
  T dx[ID], dy[ID], dz[ID];
  dmonomials<P, T>(xi[0], xi[32], xi[64], dx, dy, dz);
  const double* J = p.jinv + c * 9;
  const T* gv = (const T*)p.gv + c * ID * 4;
  if constexpr (sizeof(T) == 4) {
    // FP32: a coefficient row's four variables in one 16-byte load (the
    // scalar loads kept k_visc_facegrad at 80 % of L1 throughput; 2.1 M-cell
    // CWENO4: 52.7 -> 51.8 ms per step); each variable's sum still runs over
    // the rows in order, so the values are the same bit for bit
    T gl[4][3];
#pragma unroll
    for (int var = 0; var < 4; ++var) gl[var][0] = gl[var][1] = gl[var][2] = T(0);
#pragma unroll
    for (int d = 0; d < ID; ++d) {
      const float4 a = *(const float4*)(gv + d * 4);
      const T g[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
      for (int var = 0; var < 4; ++var) {
        gl[var][0] += g[var] * dx[d];
        gl[var][1] += g[var] * dy[d];
        gl[var][2] += g[var] * dz[d];
      }
    }
#pragma unroll
    for (int var = 0; var < 4; ++var)
#pragma unroll
      for (int k = 0; k < 3; ++k)
        out[var * 3 + k] = T(J[0 * 3 + k]) * gl[var][0] + T(J[1 * 3 + k]) * gl[var][1] + T(J[2 * 3 + k]) * gl[var][2];
  } else {
#pragma unroll
    for (int var = 0; var < 4; ++var) {
      T gl[3] = {T(0), T(0), T(0)};
#pragma unroll
      for (int d = 0; d < ID; ++d) {
        const T g = gv[d * 4 + var];
        gl[0] += g * dx[d];
        gl[1] += g * dy[d];
        gl[2] += g * dz[d];
      }
#pragma unroll
      for (int k = 0; k < 3; ++k)
        out[var * 3 + k] = T(J[0 * 3 + k]) * gl[0] + T(J[1 * 3 + k]) * gl[1] + T(J[2 * 3 + k]) * gl[2];
    }
  }
}

template <int P, typename T>
__device__ __forceinline__ void visc_facegrad(const Problem& p) {
  const int QS = p.nq_quad > p.nq_tri ? p.nq_quad : p.nq_tri;
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t i = t / QS;
  const int q = (int)(t - i * QS);
  if (i >= p.nown) return;
  const int32_t code = p.own[i];
  const int64_t c = code >> 3;
  const int f = code & 7;
  const int64_t nb = p.neigh[c * MF + f];
  if (q >= face_nq(p, p.ftype[c * MF + f])) return;
  T gl[12], gr[12];
  visc_point_grad<P, T>(p, c, f, q, QS, gl);
  if (nb >= 0) {
    visc_point_grad<P, T>(p, nb, p.nface[c * MF + f], p.qperm[(c * MF + f) * QS + q], QS, gr);
  } else {  // physical boundary: the ghost side takes the cell's own gradient
#pragma unroll
    for (int k = 0; k < 12; ++k) gr[k] = gl[k];
  }
  double2* o = (double2*)(p.fgrad + (i * QS + q) * 12);
#pragma unroll
  for (int k = 0; k < 6; ++k)
    o[k] = make_double2((double)((gl[2 * k] + gr[2 * k]) / T(2)), (double)((gl[2 * k + 1] + gr[2 * k + 1]) / T(2)));
}
// FP64 with the registers that the compiler takes (80 below IORDER 4, 128 there):
// bounded to five blocks per SM it took 96 and at IORDER 4 spilled (reconstruction
// after the least squares, CWENO4, 271,872 cells 2.065 against 2.026 ms; WENO3, 48^3
// 0.335, 0.326; WENO5, 24^3 0.367, 0.358).  FP32 eight blocks per SM: CWENO4,
// 271,872 cells 1.037 ms against 1.050 unbounded, WENO4, 32^3 0.221, 0.224, WENO3,
// 48^3 0.244, 0.241.
template <int P>
__global__ void k_visc_facegrad(Problem p) {
  visc_facegrad<P, double>(p);
}
template <int P>
__global__ void __launch_bounds__(128, 8) k_visc_facegrad_f32(Problem p) {
  visc_facegrad<P, float>(p);
}
template <int P, typename T>
void launch_visc_facegrad(const Problem& p, cudaStream_t st) {
  const int QS = p.nq_quad > p.nq_tri ? p.nq_quad : p.nq_tri;
  const unsigned b = (unsigned)((p.nown * QS + 127) / 128);
  if constexpr (sizeof(T) == 4) k_visc_facegrad_f32<P><<<b, 128, 0, st>>>(p);
  else k_visc_facegrad<P><<<b, 128, 0, st>>>(p);
}

// CHARACTERISTIC_RECONSTRUCTION (src/reconstruct_p.f90:497-758): per face, the
// eigenvectors at the average of the cell mean and the face neighbour's mean
// (or the boundary ghost of the cell mean), both in the face frame; stencil
// polynomials projected on the left eigenvectors (global-frame conserved
// variables, as the reference projects them); indicators and weights per
// characteristic variable; the face's polynomial back-projected.  The
// indicator of the projection W = G EL^T is EL_k^T (G^T S G) EL_k, so G^T S G
// is formed once per cell and stencil (k_char_forms) and each face only
// applies its eigenvectors (k_char_face).  With M_ll = ER diag(w_ll) EL the
// combined conserved polynomial is sum_ll M_ll G_ll (rows d >= 1) and its
// mean sum_ll M_ll u0, formed in FP64.
//
// Both run one block per 32-cell group (and stencil, or faces) with one warp
// per variable, lane = cell, as k_wis and k_wface do: the polynomials of one
// variable fit in registers, and the five warps read the same triangles and
// stencil polynomials at about the same time (from L1).  One lane per cell
// with all five variables (four 64-thread blocks per SM, 1-1.4 KB of spills)
// was latency-bound: 27,000 cells, WENO5 FP64: 5.92 ms -> 0.16 + 1.06 ms.
// Three blocks of k_char_forms per SM (0.52 ms with two, 0.66 with four).
//
// Rows d < IDEGFREE2 of sum_l2 lk G_l2, what CWENO takes off its central
// stencil (reconstruct_p.f90:1723-1737), of variable v into s[d][v][lane].
template <int P, typename T>
__device__ __forceinline__ void char_lower_sum(const Problem& p, const T* Gc, int adm, int v, int lane, T* s) {
  constexpr int ID = Deg<P>::ideg;
  const double lc1 = 1.0 - 1.0 / p.lwci;
  const double lk = adm > 1 ? (1.0 - lc1) / (adm - 1) : 0.0;
  for (int d = 0; d < p.ideg2; ++d) {
    T g3 = T(0);
    for (int l2 = 1; l2 < adm; ++l2) g3 = g3 + T(lk) * Gc[(int64_t)((l2 * ID + d) * NV + v) * 32];
    s[(d * NV + v) * 32 + lane] = g3;
  }
}

// G_l^T S G_l (symmetric 5x5, upper triangle row by row) of every stencil:
// block (group, stencil), warp w forms the column products with variable w.
template <int P, typename T>
__global__ void __launch_bounds__(32 * NV, 3) k_char_forms(Problem p) {
  constexpr int ID = Deg<P>::ideg;
  constexpr int VEC = Vec<T>::N;
  constexpr int L2 = ID < 9 ? ID : 9;
  __shared__ T s_a[NV * NV][32];
  __shared__ T s_g[L2 * NV * 32];
  __shared__ __align__(16) T s_tri[tri_len<T>(ID)];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, ll = blockIdx.y;
  const int64_t grp = blockIdx.x, c = grp * 32 + lane;
  const bool cell = c < p.n, full = cell && p.full[c];
  if (ll == 0 && w == 0 && cell) p.wflag[c] = full ? 0 : 1;  // CHECKSOL: FULL = 0 -> REDUCE
  const int adm = full || (cell && p.mprev) ? p.admis[c] : 0;
  const int A = p.admis_max, ID2 = p.ideg2;
  const bool cw = p.ees == 5, low = cw && ll > 0, rem = cw && ll == 0;
  const T* Gc = (const T*)p.gbuf + grp * (int64_t)(A * ID * NV) * 32 + lane;
  // where all cells of the group share a matrix set, its triangle is read as
  // broadcasts (27,000 cells, WENO5 FP64: 0.41 -> 0.16 ms)
  const int gs = p.ntile ? p.gset[grp] : -1;
  if (gs >= 0) {
    const T* src = (const T*)p.setind + gs * p.istride + (low ? p.i2off : 0);
    const int nt = low ? (int)p.istride - p.i2off : p.i2off;
    for (int i = threadIdx.x; i < nt / VEC; i += 32 * NV) ((float4*)s_tri)[i] = ((const float4*)src)[i];
  }
  if (rem) char_lower_sum<P, T>(p, Gc, adm, w, lane, s_g);
  __syncthreads();
  const T ilc = T(1.0 / (1.0 - 1.0 / p.lwci));
  auto Gp = [&](int d, int u) -> T {
    const T g = Gc[(int64_t)((ll * ID + d) * NV + u) * 32];
    return rem ? ilc * (g - (d < L2 && d < ID2 ? s_g[(d * NV + u) * 32 + lane] : T(0))) : g;
  };
  const T* Pc = (const T*)p.ind + grp * p.istride * 32 + lane * VEC;
  T a[NV];
#pragma unroll
  for (int u = 0; u < NV; ++u) a[u] = T(0);
  // a[u] += g[d][u] * sum_{e>=d} P_de g[e][w], the packed triangle as in quad_form
  auto form = [&](auto& g, const T* Pl, int nd, auto strc) {
    constexpr int ND = sizeof(g) / sizeof(T), STR = decltype(strc)::value;
#pragma unroll
    for (int d = 0; d < ND; ++d) g[d] = d < nd ? Gp(d, w) : T(0);
    int rs = 0;
#pragma unroll
    for (int d = 0; d < ND; ++d)
      if (d < nd) {
        T t = T(0);
#pragma unroll
        for (int q = 0; q < (ND - d + VEC - 1) / VEC; ++q)
          if (d + q * VEC < nd) {
            T x[VEC];
            ldv(Pl + (int64_t)(rs + q) * STR * VEC, x);
#pragma unroll
            for (int i = 0; i < VEC; ++i)
              if (d + q * VEC + i < ND) t += x[i] * g[d + q * VEC + i];
          }
        rs += (nd - d + VEC - 1) / VEC;
#pragma unroll
        for (int u = 0; u < NV; ++u) a[u] += Gp(d, u) * t;
        asm volatile("" ::: "memory");  // as in quad_form
      }
  };
  if (ll < adm) {
    if (low) {
      T g[L2];
      if (gs >= 0) form(g, s_tri, ID2, IntC<1>());
      else form(g, Pc + (int64_t)(p.i2off / VEC) * 32 * VEC, ID2, IntC<32>());
    } else {
      T g[ID];
      if (gs >= 0) form(g, s_tri, ID, IntC<1>());
      else form(g, Pc, ID, IntC<32>());
    }
  }
#pragma unroll
  for (int u = 0; u < NV; ++u) s_a[u * NV + w][lane] = a[u];
  __syncthreads();
  if (ll >= adm) return;
  double* Qc = p.qbuf + grp * (int64_t)(A * 15) * 32 + lane;
  int j = 0;
#pragma unroll
  for (int u = 0; u < NV; ++u)
#pragma unroll
    for (int k = u; k < NV; ++k, ++j)
      if (j % NV == w)
        Qc[(int64_t)(ll * 15 + j) * 32] = u == k ? (double)s_a[u * NV + u][lane]
                                                 : 0.5 * ((double)s_a[u * NV + k][lane] + (double)s_a[k * NV + u][lane]);
}

// Faces of a block, whose polynomials of one variable stay in registers
// together, so that each stencil polynomial is read once for all of them.  In
// FP64 at IORDER 4 one face: two leave no registers for loads in flight
// (27,000 cells: 1.28 ms with two, 1.06 with one and two blocks per SM, 1.38
// with three).
// At IORDER 1 and 2, whose polynomials are short, two, and more blocks per SM: with
// three and two the kernel waited for its loads (38 us a block, the 15 values of
// each stencil's form read by every warp for every face); there and in FP32 at
// IORDER 3 the forms are read once for the block's faces (lean).  Characteristic
// reconstruction after the least squares, us, FP64 and FP32: IORDER 1, 85,184
// hexahedra 672 -> 522, 508 -> 480, 48,000 tetrahedra 254 -> 192, 183 -> 159; IORDER 2
// 989 -> 871, 889 -> 676, 427 -> 388, 351 -> 262; IORDER 3 FP32 1285 -> 1204, 523 ->
// 503 (FP64 1275 -> 1309 on 32,768 hexahedra, IORDER 4 FP32 1014 -> 1063: kept out).
// One lane per cell took 651, 409, 242, 148; 2054, 859, 637, 275 (IORDER 1, 2): in FP32
// at IORDER 1 on large meshes it was faster.
template <int P, typename T>
struct CharFaces {
  static constexpr int value = P < 3 ? 2 : P < 4 || sizeof(T) == 4 ? 3 : 1;
  static constexpr bool lean = P < 3 || (P == 3 && sizeof(T) == 4);
  static constexpr int blocks = P < 3 ? (sizeof(T) == 4 ? 4 : 3) : 2;  // per SM
};
template <int P, typename T>
__host__ __device__ constexpr size_t char_face_smem(int QS) {
  constexpr int NF = CharFaces<P, T>::value, ID = Deg<P>::ideg, L2 = ID < 9 ? ID : 9;
  return (size_t)NF * (50 + 7 * NV) * 32 * 8 + ((size_t)((QS * NV) | 1) + L2 * NV) * 32 * sizeof(T);
}
template <int P, typename T>
__global__ void __launch_bounds__(32 * NV, CharFaces<P, T>::blocks)
    k_char_face(Problem p, const double* __restrict__ U) {
  constexpr int ID = Deg<P>::ideg;
  constexpr int L2 = ID < 9 ? ID : 9;
  constexpr int NF = CharFaces<P, T>::value;
  constexpr bool LEAN = CharFaces<P, T>::lean;
  constexpr int MA = 7;  // stencils per cell at most
  extern __shared__ __align__(16) unsigned char cf_smem[];
  const int QS = p.nq_quad > p.nq_tri ? p.nq_quad : p.nq_tri;
  const int FQ = MF * QS, RS = (QS * NV) | 1;
  double* s_e = (double*)cf_smem;          // [NF][50][32]: left, then right eigenvectors
  double* s_w = s_e + NF * 50 * 32;        // [NF][MA][NV][32]: weights
  T* s_g = (T*)(s_w + NF * MA * NV * 32);  // [L2][NV][32]: char_lower_sum
  T* s_o = s_g + L2 * NV * 32;             // [32][RS]: the values of one face
  const int lane = threadIdx.x & 31, v = threadIdx.x >> 5;
  const int64_t grp = blockIdx.x, c = grp * 32 + lane;
  const int f0 = blockIdx.y * NF;
  const bool cell = c < p.n;
  const bool live = cell && (p.full[c] || p.mprev);
  const int adm = live ? p.admis[c] : 0, nf = live ? p.nfaces[c] : 0;
  const int A = p.admis_max, ID2 = p.ideg2;
  const bool cw = p.ees == 5;
  const double lc1 = 1.0 - 1.0 / p.lwci;
  const double lk = adm > 1 ? (1.0 - lc1) / (adm - 1) : 0.0;
  const T* Gc = (const T*)p.gbuf + grp * (int64_t)(A * ID * NV) * 32 + lane;
  double u0[NV];
#pragma unroll
  for (int k = 0; k < NV; ++k) u0[k] = cell ? U[c * NV + k] : 1.0;
  for (int f = v; f < NF; f += NV)
    if (f0 + f < nf) {
      const int64_t cf = c * MF + f0 + f;
      double r[4], ur[NV], rl[NV], rr[NV];
#pragma unroll
      for (int k = 0; k < 4; ++k) r[k] = p.rot[cf * 4 + k];
      const int64_t nb = p.neigh[cf];
      if (nb >= 0) {
#pragma unroll
        for (int k = 0; k < NV; ++k) ur[k] = U[nb * NV + k];
      } else {
        boundary_ghost(p, p.bc[cf], r, u0, ur);
      }
      rot_f(r, u0, rl);
      rot_f(r, ur, rr);
      char_eigenvectors(p.gamma, rl, rr, s_e + f * 50 * 32 + lane, s_e + (f * 50 + 25) * 32 + lane, 32);
    }
  if (cw) char_lower_sum<P, T>(p, Gc, adm, v, lane, s_g);
  __syncthreads();
  // indicators and weights (WENOWEIGHTS, FP64) of characteristic variable v
  const double* Qc = p.qbuf + grp * (int64_t)(A * 15) * 32 + lane;
  auto weights = [&](int f, double (&w)[MA]) {  // w: the indicators
    double tau = 0.0, sum = 0.0;
    if (cw && p.wenoz) {
#pragma unroll
      for (int ll = 0; ll < MA; ++ll)
        if (ll < adm) tau += fabs(w[0] - w[ll]);
      tau = tau / (adm - 1);
    }
#pragma unroll
    for (int ll = 0; ll < MA; ++ll)
      if (ll < adm) {
        const double e = p.weno_eps + w[ll];
        const double lam = ll == 0 ? (cw ? lc1 : p.lwci) : (cw ? lk : 1.0);
        if (cw && p.wenoz) {
          double q = tau / e;
          q = q * q;
          w[ll] = lam * (1.0 + q * q);
        } else {
          const double e2 = e * e;
          w[ll] = lam / (e2 * e2);
        }
        sum += w[ll];
      }
#pragma unroll
    for (int ll = 0; ll < MA; ++ll)
      if (ll < adm) s_w[((f * MA + ll) * NV + v) * 32 + lane] = w[ll] / sum;
  };
  if constexpr (LEAN) {  // a stencil's form read once for the block's faces
    double l[NF][NV], w[NF][MA];
#pragma unroll
    for (int f = 0; f < NF; ++f)
#pragma unroll
      for (int u = 0; u < NV; ++u) l[f][u] = f0 + f < nf ? s_e[(f * 50 + v * NV + u) * 32 + lane] : 0.0;
#pragma unroll
    for (int ll = 0; ll < MA; ++ll) {
#pragma unroll
      for (int f = 0; f < NF; ++f) w[f][ll] = 0.0;
      if (ll < adm) {
        int j = 0;
#pragma unroll
        for (int u = 0; u < NV; ++u)
#pragma unroll
          for (int k = u; k < NV; ++k, ++j) {
            const double q = Qc[(int64_t)(ll * 15 + j) * 32];
#pragma unroll
            for (int f = 0; f < NF; ++f) w[f][ll] += (u == k ? 1.0 : 2.0) * l[f][u] * l[f][k] * q;
          }
      }
    }
#pragma unroll
    for (int f = 0; f < NF; ++f)
      if (f0 + f < nf) weights(f, w[f]);
  } else {
    for (int f = 0; f < NF; ++f) {
      if (f0 + f >= nf) break;
      double l[NV], w[MA];
#pragma unroll
      for (int u = 0; u < NV; ++u) l[u] = s_e[(f * 50 + v * NV + u) * 32 + lane];
#pragma unroll
      for (int ll = 0; ll < MA; ++ll) {
        w[ll] = 0.0;
        if (ll < adm) {
          double is = 0.0;
          int j = 0;
#pragma unroll
          for (int u = 0; u < NV; ++u)
#pragma unroll
            for (int k = u; k < NV; ++k, ++j)
              is += (u == k ? 1.0 : 2.0) * l[u] * l[k] * Qc[(int64_t)(ll * 15 + j) * 32];
          w[ll] = is;
        }
      }
      weights(f, w);
    }
  }
  __syncthreads();
  // the faces' polynomials of variable v
  T gh[NF][ID];
  double fm[NF];
#pragma unroll
  for (int f = 0; f < NF; ++f) {
    fm[f] = 0.0;
#pragma unroll
    for (int d = 0; d < ID; ++d) gh[f][d] = T(0);
  }
#pragma unroll 1
  for (int ll = 0; ll < adm; ++ll) {
    const int nd = cw && ll > 0 ? ID2 : ID;
    const bool rem = cw && ll == 0;
    T M[NF][NV];
#pragma unroll
    for (int f = 0; f < NF; ++f) {
#pragma unroll
      for (int u = 0; u < NV; ++u) M[f][u] = T(0);
      if (f0 + f < nf) {
        const double *EL = s_e + f * 50 * 32 + lane, *ER = EL + 25 * 32, *wf = s_w + (f * MA + ll) * NV * 32 + lane;
#pragma unroll
        for (int u = 0; u < NV; ++u) {
          double a = 0.0;
#pragma unroll
          for (int j = 0; j < NV; ++j) a += ER[(v * NV + j) * 32] * wf[j * 32] * EL[(j * NV + u) * 32];
          fm[f] += a * u0[u];
          M[f][u] = T(a);
        }
      }
    }
    const T* Gl = Gc + (int64_t)(ll * ID) * NV * 32;
#pragma unroll
    for (int d = 0; d < ID; ++d)
      if (d < nd) {
        T gu[NV];
#pragma unroll
        for (int u = 0; u < NV; ++u) {
          gu[u] = Gl[(int64_t)(d * NV + u) * 32];
          if (rem) gu[u] = T(1.0 / lc1) * (gu[u] - (d < L2 && d < ID2 ? s_g[(d * NV + u) * 32 + lane] : T(0)));
        }
#pragma unroll
        for (int f = 0; f < NF; ++f)
#pragma unroll
          for (int u = 0; u < NV; ++u) gh[f][d] += M[f][u] * gu[u];
      }
  }
  // face values, CHECKSOL and the stores, face by face
  const T* bmv = (const T*)p.bmean + grp * (int64_t)ID * 32 + lane;
  const T* xq = (const T*)p.qpts + grp * (int64_t)FQ * 3 * 32 + lane;
  double pm[NV];
  cons2prim(p.gamma, u0, pm);
  bool flag = false;
  T* out = (T*)p.dul + grp * 32 * (int64_t)FQ * NV;
  const int ncl = p.n - grp * 32 < 32 ? (int)(p.n - grp * 32) : 32;
#pragma unroll
  for (int f = 0; f < NF; ++f) {
    const int fc = f0 + f;
    if (fc >= MF) break;
    if (f) __syncthreads();  // the stores of the last face have read s_o
    const int nq = fc < nf ? face_nq(p, p.ftype[c * MF + fc]) : 0;
    T cb = T(0);
#pragma unroll
    for (int d = 0; d < ID; ++d) cb += bmv[d * 32] * gh[f][d];
    for (int q = 0; q < QS; ++q) {
      T r = T(0);
      if (q < nq) {
        const T* xi = xq + (int64_t)(fc * QS + q) * 3 * 32;
        T m[ID], t = T(0);
        monomials<P, T>(xi[0], xi[32], xi[64], m);
#pragma unroll
        for (int d = 0; d < ID; ++d) t += m[d] * gh[f][d];
        r = T((fm[f] - u0[v]) + (double)(t - cb));
      }
      s_o[lane * RS + q * NV + v] = r;
    }
    __syncthreads();
    for (int q = v; q < nq; q += NV) {  // CHECKSOL (0.85): warp v takes the points v, v + NV, ...
      double uf[NV];
#pragma unroll
      for (int k = 0; k < NV; ++k) uf[k] = u0[k] + (double)s_o[lane * RS + q * NV + k];
      flag = flag || jump_bad(p.gamma, pm, uf, 0.85);
    }
    if constexpr (LEAN) {  // a thread per value: a cell's run is short
      const int run = QS * NV;
      for (int k = threadIdx.x; k < ncl * run; k += 32 * NV) {
        const int cl = k / run, r = k - cl * run;
        out[(int64_t)cl * FQ * NV + fc * run + r] = s_o[cl * RS + r];
      }
    } else {
      for (int cl = v; cl < ncl; cl += NV)
        for (int r = lane; r < QS * NV; r += 32) out[(int64_t)cl * FQ * NV + fc * QS * NV + r] = s_o[cl * RS + r];
    }
  }
  if (flag) p.wflag[c] = 1;  // to the MUSCL fall-back (k_wpost<..., FB>)
}

// Characteristic-variable post-processing: compiled only in recon_char*.cu
// (explicit instantiations), in parallel with the other reconstruction units.
template <int P, typename T>
cudaError_t launch_wpost_char(const Problem& p, const double* U, cudaStream_t st) {
  const int QS = p.nq_quad > p.nq_tri ? p.nq_quad : p.nq_tri;
  constexpr int NF = CharFaces<P, T>::value;
  const unsigned ng = (unsigned)((p.n + 31) / 32);
  const size_t smem = char_face_smem<P, T>(QS);
  const cudaError_t e = smem_limit(k_char_face<P, T>, char_face_smem<P, T>(MQ));
  if (e != cudaSuccess) return e;
  k_char_forms<P, T><<<dim3(ng, (unsigned)p.admis_max), 32 * NV, 0, st>>>(p);
  k_char_face<P, T><<<dim3(ng, (MF + NF - 1) / NF), 32 * NV, smem, st>>>(p, U);
  k_wpost<P, T, false, true><<<(unsigned)((p.n + 127) / 128), 128, 0, st>>>(p, U);
  return cudaGetLastError();
}
#ifndef UCG_RECON_CHAR_TU
extern template cudaError_t launch_wpost_char<1, float>(const Problem&, const double*, cudaStream_t);
extern template cudaError_t launch_wpost_char<2, float>(const Problem&, const double*, cudaStream_t);
extern template cudaError_t launch_wpost_char<3, float>(const Problem&, const double*, cudaStream_t);
extern template cudaError_t launch_wpost_char<4, float>(const Problem&, const double*, cudaStream_t);
extern template cudaError_t launch_wpost_char<1, double>(const Problem&, const double*, cudaStream_t);
extern template cudaError_t launch_wpost_char<2, double>(const Problem&, const double*, cudaStream_t);
extern template cudaError_t launch_wpost_char<3, double>(const Problem&, const double*, cudaStream_t);
extern template cudaError_t launch_wpost_char<4, double>(const Problem&, const double*, cudaStream_t);
#endif

// the indicators of every cell into p.isb
template <int P, typename T>
cudaError_t launch_wis(const Problem& p, cudaStream_t st) {
  const unsigned ng = (unsigned)((p.n + 31) / 32), th = 32 * p.admis_max;
  if (!sets_give_is<P>(p)) {
    k_wis<P, T><<<ng, th, 0, st>>>(p);
    return cudaGetLastError();
  }
  const size_t smem = (size_t)p.i2off * sizeof(T);
  k_wis_set<P, T><<<dim3((unsigned)p.ntile, (unsigned)p.admis_max), SET_TILE, smem, st>>>(p);
  if (p.tiled) k_wis<P, T, true><<<ng, th, 0, st>>>(p);
  return cudaGetLastError();
}

// One reconstruction: stencil polynomials, WENO post-processing and, for
// Navier-Stokes, the viscous LSQ and face gradients.  Instantiated per
// precision and order in recon_*.cu, which nvcc compiles in parallel.
// `mark`, if not null, is recorded after the least squares (kernel timing).
template <int P, typename T>
cudaError_t launch_weno_t(const Problem& p, const double* U, bool ns, int QS, cudaStream_t st, int64_t* launches,
                          cudaEvent_t mark) {
  const unsigned b = (unsigned)((p.n + 127) / 128);
  // the per-cell records that the stencils gather cover every cell, also
  // those past the reconstructed prefix of a partition (p.n < p.nall)
  Problem pa = p;
  pa.n = p.nall > p.n ? p.nall : p.n;
  if (p.mmus) {  // the first MOOD cascade: MUSCL of the selected cells from this stage's G
    k_wpost<P, T, false, true, true><<<b, 128, 0, st>>>(p, U);
    ++*launches;
    return cudaGetLastError();
  }
  const cudaError_t el = launch_lsq<P, T>(p, U, st, launches);
  if (el != cudaSuccess) return el;
  if (mark) cudaEventRecord(mark, st);
  if (p.wenwrt == 2) {
    const cudaError_t e = launch_wpost_char<P, T>(p, U, st);
    if (e != cudaSuccess) return e;
    *launches += 2;
  } else {
    // indicators in their own kernel at IORDER 4, where the cell's packed
    // triangle (595 entries) no longer stays in L1 between the stencils of
    // one lane (64^3 WENO5: FP64 stage 17.2 -> 15.5 ms, mixed 7.80 -> 7.67 ms);
    // at IORDER 2-3 the triangle is small and the extra kernel costs more
    // than it saves (2.1 M-cell CWENO4, every cell's own triangle: 17.3 -> 19.6 ms)
    bool done = false;
    const int QS = p.nq_quad > p.nq_tri ? p.nq_quad : p.nq_tri;
    const size_t smem = wface_smem<T>(QS);
    const unsigned ng = (unsigned)((p.n + 31) / 32);
    if constexpr (P == 4) {
      if (p.isb && p.scheme == 3) {
        const cudaError_t e = launch_wis<P, T>(p, st);
        if (e != cudaSuccess) return e;
        ++*launches;
        if (p.wface) {
          const cudaError_t ef = smem_limit(k_wface<P, T>, wface_smem<T>(MQ));
          if (ef != cudaSuccess) return ef;
          k_wface<P, T><<<ng, 32 * NV, smem, st>>>(p, U);
          k_wpost<P, T, false, true><<<b, 128, 0, st>>>(p, U);
          ++*launches;
        } else {
          k_wpost<P, T, true><<<b, 128, 0, st>>>(p, U);
        }
        done = true;
      }
    } else if (wface_own<P, T>(p)) {
      const cudaError_t e = smem_limit(k_wface<P, T, true>, wface_smem<T>(MQ));
      if (e != cudaSuccess) return e;
      k_wface<P, T, true><<<ng, 32 * NV, smem, st>>>(p, U);
      k_wpost<P, T, false, true><<<b, 128, 0, st>>>(p, U);
      ++*launches;
      done = true;
    }
    if (!done) k_wpost<P, T><<<b, 128, 0, st>>>(p, U);
  }
  ++*launches;
  if (ns) {
    k_visc_prim<P, T><<<(unsigned)((pa.n + 255) / 256), 256, 0, st>>>(pa, U);
    if (p.ntile) {
      const size_t rows = (size_t)p.imax * set_stride<T>(Deg<P>::ideg) * sizeof(T);
      const cudaError_t e = smem_limit(k_visc_lsq<P, T, true>, SET_SMEM);
      if (e != cudaSuccess) return e;
      k_visc_lsq<P, T, true><<<(unsigned)(visc_lsq_own(p) + p.ntile), 128, rows, st>>>(p, U);
    } else {
      k_visc_lsq<P, T><<<(unsigned)((p.n + 127) / 128), 128, 0, st>>>(p, U);
    }
    *launches += 2;
    launch_visc_facegrad<P, T>(p, st);
    *launches += 1;
  }
  return cudaGetLastError();
}

// precision-specific entry points (recon_f32.cu + recon_f32_p4.cu, recon_f64.cu +
// recon_f64_p4.cu; characteristic post-processing in recon_char*.cu);
// iorder 1..4, anything else returns cudaErrorInvalidValue
cudaError_t launch_weno_f32(int iorder, const Problem& p, const double* U, bool ns, int QS, cudaStream_t st,
                            int64_t* launches, cudaEvent_t mark);
cudaError_t launch_weno_f32_p4(const Problem& p, const double* U, bool ns, int QS, cudaStream_t st,
                               int64_t* launches, cudaEvent_t mark);
cudaError_t launch_weno_f64(int iorder, const Problem& p, const double* U, bool ns, int QS, cudaStream_t st,
                            int64_t* launches, cudaEvent_t mark);
cudaError_t launch_weno_f64_p4(const Problem& p, const double* U, bool ns, int QS, cudaStream_t st,
                               int64_t* launches, cudaEvent_t mark);
// the stencil least squares alone (FP64 tables) into p.gbuf: G is linear in
// U, so applied to a tangent dU it gives the tangent dG (adjoint.cu)
cudaError_t launch_lsq_f64(int iorder, const Problem& p, const double* U, cudaStream_t st, int64_t* launches);
cudaError_t launch_lsq_f64_p4(const Problem& p, const double* U, cudaStream_t st, int64_t* launches);

}  // namespace ucg
