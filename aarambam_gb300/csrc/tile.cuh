// Strided line transforms (x and y passes): two register stages and one
// exchange.
//
// A pass moves tiles of N rows x W = 8 kz columns (64-byte row segments)
// between HBM and registers.  A line of N = R1 R2 points (R2 <= R1 <= 32)
// belongs to the T = R2 threads (t, w), w fastest: thread (t, w) of a tile
// loads x[t + T r], r < R1, of column w straight into registers -- a warp
// reads whole 64-byte segments of 4 rows -- runs a radix-R1 DFT, exchanges
// once through shared memory, and runs R1 / T radix-R2 DFTs whose outputs
// X[t + T b + R1 r] it stores the way it loaded (Stockham: fft.cuh).
//
// What bounds it: HBM; a tile in and a tile out is 128 KB at N = 1024 and the
// SM's share of the measured copy rate moves that in about 5900 cycles.  The
// lanes of a warp span the columns, so the global accesses need no staging
// and the exchange is the only shared-memory traffic: 2 x 64-bit accesses a
// value, conflict-free (below), where a tile staged in shared memory as
// padded lines took 6.  Measured per field against that form: y pass 2.13 ->
// 1.58 ms at 1024^3 (5.5 TB/s), 0.220 -> 0.188 ms at 512^3, 0.035 -> 0.023 ms
// at 256^3; x pass 2.09 -> 1.80, 0.231 -> 0.217, 0.037 -> 0.024 ms; the filter
// x pass (a field written per tile read from L2) 2.25 -> 1.61 ms at 1024^3.
//
// Exchange layout: row p of a column at row p + p / R1 (float2 [row][W]): the
// first stage's stores (thread t: rows t (R1 + 1) + r) of a half-warp, two
// values of t, fall on the two 64-byte halves of the banks because R1 + 1 is
// odd, and the second stage's loads (rows r (R1 + 1) + j, j consecutive over
// t) are contiguous.
#pragma once
#include "cells.cuh"
#include "fft.cuh"

namespace aar {

// asynchronous global -> shared copy of 16 bytes (cp.async), past L1
__device__ __forceinline__ void cp_async16(void* smem, const void* gmem) {
  unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async4(void* smem, const void* gmem) {  // of 4 bytes
  unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int K>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(K) : "memory");
}

template <int N>
struct TileCfg {
  static constexpr int W = 8;
  static constexpr int R1 = two_stage_r1(N);
  static constexpr int R2 = N / R1;
  static constexpr int T = R2;       // threads per line
  static constexpr int G = R1 / T;   // second-stage DFTs per thread
  static_assert(R1 * R2 == N && R1 % T == 0 && T % kXB == 0);
  static constexpr int THREADS = T * W;
  static constexpr size_t SMEM = sizeof(float2) * (size_t)T * (R1 + 1) * W;
  static constexpr int HP = ((N / 2 + 1) + 7) / 8 * 8;  // the plan's padded row length
  static constexpr int NCOL = HP / W;
  static constexpr int TILES = N * NCOL;  // tiles of a field
  // resident blocks per SM aimed at: 32 values per lane need 128 registers,
  // 16 take 64
  static constexpr int MINB = R1 == 32 ? 512 / THREADS : R1 == 16 ? 1024 / THREADS : 16;
};

// Offsets of a thread's values in a field (x-blocked row order row_of).
// AXIS 0: rows n = x at y = o; AXIS 1: rows n = y at x = o.  An index step of
// a multiple of kXB moves by a constant stride.
template <int N, int AXIS>
struct TileMap {
  using C = TileCfg<N>;
  static constexpr int64_t STEP = AXIS == 0 ? (int64_t)N * C::HP : (int64_t)kXB * C::HP;  // per unit of n
  int64_t base;  // element (t, w)
  __device__ __forceinline__ TileMap(int o, int c0, int t, int w) {
    base = (AXIS == 0 ? row_of(t, o, N, kXB) : row_of(o, t, N, kXB)) * C::HP + c0 + w;
  }
  static __device__ __forceinline__ int64_t off(int dn) { return (int64_t)dn * STEP; }  // dn a multiple of kXB
};

// The same in the caller's natural order, complex [N][N][N/2+1] (x passes): its
// row segments start on any 8 bytes.
template <int N>
struct NatMap {
  static constexpr int K = N / 2 + 1;
  static __device__ __forceinline__ int64_t base(int o, int c0, int t, int w) {
    return ((int64_t)t * N + o) * K + c0 + w;
  }
  static __device__ __forceinline__ int64_t off(int dn) { return (int64_t)dn * N * K; }
};

// Line index of value i of thread t before a transform (x[t + T i]) and, at
// v[b R2 + r], after it (X[t + T b + R1 r]): the same indices, value i = b +
// (R1 / T) r.
template <int N>
__device__ __forceinline__ int tile_n(int t, int i) {
  return t + TileCfg<N>::T * i;
}
template <int N>
__device__ __forceinline__ constexpr int tile_out_i(int b, int r) {
  return b + TileCfg<N>::G * r;
}

// The transform of a thread's line values: v[r] = x[t + T r] in, v[b R2 + r]
// = X[t + T b + R1 r] out.  tw2[r R1 + j] = exp(-2 pi i r j / N).  All threads
// of the block call it; the caller synchronises before ex is used again.
template <int N, int SIGN>
__device__ __forceinline__ void tile_fft2(float2* v, float2* ex, int t, int w, const float2* __restrict__ tw2) {
  using C = TileCfg<N>;
  DFT<C::R1, SIGN>::run(v);
  float2* s = ex + t * (C::R1 + 1) * C::W + w;
#pragma unroll
  for (int r = 0; r < C::R1; ++r) s[r * C::W] = v[r];
  __syncthreads();
  const float2* q = ex + t * C::W + w;
#pragma unroll
  for (int b = 0; b < C::G; ++b)
#pragma unroll
    for (int r = 0; r < C::R2; ++r) v[b * C::R2 + r] = q[(r * (C::R1 + 1) + C::T * b) * C::W];
#pragma unroll
  for (int b = 0; b < C::G; ++b) {
    const float2* tw = tw2 + t + C::T * b;
#pragma unroll
    for (int r = 1; r < C::R2; ++r) v[b * C::R2 + r] = cmul(v[b * C::R2 + r], tw_load<SIGN>(tw, r * C::R1));
    DFT<C::R2, SIGN>::run(v + b * C::R2);
  }
}

// Issue the asynchronous copy of a tile into shared memory as [n][W] (its
// 64-byte row segments as they lie in memory).
template <int N, int AXIS>
__device__ __forceinline__ void tile_stage_load(float2* stage, const float2* __restrict__ f, int o, int c0) {
  using C = TileCfg<N>;
  constexpr int ROWS = C::THREADS / 4;  // rows of one copy per thread
  static_assert(ROWS % kXB == 0 && N % ROWS == 0);
  const int n = threadIdx.x >> 2, part = (threadIdx.x & 3) * 2;
  const float2* src = f + TileMap<N, AXIS>(o, c0, n, part).base;
  float2* dst = stage + n * C::W + part;
#pragma unroll
  for (int j = 0; j < N / ROWS; ++j) cp_async16(dst + j * ROWS * C::W, src + TileMap<N, AXIS>::off(j * ROWS));
}

// Packed FP32 sums of a complex value's two parts (one issue slot each; the
// FP32 pipe takes as long as two scalar ones).
__device__ __forceinline__ float2 add2(float2 a, float2 b) {
  unsigned long long r;
  asm("add.rn.f32x2 %0, %1, %2;"
      : "=l"(r)
      : "l"(reinterpret_cast<unsigned long long&>(a)), "l"(reinterpret_cast<unsigned long long&>(b)));
  return reinterpret_cast<float2&>(r);
}
__device__ __forceinline__ float2 sub2(float2 a, float2 b) {
  unsigned long long r;
  asm("sub.rn.f32x2 %0, %1, %2;"
      : "=l"(r)
      : "l"(reinterpret_cast<unsigned long long&>(a)), "l"(reinterpret_cast<unsigned long long&>(b)));
  return reinterpret_cast<float2&>(r);
}
// Knuth's two-sum: s + c carries the running sum of the t's, the rounding
// error of s + t exactly (as Neumaier's step, without its comparison)
__device__ __forceinline__ void two_sum2(float2& s, float2& c, float2 t) {
  const float2 u = add2(s, t), b = sub2(u, s);
  c = add2(c, add2(sub2(s, sub2(u, b)), sub2(t, b)));
  s = u;
}

}  // namespace aar
