// FP32 FFTs for sm_103a: register DFTs of radix 2..32 with compile-time
// twiddles, and the two-stage line transform of the folded rows.
//
// Stage formulation (here, tile.cuh, rows.cuh): Govindaraju et al., "High
// performance discrete Fourier transforms on graphics processors", SC'08, Fig. 2
// (iteration j, radix R, span Ns: inputs x[j + r N/R], twiddle exp(s 2 pi i r
// (j mod Ns)/(Ns R)), outputs y[(j/Ns) Ns R + (j mod Ns) + r Ns]).
#pragma once
#ifndef __CUDACC_RTC__
#include <cuda_runtime.h>
#include <stdint.h>
#else
typedef long long int64_t;
typedef unsigned int uint32_t;
#endif

namespace aar {

// ---------------------------------------------------------------- complex
__device__ __forceinline__ float2 cadd(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ float2 csub(float2 a, float2 b) { return make_float2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ float2 cmul(float2 a, float2 b) {
  return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ float2 cconj(float2 a) { return make_float2(a.x, -a.y); }
__device__ __forceinline__ float2 cscale(float2 a, float s) { return make_float2(a.x * s, a.y * s); }

// --------------------------------------------- compile-time trigonometry
// cos / sin of 2 pi k / n evaluated by quadrant reduction and Taylor series
// in double precision during compilation.
__host__ __device__ constexpr double ce_sin_small(double x) {
  double x2 = x * x, term = x, sum = x;
  for (int n = 1; n < 14; ++n) {
    term *= -x2 / ((2.0 * n) * (2.0 * n + 1));
    sum += term;
  }
  return sum;
}
__host__ __device__ constexpr double ce_cos_small(double x) {
  double x2 = x * x, term = 1, sum = 1;
  for (int n = 1; n < 14; ++n) {
    term *= -x2 / ((2.0 * n - 1) * (2.0 * n));
    sum += term;
  }
  return sum;
}
__host__ __device__ constexpr double ce_cos2pi(long k, long n) {
  long t = ((k % n) + n) % n;
  long q = (4 * t) / n, r = 4 * t - q * n;
  double a = 1.5707963267948966192313216916397514 * (double)r / (double)n;
  double c = ce_cos_small(a), s = ce_sin_small(a);
  return q == 0 ? c : q == 1 ? -s : q == 2 ? -c : s;
}
__host__ __device__ constexpr double ce_sin2pi(long k, long n) {
  long t = ((k % n) + n) % n;
  long q = (4 * t) / n, r = 4 * t - q * n;
  double a = 1.5707963267948966192313216916397514 * (double)r / (double)n;
  double c = ce_cos_small(a), s = ce_sin_small(a);
  return q == 0 ? s : q == 1 ? c : q == 2 ? -s : -c;
}

// multiply by exp(SIGN * 2 pi i K / R) with the trivial angles special-cased
template <int R, int K, int SIGN>
__device__ __forceinline__ float2 twiddle_ct(float2 v) {
  constexpr int k = ((K % R) + R) % R;
  if constexpr (k == 0) {
    return v;
  } else if constexpr (4 * k == R) {  // SIGN * i
    return SIGN < 0 ? make_float2(v.y, -v.x) : make_float2(-v.y, v.x);
  } else if constexpr (2 * k == R) {
    return make_float2(-v.x, -v.y);
  } else if constexpr (4 * k == 3 * R) {  // -SIGN * i
    return SIGN < 0 ? make_float2(-v.y, v.x) : make_float2(v.y, -v.x);
  } else {
    constexpr float c = (float)ce_cos2pi(k, R);
    constexpr float s = (float)(SIGN * ce_sin2pi(k, R));
    return make_float2(v.x * c - v.y * s, v.x * s + v.y * c);
  }
}

// ------------------------------------------------------ register DFTs
// In-place DFT of R values, natural order in and out: X_k = sum x_r w^{rk},
// w = exp(SIGN 2 pi i / R).  Radix-2 decimation in time, fully unrolled.
template <int R, int SIGN>
struct DFT {
  template <int K>
  static __device__ __forceinline__ void combine(float2* v, const float2* e, const float2* o) {
    if constexpr (K < R / 2) {
      float2 t = twiddle_ct<R, K, SIGN>(o[K]);
      v[K] = cadd(e[K], t);
      v[K + R / 2] = csub(e[K], t);
      combine<K + 1>(v, e, o);
    }
  }
  static __device__ __forceinline__ void run(float2* v) {
    if constexpr (R == 1) {
      return;
    } else if constexpr (R == 2) {
      float2 a = v[0], b = v[1];
      v[0] = cadd(a, b);
      v[1] = csub(a, b);
    } else if constexpr (R == 4) {
      float2 s0 = cadd(v[0], v[2]), d0 = csub(v[0], v[2]);
      float2 s1 = cadd(v[1], v[3]), d1 = csub(v[1], v[3]);
      float2 rd1 = twiddle_ct<4, 1, SIGN>(d1);
      v[0] = cadd(s0, s1);
      v[2] = csub(s0, s1);
      v[1] = cadd(d0, rd1);
      v[3] = csub(d0, rd1);
    } else {
      float2 e[R / 2], o[R / 2];
#pragma unroll
      for (int i = 0; i < R / 2; ++i) {
        e[i] = v[2 * i];
        o[i] = v[2 * i + 1];
      }
      DFT<R / 2, SIGN>::run(e);
      DFT<R / 2, SIGN>::run(o);
      combine<0>(v, e, o);
    }
  }
};

// First radix of the two-stage transforms (tile.cuh, rows.cuh): N = R1 R2,
// R2 <= R1 <= 32.
__host__ __device__ constexpr int two_stage_r1(int N) { return N >= 512 ? 32 : N >= 128 ? 16 : N >= 32 ? 8 : 4; }

// padded shared-memory index: one spare slot per 16 entries, so that the
// first stage's stores (lane t writes 16 t + r) and the natural-order loads both
// fall on distinct banks within a half-warp
__device__ __forceinline__ int spad(int i) { return i + (i >> 4); }
__host__ __device__ constexpr int spad_len(int n) { return n + n / 16 + 4; }

// Runtime twiddle exp(SIGN 2 pi i m / N) from a table tw[m] = exp(-2 pi i m / N)
// in global memory.
template <int SIGN>
__device__ __forceinline__ float2 tw_load(const float2* __restrict__ tw, int m) {
  float2 w = __ldg(tw + m);
  return SIGN < 0 ? w : make_float2(w.x, -w.y);
}

// ------------------------------------------------- 256-point lines
// A line of R R points (R = 16) in a padded shared-memory buffer, R lanes of a
// warp with R values each, two stages.  The second stage multiplies input r of
// lane k by exp(SIGN 2 pi i r k / R^2); a block keeps these in shared memory as
// lt[(r - 1) R + k] (lt_fill, once per block), so a lane reads its R - 1 factors
// as conflict-free shared loads instead of as many global loads per line at
// lane-scattered indices, which made the twiddles the largest source of L1
// wavefronts of the row kernel after its shared-memory stages.
constexpr int kLineR = 16;
constexpr int kLineTw = (kLineR - 1) * kLineR;  // entries of the lane twiddle table

// the table from tw, the table of a line TWS times as long, by the block's
// nthreads threads
template <int TWS>
__device__ __forceinline__ void lt_fill(float2* lt, const float2* __restrict__ tw, int tid, int nthreads) {
  for (int i = tid; i < kLineTw; i += nthreads) lt[i] = __ldg(tw + (i / kLineR + 1) * (i % kLineR) * TWS);
}

// The transform in place, natural order in and out (padded indices).  The R
// lanes of the line call it together, in whole warps.
template <int SIGN>
__device__ __forceinline__ void line_fft(float2* s, int t, const float2* __restrict__ lt) {
  constexpr int R = kLineR;
  float2 v[R];
  float2* p = s + t;  // element t + R r at spad = t + (R + 1) r
#pragma unroll
  for (int r = 0; r < R; ++r) v[r] = p[(R + 1) * r];
  __syncwarp();
  DFT<R, SIGN>::run(v);
#pragma unroll
  for (int r = 0; r < R; ++r) s[(R + 1) * t + r] = v[r];
  __syncwarp();
#pragma unroll
  for (int r = 0; r < R; ++r) v[r] = p[(R + 1) * r];
  __syncwarp();
#pragma unroll
  for (int r = 1; r < R; ++r) {
    const float2 w = lt[(r - 1) * R + t];
    v[r] = cmul(v[r], SIGN < 0 ? w : make_float2(w.x, -w.y));
  }
  DFT<R, SIGN>::run(v);
#pragma unroll
  for (int r = 0; r < R; ++r) p[(R + 1) * r] = v[r];
  __syncwarp();
}

}  // namespace aar
