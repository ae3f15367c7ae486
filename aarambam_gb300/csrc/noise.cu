// Seed table and Gaussian potential (white noise) kernels.
//
// Seed table (Aarambam/LPT/Basis/main.c:317-349): one ranlxd1 stream seeded
// with Seed delivers N^2 uniforms, stored as (unsigned)(0x7fffffff * u) in
// eight "shell" segments per i < N/2.  One thread takes one refill (12
// draws): it rebuilds the refill's starting state with the exact skip-ahead of
// ranlux.cuh and scatters its draws (the shell order is a permutation of the
// table, so the scatter has no write conflicts).
//
// Noise (main.c:382-524): one thread per (i, j) column reseeds ranlxd1 with
// seedtable[i][j] and draws (phase, amplitude) pairs for k < N/2, skipping the
// Nyquist indices and DC after the draws, keeping the cube/sphere cut, and
// writing the k = 0 plane with its Hermitian partner (k_noise32: the lanes of a
// warp share its columns' cells).  The fused plan's
// spectrum is written in its x-blocked row order; the plain form and the
// caller's buffers in the natural one.
#include <cuda_runtime.h>
#include <stdint.h>

#include <mutex>
#include <string>
#include <type_traits>
#include <vector>

#include "aar_internal.cuh"
#include "ranlux.cuh"

namespace aar {

__device__ __forceinline__ int shell_pos(int d, int N) {
  // draws before shell i: 4 i^2; segment lengths i, i+1, i, i+1, ...
  int i = (int)sqrtf((float)d) / 2;
  while (4 * (i + 1) * (i + 1) <= d) ++i;
  while (4 * i * i > d) --i;
  int o = d - 4 * i * i;
  const int n = N;
  if (o < i) return i * n + o;
  o -= i;
  if (o < i + 1) return o * n + i;
  o -= i + 1;
  if (o < i) return (n - 1 - i) * n + o;
  o -= i;
  if (o < i + 1) return (n - 1 - o) * n + i;
  o -= i + 1;
  if (o < i) return i * n + (n - 1 - o);
  o -= i;
  if (o < i + 1) return o * n + (n - 1 - i);
  o -= i + 1;
  if (o < i) return (n - 1 - i) * n + (n - 1 - o);
  o -= i;
  return (n - 1 - o) * n + (n - 1 - i);
}

// What bounds it: the latency of one thread's chain of 576-bit products and
// of the 202 steps, at every grid size (N^2 / 12 threads).  So the chain is
// short: the seeded state and its residue come from the host, the power of
// the g-th refill is a product of at most three table entries (g's base-256
// digits; the binary powers took up to 17), and a thread does one refill.
// N = 64 0.023 ms, N = 1024 0.065 ms; with 8 refills per thread, seeding on
// the device and binary powers 0.137 and 0.161 ms.
static __device__ const U576 kSkip[kRlxLevels * kRlxRadix] = {
#include "ranlux_powers.h"  // level l, digit d: b^{-202 d 256^l} mod m (generated by build.py)
};
struct SeedStart {
  Rlx s;   // the seeded state
  U576 r;  // its residue
};
__global__ void __launch_bounds__(32) k_seedtable(const __grid_constant__ SeedStart st, int N,
                                                  uint32_t* __restrict__ table) {
  const int g = blockIdx.x * 32 + threadIdx.x;
  const int total = N * N, d0 = 12 * g;
  if (d0 >= total) return;
  Rlx s;
  if (g == 0) {
    s = st.s;
  } else {
    U576 r = st.r;
    for (int l = 0, h = g; h; ++l, h >>= 8)
      if (h & 255) r = modmul576(r, kSkip[l * kRlxRadix + (h & 255)]);
    rlx_from_residue(r, s);
  }
  rlx_refill(s);
#pragma unroll
  for (int i = 0; i < 12; ++i) {
    if (d0 + i >= total) break;
    const double u = (double)s.x[i] * 3.5527136788005009e-15;  // 2^-48
    table[shell_pos(d0 + i, N)] = __double2uint_rz(__dmul_rn(2147483647.0, u));
  }
}

static void run_seedtable(Plan* p, uint32_t* d_out, cudaStream_t st) {
  SeedStart s0;
  rlx_seed(s0.s, (uint32_t)p->prm.seed);
  s0.r = rlx_window_residue(s0.s);
  const int64_t nthr = ((int64_t)p->N * p->N + 11) / 12;
  k_seedtable<<<(unsigned)((nthr + 31) / 32), 32, 0, st>>>(s0, p->N, d_out);
}

int launch_seedtable(Plan* p, uint32_t* d_out, cudaStream_t st) {
  {
    ProfScope ps_(p, "seedtable", st);
    run_seedtable(p, d_out, st);
  }
  AAR_CUDA_TRY(p, cudaGetLastError());
  p->last_launches += 1;
  return AAR_OK;
}

// ------------------------------------------------------------ noise
struct NoiseArgs {
  Grid g;
  int xb;  // row order of the output: row_of(i, j, N, xb)
  int phase_flip, fixed_amp;
  int one_draw;  // every column one draw at a time (AAR_NOISE_ONE_DRAW=1: checks the six-cell blocks)
  // FP64 form: the reference's own formula
  double anorm, ns, fac, beta;
  aar_params prm;  // variant and ResBasis oscillation (noise_osc)
  // FP32 form: amplitude per n^2 = sqrt(Anorm k^ns osc) fac Beta / k^2
  const float* amp;
};

// -ln(u) for u = U 2^-48 in (0, 1), FP32: U = f + l with f its nearest float
// and l the exact rest (|l| <= 2^-25 f), so ln u = ln(f 2^-48) + l / f to
// 2^-50; for u next to 1, where ln f cancels or vanishes, l / f carries the
// digits of 1 - u.
__device__ __forceinline__ float neg_log_u48(uint64_t U) {
  const float h = (float)(uint32_t)(U >> 24), g = (float)(uint32_t)(U & 0xFFFFFFu);
  const float f = fmaf(h, 16777216.f, g);
  const float l = g - fmaf(-h, 16777216.f, f);
  return -(logf(f * 3.5527136788005009e-15f) + __fdividef(l, f));
}

// cos / sin of 2 pi u (+ pi when flipped) for u = U 2^-48, FP32: the exact
// split U = H 2^24 + L gives sincospi(H 2^-23) plus a first-order correction.
__device__ __forceinline__ void sincos_u48(uint64_t U, bool flip, float& c, float& s) {
  uint32_t H = (uint32_t)(U >> 24), L = (uint32_t)(U & 0xFFFFFFu);
  float a = (float)H * 1.1920928955078125e-07f;  // H 2^-23 (exact)
  float s0, c0;
  sincospif(a, &s0, &c0);
  float d = (float)L * (float)(3.14159265358979323846 / 140737488355328.0);
  c = c0 - d * s0;
  s = s0 + d * c0;
  if (flip) {
    c = -c;
    s = -s;
  }
}

// Where cell (i, j, k) of a column goes and with what: the k = 0 plane is
// Hermitian, its cell (i, j) drawn for i = 0, j < N/2 and for 0 < i < N/2 and
// conjugated into (-i, -j) (main.c:463-520).  c1 < 0: the cell belongs to its
// partner's column.
__device__ __forceinline__ void noise_place(const NoiseArgs& a, int i, int j, int k, int HP, int64_t& c1, int64_t& c2) {
  const int N = a.g.N;
  c1 = c2 = -1;
  if (k > 0) {
    c1 = row_of(i, j, N, a.xb) * HP + k;
  } else if (i == 0) {
    if (j >= N / 2) return;
    c1 = row_of(0, j, N, a.xb) * HP;
    if (j > 0) c2 = row_of(0, N - j, N, a.xb) * HP;
  } else {
    if (i >= N / 2) return;
    c1 = row_of(i, j, N, a.xb) * HP;
    c2 = row_of(N - i, (N - j) % N, N, a.xb) * HP;
  }
}

// One cell by the reference's FP64 formula (main.c:443-459) from its two
// uniforms U1 (phase), U2 (amplitude), into a buffer that starts at zero: the
// Nyquist / DC skips after the draws, the cut.  OUT64: double2 output (the
// plain forms), else float2.
template <bool OUT64>
__device__ __forceinline__ void noise_cell64(const NoiseArgs& a, int i, int j, int k, uint64_t U1, uint64_t U2, double fx,
                                             double fy, void* __restrict__ out, int HP) {
  const int N = a.g.N;
  if (i == N / 2 || j == N / 2) return;
  if (i == 0 && j == 0 && k == 0) return;
  const int kx = sidx(i, N), ky = sidx(j, N);
  if (!keep_cell(a.g, kx, ky, k)) return;
  const double fz = __ddiv_rn(__dmul_rn((double)(2 * k), kPi), a.g.box);
  const double k2 = __dadd_rn(__dadd_rn(__dmul_rn(fx, fx), __dmul_rn(fy, fy)), __dmul_rn(fz, fz));
  const double km = sqrt(k2);
  double phase = __dmul_rn(__dmul_rn((double)U1 * 3.5527136788005009e-15, 2.0), kPi);
  if (a.phase_flip) phase = __dadd_rn(phase, kPi);
  const double ampl = (double)U2 * 3.5527136788005009e-15;
  double phig = noise_osc(a.prm, a.anorm * exp(a.ns * log(km)), km);
  if (!a.fixed_amp) phig *= -log(ampl);
  phig = sqrt(phig) * a.fac * a.beta / k2;
  double sn, cs;
  sincos(phase, &sn, &cs);
  const double re = phig * cs, im = phig * sn;
  int64_t c1, c2;
  noise_place(a, i, j, k, HP, c1, c2);
  if (c1 < 0) return;
  if (OUT64) {
    double2* o = (double2*)out;
    o[c1] = make_double2(re, im);
    if (c2 >= 0) o[c2] = make_double2(re, -im);
  } else {
    float2* o = (float2*)out;
    o[c1] = make_float2((float)re, (float)im);
    if (c2 >= 0) o[c2] = make_float2((float)re, -(float)im);
  }
}

// The drawn value of a cell of |k|^2 = n2 in FP32
__device__ __forceinline__ float2 noise_draw32(const NoiseArgs& a, int n2, uint64_t U1, uint64_t U2) {
  float amp = __ldg(a.amp + n2);
  if (!a.fixed_amp) amp *= sqrtf(neg_log_u48(U2));
  float c, sn;
  sincos_u48(U1, a.phase_flip != 0, c, sn);
  return make_float2(amp * c, amp * sn);
}

// One cell in FP32 from the per-|k|^2 amplitudes, zero where nothing is drawn:
// every cell k < N/2 of the spectrum is written by exactly one column, so the
// buffer needs no clearing.
__device__ __forceinline__ void noise_cell32(const NoiseArgs& a, int i, int j, int k, uint64_t U1, uint64_t U2,
                                             float2* __restrict__ o, int HP) {
  const int N = a.g.N;
  const int kx = sidx(i, N), ky = sidx(j, N), n2 = kx * kx + ky * ky + k * k;
  float2 r = make_float2(0.f, 0.f);
  if (i != N / 2 && j != N / 2 && n2 != 0 && keep_cell(a.g, kx, ky, k)) r = noise_draw32(a, n2, U1, U2);
  int64_t c1, c2;
  noise_place(a, i, j, k, HP, c1, c2);
  if (c1 < 0) {
    // (N/2, j, 0) and (0, N/2, 0) are their own or each other's partners: zero
    if (i != N / 2 && !(i == 0 && j == N / 2)) return;
    c1 = row_of(i, j, N, a.xb) * HP;
  }
  o[c1] = r;
  if (c2 >= 0) o[c2] = make_float2(r.x, -r.y);
}

template <bool FP64, bool OUT64>
__device__ __forceinline__ void noise_cell(const NoiseArgs& a, int i, int j, int k, uint64_t U1, uint64_t U2, double fx,
                                           double fy, void* __restrict__ out, int HP) {
  if constexpr (FP64) noise_cell64<OUT64>(a, i, j, k, U1, U2, fx, fy, out, HP);
  else noise_cell32(a, i, j, k, U1, U2, (float2*)out, HP);
}

// The rest of a column from cell k on with the generator as it stands:
// draws one by one (U2 == 0 redrawn, main.c:401-403).  Taken from the
// start of the first refill block whose pairing a redraw would shift -- a
// zero U2 has probability 2^-48 -- and never otherwise.  Not inlined: the
// state indexed by its running position lives in local memory here only.
template <bool FP64, bool OUT64>
__device__ __noinline__ void noise_column_rest(NoiseArgs a, Rlx s, int i, int j, int k, double fx, double fy,
                                                void* __restrict__ out, int HP) {
  for (; k < a.g.N / 2; ++k) {
    const uint64_t U1 = rlx_next48(s);
    uint64_t U2;
    do U2 = rlx_next48(s);
    while (U2 == 0);
    noise_cell<FP64, OUT64>(a, i, j, k, U1, U2, fx, fy, out, HP);
  }
}

// The FP64 amplitudes: one thread per (i, j) column.  A refill of ranlxd1 gives
// 12 uniforms, the (U1, U2) pairs of six cells while no U2 is zero: the column
// runs in blocks of six cells reading the refilled state at compile-time
// indices (it stays in registers), and a block with a zero U2 hands the column
// from its first draw to noise_column_rest.  Same draws, same cells as one
// draw at a time.
template <bool OUT64>
__global__ void k_noise64(NoiseArgs a, const uint32_t* __restrict__ seedtable, void* __restrict__ out, int HP) {
  const int N = a.g.N;
  int64_t col = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (col >= (int64_t)N * N) return;
  const int i = (int)(col / N), j = (int)(col % N);
  Rlx s;
  rlx_seed(s, seedtable[col]);
  const double fx = __ddiv_rn(__dmul_rn((double)(2 * sidx(i, N)), kPi), a.g.box);
  const double fy = __ddiv_rn(__dmul_rn((double)(2 * sidx(j, N)), kPi), a.g.box);
  if (a.one_draw) {
    noise_column_rest<true, OUT64>(a, s, i, j, 0, fx, fy, out, HP);
    return;
  }
  for (int k = 0; k < N / 2; k += 6) {
    rlx_refill(s);  // every block consumes whole refills: the position is 12 here
    const int nk = min(6, N / 2 - k);
    bool zero = false;
#pragma unroll
    for (int c = 0; c < 6; ++c) zero |= c < nk && s.x[2 * c + 1] == 0;
    if (zero) {
      noise_column_rest<true, OUT64>(a, s, i, j, k, fx, fy, out, HP);
      return;
    }
#pragma unroll
    for (int c = 0; c < 6; ++c)
      if (c < nk) noise_cell64<OUT64>(a, i, j, k + c, s.x[2 * c], s.x[2 * c + 1], fx, fy, out, HP);
  }
}

// The FP32 amplitudes: a warp takes COLS consecutive columns, a lane each for
// the generator.  Two refills give a column's next twelve cells; their uniforms
// cross the warp through shared memory so that all 32 lanes form the cells, 12
// consecutive lanes a column's (96-byte runs), and N/2 .. HP - 1 are cleared at
// the end.  A column with a zero U2, which shifts the pairing of its later
// draws (probability 2^-48 per draw), leaves the warp and is made from its
// start by noise_column_rest.
//
// What bounds it: the generator's serial steps -- their latency while there
// are few columns, their issue with many -- and the cells' logarithm, sine and
// cosine.  A column per thread, each storing 8 bytes a row, on a cleared
// buffer: 8.2 ms at 1024^3 with the clearing, this form 7.0; 1.15 -> 0.99 at
// 512^3, 0.060 -> 0.049 at 128^3, 0.035 -> 0.023 at 64^3.
constexpr int kNoiseWarps = 4;
template <int COLS>
__global__ void __launch_bounds__(32 * kNoiseWarps, 6) k_noise32(const __grid_constant__ NoiseArgs a,
                                                             const uint32_t* __restrict__ seedtable,
                                                             float2* __restrict__ out, int HP) {
  constexpr int LD = 25;  // odd: the columns' 8-byte rows fall on different banks
  __shared__ uint64_t raw_all[kNoiseWarps][COLS * LD];
  __shared__ int64_t base_all[kNoiseWarps][COLS];  // a column's row in `out`
  __shared__ int kk_all[kNoiseWarps][COLS];        // kx^2 + ky^2, negative: nothing drawn in the column
  __shared__ int kxy_all[kNoiseWarps][COLS];       // kx, ky of the sphere's cut, 16 bits each
  const int N = a.g.N, lane = threadIdx.x & 31;
  uint64_t* raw = raw_all[threadIdx.x >> 5];
  const int64_t col0 = ((int64_t)blockIdx.x * kNoiseWarps + (threadIdx.x >> 5)) * COLS, ncol = (int64_t)N * N;
  if (col0 >= ncol) return;
  const int here = (int)min((int64_t)COLS, ncol - col0);  // N not a multiple of 8: a short last warp
  const bool own = lane < here;
  const int oi = (int)((unsigned)(col0 + lane) / (unsigned)N), oj = (int)(col0 + lane) - oi * N;
  int64_t* base = base_all[threadIdx.x >> 5];
  int* kk = kk_all[threadIdx.x >> 5];
  int* kxy = kxy_all[threadIdx.x >> 5];
  if (own) {
    const int kx = sidx(oi, N), ky = sidx(oj, N);
    const bool in = oi != N / 2 && oj != N / 2 && (a.g.sphere || (abs(kx) <= a.g.kcut && abs(ky) <= a.g.kcut));
    base[lane] = row_of(oi, oj, N, a.xb) * HP;
    kk[lane] = in ? kx * kx + ky * ky : -1;
    kxy[lane] = (kx & 0xffff) | (int)((unsigned)ky << 16);
  }
  Rlx s;
  rlx_seed(s, own ? seedtable[col0 + lane] : 1u);
  if (a.one_draw) {
    if (own) noise_column_rest<false, false>(a, s, oi, oj, 0, 0, 0, out, HP);
  } else {
    unsigned dead = 0;  // columns that left the warp
    for (int k = 0; k < N / 2; k += 12) {
      const int nk = min(12, N / 2 - k);
      bool zero = false;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        rlx_refill(s);
        if (own) {
#pragma unroll
          for (int c = 0; c < 12; ++c) raw[lane * LD + 12 * h + c] = s.x[c];
        }
#pragma unroll
        for (int c = 0; c < 6; ++c) zero |= 6 * h + c < nk && s.x[2 * c + 1] == 0;
      }
      dead |= __ballot_sync(0xffffffffu, own && zero);  // also orders the stores before the loads
      __syncwarp();
#pragma unroll 2
      for (int q = lane; q < here * 12; q += 32) {
        const int cl = q / 12, c = q - 12 * cl;
        if (c >= nk || (dead >> cl) & 1u) continue;
        const uint64_t U1 = raw[cl * LD + 2 * c], U2 = raw[cl * LD + 2 * c + 1];
        const int kz = k + c;
        if (kz == 0) {
          const unsigned col = (unsigned)(col0 + cl);
          noise_cell32(a, (int)(col / N), (int)(col % N), 0, U1, U2, out, HP);
          continue;
        }
        const int k2 = kk[cl], n2 = k2 + kz * kz;
        bool on = k2 >= 0;
        if (!a.g.sphere) on = on && kz <= a.g.kcut;
        else if (on) on = keep_cell(a.g, (int)(short)kxy[cl], kxy[cl] >> 16, kz);
        out[base[cl] + kz] = on ? noise_draw32(a, n2, U1, U2) : make_float2(0.f, 0.f);
      }
      __syncwarp();
    }
    if (own && (dead >> lane) & 1u) {
      rlx_seed(s, seedtable[col0 + lane]);
      noise_column_rest<false, false>(a, s, oi, oj, 0, 0, 0, out, HP);
    }
  }
  __syncwarp();
  const int tail = HP - N / 2;  // the kz = N/2 plane and the padding columns
  for (int q = lane; q < here * tail; q += 32) {
    const int cl = q / tail;
    out[base[cl] + N / 2 + (q - cl * tail)] = make_float2(0.f, 0.f);
  }
}

static NoiseArgs noise_args(Plan* p, int xb) {
  NoiseArgs a;
  a.g = p->grid;
  a.xb = xb;
  a.phase_flip = p->prm.phase_flip == 1;
  a.fixed_amp = p->prm.fixed_amplitude != 0;
  a.one_draw = p->noise_one_draw;
  a.anorm = p->Anorm;
  a.ns = p->prm.primordial_index;
  a.fac = pow(2 * kPi / p->prm.box, 1.5);
  a.beta = p->Beta;
  a.prm = p->prm;
  a.amp = p->d_amp;
  return a;
}

// The FP32 form's Gaussian spectrum, row order xb, into out (rows of hp)
static int run_noise32(Plan* p, const uint32_t* d_seed, float2* out, int hp, int xb, cudaStream_t st) {
  const int64_t cols = (int64_t)p->N * p->N;
  if (p->prm.noise_fp64) {
    AAR_CUDA_TRY(p, cudaMemsetAsync(out, 0, sizeof(float2) * (size_t)cols * hp, st));
    k_noise64<false><<<(unsigned)((cols + 127) / 128), 128, 0, st>>>(noise_args(p, xb), d_seed, out, hp);
    return AAR_OK;
  }
  // columns per warp: fewer lanes run the generator where there are few warps
  // to hide its latency, at the price of its issue slots: 64^3 0.0226 ms with
  // 8, 0.0275 with 16; 128^3 0.049 with 16, 0.058 with 32.  That is one plan by
  // itself; the rule knows nothing of other plans on the device.  Six 128^3
  // plans in one graph took 2615 us with 16 and 2584 with 32.
  auto go = [&](auto c) {
    constexpr int COLS = decltype(c)::value, per = COLS * kNoiseWarps;
    k_noise32<COLS><<<(unsigned)((cols + per - 1) / per), 32 * kNoiseWarps, 0, st>>>(noise_args(p, xb), d_seed, out, hp);
  };
  if (p->N <= 64) go(std::integral_constant<int, 8>{});
  else if (p->N <= 128) go(std::integral_constant<int, 16>{});
  else go(std::integral_constant<int, 32>{});
  return AAR_OK;
}

int launch_noise_fp32(Plan* p, const uint32_t* d_seed, float2* d_phik, cudaStream_t st) {
  {
    ProfScope ps_(p, "noise", st);
    int rc = run_noise32(p, d_seed, d_phik, p->HP, kXB, st);
    if (rc) return rc;
  }
  AAR_CUDA_TRY(p, cudaGetLastError());
  p->last_launches += 1;
  return AAR_OK;
}

int launch_noise_fp64(Plan* p, const uint32_t* d_seed, double2* d_phik, int hp, cudaStream_t st) {
  size_t bytes = sizeof(double2) * (size_t)p->N * p->N * hp;
  AAR_CUDA_TRY(p, cudaMemsetAsync(d_phik, 0, bytes, st));
  int64_t cols = (int64_t)p->N * p->N;
  int bs = 128;
  { ProfScope ps_(p, "noise", st);
  k_noise64<true><<<(unsigned)((cols + bs - 1) / bs), bs, 0, st>>>(noise_args(p, 1), d_seed, d_phik, hp);
  }
  AAR_CUDA_TRY(p, cudaGetLastError());
  p->last_launches += 1;
  return AAR_OK;
}

// ------------------------------------------- no-allocation Gaussian spectrum
// Scratch of aar_gaussian_spectrum_noalloc: the seed table, one uint32 per
// (x, y) column of an Nmesh <= kNoAllocMaxN grid (4 MiB).  It is static
// device memory of this library, reserved when the CUDA module is loaded, so
// the call itself allocates nothing.  k_seedtable writes every entry before
// k_noise reads any, so nothing in it has to start at zero.  There is one
// scratch per device: calls that overlap on one device race on it.
constexpr int kNoAllocMaxN = 1024;
static __device__ __align__(256) uint32_t g_noalloc_seed[kNoAllocMaxN * kNoAllocMaxN];

// Address of the scratch on the plan's device, resolved once per device with
// cudaGetSymbolAddress (the first call on a device does this set-up).
static int noalloc_scratch(Plan* p, uint32_t** out) {
  constexpr int kMaxDev = 64;
  static std::mutex mu;
  static uint32_t* addr[kMaxDev] = {};
  int dev = -1;
  AAR_CUDA_TRY(p, cudaGetDevice(&dev));
  if (dev != p->dev) return set_err(p, "the current device is not the plan's device"), AAR_ERR_ARG;
  if (dev < 0 || dev >= kMaxDev) return set_err(p, "device ordinal out of range"), AAR_ERR_ARG;
  std::lock_guard<std::mutex> lock(mu);
  if (!addr[dev]) {
    void* a = nullptr;
    AAR_CUDA_TRY(p, cudaGetSymbolAddress(&a, g_noalloc_seed));
    addr[dev] = (uint32_t*)a;
  }
  *out = addr[dev];
  return AAR_OK;
}

// The Gaussian potential spectrum of the plan's seed straight into the
// caller's complex [N][N][N/2+1] buffer (float32 pairs for the fused form,
// float64 for the plain form), with the seed table in the static scratch
// instead of the plan's seed-table buffer.  Same kernels and arguments as
// launch_seedtable + launch_noise_fp32 / _fp64.
int noalloc_gaussian(Plan* p, void* d_out, cudaStream_t st) {
  const int N = p->N;
  if (N > kNoAllocMaxN)
    return set_err(p, "Nmesh " + std::to_string(N) + " exceeds the no-allocation scratch (Nmesh <= " +
                          std::to_string(kNoAllocMaxN) + ")"),
           AAR_ERR_ARG;
  uint32_t* seed = nullptr;
  int rc = noalloc_scratch(p, &seed);
  if (rc) return rc;
  const int64_t total = (int64_t)N * N;
  run_seedtable(p, seed, st);
  AAR_CUDA_TRY(p, cudaGetLastError());
  const int hp = N / 2 + 1;
  if (is_plain(p->prm)) {
    AAR_CUDA_TRY(p, cudaMemsetAsync(d_out, 0, sizeof(double2) * (size_t)total * hp, st));
    k_noise64<true><<<(unsigned)((total + 127) / 128), 128, 0, st>>>(noise_args(p, 1), seed, d_out, hp);
  } else if ((rc = run_noise32(p, seed, (float2*)d_out, hp, 1, st))) {
    return rc;
  }
  AAR_CUDA_TRY(p, cudaGetLastError());
  p->last_launches = 2;
  return AAR_OK;
}

}  // namespace aar
