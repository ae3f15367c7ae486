// Fused FP32 form of the Aarambam IC path on sm_103a.
//
// Fields live in HBM as complex half spectra float2 [N][N][HP] (HP >= N/2+1,
// a multiple of 8 so rows are 64-byte aligned); after a c2r the same buffer
// holds the real field as float [N][N][2 HP] (z fastest).  A 3-D transform is
// three passes, each reading and writing a field once:
//   x pass / y pass  -- strided complex FFTs on tiles of 8 consecutive kz
//                       columns x N rows, held in registers (tile.cuh);
//   z pass (rows)    -- the real<->half-complex transform of contiguous rows,
//                       two real rows as one N-point complex line (N = 1024
//                       with many lines: folded single rows; rows.cuh).
// The reference's per-pass work is fused into these passes:
//   modal potential (Aarambam/LPT/Basis/main.c:564-1151) regrouped exactly by
//   linearity of the DFT: acc = sum_r rho_r(k) r2c[ g_r ],
//   g_r(x) = sum_{p<=q} a'_{pqr} f_p(x) f_q(x), f_p = c2r[ q_p(k) phi(k) ],
//   with a' = alpha on sorted triples plus the two counter-terms of
//   main.c:1045-1050.  The x pass that starts every f_p reads phi once and
//   applies q_p; one row kernel does all c2r's, products and r2c's of a row;
//   the last x pass applies rho_r, sums over r and adds Fnl acc / N^3.
//   2LPT (main.c:1156-1381): one factor per axis (x passes, fan-out y passes,
//   c2r rows), the source in the row kernel, 1/k^2 in its forward x pass.
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include <stddef.h>

#include <algorithm>
#include <vector>

#include "aar_internal.cuh"
#include "fft.cuh"
#include "rows.cuh"
#include "spectral.cuh"
#include "tile.cuh"

namespace aar {

// ----------------------------------------------------------- row passes
// (rows.cuh: rows_pairs, rows_fold)
template <int N>
constexpr int pair_min_blocks(int threads) {
  const int regs = two_stage_r1(N) == 32 ? 128 : 64;
  return 65536 / regs / threads > 0 ? 65536 / regs / threads : 1;
}
constexpr int kPairThreads = 256;
// Modal rows at radix 16 (N = 128, 256): 80 registers and three blocks; the 64 of
// four blocks spill 380 bytes a thread (128^3, 3 read modes: 19 vs 15 us with
// events), and two blocks measured the same as three.
template <int N>
constexpr int modal_min_blocks() {
  return two_stage_r1(N) == 16 ? 3 : pair_min_blocks<N>(kPairThreads);
}
template <int N, class Op>
__global__ void __launch_bounds__(kPairThreads, modal_min_blocks<N>())
    k_rows_pairs(const __grid_constant__ Op op, float2* work, int64_t fs, int HP, int64_t nrows, int pr,
                 const float2* __restrict__ tw2) {
  rows_pairs<N, Op, kPairThreads>(op, work, fs, HP, nrows, tw2, pr);
}
template <int N, class Op>
__global__ void __launch_bounds__(kRowThreads, 2) k_rows_fold(const __grid_constant__ Op op, float2* work, int64_t fs,
                                                              int HP, const float2* __restrict__ twN,
                                                              const float2* __restrict__ twH) {
  rows_fold<N>(op, work, fs, HP, twN, twH);
}
// The source rows: 6 lines per pair, PR = 32 / T pairs, 192 threads.
constexpr int kSixThreads = 192;
// resident blocks: 96 registers hold 32 values per lane in these kernels
// without spills (three blocks against two with 138-146: source rows 8.9 vs
// 10.7 ms at 1024^3, 1.10 vs 1.31 at 512^3)
template <int N>
constexpr int six_min_blocks() {
  return two_stage_r1(N) == 32 ? 3 : 5;
}
template <int N, class Op>
__global__ void __launch_bounds__(kSixThreads, six_min_blocks<N>())
    k_rows_six(const __grid_constant__ Op op, float2* work, int64_t fs, int HP, int64_t nrows,
               const float2* __restrict__ tw2) {
  rows_pairs<N, Op, kSixThreads>(op, work, fs, HP, nrows, tw2, 32 / PairCfg<N>::T);
}

// A term in factored order (factor_terms) as a kernel parameter: the shared-
// memory offsets of the lines of f_o and f_F, and bit 31 at its group's end.
struct TermC {
  uint32_t off;  // o LS | (F LS) << 16 | end << 31
  float c;
};

// modal products: the line of p holds f_p; the line of r is overwritten by g_r.  The
// term list travels in the kernel's parameter space, so every thread reads
// a term through the uniform constant path; each thread forms two positions
// per term.  Bound by issue slots (60-70 % issued at 128^3), most of them
// addresses and loop control: in factored order a term takes one field's load
// and one multiply-add per component and a group one more of each, where f_p,
// f_q and three operations were taken for every term (six templates of 6-20
// modes at 128^3, in one graph: 1038 -> 871 us of this kernel; a 64^3 run of 10
// modes 152 -> 145 us).  Two neighbouring
// positions in one 16-byte access take a fifth fewer instructions but leave
// half the warps without work at 64^3 (21 -> 26 us) and gain nothing at 128^3.
struct ModalRowOp {
  static constexpr bool kZfac = false;
  static constexpr bool kPairs = true;
  int ni, nr, nl;
  int in_mode[kMaxModes], line_in[kMaxModes];
  int r_of_slot[kMaxModes], line_out[kMaxModes];
  int begin[kMaxModes + 1];
  TermC early;  // the counter-term, c = 0 where there is none
  TermC t[kMaxTerms];
  __device__ int nin() const { return ni; }
  __device__ int nlines() const { return nl; }
  __device__ int in_slot(int l) const { return in_mode[l]; }
  __device__ int in_line(int l) const { return line_in[l]; }
  __device__ int nout() const { return nr; }
  __device__ int out_line(int l) const { return line_out[l]; }
  __device__ int out_slot(int l) const { return r_of_slot[l]; }
  // Slots in descending r: g_r only needs f_p f_q with p <= q <= r, so once
  // g_r is formed nothing later reads f_r and it is stored over it at once.
  // (The counter-term f_0 f_2 -> g_1 reads f_2 after g_2 has replaced it;
  // that term is evaluated first, into registers.)
  template <int K>
  __device__ void combine(float2* sm, const int* pos, int LS) const {
    float2 g1_extra[K];
#pragma unroll
    for (int i = 0; i < K; ++i) g1_extra[i] = make_float2(0.f, 0.f);
    if (early.c != 0.f) {
      const int po = (int)(early.off & 0xFFFFu), qo = (int)(early.off >> 16);
#pragma unroll
      for (int i = 0; i < K; ++i) {
        const float2 fp = sm[po + pos[i]], fq = sm[qo + pos[i]];
        g1_extra[i] = make_float2(early.c * fp.x * fq.x, early.c * fp.y * fq.y);
      }
    }
    for (int s = nr - 1; s >= 0; --s) {
      float2 acc[K], h[K];
#pragma unroll
      for (int i = 0; i < K; ++i) {
        acc[i] = r_of_slot[s] == 1 ? g1_extra[i] : make_float2(0.f, 0.f);
        h[i] = make_float2(0.f, 0.f);
      }
      const int tb = begin[s], te = begin[s + 1];
#pragma unroll 4
      for (int ti = tb; ti < te; ++ti) {
        const TermC tm = t[ti];
        const int oo = (int)(tm.off & 0xFFFFu);
#pragma unroll
        for (int i = 0; i < K; ++i) {
          const float2 fo = sm[oo + pos[i]];
          h[i].x = fmaf(tm.c, fo.x, h[i].x);
          h[i].y = fmaf(tm.c, fo.y, h[i].y);
        }
        if ((tm.off >> 31) != 0u) {
          const int Fo = (int)((tm.off >> 16) & 0x7FFFu);
#pragma unroll
          for (int i = 0; i < K; ++i) {
            const float2 fF = sm[Fo + pos[i]];
            acc[i].x = fmaf(fF.x, h[i].x, acc[i].x);
            acc[i].y = fmaf(fF.y, h[i].y, acc[i].y);
            h[i] = make_float2(0.f, 0.f);
          }
        }
      }
#pragma unroll
      for (int i = 0; i < K; ++i) sm[line_out[s] * LS + pos[i]] = acc[i];
    }
  }
};

// 2LPT source (main.c:1284-1294): lines 0..5 hold d00 d01 d02 d11 d12 d22;
// the source goes to line 0, written to slot `out`.
struct SourceRowOp {
  static constexpr bool kPairs = true;
  static constexpr bool kZfac = true;  // z factors of the Hessians (1, 1, kz, 1, kz, kz^2)
  int out;
  float kF;
  const float* isinc2;
  __device__ ZFac zfac(int l) const { return ZFac{l == 2 || l == 4 ? 1 : l == 5 ? 2 : 0, kF, isinc2}; }
  __device__ int nin() const { return 6; }
  __device__ int nlines() const { return 6; }
  __device__ int in_slot(int l) const { return l; }
  __device__ int in_line(int l) const { return l; }
  __device__ int nout() const { return 1; }
  __device__ int out_line(int) const { return 0; }
  __device__ int out_slot(int) const { return out; }
  template <int K>
  __device__ void combine(float2* sm, const int* pos, int LS) const {
#pragma unroll
    for (int i = 0; i < K; ++i) {
      float2 d[6];
#pragma unroll
      for (int c = 0; c < 6; ++c) d[c] = sm[c * LS + pos[i]];
      float2 s;
      s.x = d[0].x * (d[3].x + d[5].x) + d[3].x * d[5].x - d[1].x * d[1].x - d[2].x * d[2].x - d[4].x * d[4].x;
      s.y = d[0].y * (d[3].y + d[5].y) + d[3].y * d[5].y - d[1].y * d[1].y - d[2].y * d[2].y - d[4].y * d[4].y;
      sm[pos[i]] = s;
    }
  }
};

// c2r of one field per blockIdx.y (slot = first + blockIdx.y), each with
// its z factor (ZFac type ztype[blockIdx.y]; 0 = plain c2r)
struct ZTypes {
  int t[6];
  float kF;
  const float* isinc2;
  // t[i] by selects (a dynamic index into the parameter block would copy it
  // to local memory)
  __device__ __forceinline__ int at(int i) const {
    int r = t[0];
#pragma unroll
    for (int j = 1; j < 6; ++j) r = i == j ? t[j] : r;
    return i < 6 ? r : 0;
  }
};
constexpr int kC2rThreads = 128;
template <int N>
constexpr unsigned c2r_blocks() {  // of a field's N^2 rows
  constexpr int rows = 2 * (kC2rThreads / PairCfg<N>::T);
  return (unsigned)(((int64_t)N * N + rows - 1) / rows);
}
template <int N>
constexpr size_t pair_line_smem(int threads) {  // one line buffer per T threads
  return sizeof(float2) * (size_t)(threads / PairCfg<N>::T) * PairCfg<N>::LS;
}
// Start of memory row m's row in the caller's natural order, in rows
template <int N>
__device__ __forceinline__ int64_t nat_row(int64_t m) {
  int x, y;
  row_xy(m, N, kXB, x, y);
  return (int64_t)x * N + y;
}
// NAT: the real rows go to `nat` in the caller's natural order, real
// [N][N][N], else in place of the spectra.
template <int N, bool NAT>
__global__ void __launch_bounds__(kC2rThreads, pair_min_blocks<N>(kC2rThreads))
    k_rows_c2r(float2* work, int64_t fs, int HP, int first, int64_t nrows, const float2* __restrict__ tw2, ZTypes zt,
               float* nat) {
  using C = PairCfg<N>;
  extern __shared__ float2 sm[];
  const int u = threadIdx.x / C::T, t = threadIdx.x % C::T;
  const int64_t row = 2 * ((int64_t)blockIdx.x * (kC2rThreads / C::T) + u);
  const bool act = row < nrows;
  float2* f = work + (int64_t)(first + blockIdx.y) * fs + (act ? row : 0) * HP;
  const ZFac zf{zt.at(blockIdx.y), zt.kF, zt.isinc2};
  float2 v[C::R1];
  pair_spectrum<N, true>(v, f, row + 1 < nrows ? f + HP : nullptr, t, zf, act);
  pair_fft<N, +1>(v, sm + u * C::LS, t, tw2, act);  // every lane of the line has read its rows
  if (act) {
    float* a = NAT ? nat + nat_row<N>(row) * N : reinterpret_cast<float*>(f);
#pragma unroll
    for (int i = 0; i < C::R1; ++i) a[t + C::T * i] = v[i].x;
    if (row + 1 < nrows) {
      float* b = NAT ? nat + nat_row<N>(row + 1) * N : a + 2 * HP;
#pragma unroll
      for (int i = 0; i < C::R1; ++i) b[t + C::T * i] = v[i].y;
    }
  }
}

// ----------------------------------------------------------- strided passes
#include "passes.cuh"

// ----------------------------------------------------------- read-out
// Trilinear read-out (main.c:1440-1516).  Fields: slots 0..5 of `work` as
// real rows (float, row stride 2 HP); psi2 slots hold N^3 x the 2LPT field.
struct ReadArgs {
  int N, HP;
  int64_t fs;           // field stride in floats
  float box, inv_n3, vp1, vp2;
  float nb_hi, nb_lo;  // N / Box as a two-float sum
};

// Cell index and fraction of one coordinate: u = Pos N / Box
// (main.c:1444-1446) to ~1e-7 of a cell in FP32 -- the product with a
// two-float split of N/Box -- then the cell index and the fraction with the
// reference's clamps (main.c:1452-1463).
__device__ __forceinline__ void cell_coord(const ReadArgs& a, float p, int& i, float& f) {
  const int N = a.N;
  float hi = p * a.nb_hi;
  float lo = fmaf(p, a.nb_hi, -hi) + p * a.nb_lo;
  if (!(hi >= 0.f)) {  // also catches NaN: the cell index stays inside the grid
    hi = 0.f;
    lo = 0.f;
  }
  if (hi > (float)N) {
    hi = (float)N;
    lo = 0.f;
  }
  const float fl = floorf(hi);
  i = (int)fl;
  f = (hi - fl) + lo;  // hi - fl is exact
  if (f < 0.f) {
    i -= 1;
    f += 1.f;
  } else if (f >= 1.f) {
    i += 1;
    f -= 1.f;
  }
  if (i < 0) {  // (int) truncates: u in (-1, 0) reads cell 0 with a negative fraction
    f = (float)i + f;
    i = 0;
  }
  if (i >= N) {
    f += (float)(i - (N - 1));
    i = N - 1;
  }
}

// Position and velocity of a particle at Lagrangian coordinate p from its
// ZA and 2LPT displacements d1, d2 (main.c:1486-1509): Pos += dis - 3/7
// dis2 / N^3 with the periodic wrap, Vel = dis vp1 - 3/7 dis2 / N^3 vp2.
__device__ __forceinline__ void move_particle(const ReadArgs& a, const float* p, const float* dis, const float* dis2,
                                              float* op, float* ov) {
  for (int ax = 0; ax < 3; ++ax) {
    const float d1 = dis[ax], d2 = dis2[ax] * a.inv_n3;
    float d = d1 - (3.f / 7.f) * d2;
    float x = p[ax] + d;
    if (x < 0.f) x += a.box;
    if (x >= a.box) x -= a.box;
    op[ax] = x;
    ov[ax] = d1 * a.vp1 - (3.f / 7.f) * d2 * a.vp2;
  }
}

__device__ __forceinline__ void readout_one(const ReadArgs& a, const float* __restrict__ F, float px, float py,
                                            float pz, float* op, float* ov) {
  const int N = a.N;
  float p[3] = {px, py, pz};
  int ii[3], jj[3];
  float fr[3];
  for (int d = 0; d < 3; ++d) {
    cell_coord(a, p[d], ii[d], fr[d]);
    jj[d] = (ii[d] + 1 == N) ? 0 : ii[d] + 1;
  }
  const int64_t rs = 2 * (int64_t)a.HP;
  float u = fr[0], v = fr[1], w = fr[2];
  float dis[3], dis2[3];
  if (u == 0.f && v == 0.f && w == 0.f) {
    // on a grid point (a regular lattice whose spacing Box/N is a binary
    // fraction): weights f1 = 1, f2..f8 = 0, so the 8-point sum is the one
    // corner value exactly (finite fields) and the other 7 loads are skipped
    const int64_t o = row_of(ii[0], ii[1], N, kXB) * rs + ii[2];
#pragma unroll
    for (int ax = 0; ax < 3; ++ax) {
      dis[ax] = F[ax * a.fs + o];
      dis2[ax] = F[(3 + ax) * a.fs + o];
    }
  } else {
    int64_t o000 = row_of(ii[0], ii[1], N, kXB) * rs, o010 = row_of(ii[0], jj[1], N, kXB) * rs;
    int64_t o100 = row_of(jj[0], ii[1], N, kXB) * rs, o110 = row_of(jj[0], jj[1], N, kXB) * rs;
    float f1 = (1 - u) * (1 - v) * (1 - w), f2 = (1 - u) * (1 - v) * w, f3 = (1 - u) * v * (1 - w),
          f4 = (1 - u) * v * w, f5 = u * (1 - v) * (1 - w), f6 = u * (1 - v) * w, f7 = u * v * (1 - w),
          f8 = u * v * w;
    int k0 = ii[2], k1 = jj[2];
    for (int ax = 0; ax < 3; ++ax) {
      const float* d1 = F + ax * a.fs;
      const float* d2 = F + (3 + ax) * a.fs;
      dis[ax] = d1[o000 + k0] * f1 + d1[o000 + k1] * f2 + d1[o010 + k0] * f3 + d1[o010 + k1] * f4 +
                d1[o100 + k0] * f5 + d1[o100 + k1] * f6 + d1[o110 + k0] * f7 + d1[o110 + k1] * f8;
      dis2[ax] = d2[o000 + k0] * f1 + d2[o000 + k1] * f2 + d2[o010 + k0] * f3 + d2[o010 + k1] * f4 +
                 d2[o100 + k0] * f5 + d2[o100 + k1] * f6 + d2[o110 + k0] * f7 + d2[o110 + k1] * f8;
    }
  }
  move_particle(a, p, dis, dis2, op, ov);
}

// One particle per thread.  (Measured at 1024^3 on a lattice: four
// particles per thread with 16-byte loads and stores, 79 registers and three
// blocks per SM, 27.0 vs 19.6 ms; at 128^3 the stores staged through shared
// memory as below, 51 vs 47 us: the gather's latency counts, and the barrier
// makes a block wait for its slowest warp.)
__global__ void __launch_bounds__(256, 6) k_readout(ReadArgs a, const float* __restrict__ F, const float* __restrict__ lagr, int64_t np,
                          float* pos, float* vel) {
  int64_t n = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (n >= np) return;
  float op[3], ov[3];
  readout_one(a, F, lagr[3 * n], lagr[3 * n + 1], lagr[3 * n + 2], op, ov);
  for (int d = 0; d < 3; ++d) {
    pos[3 * n + d] = op[d];
    vel[3 * n + d] = ov[d];
  }
}

// Lagrangian positions from a glass tiled tile^3 times (read_glass.c:129-214):
// Pos = glass / glass_box * (Box / tile) + t * (Box / tile) in FP64 with
// unfused operations, rounded to float.  The two products depend only on
// the glass particle and on the tile index, so k_glass_scale makes them once
// per call (3 nglass + tile doubles) and a particle costs one FP64 add per
// axis (GB300's FP64 rate is a small fraction of its FP32 rate).
__global__ void k_glass_scale(const float* __restrict__ glass, int64_t nglass, double glass_box, int tile,
                              double box_over_tile, double* __restrict__ gs) {
  const int64_t n = 3 * nglass + tile;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    gs[i] = i < 3 * nglass ? __dmul_rn(__ddiv_rn((double)glass[i], glass_box), box_over_tile)
                           : __dmul_rn((double)(i - 3 * nglass), box_over_tile);
}

// Particles n0 <= n < n1 (indices of the whole tiled set, particle order of
// read_glass.c:181-214: tile index outer, glass index inner).  A block's
// positions and velocities go through shared memory and out as 16-byte
// stores of whole lines: the outputs may be page-locked host memory written
// over the host link (4-byte stores 12 bytes apart: 37 GB/s at 1536^3; whole
// lines 41-47 GB/s, the rate the copy engines reach on the same link).
constexpr int kReadoutThreads = 256;
__global__ void __launch_bounds__(kReadoutThreads) k_readout_glass(ReadArgs a, const float* __restrict__ F,
                                                                   const double* __restrict__ gs, int64_t nglass,
                                                                   int tile, float* pos, float* vel, int* ids,
                                                                   int64_t n0, int64_t n1) {
  __shared__ float4 sp4[3 * kReadoutThreads / 4], sv4[3 * kReadoutThreads / 4];
  float* sp = (float*)sp4;
  float* sv = (float*)sv4;
  const int64_t base = n0 + (int64_t)blockIdx.x * kReadoutThreads;
  const int64_t n = base + threadIdx.x;
  if (n < n1) {
    int64_t gi = n % nglass, t = n / nglass;
    int ti = (int)(t / ((int64_t)tile * tile)), tj = (int)((t / tile) % tile), tk = (int)(t % tile);
    int tt[3] = {ti, tj, tk};
    const double* toff = gs + 3 * nglass;
    float lp[3];
    for (int d = 0; d < 3; ++d) lp[d] = (float)__dadd_rn(gs[3 * gi + d], toff[tt[d]]);
    float op[3], ov[3];
    readout_one(a, F, lp[0], lp[1], lp[2], op, ov);
    for (int d = 0; d < 3; ++d) {
      sp[3 * threadIdx.x + d] = op[d];
      sv[3 * threadIdx.x + d] = ov[d];
    }
    if (ids) ids[n] = (int)(n + 1);
  }
  __syncthreads();
  const int cnt = (int)min((int64_t)kReadoutThreads, n1 - base);
  float* po = pos + 3 * base;
  float* vo = vel + 3 * base;
  if (cnt == kReadoutThreads && ((reinterpret_cast<uintptr_t>(po) | reinterpret_cast<uintptr_t>(vo)) & 15) == 0) {
    for (int i = threadIdx.x; i < 3 * kReadoutThreads / 4; i += kReadoutThreads) {
      reinterpret_cast<float4*>(po)[i] = sp4[i];
      reinterpret_cast<float4*>(vo)[i] = sv4[i];
    }
  } else {
    for (int i = threadIdx.x; i < 3 * cnt; i += kReadoutThreads) {
      po[i] = sp[i];
      vo[i] = sv[i];
    }
  }
}

// ----------------------------------------------------------- lattice read-out
// Particles of the regular g^3 lattice glass (per-axis glass coordinate
// (float)(i * glass_box / g), the particle order of read_glass.c:181-214)
// tiled tile^3 times.  k_lattice_axis makes the Lagrangian coordinate of
// every lattice index of one axis with the operations of the general glass
// path (k_glass_scale + k_readout_glass) and flags any that is not exactly
// on its own grid point by the reference's own FP64 cell coordinate u = Pos
// / Box * Nmesh (main.c:1444-1446): u must equal the index.  When none is
// flagged and g tile = Nmesh, every particle sits on a grid point and reads
// just the grid value under it (the weights of the other seven corners are
// zero), so the read-out can be fused into the displacement rows:
// k_rows_lattice.  (The FP32 read-out's two-float coordinate can leave a
// fraction of ~1e-12 at such a point, which weights the neighbour by as
// much; the fused read-out takes the grid value, as the FP64 reference
// does.)
__global__ void k_lattice_axis(int N, double box, int g, double gsp, double glass_box, double bot, float* lpa,
                               int* off_grid) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= N) return;
  const int gi = i % g, ti = i / g;
  const float gc = (float)__dmul_rn((double)gi, gsp);
  const float lp = (float)__dadd_rn(__dmul_rn(__ddiv_rn((double)gc, glass_box), bot), __dmul_rn((double)ti, bot));
  lpa[i] = lp;
  const double u = __dmul_rn(__ddiv_rn((double)lp, box), (double)N);
  if (u != (double)i) atomicOr(off_grid, 1);
}

// The lattice glass itself (3 g^3 floats), for the general read-out.
__global__ void k_lattice_glass(int g, double gsp, float* glass) {
  const int64_t n = (int64_t)g * g * g;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t ix = i / ((int64_t)g * g), iy = (i / g) % g, iz = i % g;
    glass[3 * i] = (float)__dmul_rn((double)ix, gsp);
    glass[3 * i + 1] = (float)__dmul_rn((double)iy, gsp);
    glass[3 * i + 2] = (float)__dmul_rn((double)iz, gsp);
  }
}

// The six displacement rows of PR = 32 / T pairs of memory rows (c2r with the
// z factors, as k_rows_c2r; one line per T threads), then the particles on the
// rows' grid points: Pos / Vel from the grid values (readout_one's on-grid
// branch, main.c:1486-1509) and IDs, written at their tiled-glass particle
// index.  A warp's 32 consecutive grid points are 32 consecutive particles
// unless a tile edge falls between them: their Pos and Vel go through shared
// memory and out as whole lines (stores 12 bytes apart write every sector
// three times).  Rows [row0, row0 + nrows) of the x-blocked order, row0 even.
template <int N>
struct LatticeCfg {
  static constexpr int PR = 32 / PairCfg<N>::T;
  static constexpr int LINES = 6 * PR;
  static constexpr size_t SMEM = sizeof(float2) * (size_t)LINES * PairCfg<N>::LS + sizeof(float) * kSixThreads * 6;
};
template <int N>
__global__ void __launch_bounds__(kSixThreads, six_min_blocks<N>())
    k_rows_lattice(const float2* __restrict__ work, int64_t fs, int HP, const float2* __restrict__ tw2, ZTypes zt,
                   ReadArgs ra, int g, int tile, const float* __restrict__ lpa, float* pos, float* vel, int* ids,
                   int64_t row0, int64_t nrows) {
  using C = PairCfg<N>;
  using L = LatticeCfg<N>;
  static_assert(kXB % 2 == 0, "the rows of a pair are (x, y) and (x + 1, y)");
  extern __shared__ float2 sm[];  // [PR][6][LS], then the warps' particle staging
  const int64_t rbase = row0 + (int64_t)blockIdx.x * (2 * L::PR), rend = row0 + nrows;
  {
    const int u = threadIdx.x / C::T, t = threadIdx.x % C::T;
    const int pr = u / 6, c = u - 6 * pr;
    const int64_t row = rbase + 2 * pr;
    const bool act = row < rend;
    const ZFac zf{zt.at(c), zt.kF, zt.isinc2};
    const float2* X = work + (int64_t)c * fs + (act ? row : 0) * HP;
    float2* ln = sm + u * C::LS;
    float2 v[C::R1];
    pair_spectrum<N, true>(v, X, row + 1 < rend ? X + HP : nullptr, t, zf, act);
    pair_fft<N, +1>(v, ln, t, tw2, act);
    if (act) {
#pragma unroll
      for (int i = 0; i < C::R1; ++i) ln[t + C::T * i] = v[i];
    }
  }
  __syncthreads();
  // a warp takes 32 consecutive grid points of a row pair at a time (N = 16:
  // of two pairs)
  const int64_t g3 = (int64_t)g * g * g;
  const int lane = threadIdx.x & 31;
  float* stp = reinterpret_cast<float*>(sm + L::LINES * C::LS) + (threadIdx.x >> 5) * 192;
  float* stv = stp + 96;
  for (int q0 = threadIdx.x - lane; q0 < L::PR * N; q0 += kSixThreads) {  // uniform over the warp
    const int q = q0 + lane, pr = q / N, z = q - pr * N;
    const int64_t row = rbase + 2 * pr;
    const bool live = q < L::PR * N && row < rend;
    const int tk = z / g, gk = z - tk * g;
    int x = 0, y = 0;
    float2 d2[6];
    if (live) {
      row_xy(row, N, kXB, x, y);
#pragma unroll
      for (int c = 0; c < 6; ++c) d2[c] = sm[(pr * 6 + c) * C::LS + z];
    }
    const float py = lpa[y], pz = lpa[z];
    const int tj = y / g, gj = y - tj * g;
    const bool line = N >= 32 && __all_sync(0xffffffffu, live && gk >= lane);  // one tile cell along z
#pragma unroll
    for (int s = 0; s < 2; ++s) {
      const bool on = live && row + s < rend;
      float op[3], ov[3];
      const int ti = (x + s) / g, gi = x + s - ti * g;
      const int64_t n = (((int64_t)ti * tile + tj) * tile + tk) * g3 + ((int64_t)gi * g + gj) * g + gk;
      if (on) {
        float d[6];
#pragma unroll
        for (int c = 0; c < 6; ++c) d[c] = s ? d2[c].y : d2[c].x;
        const float p[3] = {lpa[x + s], py, pz};
        move_particle(ra, p, d, d + 3, op, ov);
        if (ids) ids[n] = (int)(n + 1);
      }
      if (line && __all_sync(0xffffffffu, on)) {
        __syncwarp();
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          stp[3 * lane + c] = op[c];
          stv[3 * lane + c] = ov[c];
        }
        __syncwarp();
        float* po = pos + 3 * (n - lane);
        float* vo = vel + 3 * (n - lane);
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          po[lane + 32 * c] = stp[lane + 32 * c];
          vo[lane + 32 * c] = stv[lane + 32 * c];
        }
      } else if (on) {
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          pos[3 * n + c] = op[c];
          vel[3 * n + c] = ov[c];
        }
      }
    }
  }
}

// ----------------------------------------------------------- host side
// Launch a strided pass, one block per item.
template <int N, int AXIS, int SIGN, class Op>
static int run_pass(Plan* p, const Op& op, int64_t nitems, cudaStream_t st, const char* name) {
  using C = TileCfg<N>;
  auto kern = k_pass<N, AXIS, SIGN, Op>;
  AAR_CUDA_TRY(p, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)C::SMEM));
  if (nitems < 1) return AAR_OK;
  if (nitems > 0x7fffffff) return set_err(p, std::string(name) + ": too many work items"), AAR_ERR_ARG;
  {
    ProfScope ps_(p, name, st);
    kern<<<(unsigned)nitems, C::THREADS, C::SMEM, st>>>(op, p->d_tw2);
  }
  AAR_CUDA_TRY(p, cudaGetLastError());
  p->last_launches += 1;
  return AAR_OK;
}

template <int N>
struct Launch {
  static constexpr int64_t kTiles = TileCfg<N>::TILES;
  static int64_t fstride(Plan* p) { return (int64_t)N * N * p->HP; }
  static unsigned group(Plan* p) { return (unsigned)std::min<int64_t>(p->xpass_group, kTiles); }
  static constexpr size_t pair_smem(int lines) { return sizeof(float2) * (size_t)lines * PairCfg<N>::LS; }
  static constexpr size_t kSixSmem = pair_smem(6 * (32 / PairCfg<N>::T));
  // dynamic shared memory of k_rows_pairs: several row pairs up to kPairSmem,
  // one whatever its lines
  static constexpr size_t kPairSmem = 100 * 1024;
  static constexpr size_t kPairSmemMax = std::max(kPairSmem, pair_smem(N < 1024 ? kMaxModes : 8));
  static int configure(Plan* p) {
    AAR_CUDA_TRY(p, cudaFuncSetAttribute(k_rows_pairs<N, ModalRowOp>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)kPairSmemMax));
    AAR_CUDA_TRY(p, cudaFuncSetAttribute(k_rows_six<N, SourceRowOp>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)kSixSmem));
    if constexpr (N == 1024)
      AAR_CUDA_TRY(p, cudaFuncSetAttribute(k_rows_fold<N, ModalRowOp>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           (int)fold_smem(kMaxModes)));
    return AAR_OK;
  }
  static constexpr size_t fold_smem(int nlines) {
    if constexpr (N == 1024) return sizeof(float2) * ((size_t)nlines * FoldCfg<N>::LS + FoldCfg<N>::LT);
    else return 0;
  }
  static Slots slots(const int* s, int n) {
    Slots r{};
    for (int i = 0; i < n; ++i) r.s[i] = s[i];
    return r;
  }
  // transform of nf fields of `base` along AXIS in place
  template <int AXIS, int SIGN>
  static int axis_pass(Plan* p, float2* base, int nf, const Slots& sl, cudaStream_t st, const char* name) {
    return run_pass<N, AXIS, SIGN>(p, AxisOp<N>{base, fstride(p), sl}, nf * kTiles, st, name);
  }
  static const TermList& terms(Plan* p) { return *(const TermList*)p->host_terms.data(); }
  // the generic row kernel's term list as a kernel parameter, for lines LS
  // float2 apart
  static ModalRowOp row_op(Plan* p, int LS) {
    static_assert(sizeof(ModalRowOp) < 32000, "kernel parameter space");
    const TermList& tl = terms(p);
    const Term* ft = (const Term*)(p->host_terms.data() + sizeof(TermList));
    static_assert(kMaxModes * PairCfg<512>::LS < 0x8000 && 8 * PairCfg<1024>::LS < 0x8000 &&
                  kMaxModes * FoldCfg<1024>::LS < 0x8000, "line offsets fit 15 bits");
    ModalRowOp op;
    op.ni = tl.nin;
    op.nr = tl.nr;
    op.nl = tl.nlines;
    for (int i = 0; i < tl.nin; ++i) op.in_mode[i] = tl.in_mode[i], op.line_in[i] = tl.line[tl.in_mode[i]];
    for (int i = 0; i < tl.nr; ++i) op.r_of_slot[i] = tl.r_of_slot[i], op.line_out[i] = tl.line[tl.r_of_slot[i]];
    op.early = {0u, 0.f};
    const TermF* tf = (const TermF*)(ft + tl.nterms);
    auto term = [&](int o, int F, bool end, float c) {
      return TermC{(uint32_t)(tl.line[o] * LS) | ((uint32_t)(tl.line[F] * LS) << 16) | (end ? 1u << 31 : 0u), c};
    };
    int n = 0;
    for (int sl = 0; sl < tl.nr; ++sl) {
      op.begin[sl] = n;
      for (int i = tl.begin[sl]; i < tl.begin[sl + 1]; ++i) {
        const TermF& f = tf[i];
        if (f.t >= 0) op.t[n++] = term(f.o, f.F, f.end, ft[f.t].c);
        else op.early = term(ft[~f.t].p, ft[~f.t].q, false, ft[~f.t].c);
      }
    }
    op.begin[tl.nr] = n;
    return op;
  }
  static int modal_rows(Plan* p, float2* work, int64_t fs, int64_t nrows, cudaStream_t st) {
    const TermList& tl = terms(p);
    {
      ProfScope ps_(p, "modal_rows", st);
      if (rows_use_pairs(N, tl.nlines)) {
        // as many row pairs as give every T threads of a block a line, while
        // two blocks' lines fit an SM
        constexpr int slots = kPairThreads / PairCfg<N>::T;
        int pr = std::max(1, slots / std::max(tl.nin, tl.nr));
        while (pr > 1 && pair_smem(pr * tl.nlines) > kPairSmem) --pr;
        k_rows_pairs<N, ModalRowOp><<<(unsigned)((nrows + 2 * pr - 1) / (2 * pr)), kPairThreads,
                                      pair_smem(pr * tl.nlines), st>>>(row_op(p, PairCfg<N>::LS), work, fs, p->HP,
                                                                       nrows, pr, p->d_tw2);
      } else if constexpr (N == 1024) {
        k_rows_fold<N, ModalRowOp><<<(unsigned)nrows, kRowThreads, fold_smem(tl.nlines), st>>>(
            row_op(p, FoldCfg<N>::LS), work, fs, p->HP, p->d_twN, p->d_twH);
      }
    }
    AAR_CUDA_TRY(p, cudaGetLastError());
    p->last_launches += 1;
    return AAR_OK;
  }
  static int modal(Plan* p, const ModalArgs& a, cudaStream_t st) {
    const int64_t fs = fstride(p);
    const TermList& tl = terms(p);
    const Slots in = slots(tl.in_mode, tl.nin), out = slots(tl.r_of_slot, tl.nr);
    XinvOp<N> xo{p->d_phik, p->d_work, fs, tl.nin, in, group(p), 0, p->M, p->d_qcube};
    int rc = run_pass<N, 0, +1>(p, xo, kTiles * tl.nin, st, "modal_xinv");
    if (rc) return rc;
    if ((rc = axis_pass<1, +1>(p, p->d_work, tl.nin, in, st, "modal_ypass_inv"))) return rc;
    if ((rc = p->jit ? jit_modal_rows(p, p->d_work, fs, st) : modal_rows(p, p->d_work, fs, (int64_t)N * N, st))) return rc;
    if ((rc = axis_pass<1, -1>(p, p->d_work, tl.nr, out, st, "modal_ypass_fwd"))) return rc;
    const float fnl_n3 = (float)(p->prm.fnl / ((double)N * N * N));
    // one slot (r = 3): 2.53 ms against k_xacc's 4.39 at 1024^3, whose registers
    // leave one block per SM; with 16 values per lane and fewer k_xacc is as fast
    // (0.0122 against 0.0132 ms at 128^3)
    if constexpr (TileCfg<N>::R1 == 32) {
      if (tl.nr == 1) {
        const int r = out.s[0];
        auto add = [&](auto one) {
          const XaddOp<N, decltype(one)::value> xo1{a.g, p->d_phik, p->d_work + r * fs, p->d_rtab + r * p->nsq, fnl_n3};
          return run_pass<N, 0, -1>(p, xo1, kTiles, st, "modal_xacc");
        };
        return r == 3 ? add(std::true_type{}) : add(std::false_type{});
      }
    }
    Slots order{};  // r = 3 last
    int nw = 0;
    for (int i = 0; i < tl.nr; ++i)
      if (out.s[i] != 3) order.s[nw++] = out.s[i];
    if (nw < tl.nr) order.s[nw] = 3;
    const XaccArgs<N> xa{a.g, p->d_phik, p->d_work, fs, tl.nr, nw, order, p->M, p->d_qcube, p->d_rtab, fnl_n3, nullptr, nullptr};
    AAR_CUDA_TRY(p, cudaFuncSetAttribute(k_xacc<N, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)XaccCfg<N>::SMEM));
    {
      ProfScope ps_(p, "modal_xacc", st);
      k_xacc<N, false><<<(unsigned)kTiles, TileCfg<N>::THREADS, XaccCfg<N>::SMEM, st>>>(xa, p->d_tw2);
    }
    AAR_CUDA_TRY(p, cudaGetLastError());
    p->last_launches += 1;
    return AAR_OK;
  }
  // 2LPT (main.c:1180-1431).  Work slots: Hessians d_ab in 0..5 (00 01 02 11
  // 12 22) via x outputs P = -kF^2 kx^2 phi_T -> 0, Q = -kF^2 kx phi_T -> 8, R =
  // -kF^2 phi_T -> 6 (phi_T = T/(D Beta) phi) and the y fan-out (xy, yz: ky;
  // yy: ky^2); the source rows apply the z factors (xz, yz: kz; zz: kz^2) and
  // write S to 6; psi1 (0..2) and psi2 (3..5) likewise from x outputs in 0, 8
  // (psi1) and 3, 7 (psi2).
  static int lpt(Plan* p, const LptArgs& a, cudaStream_t st, bool rows = true) {
    const int64_t fs = fstride(p);
    const float kF = a.m.g.kF;
    int rc;
    {
      LptXOp<N, 0> ho{p->d_phik, nullptr, p->d_work, fs, {0, 8, 6, 0}, group(p), kF, a.isinc2, p->d_tcube, p->d_twb};
      if ((rc = run_pass<N, 0, +1>(p, ho, kTiles * 3, st, "lpt_xinv_hess"))) return rc;
      YFanOp<N> yf{p->d_work, fs, {0, 8, 8, 6, 6, 6}, {0, 1, 2, 3, 4, 5}, {0, 1, 0, 2, 1, 0}, 1, kF, a.isinc2};
      if ((rc = run_pass<N, 1, +1>(p, yf, kTiles * 6, st, "lpt_ypass_inv_hess"))) return rc;
    }
    const SourceRowOp op{6, a.m.g.kF, a.isinc2};
    {
      ProfScope ps_(p, "lpt_rows_source", st);
      constexpr int rows = 2 * (32 / PairCfg<N>::T);  // of a block
      k_rows_six<N, SourceRowOp><<<(unsigned)(((int64_t)N * N + rows - 1) / rows), kSixThreads, kSixSmem, st>>>(
          op, p->d_work, fs, p->HP, (int64_t)N * N, p->d_tw2);
    }
    AAR_CUDA_TRY(p, cudaGetLastError());
    p->last_launches += 1;
    if ((rc = axis_pass<1, -1>(p, p->d_work, 1, Slots{{6}}, st, "lpt_ypass_fwd_source"))) return rc;
    // forward x of the source in place with -1/k^2, then the displacement x passes
    {
      XfwdInvK2Op<N> xs{p->d_work + 6 * fs, kF};
      if ((rc = run_pass<N, 0, -1>(p, xs, kTiles, st, "lpt_xfwd_source"))) return rc;
    }
    {
      LptXOp<N, 1> mo{p->d_phik, p->d_work + 6 * fs, p->d_work, fs, {0, 8, 3, 7}, group(p), kF, a.isinc2, p->d_tcube, p->d_twb};
      if ((rc = run_pass<N, 0, +1>(p, mo, kTiles * 4, st, "lpt_xpsi"))) return rc;
      YFanOp<N> yf{p->d_work, fs, {0, 8, 8, 3, 7, 7}, {0, 1, 2, 3, 4, 5}, {3, 4, 3, 3, 4, 3}, 1, kF, a.isinc2};
      if ((rc = run_pass<N, 1, +1>(p, yf, kTiles * 6, st, "lpt_ypass_inv_disp"))) return rc;
    }
    // the displacement rows: here, or fused with the lattice read-out
    // (fused_rows_lattice), which leaves no real fields behind
    p->disp_real = rows;
    if (!rows) return AAR_OK;
    const ZTypes zt{{3, 3, 4, 3, 3, 4}, a.m.g.kF, a.isinc2};
    {
      ProfScope ps_(p, "lpt_rows_c2r", st);
      k_rows_c2r<N, false><<<dim3(c2r_blocks<N>(), 6), kC2rThreads, pair_line_smem<N>(kC2rThreads), st>>>(
          p->d_work, fs, p->HP, 0, (int64_t)N * N, p->d_tw2, zt, nullptr);
    }
    AAR_CUDA_TRY(p, cudaGetLastError());
    p->last_launches += 1;
    return AAR_OK;
  }
};

template <class F>
static int dispatch_n(int N, F&& f) {
  switch (N) {
    case 16: return f(std::integral_constant<int, 16>{});
    case 32: return f(std::integral_constant<int, 32>{});
    case 64: return f(std::integral_constant<int, 64>{});
    case 128: return f(std::integral_constant<int, 128>{});
    case 256: return f(std::integral_constant<int, 256>{});
    case 512: return f(std::integral_constant<int, 512>{});
    case 1024: return f(std::integral_constant<int, 1024>{});
    default: return AAR_ERR_ARG;
  }
}

int fused_tile_r1(int N) {
  int r1 = 0;
  dispatch_n(N, [&](auto nc) { return r1 = TileCfg<decltype(nc)::value>::R1, AAR_OK; });
  return r1;
}

ModalArgs modal_args(Plan* p) {
  ModalArgs a;
  a.g = p->grid;
  a.M = p->M;
  return a;
}

// The regrouped term list by output slot: sorted triples p <= q <= r with
// alpha != 0 contribute a f_p f_q to g_r (main.c:833-867); the
// counter-terms of main.c:1045-1050 add -a012 t012 f_0 f_1 to g_2 and
// +a012 t012 f_0 f_2 to g_1.  The second one sits in the list of r = 2 (its
// target r stays 1): the row kernels form the slots in descending r and g_2
// replaces f_2 in place, so f_0 f_2 is taken before that.
std::vector<std::vector<Term>> regrouped_terms(const std::vector<double>& alpha, int M) {
  auto A = [&](int i, int j, int k) { return alpha[((size_t)i * M + j) * M + k]; };
  std::vector<std::vector<Term>> by_r(M);
  for (int i = 0; i < M; ++i)
    for (int j = i; j < M; ++j)
      for (int k = j; k < M; ++k)
        if (A(i, j, k) != 0) by_r[k].push_back(Term{i, j, k, (float)A(i, j, k)});
  if (M > 2 && A(0, 1, 2) != 0) {
    double t012 = -A(1, 1, 1) / A(0, 1, 2);
    double c = A(0, 1, 2) * t012;
    by_r[2].push_back(Term{0, 1, 2, (float)(-c)});
    by_r[2].push_back(Term{0, 2, 1, (float)(c)});
    if (by_r[1].empty()) by_r[1].push_back(Term{0, 0, 1, 0.f});  // keep a slot for r = 1
  }
  return by_r;
}

// Split of the active r over nparts cooperating plans, balanced by the
// number of product terms each g_r takes: the r in decreasing term count
// (ties: lower r first) each go to the part with the fewest terms so far
// (ties: lower part).  part_of_r[r] = -1 for an r without terms.
std::vector<int> modal_partition(const std::vector<std::vector<Term>>& by_r, int nparts) {
  const int M = (int)by_r.size();
  std::vector<int> cnt(M, 0), part(M, -1);
  for (const auto& lst : by_r)
    for (const Term& t : lst) cnt[t.r] += 1;
  std::vector<int> order;
  for (int r = 0; r < M; ++r)
    if (!by_r[r].empty() || cnt[r] > 0) order.push_back(r);
  std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return cnt[a] > cnt[b]; });
  std::vector<long> load(std::max(nparts, 1), 0);
  for (int r : order) {
    int best = 0;
    for (int q = 1; q < nparts; ++q)
      if (load[q] < load[best]) best = q;
    part[r] = best;
    load[best] += cnt[r];
  }
  return part;
}

// The terms `rem` of one target in factored order: greedily, the field that
// occurs in most remaining terms is taken out, g_r += f_F (sum_t c_t f_o), so a
// term costs one multiply-add and a group one more (at 20 modes 212 operations
// for the 134 terms instead of 268).
void factor_terms(const Term* t, std::vector<int> rem, int M, std::vector<TermF>& out) {
  while (!rem.empty()) {
    std::vector<int> cnt(M, 0), keep;
    for (int i : rem) {
      cnt[t[i].p] += 1;
      if (t[i].q != t[i].p) cnt[t[i].q] += 1;
    }
    const int F = (int)(std::max_element(cnt.begin(), cnt.end()) - cnt.begin());
    for (int i : rem) {
      if (t[i].p != F && t[i].q != F) keep.push_back(i);
      else out.push_back({i, t[i].p == F ? t[i].q : t[i].p, F, 0});
    }
    out.back().end = 1;
    rem.swap(keep);
  }
}

// The plan's term list: the regrouped terms, or
// with a modal partition only the slots of the plan's part.  A split keeps
// the counter-term f_0 f_2 -> g_1 with the part of r = 1: as a term read
// before g_2 replaces f_2 when r = 2 is in the same part, else as an
// ordinary term of r = 1 (f_2 is never replaced in that part).
static int build_terms(Plan* p) {
  int M = p->M;
  std::vector<std::vector<Term>> by_r = regrouped_terms(p->alpha, M);
  if (p->modal_nparts > 1) {
    const std::vector<int> part = modal_partition(by_r, p->modal_nparts);
    const int me = p->modal_part;
    std::vector<std::vector<Term>> mine(M);
    for (int r = 0; r < M; ++r)
      for (const Term& t : by_r[r]) {
        if (part[t.r] != me) continue;
        if (t.r != r && part[r] != me) mine[t.r].push_back(t);  // counter-term moves to its own slot
        else mine[r].push_back(t);
      }
    by_r.swap(mine);
  }
  TermList tl{};
  std::vector<Term> flat;
  int nr = 0;
  for (int r = 0; r < M; ++r) {
    if (by_r[r].empty()) continue;
    tl.r_of_slot[nr] = r;
    tl.begin[nr] = (int)flat.size();
    for (auto& t : by_r[r]) flat.push_back(t);
    ++nr;
  }
  tl.begin[nr] = (int)flat.size();
  tl.nr = nr;
  tl.nterms = (int)flat.size();
  bool read[kMaxModes] = {}, active[kMaxModes] = {};
  for (const Term& t : flat) read[t.p] = read[t.q] = true;
  for (int i = 0; i < nr; ++i) active[tl.r_of_slot[i]] = true;
  for (int m = 0; m < M; ++m) {
    if (read[m]) tl.in_mode[tl.nin++] = m;
    tl.line[m] = read[m] || active[m] ? tl.nlines++ : -1;
  }
  if (tl.nterms > kMaxTerms) return set_err(p, "too many alpha terms"), AAR_ERR_ARG;
  p->host_terms.assign((const char*)&tl, (const char*)&tl + sizeof(tl));
  p->host_terms.insert(p->host_terms.end(), (const char*)flat.data(), (const char*)(flat.data() + flat.size()));
  // the generic row kernel's order: a slot's own terms factored, then the
  // counter-term of g_1 among those of r = 2, as ~index
  std::vector<TermF> fac;
  for (int i = 0; i < nr; ++i) {
    std::vector<int> own;
    for (int t = tl.begin[i]; t < tl.begin[i + 1]; ++t)
      if (flat[t].r == tl.r_of_slot[i]) own.push_back(t);
    factor_terms(flat.data(), own, M, fac);
    for (int t = tl.begin[i]; t < tl.begin[i + 1]; ++t)
      if (flat[t].r != tl.r_of_slot[i]) fac.push_back({~t, 0, 0, 0});
  }
  p->host_terms.insert(p->host_terms.end(), (const char*)fac.data(), (const char*)(fac.data() + fac.size()));
  p->nterms = tl.nterms;
  p->nr_active = nr;
  p->chain_stale = true;
  return AAR_OK;
}

// The filter cube of the modal passes: the plan's per-|k|^2 filters
// (mode_tables: FP64 formulas rounded once to float) over 0 <= |kx|, |ky| <=
// N/2 and 0 <= kz <= N/2, zero on the cut and at k = 0 (keep_cell depends on
// |k_a| only), in the order of CubeMap (passes.cuh), p the mode.  Every mode has its
// plane, read by a term or not: the products' gradients take them all, and the
// cube keeps its address while the mode count does.
__global__ void __launch_bounds__(256) k_qcube(Grid g, int M, const float* __restrict__ qtab, int64_t nsq,
                                               float* __restrict__ q) {
  const CubeMap cm{g.N / 2 + 1, M};
  const int64_t per = (int64_t)cm.K * cm.K * cm.K;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < per; i += (int64_t)gridDim.x * blockDim.x) {
    int ax, ay, kz;
    cm.cell(i, ax, ay, kz);
    const int n2 = ax * ax + ay * ay + kz * kz;
    const bool on = n2 != 0 && keep_cell(g, ax, ay, kz);
    for (int c = 0; c < M; ++c) q[cm.at(c, ay, kz, ax)] = on ? __ldg(qtab + (int64_t)c * nsq + n2) : 0.f;
  }
}

int qcube_build(Plan* p) {
  if (!p->have_tables || (!p->qcube_stale && p->d_qcube)) return AAR_OK;  // no tables yet: nothing reads filters
  const int64_t K = p->N / 2 + 1, per = K * K * K;
  if (!p->d_qcube || p->qcube_m != p->M) {
    if (p->d_qcube) {
      AAR_CUDA_TRY(p, cudaDeviceSynchronize());
      cudaFree(p->d_qcube), p->used_bytes -= sizeof(float) * (size_t)per * p->qcube_m;
    }
    p->d_qcube = nullptr;
    p->qcube_m = 0;
    int rc = plan_alloc(p, (void**)&p->d_qcube, sizeof(float) * (size_t)per * p->M);
    if (rc) return rc;
    p->qcube_m = p->M;
  }
  k_qcube<<<(unsigned)(p->num_sms * 8), 256>>>(p->grid, p->M, p->d_qtab, p->nsq, p->d_qcube);
  AAR_CUDA_TRY(p, cudaGetLastError());
  // made on the legacy stream once per table set; runs on the caller's
  // streams read it afterwards
  AAR_CUDA_TRY(p, cudaDeviceSynchronize());
  p->qcube_stale = false;
  return AAR_OK;
}

// The transfer cube of the 2LPT x passes: T/(D Beta) in the filter cube's
// layout, no cut.  It takes an eighth of a field
// that a caller's memory limit does not know of, so plans with a limit, and
// those whose device has no room, read the per-|n|^2 table in its place.
__global__ void __launch_bounds__(256) k_tcube(int K, const float* __restrict__ twb, float* __restrict__ q) {
  const CubeMap cm{K, 1};
  const int64_t per = (int64_t)K * K * K;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < per; i += (int64_t)gridDim.x * blockDim.x) {
    int ax, ay, kz;
    cm.cell(i, ax, ay, kz);
    q[cm.at(0, ay, kz, ax)] = __ldg(twb + ax * ax + ay * ay + kz * kz);
  }
}

int tcube_build(Plan* p) {
  if (!p->tcube_stale || !p->have_transfer) return AAR_OK;
  const int64_t K = p->N / 2 + 1, per = K * K * K;
  p->tcube_stale = false;
  if (p->prm.mem_limit_bytes > 0) return AAR_OK;
  if (!p->d_tcube && plan_alloc(p, (void**)&p->d_tcube, sizeof(float) * (size_t)per)) return AAR_OK;
  k_tcube<<<(unsigned)(p->num_sms * 8), 256>>>((int)K, p->d_twb, p->d_tcube);
  AAR_CUDA_TRY(p, cudaGetLastError());
  AAR_CUDA_TRY(p, cudaDeviceSynchronize());  // as qcube_build
  return AAR_OK;
}

int build_term_list(Plan* p) {
  if (p->M > kMaxModes) return set_err(p, "N_modes above 32 is not supported"), AAR_ERR_ARG;
  return build_terms(p);
}

int fused_prepare(Plan* p) {
  if (p->M > kMaxModes) return set_err(p, "N_modes above 32 is not supported"), AAR_ERR_ARG;
  int rc = build_terms(p);
  if (rc) return rc;
  if ((rc = dispatch_n(p->N, [&](auto nc) {
         return Launch<decltype(nc)::value>::configure(p);
       })))
    return rc;
  return jit_prepare(p);
}

// The plan's modal row kernel (NVRTC or generic) on nrows rows of caller
// fields laid out with field stride nrows * HP: a harness that profiles the
// row kernel on a few thousand rows without full-size fields.
int profile_modal_rows(Plan* p, float2* work, int64_t nrows, cudaStream_t st) {
  if (nrows < 1 || nrows > (int64_t)p->N * p->N) return set_err(p, "profile rows: 1 <= nrows <= N^2"), AAR_ERR_ARG;
  if (p->nr_active == 0) return set_err(p, "profile rows: no modal terms"), AAR_ERR_STATE;
  const int64_t fs = nrows * p->HP;
  if (p->jit) return jit_modal_rows(p, work, fs, st, nrows);
  return dispatch_n(p->N, [&](auto nc) { return Launch<decltype(nc)::value>::modal_rows(p, work, fs, nrows, st); });
}

int fused_modal(Plan* p, cudaStream_t st) {
  ModalArgs a = modal_args(p);
  if (p->nr_active == 0 || p->prm.fnl == 0) return AAR_OK;  // no non-Gaussian term at all
  return dispatch_n(p->N, [&](auto nc) { return Launch<decltype(nc)::value>::modal(p, a, st); });
}

LptArgs lpt_args(Plan* p) {
  LptArgs a;
  a.m = modal_args(p);
  a.twb = p->d_twb;
  a.sinc = p->d_sinc;
  a.isinc2 = p->d_isinc2;
  return a;
}

int fused_lpt(Plan* p, cudaStream_t st, bool rows) {
  LptArgs a = lpt_args(p);
  return dispatch_n(p->N, [&](auto nc) { return Launch<decltype(nc)::value>::lpt(p, a, st, rows); });
}

static ReadArgs read_args(Plan* p) {
  ReadArgs a;
  a.N = p->N;
  a.HP = p->HP;
  a.fs = 2 * (int64_t)p->N * p->N * p->HP;
  a.box = (float)p->prm.box;
  unsigned int n3 = (unsigned int)p->N * (unsigned int)p->N * (unsigned int)p->N;
  a.inv_n3 = (float)(1.0 / (double)(float)n3);
  a.vp1 = (float)p->vel_prefac;
  a.vp2 = (float)p->vel_prefac2;
  const double nb = (double)p->N / p->prm.box;
  a.nb_hi = (float)nb;
  a.nb_lo = (float)(nb - (double)a.nb_hi);
  return a;
}

int fused_readout(Plan* p, const float* d_lagr, int64_t npart, float* d_pos, float* d_vel, cudaStream_t st) {
  if (npart == 0) return AAR_OK;
  int bs = 256;
  { ProfScope ps_(p, "readout", st);
  k_readout<<<(unsigned)((npart + bs - 1) / bs), bs, 0, st>>>(read_args(p), (const float*)p->d_work, d_lagr, npart,
                                                               d_pos, d_vel);
  }
  AAR_CUDA_TRY(p, cudaGetLastError());
  p->last_launches += 1;
  return AAR_OK;
}

// Lattice read-out set-up for (g, glass_box, tile): the per-axis Lagrangian
// coordinates and whether the rows can read out (see k_lattice_axis); made
// once per parameter set (one synchronisation), then cached.
int lattice_prepare(Plan* p, int g, double glass_box, int tile, cudaStream_t st, bool& fused) {
  fused = false;
  if ((int64_t)g * tile != p->N) return AAR_OK;
  if (p->lat_g == g && p->lat_box == glass_box && p->lat_tile == tile) {
    fused = p->lat_fused;
    return AAR_OK;
  }
  int rc;
  if (!p->d_lpa && (rc = plan_alloc(p, (void**)&p->d_lpa, sizeof(float) * (p->N + 1)))) return rc;
  int* d_flag = (int*)(p->d_lpa + p->N);
  AAR_CUDA_TRY(p, cudaMemsetAsync(d_flag, 0, sizeof(int), st));
  k_lattice_axis<<<(p->N + 255) / 256, 256, 0, st>>>(p->N, p->prm.box, g, glass_box / g, glass_box, p->prm.box / tile,
                                                      p->d_lpa, d_flag);
  AAR_CUDA_TRY(p, cudaGetLastError());
  int flag = 1;
  AAR_CUDA_TRY(p, cudaMemcpyAsync(&flag, d_flag, sizeof(int), cudaMemcpyDeviceToHost, st));
  AAR_CUDA_TRY(p, cudaStreamSynchronize(st));
  p->lat_g = g;
  p->lat_box = glass_box;
  p->lat_tile = tile;
  p->lat_fused = flag == 0;
  fused = p->lat_fused;
  return AAR_OK;
}

int lattice_glass(Plan* p, int g, double glass_box, float* d_glass, cudaStream_t st) {
  const int64_t n = (int64_t)g * g * g;
  k_lattice_glass<<<(unsigned)std::min<int64_t>((n + 255) / 256, (int64_t)p->num_sms * 8), 256, 0, st>>>(
      g, glass_box / g, d_glass);
  AAR_CUDA_TRY(p, cudaGetLastError());
  p->last_launches += 1;
  return AAR_OK;
}

// The displacement rows with the lattice read-out fused (rows [row0, row0 +
// nrows) of the x-blocked order; lattice_prepare said fused).
int fused_rows_lattice(Plan* p, int g, int tile, float* d_pos, float* d_vel, int* d_ids, int64_t row0, int64_t nrows,
                       cudaStream_t st) {
  if (nrows <= 0) return AAR_OK;
  const LptArgs la = lpt_args(p);
  const ZTypes zt{{3, 3, 4, 3, 3, 4}, la.m.g.kF, la.isinc2};
  return dispatch_n(p->N, [&](auto nc) {
    constexpr int N = decltype(nc)::value;
    using L = LatticeCfg<N>;
    AAR_CUDA_TRY(p, cudaFuncSetAttribute(k_rows_lattice<N>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)L::SMEM));
    {
      ProfScope ps_(p, "lpt_rows_readout", st);
      k_rows_lattice<N><<<(unsigned)((nrows + 2 * L::PR - 1) / (2 * L::PR)), kSixThreads, L::SMEM, st>>>(
          p->d_work, (int64_t)N * N * p->HP, p->HP, p->d_tw2, zt, read_args(p), g, tile, p->d_lpa, d_pos, d_vel, d_ids,
          row0, nrows);
    }
    AAR_CUDA_TRY(p, cudaGetLastError());
    p->last_launches += 1;
    return AAR_OK;
  });
}

int glass_prepare(Plan* p, const float* d_glass, int64_t nglass, double glass_box, int tile, cudaStream_t st) {
  const int64_t need = 3 * nglass + tile;
  if (need > p->gscale_cap) {
    AAR_CUDA_TRY(p, cudaDeviceSynchronize());  // an earlier read-out may still read the old buffer
    if (p->d_gscale) cudaFree(p->d_gscale), p->used_bytes -= sizeof(double) * (size_t)p->gscale_cap;
    p->d_gscale = nullptr;
    p->gscale_cap = 0;
    int rc = plan_alloc(p, (void**)&p->d_gscale, sizeof(double) * (size_t)need);
    if (rc) return rc;
    p->gscale_cap = need;
  }
  k_glass_scale<<<(unsigned)std::min<int64_t>((need + 255) / 256, (int64_t)p->num_sms * 8), 256, 0, st>>>(
      d_glass, nglass, glass_box, tile, p->prm.box / tile, p->d_gscale);
  AAR_CUDA_TRY(p, cudaGetLastError());
  p->last_launches += 1;
  return AAR_OK;
}

int fused_readout_glass(Plan* p, int64_t nglass, int tile, float* d_pos, float* d_vel, int* d_ids, cudaStream_t st,
                        int64_t n0, int64_t n1) {
  const int64_t np = nglass * tile * tile * tile;
  if (n1 < 0 || n1 > np) n1 = np;
  if (n1 <= n0) return AAR_OK;
  const int bs = kReadoutThreads;
  const int64_t cnt = n1 - n0;
  { ProfScope ps_(p, "readout_glass", st);
  k_readout_glass<<<(unsigned)((cnt + bs - 1) / bs), bs, 0, st>>>(read_args(p), (const float*)p->d_work, p->d_gscale,
                                                                   nglass, tile, d_pos, d_vel, d_ids, n0, n1);
  }
  AAR_CUDA_TRY(p, cudaGetLastError());
  p->last_launches += 1;
  return AAR_OK;
}

}  // namespace aar

// ----------------------------------------------------------- standalone 3-D transforms
namespace aar {

// r2c of real fields into plan fields fs apart, blockIdx.y of them: NAT, the
// caller's natural-order ones at `nat`, N^3 apart, else in place
template <int N, bool NAT>
__global__ void __launch_bounds__(kC2rThreads, pair_min_blocks<N>(kC2rThreads))
    k_rows_r2c(const float* nat, float2* f, int64_t fs, int HP, int64_t nrows, const float2* __restrict__ tw2) {
  using C = PairCfg<N>;
  extern __shared__ float2 sm[];
  const int u = threadIdx.x / C::T, t = threadIdx.x % C::T;
  const int64_t row = 2 * ((int64_t)blockIdx.x * (kC2rThreads / C::T) + u);
  const bool act = row < nrows, two = row + 1 < nrows;
  f += blockIdx.y * fs + (act ? row : 0) * HP;
  if (NAT) nat += blockIdx.y * ((int64_t)N * N * N);
  const float* a = NAT ? nat + nat_row<N>(act ? row : 0) * N : reinterpret_cast<const float*>(f);
  const float* b = NAT ? nat + nat_row<N>(two ? row + 1 : 0) * N : a + (two ? 2 * HP : 0);
  float2 v[C::R1];
#pragma unroll
  for (int i = 0; i < C::R1; ++i) {
    const int n = t + C::T * i;
    v[i] = make_float2(act ? a[n] : 0.f, two ? b[n] : 0.f);
  }
  pair_fft<N, -1>(v, sm + u * C::LS, t, tw2, act);
  pair_split<N>(v, f, HP, t, act, two);
}

// The 3-D transforms of a caller's field through work slot 0: the first pass
// reads the caller's order, the last one writes it (with copies between the
// two orders before and after an r2c and a c2r at 512^3 took 3.5 ms, now 1.2).
template <int N>
struct Xform {
  static constexpr int64_t tiles = TileCfg<N>::TILES;
  static constexpr size_t kSmem = pair_line_smem<N>(kC2rThreads);
  static int c2r(Plan* p, const float2* in, float* out, cudaStream_t st) {
    float2* slot = p->d_work;
    int rc = run_pass<N, 0, +1>(p, XNatInOp<N>{in, slot}, tiles, st, "xform_x");
    if (rc) return rc;
    if ((rc = run_pass<N, 1, +1>(p, AxisOp<N>{slot, 0, Slots{}}, tiles, st, "xform_y"))) return rc;
    {
      ProfScope ps_(p, "xform_rows", st);
      k_rows_c2r<N, true><<<c2r_blocks<N>(), kC2rThreads, kSmem, st>>>(slot, 0, p->HP, 0, (int64_t)N * N, p->d_tw2,
                                                                       ZTypes{{0, 0, 0, 0, 0, 0}, 0.f, nullptr}, out);
    }
    AAR_CUDA_TRY(p, cudaGetLastError());
    p->last_launches += 1;
    return AAR_OK;
  }
  static int r2c(Plan* p, const float* in, float2* out, cudaStream_t st) {
    float2* slot = p->d_work;
    {
      ProfScope ps_(p, "xform_rows", st);
      k_rows_r2c<N, true><<<c2r_blocks<N>(), kC2rThreads, kSmem, st>>>(in, slot, 0, p->HP, (int64_t)N * N, p->d_tw2);
    }
    AAR_CUDA_TRY(p, cudaGetLastError());
    p->last_launches += 1;
    int rc = run_pass<N, 1, -1>(p, AxisOp<N>{slot, 0, Slots{}}, tiles, st, "xform_y");
    if (rc) return rc;
    return run_pass<N, 0, -1>(p, XNatOutOp<N>{slot, out}, tiles, st, "xform_x");
  }
};

// Row copy between row orders: row (x, y) of src (order src_xb, ld src_ld
// elements) to row (x, y) of dst, the first ncols elements of each row, a warp
// per row.  Moves fields between the caller's natural [x][y] buffers and the
// plan's x-blocked ones.
template <class T>
__global__ void __launch_bounds__(256) k_copy_rows(T* __restrict__ dst, int64_t dst_ld, int dst_xb,
                                                   const T* __restrict__ src, int64_t src_ld, int src_xb, int N,
                                                   int ncols) {
  const int lane = threadIdx.x & 31;
  const int64_t rows = (int64_t)N * N, step = (int64_t)gridDim.x * (blockDim.x >> 5);
  for (int64_t r = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); r < rows; r += step) {
    const int x = (int)(r / N), y = (int)(r - (int64_t)x * N);
    T* d = dst + row_of(x, y, N, dst_xb) * dst_ld;
    const T* s = src + row_of(x, y, N, src_xb) * src_ld;
#pragma unroll 4
    for (int c = lane; c < ncols; c += 32) d[c] = s[c];
  }
}

int copy_rows(Plan* p, void* dst, int64_t dst_ld, int dst_xb, const void* src, int64_t src_ld, int src_xb, int ncols,
              size_t elem, cudaStream_t st) {
  const unsigned nb = (unsigned)std::min<int64_t>(((int64_t)p->N * p->N + 7) / 8, (int64_t)p->num_sms * 8);
  if (elem == sizeof(float2))
    k_copy_rows<float2><<<nb, 256, 0, st>>>((float2*)dst, dst_ld, dst_xb, (const float2*)src, src_ld, src_xb, p->N,
                                            ncols);
  else
    k_copy_rows<float><<<nb, 256, 0, st>>>((float*)dst, dst_ld, dst_xb, (const float*)src, src_ld, src_xb, p->N,
                                           ncols);
  AAR_CUDA_TRY(p, cudaGetLastError());
  return AAR_OK;
}

// unnormalised FFTW-convention transforms
int fused_c2r(Plan* p, const float2* in, float* out, cudaStream_t st) {
  return dispatch_n(p->N, [&](auto nc) { return Xform<decltype(nc)::value>::c2r(p, in, out, st); });
}

int fused_r2c(Plan* p, const float* in, float2* out, cudaStream_t st) {
  return dispatch_n(p->N, [&](auto nc) { return Xform<decltype(nc)::value>::r2c(p, in, out, st); });
}

#include "chain.cuh"

// Device tables of the chain's products (entries, groups); made once per table
// set.
struct ChainTables {
  AdjEntry* ent;
  AdjGroup* grp;
  int nent, ngrp;
};
static int chain_tables(Plan* p, ChainTables& ct) {
  const int M = p->M;
  if (p->chain_stale) {
    const TermList& tl = *(const TermList*)p->host_terms.data();
    const Term* ft = (const Term*)(p->host_terms.data() + sizeof(TermList));
    std::vector<std::vector<AdjEntry>> by((size_t)M * M);  // [p][r]
    for (int i = 0; i < tl.nterms; ++i) {
      if (ft[i].c == 0.f) continue;
      by[(size_t)ft[i].p * M + ft[i].r].push_back(AdjEntry{ft[i].c, ft[i].q});
      by[(size_t)ft[i].q * M + ft[i].r].push_back(AdjEntry{ft[i].c, ft[i].p});
    }
    std::vector<AdjEntry> ent;
    std::vector<AdjGroup> grp;
    for (int i = 0; i < M * M; ++i) {
      if (by[i].empty()) continue;
      grp.push_back(AdjGroup{i / M, i % M, (int)ent.size(), (int)(ent.size() + by[i].size())});
      ent.insert(ent.end(), by[i].begin(), by[i].end());
    }
    const size_t o_ent = sizeof(AdjGroup) * grp.size(), need = o_ent + sizeof(AdjEntry) * ent.size();
    AAR_CUDA_TRY(p, cudaDeviceSynchronize());  // an earlier pass may still read the old tables
    if (p->chain_bytes < need) {
      if (p->d_chain) cudaFree(p->d_chain), p->used_bytes -= p->chain_bytes;
      p->d_chain = nullptr;
      p->chain_bytes = 0;
      int rc = plan_alloc(p, &p->d_chain, need);
      if (rc) return rc;
      p->chain_bytes = need;
    }
    std::vector<char> host(need);
    std::copy(grp.begin(), grp.end(), (AdjGroup*)host.data());
    std::copy(ent.begin(), ent.end(), (AdjEntry*)(host.data() + o_ent));
    if (int rc_ = upload(p, p->d_chain, host.data(), need)) return rc_;
    p->chain_nent = (int)ent.size();
    p->chain_ngrp = (int)grp.size();
    p->chain_stale = false;
  }
  ct.grp = (AdjGroup*)p->d_chain;
  ct.ent = (AdjEntry*)(ct.grp + p->chain_ngrp);
  ct.nent = p->chain_nent;
  ct.ngrp = p->chain_ngrp;
  return AAR_OK;
}

// Fields of the gradient's scratch: G, T, then the larger of the Hessian
// stage's nine and the products' 2 M; the sums of the products follow them (in
// the caller's scratch, not the plan's memory: calls on different streams may
// overlap).
static int chain_fields(int M) { return 2 + std::max(9, 2 * M); }

template <int N>
struct Chain {
  using L = Launch<N>;
  static constexpr int64_t kTiles = TileCfg<N>::TILES;
  static constexpr size_t kLineSmem = pair_line_smem<N>(kC2rThreads);
  static constexpr size_t kSevenSmem = L::pair_smem(7 * (32 / PairCfg<N>::T));
  // shared memory of the products' kernels; shares of a chunk that the threads
  // of k_chain_sums split into, as many as its items leave
  static constexpr int sums_share(int M, int nrb) {
    const int items = M * (M + 1) / 2 * nrb;
    return items <= 32 ? 4 : items <= 64 ? 2 : 1;
  }
  static constexpr size_t sums_smem(int M, int share) {
    return sizeof(double) * ((share * chain_ntrip(M) + 1) / 2 * 2) + sizeof(float) * 2 * M * kChainLd;
  }
  static constexpr size_t gf_smem(int M, int nent, int ngrp) {
    return sizeof(float2) * 2 * M * kChainThreads + sizeof(AdjEntry) * ((nent + 1) / 2 * 2) + sizeof(AdjGroup) * ngrp;
  }
  // The limits belong to the functions, which all plans of a grid size share:
  // set to what the largest table takes, never to a plan's own need (one thread
  // could lower it between another's setting and its launch).
  static int configure(Plan* p) {
    auto limit = [&](auto kern, size_t smem) {
      AAR_CUDA_TRY(p, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
      return AAR_OK;
    };
    constexpr size_t sums = sums_smem(kMaxModes, 1), gf = gf_smem(kMaxModes, 2 * kMaxTerms, kMaxModes * kMaxModes);
    static_assert(sums >= sums_smem(10, 2) && sums >= sums_smem(7, 4) && sums_share(kMaxModes, 2) == 1 &&
                  sums_share(11, 1) == 1 && sums_share(8, 1) == 2 && gf <= 227 * 1024);
    int rc;
    if ((rc = limit(k_chain_sums<N, 4>, sums)) || (rc = limit(k_chain_sums<N, 8>, sums)) ||
        (rc = limit(k_chain_sums<N, 12>, sums)) || (rc = limit(k_chain_sums<N, 16>, sums)) ||
        (rc = limit(k_chain_gf<N>, gf)) || (rc = limit(k_rows_source_adj<N>, kSevenSmem)))
      return rc;
    return limit(k_xacc<N, true>, XaccCfg<N>::SMEM);
  }
  static unsigned cells(Plan* p) { return (unsigned)(p->num_sms * 8); }
  static int done(Plan* p) {
    AAR_CUDA_TRY(p, cudaGetLastError());
    p->last_launches += 1;
    return AAR_OK;
  }
  static Slots run(int first, int n) {
    Slots s{};
    for (int i = 0; i < n; ++i) s.s[i] = first + i;
    return s;
  }
  static int forward(Plan* p, const float2* w, float* disp, float2* phig, float2* phi, cudaStream_t st) {
    int rc;
    k_chain_gauss<N><<<cells(p), 256, 0, st>>>(p->grid, p->d_amp, w, p->d_phik, phig);
    if ((rc = done(p)) || (rc = fused_modal(p, st))) return rc;
    if ((rc = copy_rows(p, phi, N / 2 + 1, 1, p->d_phik, p->HP, kXB, N / 2 + 1, sizeof(float2), st))) return rc;
    if ((rc = fused_lpt(p, st))) return rc;
    k_chain_disp<N><<<dim3(cells(p), 3), 256, 0, st>>>((const float*)p->d_work, 2 * L::fstride(p), p->HP,
                                                       (float)(-(3.0 / 7.0) / ((double)N * N * N)), disp);
    return done(p);
  }
  static int backward(Plan* p, const float2* phig, const float2* phi, const float* gdisp, float2* gw, double* galpha,
                      float2* scratch, cudaStream_t st) {
    const int64_t fs = L::fstride(p), rows = (int64_t)N * N;
    const int M = p->M;
    float2 *G = scratch, *T = scratch + fs, *W = scratch + 2 * fs;
    const LptArgs a = lpt_args(p);
    const float kF = a.m.g.kF;
    const ZTypes none{{0, 0, 0, 0, 0, 0}, 0.f, nullptr};
    const float fnl_n3 = (float)(p->prm.fnl / ((double)N * N * N));
    double* sum = (double*)(scratch + chain_fields(M) * fs);
    ChainTables ct;
    int rc;
    if ((rc = chain_tables(p, ct))) return rc;
    AAR_CUDA_TRY(p, cudaMemsetAsync(sum, 0, sizeof(double) * chain_ntrip(M), st));
    // displacement fields
    k_rows_r2c<N, true><<<dim3(c2r_blocks<N>(), 3), kC2rThreads, kLineSmem, st>>>(gdisp, W, fs, p->HP, rows, p->d_tw2);
    if ((rc = done(p))) return rc;
    if ((rc = L::template axis_pass<1, -1>(p, W, 3, run(0, 3), st, "grad_y"))) return rc;
    if ((rc = L::template axis_pass<0, -1>(p, W, 3, run(0, 3), st, "grad_x"))) return rc;
    k_chain_div<N><<<cells(p), 256, 0, st>>>(a, W, fs, (float)(-(3.0 / 7.0) / ((double)N * N * N)), G, T);
    if ((rc = done(p))) return rc;
    if ((rc = L::template axis_pass<0, +1>(p, T, 1, run(0, 1), st, "grad_x"))) return rc;
    if ((rc = L::template axis_pass<1, +1>(p, T, 1, run(0, 1), st, "grad_y"))) return rc;
    // the source, its Hessians made again from phi
    const LptXNatOp<N> ho{{phi, nullptr, W, fs, {0, 8, 6, 0}, 1, kF, a.isinc2, p->d_tcube, p->d_twb}};
    if ((rc = run_pass<N, 0, +1>(p, ho, kTiles * 3, st, "grad_xhess"))) return rc;
    const YFanOp<N> yf{W, fs, {0, 8, 8, 6, 6, 6}, {0, 1, 2, 3, 4, 5}, {0, 1, 0, 2, 1, 0}, 1, kF, a.isinc2};
    if ((rc = run_pass<N, 1, +1>(p, yf, kTiles * 6, st, "grad_yhess"))) return rc;
    {
      ProfScope ps_(p, "grad_rows_source", st);
      constexpr int per = 2 * (32 / PairCfg<N>::T);  // rows of a block
      k_rows_source_adj<N><<<(unsigned)((rows + per - 1) / per), kSevenThreads, kSevenSmem, st>>>(
          SourceAdjRowOp{-1, kF, a.isinc2}, W, fs, p->HP, rows, p->d_tw2);
    }
    if ((rc = done(p))) return rc;
    if ((rc = run_pass<N, 1, -1>(p, YAdjOp<N>{W, fs, Slots{{0, 1, 0, 2, 1, 0}}}, kTiles * 6, st, "grad_y"))) return rc;
    if ((rc = run_pass<N, 0, -1>(p, XSumOp<N>{W, fs, {0, 1, 3}, {1, 2, 3}}, kTiles * 3, st, "grad_x"))) return rc;
    k_chain_hess<N><<<cells(p), 256, 0, st>>>(a, W, fs, p->d_rtab, fnl_n3, G, T);
    if ((rc = done(p))) return rc;
    // the modal products, their fields made again from phig
    const XinvGradOp<N> xg{{T, W, fs, M, run(0, M), 1, M, M, p->d_qcube}, G, fnl_n3};
    if ((rc = run_pass<N, 0, +1>(p, xg, kTiles * M, st, "grad_xinv"))) return rc;
    const XinvNatOp<N> xf{{phig, W, fs, M, run(0, M), 1, 0, M, p->d_qcube}};
    if ((rc = run_pass<N, 0, +1>(p, xf, kTiles * M, st, "grad_xinv"))) return rc;
    for (int h = 0; h < 2; ++h)
      if ((rc = L::template axis_pass<1, +1>(p, W, M, run(h * M, M), st, "grad_y"))) return rc;
    {
      ProfScope ps_(p, "grad_rows", st);
      k_rows_c2r<N, false><<<dim3(c2r_blocks<N>(), 2 * M), kC2rThreads, kLineSmem, st>>>(W, fs, p->HP, 0, rows, p->d_tw2,
                                                                                        none, nullptr);
    }
    if ((rc = done(p))) return rc;
    {
      ProfScope ps_(p, "grad_sums", st);
      // r in as few blocks of at most 16 as hold them, the threads in as many
      // shares of a chunk as the items leave
      const int nrb = (M + 15) / 16, rb = (M + nrb - 1) / nrb;
      const int share = sums_share(M, nrb);
      const size_t smem = sums_smem(M, share);
      const unsigned blocks = (unsigned)std::min<int64_t>((int64_t)N * N * N / kChainChunk, (int64_t)p->num_sms * 8);
      auto go = [&](auto rbc) {
        k_chain_sums<N, decltype(rbc)::value>
            <<<blocks, kChainThreads, smem, st>>>((const float*)W, 2 * fs, p->HP, M, share, sum);
      };
      if (rb <= 4) go(std::integral_constant<int, 4>{});
      else if (rb <= 8) go(std::integral_constant<int, 8>{});
      else if (rb <= 12) go(std::integral_constant<int, 12>{});
      else go(std::integral_constant<int, 16>{});
    }
    if ((rc = done(p))) return rc;
    {
      ProfScope ps_(p, "grad_gf", st);
      const size_t smem = gf_smem(M, ct.nent, ct.ngrp);
      const int64_t n2 = (int64_t)N * N * N / 2;
      k_chain_gf<N><<<(unsigned)std::min<int64_t>((n2 + kChainThreads - 1) / kChainThreads, (int64_t)p->num_sms * 16),
                      kChainThreads, smem, st>>>((float*)W, 2 * fs, p->HP, M, ct.ent, ct.nent, ct.grp, ct.ngrp);
    }
    if ((rc = done(p))) return rc;
    const int counter = M > 2 && p->alpha[(size_t)1 * M + 2] != 0;
    k_chain_galpha<<<1, 256, 0, st>>>(sum, M, counter, galpha);
    if ((rc = done(p))) return rc;
    {
      ProfScope ps_(p, "grad_rows", st);
      k_rows_r2c<N, false><<<dim3(c2r_blocks<N>(), M), kC2rThreads, kLineSmem, st>>>(nullptr, W, fs, p->HP, rows, p->d_tw2);
    }
    if ((rc = done(p))) return rc;
    if ((rc = L::template axis_pass<1, -1>(p, W, M, run(0, M), st, "grad_y"))) return rc;
    const XaccArgs<N> xa{p->grid, G, W, fs, M, M, run(0, M), M, p->d_qcube, nullptr, 0.f, p->d_amp, gw};
    {
      ProfScope ps_(p, "grad_xacc", st);
      k_xacc<N, true><<<(unsigned)kTiles, TileCfg<N>::THREADS, XaccCfg<N>::SMEM, st>>>(xa, p->d_tw2);
    }
    return done(p);
  }
};

size_t chain_scratch_bytes(const Plan* p) {
  return sizeof(float2) * (size_t)p->N * p->N * p->HP * chain_fields(p->M) + sizeof(double) * chain_ntrip(p->M);
}
int chain_forward(Plan* p, const float2* w, float* disp, float2* phig, float2* phi, cudaStream_t st) {
  return dispatch_n(p->N, [&](auto nc) { return Chain<decltype(nc)::value>::forward(p, w, disp, phig, phi, st); });
}
int chain_backward(Plan* p, const float2* phig, const float2* phi, const float* gdisp, float2* gw, double* galpha,
                   float2* scratch, cudaStream_t st) {
  return dispatch_n(p->N, [&](auto nc) {
    return Chain<decltype(nc)::value>::backward(p, phig, phi, gdisp, gw, galpha, scratch, st);
  });
}

int fused_configure_xform(Plan* p) {
  return dispatch_n(p->N, [&](auto nc) {
    constexpr int N = decltype(nc)::value;
    const int smem = (int)pair_line_smem<N>(kC2rThreads);
    AAR_CUDA_TRY(p, cudaFuncSetAttribute(k_rows_c2r<N, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    AAR_CUDA_TRY(p, cudaFuncSetAttribute(k_rows_c2r<N, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    AAR_CUDA_TRY(p, cudaFuncSetAttribute(k_rows_r2c<N, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    AAR_CUDA_TRY(p, cudaFuncSetAttribute(k_rows_r2c<N, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    const int rc = Chain<N>::configure(p);
    return rc ? rc : Launch<N>::configure(p);
  });
}

}  // namespace aar
