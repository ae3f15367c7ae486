// Row (z) kernels: the real <-> half-complex transform of contiguous rows
// and the generic per-row "c2r, combine, r2c" body.  Device code only, so
// that it compiles both in this library and in the run-time specialised
// row kernel (jit.cu, NVRTC).
#pragma once
#include "fft.cuh"

namespace aar {

// Per-axis real factor of the 2LPT y pass and c2r rows (index k along the
// axis; y uses the signed index, z the column index kz = 0..N/2): 0: 1,
// 1: k, 2: k^2, 3: 1/sinc^2, 4: kF k / sinc^2, as the product of a table value
// (isinc2 = 1/sinc^2 per grid index; types 3 and 4) and a polynomial.  A
// thread's table loads go out together, without a branch per value.
__device__ __forceinline__ float axis_table(int type, const float* __restrict__ isinc2, int gi) {
  return type >= 3 ? __ldg(isinc2 + gi) : 1.f;
}
__device__ __forceinline__ float axis_poly(int type, float k, float kF) {
  return type == 1 ? k : type == 2 ? k * k : type == 4 ? kF * k : 1.f;
}

// z factor of a row's spectrum, applied as the c2r reads X_k
struct ZFac {
  int type;  // 0 = none
  float kF;
  const float* isinc2;
};

// Row layout: complex row X[0..N/2] at field + m HP, m the row's memory
// index (the plan's row order maps (x, y) to m); the real row x[0..N-1]
// occupies the same bytes.  The row steps are the same for every row, so the
// kernels run over memory rows.

// ---------------------------------------------------------------------
// Rows in pairs.  Two real rows a, b travel as one complex line a + i b: its
// N-point spectrum is C_k = A_k + i B_k, C_{N-k} = conj A_k + i conj B_k, so
// a c2r of both is one complex inverse transform of C and an r2c of both one
// forward transform and C's even / odd split -- no half-length twiddle steps.
// The rows of a pair are neighbours of the same field (memory rows m, m + 1).
// The FP32 rounding of a line is relative to the larger of the two; the x and y
// passes mix all rows anyway, so the error of a 3-D transform relative to its
// norm is that of single rows, whatever the field.
//
// A line is transformed by T threads with R1 = N / T values each in two
// register stages and one exchange through the line's own shared memory
// (R1 R2 = N, T = R2; fft.cuh: two_stage_r1): lane t holds C_{t + T i}, i < R1,
// before and after, so the partner C_{N-k} of k = t + T i is value R1 - 1 - i
// of lane T - t: a shuffle (lane 0 has its own partners).  The samples come
// out at positions t + T i again, and go through shared memory once for the
// pointwise combine, which needs every line at one position.
//
// What bounds it: instruction issue (FP32) and shared-memory wavefronts, then
// HBM.  Measured against half-length transforms of single rows staged in
// shared memory (folded radix 2 at N = 1024): modal rows 5.81 -> 3.90 ms
// (512^3, 12 modes), 0.82 -> 0.48 (256^3, 13 modes), 0.089 -> 0.019 (128^3,
// generic kernel, 3 read modes); source rows 10.3 -> 9.0 (1024^3), 2.34 ->
// 1.10 (512^3), 0.317 -> 0.115 (256^3); displacement rows 12.9 -> 9.3
// (1024^3); rows with the lattice read-out 13.3 -> 12.9 (1024^3), 2.47 -> 1.65
// (512^3).
template <int N>
struct PairCfg {
  static constexpr int R1 = two_stage_r1(N);
  static constexpr int R2 = N / R1;
  static constexpr int T = R2;           // threads per line
  static constexpr int G = R1 / T;       // second-stage DFTs per thread
  static constexpr int LPW = 32 / T;     // lines per warp
  static constexpr int LS = N + T;       // exchange entries of a line
  static constexpr int HR = R1 / 2;
};

// The modal rows' path: pairs, except at N = 1024 with more than 8 lines,
// where a block of a row pair leaves too few warps on the SM for its 32
// values per lane (1024^3, NVRTC kernel, pairs against one folded row per
// block: 4 modes 7.5 / 10.7 ms, 6 12.4 / 14.6, 8 17.1 / 18.7, 10 28.7 / 27.2,
// 13 36.6 / 36.0).
__host__ __device__ constexpr bool rows_use_pairs(int N, int nlines) { return N < 1024 || nlines <= 8; }

// The transform of a lane's line values, v[i] = x[t + T i] in and out
// (reordered), through the line buffer ln.  tw2[r R1 + j] = exp(-2 pi i r j /
// N).  The T lanes of a line call it together (whole warps); lanes without a
// line (act false) take part in the barriers only.  Conflict-free: the first
// stage's stores are R1 + 1 (odd) entries apart between lanes, its loads
// contiguous.
template <int N, int SIGN>
__device__ __forceinline__ void pair_fft(float2* v, float2* ln, int t, const float2* __restrict__ tw2, bool act) {
  using C = PairCfg<N>;
  DFT<C::R1, SIGN>::run(v);
  __syncwarp();  // the line's earlier readers are done
  if (act) {
#pragma unroll
    for (int r = 0; r < C::R1; ++r) ln[t * (C::R1 + 1) + r] = v[r];
  }
  __syncwarp();
  float2 u[C::R1];
  if (act) {
#pragma unroll
    for (int b = 0; b < C::G; ++b)
#pragma unroll
      for (int r = 0; r < C::R2; ++r) u[b * C::R2 + r] = ln[r * (C::R1 + 1) + t + C::T * b];
  }
#pragma unroll
  for (int b = 0; b < C::G; ++b) {
#pragma unroll
    for (int r = 1; r < C::R2; ++r)
      u[b * C::R2 + r] = cmul(u[b * C::R2 + r], tw_load<SIGN>(tw2 + t + C::T * b, r * C::R1));
    DFT<C::R2, SIGN>::run(u + b * C::R2);
  }
  __syncwarp();  // the exchange has been read
#pragma unroll
  for (int b = 0; b < C::G; ++b)
#pragma unroll
    for (int r = 0; r < C::R2; ++r) v[b + C::G * r] = u[b * C::R2 + r];
}

// Lane t's line values C_{t + T i} of the pair's half spectra A, B (B null:
// zero), with the z factor of the field.  FFTW c2r: Im X_0, Im X_{N/2} of
// each row are dropped.
template <int N, bool ZF>
__device__ __forceinline__ void pair_spectrum(float2* v, const float2* __restrict__ A, const float2* __restrict__ B,
                                              int t, ZFac zf, bool act) {
  using C = PairCfg<N>;
  float2 a[C::HR], b[C::HR];
  float2 ah = make_float2(0.f, 0.f), bh = ah;
#pragma unroll
  for (int i = 0; i < C::HR; ++i) {
    a[i] = act ? A[t + C::T * i] : make_float2(0.f, 0.f);
    b[i] = act && B ? B[t + C::T * i] : make_float2(0.f, 0.f);
  }
  if (act && t == 0) {
    ah = A[N / 2];
    if (B) bh = B[N / 2];
  }
  if constexpr (ZF) {
    float f[C::HR];
#pragma unroll
    for (int i = 0; i < C::HR; ++i) f[i] = axis_table(zf.type, zf.isinc2, t + C::T * i);
    const float fh = axis_table(zf.type, zf.isinc2, N / 2) * axis_poly(zf.type, (float)(N / 2), zf.kF);
#pragma unroll
    for (int i = 0; i < C::HR; ++i) {
      f[i] *= axis_poly(zf.type, (float)(t + C::T * i), zf.kF);
      a[i] = cscale(a[i], f[i]);
      b[i] = cscale(b[i], f[i]);
    }
    ah.x *= fh;
    bh.x *= fh;
  }
  float2 u[C::HR];  // conj A + i conj B: the value at N - k
#pragma unroll
  for (int i = 0; i < C::HR; ++i) {
    v[i] = make_float2(a[i].x - b[i].y, a[i].y + b[i].x);
    u[i] = make_float2(a[i].x + b[i].y, b[i].x - a[i].y);
  }
  if (t == 0) v[0] = make_float2(a[0].x, b[0].x);
  const int lane = threadIdx.x & 31;
  const int src = (lane & ~(C::T - 1)) | ((C::T - t) & (C::T - 1));
#pragma unroll
  for (int i = 0; i < C::HR; ++i) {
    const float2 w = make_float2(__shfl_sync(0xffffffffu, u[i].x, src), __shfl_sync(0xffffffffu, u[i].y, src));
    const float2 own = i + 1 < C::HR ? u[i + 1 < C::HR ? i + 1 : 0] : make_float2(ah.x, bh.x);
    v[C::R1 - 1 - i] = t == 0 ? own : w;
  }
}

// Half spectra of the pair from lane t's transformed values C_{t + T i}, into
// X (row a) and X + HP (row b, when two), with the z factor of the field (ZF).
template <int N, bool ZF = false>
__device__ __forceinline__ void pair_split(const float2* v, float2* __restrict__ X, int HP, int t, bool act, bool two,
                                           ZFac zf = ZFac{0, 0.f, nullptr}) {
  using C = PairCfg<N>;
  const int lane = threadIdx.x & 31;
  const int src = (lane & ~(C::T - 1)) | ((C::T - t) & (C::T - 1));
#pragma unroll
  for (int i = 0; i < C::HR; ++i) {
    const float2 c = v[i];
    float2 p = make_float2(__shfl_sync(0xffffffffu, v[C::R1 - 1 - i].x, src),
                           __shfl_sync(0xffffffffu, v[C::R1 - 1 - i].y, src));
    if (t == 0) p = v[i == 0 ? 0 : C::R1 - i];
    const float h = ZF ? 0.5f * axis_poly(zf.type, (float)(t + C::T * i), zf.kF) : 0.5f;  // types 0..2
    if (act) {
      X[t + C::T * i] = make_float2(h * (c.x + p.x), h * (c.y - p.y));
      if (two) X[HP + t + C::T * i] = make_float2(h * (c.y + p.y), h * (p.x - c.x));
    }
  }
  if (act && t == 0) {
    const float h = ZF ? axis_poly(zf.type, (float)(N / 2), zf.kF) : 1.f;
    X[N / 2] = make_float2(h * v[C::HR].x, 0.f);
    if (two) X[HP + N / 2] = make_float2(h * v[C::HR].y, 0.f);
  }
}

// Row kernel on pairs: block b takes the PR row pairs from memory row 2 PR b
// on.  Phase 1: inverse transforms of every (pair, input) line, one line per
// T threads; phase 2: the combine, a float2 position holding the two rows'
// samples; phase 3: forward transforms of every (pair, output) line.
template <int N, class Op, int THREADS>
__device__ __forceinline__ void rows_pairs(const Op& op, float2* work, int64_t fs, int HP, int64_t nrows,
                                           const float2* __restrict__ tw2, const int PR) {
  using C = PairCfg<N>;
  extern __shared__ float2 sm_all[];
  float2* sm = sm_all;  // [PR][op.nlines()][LS]
  const int64_t row0 = (int64_t)blockIdx.x * (2 * PR);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int sub = lane / C::T, t = lane % C::T;
  constexpr int STEP = THREADS / 32 * C::LPW;
  const int stride = op.nlines() * C::LS;  // of a row pair
  for (int u0 = warp * C::LPW; u0 < PR * op.nin(); u0 += STEP) {
    const int u = u0 + sub, pr = PR == 1 ? 0 : u / op.nin(), l = PR == 1 ? u : u - pr * op.nin();
    const int64_t row = row0 + 2 * pr;
    const bool act = u < PR * op.nin() && row < nrows;
    float2* ln = sm + (act ? pr * stride + op.in_line(l) * C::LS : 0);
    const float2* X = work + (act ? (int64_t)op.in_slot(l) * fs + row * HP : 0);
    float2 v[C::R1];
    ZFac zf{0, 0.f, nullptr};
    if constexpr (Op::kZfac) zf = op.zfac(act ? l : 0);
    pair_spectrum<N, Op::kZfac>(v, X, row + 1 < nrows ? X + HP : nullptr, t, zf, act);
    pair_fft<N, +1>(v, ln, t, tw2, act);
    if (act) {
#pragma unroll
      for (int i = 0; i < C::R1; ++i) ln[t + C::T * i] = v[i];
    }
  }
  __syncthreads();
  constexpr int K = Op::kPairs ? 2 : 1;
  for (int n = threadIdx.x; n < PR * N; n += K * THREADS) {
    const int o0 = (PR == 1 ? 0 : n / N * stride) + n % N;
    if (K == 2 && n + THREADS < PR * N) {
      const int m = n + THREADS;
      const int pos[2] = {o0, (PR == 1 ? 0 : m / N * stride) + m % N};
      op.template combine<2>(sm, pos, C::LS);
    } else {
      const int pos[1] = {o0};
      op.template combine<1>(sm, pos, C::LS);
    }
  }
  __syncthreads();
  for (int u0 = warp * C::LPW; u0 < PR * op.nout(); u0 += STEP) {
    const int u = u0 + sub, pr = PR == 1 ? 0 : u / op.nout(), l = PR == 1 ? u : u - pr * op.nout();
    const int64_t row = row0 + 2 * pr;
    const bool act = u < PR * op.nout() && row < nrows;
    float2* ln = sm + (act ? pr * stride + op.out_line(l) * C::LS : 0);
    float2 v[C::R1];
#pragma unroll
    for (int i = 0; i < C::R1; ++i) v[i] = act ? ln[t + C::T * i] : make_float2(0.f, 0.f);
    pair_fft<N, -1>(v, ln, t, tw2, act);
    float2* X = work + (act ? (int64_t)op.out_slot(l) * fs + row * HP : 0);
    if constexpr (requires { Op::kZfacOut; }) pair_split<N, true>(v, X, HP, t, act, row + 1 < nrows, op.zfac(act ? l : 0));
    else pair_split<N>(v, X, HP, t, act, row + 1 < nrows);
  }
}

// ---------------------------------------------------------------------
// Rows of N = 1024 (half-length H = 512) fold the radix-2 step of the
// half-length transform into the c2r pre-step and the r2c post-step, so a
// line takes two shared-memory stages (two H/2-point transforms of radix
// 16 x 16 on the half-warps) instead of three (16 x 16 x 2).  Lane `lane`
// of the warp owns the quads of positions k, h-k, h+k, H-k (h = H/2,
// k = lane + 32 i <= H/4); the quads partition 0..H, so the steps work in
// place without a barrier.
//
// Inverse: Z_n from X (the pre-step), then decimation in frequency:
// u_n = Z_n + Z_{n+h} to position n and (Z_n - Z_{n+h}) e^{2 pi i n/H} to
// n + h, n < h.  Inverse h-point transforms of the two halves leave z_{2m}
// at m and z_{2m+1} at h + m (z_n = (x_{2n}, x_{2n+1})): the line's samples
// in a permuted order, which the pointwise combine does not see.
// Forward, from that order: E_k (first half) and O_k (second half) after
// the h-point transforms, Z_k = E_k + e^{-2 pi i k/H} O_k and Z_{k+h} =
// E_k - e^{-2 pi i k/H} O_k, then the post-step X_k from Z_k, Z_{H-k}.
template <int N>
struct FoldCfg {
  static_assert(N == 1024 && N / 4 == kLineR * kLineR, "folded rows: one warp per 512-point half line");
  static constexpr int LS = spad_len(N / 2);
  // float2 slots of the lane twiddle table (fft.cuh) of the H/2-point
  // half-line transforms, at the start of the shared memory, filled once per
  // block (the modal rows at 1024^3 with 20 modes 67.9 -> 60.8 ms)
  static constexpr int LT = kLineTw;
};

// Z_j of the c2r pre-step from a = X_j, b = X_{H-j}, w = e^{+2 pi i j/N}:
// E + i O with E = a + conj b, O = (a - conj b) w
__device__ __forceinline__ float2 pre1(float2 a, float2 b, float2 w) {
  const float2 e = make_float2(a.x + b.x, a.y - b.y);
  const float2 o = cmul(make_float2(a.x - b.x, a.y + b.y), w);
  return make_float2(e.x - o.y, e.y + o.x);
}
// X_j of the r2c post-step from z = Z_j, zr = Z_{H-j}, w = e^{-2 pi i j/N}
__device__ __forceinline__ float2 post1(float2 z, float2 zr, float2 w) {
  const float2 e = make_float2(0.5f * (z.x + zr.x), 0.5f * (z.y - zr.y));
  const float2 od = cmul(make_float2(0.5f * (z.x - zr.x), 0.5f * (z.y + zr.y)), w);
  return make_float2(e.x + od.y, e.y - od.x);
}

// The folded steps walk the quads k = lane + 32 it < Q in Q / 32 rounds; the
// quad k = Q, which has two outputs only (positions Q and H - Q, where its
// first and second output pairs coincide), rides with lane 0's first quad
// k = 0, which has no second pair: lane 0 computes that pair from the quad
// k = Q instead.  (With k = Q a round of its own, a fifth round ran a whole
// warp for one quad.)  At j = Q the twiddles of the two pair formulas agree:
// conj w_Q = i w_Q and -v_Q = conj v_Q (w_Q = e^{-i pi/4}, v_Q = -i).

// Inverse pre-step into the line buffer, from X in global memory (src):
// first pair (Z_k + Z_{k+h}, (Z_k - Z_{k+h}) e^{2 pi i k/H}) to positions k
// and h + k from the quad at k; second pair to positions h - k2 and H - k2
// from the quad at k2 (k2 = k, or Q for lane 0's first quad).
template <int N>
__device__ __forceinline__ void row_c2r_pre_fold(float2* line, int lane, const float2* __restrict__ twN,
                                                 const float2* __restrict__ twH,
                                                 const float2* __restrict__ src) {
  constexpr int H = N / 2, h = H / 2, Q = H / 4;
  static_assert(Q % 32 == 0, "folded rows: whole rounds of quads");
  constexpr int NIT = Q / 32;
  // all of the lane's loads first (independent, in flight together), then
  // the quads: the loads of one quad do not wait for the previous quad's
  // arithmetic and stores
  float2 qa[NIT], qb[NIT], qc[NIT], qd[NIT];
#pragma unroll
  for (int it = 0; it < NIT; ++it) {
    const int k = lane + 32 * it;
    qa[it] = src[k];
    qb[it] = src[H - k];
    qc[it] = src[h - k];
    qd[it] = src[h + k];
  }
  const float2 xq = src[Q], x3q = src[H - Q];  // the quad k = Q: X_Q, X_{H-Q} (= X_{h-Q}, X_{h+Q})
  const float2 wQ = __ldg(twN + Q), vQ = __ldg(twH + Q);
#pragma unroll
  for (int it = 0; it < NIT; ++it) {
    const int k = lane + 32 * it;
    const bool l0 = it == 0 && lane == 0;
    float2 a = qa[it], b = qb[it], c = qc[it], d = qd[it];
    const int k2 = l0 ? Q : k;
    const float2 wk = __ldg(twN + k), vk = __ldg(twH + k);
    const float2 w2 = l0 ? wQ : wk, v2 = l0 ? vQ : vk;
    float2 a2 = l0 ? xq : a, b2 = l0 ? x3q : b, c2 = l0 ? xq : c, d2 = l0 ? x3q : d;
    if (k == 0) {  // FFTW c2r: Im X_0, Im X_{N/2} dropped
      a.y = 0.f;
      b.y = 0.f;
    }
    // e^{+2 pi i j/N} at j = k, h+k: conj w, i conj w; at j = H-k2, h-k2: -w, i w
    const float2 zk = pre1(a, b, make_float2(wk.x, -wk.y));
    const float2 zhp = pre1(d, c, make_float2(wk.y, wk.x));
    const float2 zHk = pre1(b2, a2, make_float2(-w2.x, -w2.y));
    const float2 zhm = pre1(c2, d2, make_float2(-w2.y, w2.x));
    // butterflies n = k and n = h - k2; e^{2 pi i n/H}: conj v, -v
    line[spad(k)] = cadd(zk, zhp);
    line[spad(h + k)] = cmul(csub(zk, zhp), make_float2(vk.x, -vk.y));
    line[spad(h - k2)] = cadd(zhm, zHk);
    line[spad(H - k2)] = cmul(csub(zhm, zHk), make_float2(-v2.x, -v2.y));
  }
}

// Forward post-step from the line buffer to X (global): per quad k the four
// outputs X_k, X_{H-k}, X_{h-k}, X_{h+k}; lane 0's first quad gives X_0,
// X_H, X_h from k = 0 (Z_0 = E_0 + O_0 = Z_H, Z_h = E_0 - O_0) in the same
// three formulas with its operands selected, and X_Q, X_{H-Q} from the quad
// k = Q in the fourth and a fifth.
template <int N>
__device__ __forceinline__ void row_r2c_post_fold(const float2* line, float2* __restrict__ X, int lane,
                                                  const float2* __restrict__ twN, const float2* __restrict__ twH) {
  constexpr int H = N / 2, h = H / 2, Q = H / 4;
  static_assert(Q % 32 == 0, "folded rows: whole rounds of quads");
  constexpr int NIT = Q / 32;
  const float2 wQ = __ldg(twN + Q), vQ = __ldg(twH + Q);
#pragma unroll
  for (int it = 0; it < NIT; ++it) {
    const int k = lane + 32 * it;
    const bool l0 = it == 0 && lane == 0;
    const int k2 = l0 ? Q : k;
    const float2 wk = __ldg(twN + k), vk = __ldg(twH + k);
    const float2 v2 = l0 ? vQ : vk;
    const float2 ek = line[spad(k)], ok = cmul(line[spad(h + k)], vk);
    const float2 zk = cadd(ek, ok), zhp = csub(ek, ok);
    // Z_{h-k2} = E - conj(v) O, Z_{H-k2} = E + conj(v) O from positions h - k2, H - k2
    const float2 em = line[spad(h - k2)], om = cmul(line[spad(H - k2)], make_float2(v2.x, -v2.y));
    const float2 zhm = csub(em, om), zHk = cadd(em, om);
    // e^{-2 pi i j/N} at j = k, H-k, h-k, h+k: w, -conj w, -i conj w, -i w
    X[k] = post1(zk, l0 ? zk : zHk, wk);
    X[H - k] = post1(l0 ? zk : zHk, zk, make_float2(-wk.x, wk.y));
    X[h - k] = post1(l0 ? zhp : zhm, zhp, make_float2(-wk.y, -wk.x));
    if (l0) {
      X[Q] = post1(zhm, zHk, wQ);
      X[H - Q] = post1(zHk, zhm, make_float2(-wQ.x, wQ.y));
    } else {
      X[h + k] = post1(zhp, zhm, make_float2(wk.y, -wk.x));
    }
  }
}

// One row per block, folded (N = 1024): c2r of the input fields into their
// lines, one warp per line at a time, the combine, r2c of the output lines.
// For plans whose lines of a row pair do not leave room for two resident
// blocks (rows_use_pairs); 256 threads, or 320 where ten warps take the
// input lines in fewer rounds than eight, two resident blocks per SM.
constexpr int kRowThreads = 256;
template <int N, class Op, int THREADS = kRowThreads>
__device__ __forceinline__ void rows_fold(const Op& op, float2* work, int64_t fs, int HP,
                                          const float2* __restrict__ twN, const float2* __restrict__ twH) {
  using C = FoldCfg<N>;
  constexpr int H = N / 2, h = H / 2, HO = h + h / 16;  // spad(h + i) = spad(i) + HO
  extern __shared__ float2 sm_all[];
  float2* sm = sm_all + C::LT;  // line buffers after the lane twiddles
  const int64_t row = blockIdx.x;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  constexpr int nwarps = THREADS / 32;
  const int half = lane >> 4, t16 = lane & 15;
  const float2* lt = sm_all;
  lt_fill<2>(sm_all, twH, threadIdx.x, THREADS);
  __syncthreads();
  for (int l = warp; l < op.nin(); l += nwarps) {
    float2* line = sm + op.in_line(l) * C::LS;
    row_c2r_pre_fold<N>(line, lane, twN, twH, work + (int64_t)op.in_slot(l) * fs + row * HP);
    __syncwarp();
    line_fft<+1>(line + half * HO, t16, lt);
  }
  __syncthreads();
  for (int n = threadIdx.x; n < H; n += (Op::kPairs ? 2 : 1) * THREADS) {
    if (Op::kPairs && n + THREADS < H) {
      const int pos[2] = {spad(n), spad(n + THREADS)};
      op.template combine<2>(sm, pos, C::LS);
    } else {
      const int pos[1] = {spad(n)};
      op.template combine<1>(sm, pos, C::LS);
    }
  }
  __syncthreads();
  for (int l = warp; l < op.nout(); l += nwarps) {
    float2* line = sm + op.out_line(l) * C::LS;
    line_fft<-1>(line + half * HO, t16, lt);
    row_r2c_post_fold<N>(line, work + (int64_t)op.out_slot(l) * fs + row * HP, lane, twN, twH);
    __syncwarp();
  }
}

}  // namespace aar
