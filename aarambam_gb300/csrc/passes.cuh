// Strided passes (included by fused.cu): one block per work item (tile x
// field or component), the tile in registers throughout (tile.cuh).  An Op
// supplies
//   coords(item, o, c0, c)  the item's tile (other index o, first column c0)
//                           and component c
//   src(c), dst(c)          its input and output fields
//   pre(v, ...)             spectral factors on the loaded values (kPre)
//   post(v, ...)            factors on the transformed values (kPost)
// and may name its input (kNatIn) or output (kNatOut) as a caller's field in
// natural order.
// Consecutive items run at the same time on consecutive blocks, so items
// that share an input tile (one phi tile for the M filters, the 2LPT
// components) are next to each other and hit L2.
#pragma once
// (included inside namespace aar)

template <int N, int AXIS, int SIGN, class Op>
__global__ void __launch_bounds__(TileCfg<N>::THREADS, TileCfg<N>::MINB) k_pass(const __grid_constant__ Op op,
                                                                                       const float2* __restrict__ tw2) {
  using C = TileCfg<N>;
  extern __shared__ float2 ex[];
  const int w = threadIdx.x % C::W, t = threadIdx.x / C::W;
  int o, c0, c;
  op.coords(blockIdx.x, o, c0, c);
  const TileMap<N, AXIS> tm(o, c0, t, w);
  float2 v[C::R1];
  if constexpr (requires { Op::kNatIn; }) {
    static_assert(AXIS == 0);
    const bool in = c0 + w <= N / 2;
    const float2* src = op.src(c) + NatMap<N>::base(o, c0, t, w);
#pragma unroll
    for (int r = 0; r < C::R1; ++r) v[r] = in ? src[NatMap<N>::off(C::T * r)] : make_float2(0.f, 0.f);
  } else {
    const float2* src = op.src(c) + tm.base;
#pragma unroll
    for (int r = 0; r < C::R1; ++r) v[r] = src[TileMap<N, AXIS>::off(C::T * r)];
  }
  if constexpr (Op::kPre) op.pre(v, o, c0 + w, c, t);
  tile_fft2<N, SIGN>(v, ex, t, w, tw2);
  if constexpr (Op::kPost) op.post(v, o, c0 + w, c, t);
  if constexpr (requires { Op::kNatOut; }) {
    static_assert(AXIS == 0);
    if (c0 + w > N / 2) return;
    float2* dst = op.dst(c) + NatMap<N>::base(o, c0, t, w);
#pragma unroll
    for (int b = 0; b < C::G; ++b)
#pragma unroll
      for (int r = 0; r < C::R2; ++r) dst[NatMap<N>::off(C::T * b + C::R1 * r)] = v[b * C::R2 + r];
  } else {
    float2* dst = op.dst(c) + tm.base;
#pragma unroll
    for (int b = 0; b < C::G; ++b)
#pragma unroll
      for (int r = 0; r < C::R2; ++r) dst[TileMap<N, AXIS>::off(C::T * b + C::R1 * r)] = v[b * C::R2 + r];
  }
}

__device__ __forceinline__ float half_weight(int kz, int N) { return kz == 0 || kz == N / 2 ? 1.f : 2.f; }

// Noise amplitude of the cells the draw writes (main.c:405-459), else 0
__device__ __forceinline__ float gauss_amp(const Grid& g, const float* __restrict__ amp, int x, int y, int kx, int ky,
                                           int kz) {
  const int N = g.N, n2 = kx * kx + ky * ky + kz * kz;
  const bool on = x != N / 2 && y != N / 2 && kz < N / 2 && n2 != 0 && keep_cell(g, kx, ky, kz);
  return on ? __ldg(amp + n2) : 0.f;
}

template <int N>
__device__ __forceinline__ void tile_coords(unsigned tile, int& o, int& c0) {
  o = (int)(tile / TileCfg<N>::NCOL);
  c0 = (int)(tile % TileCfg<N>::NCOL) * TileCfg<N>::W;
}

// Field slots of a pass (indexed in the kernel's parameter space).
struct Slots {
  int s[kMaxModes];
};

// In-place complex FFT of the fields slot.s[f], items f * tiles + tile.
template <int N>
struct AxisOp {
  static constexpr bool kPre = false, kPost = false;
  float2* base;
  int64_t fs;
  Slots slot;
  __device__ void coords(unsigned item, int& o, int& c0, int& c) const {
    const unsigned f = item / TileCfg<N>::TILES;
    tile_coords<N>(item - f * TileCfg<N>::TILES, o, c0);
    c = slot.s[f];
  }
  __device__ const float2* src(int c) const { return base + (int64_t)c * fs; }
  __device__ float2* dst(int c) const { return base + (int64_t)c * fs; }
};

// x pass from a caller's natural-order spectrum into a plan field, and from a
// plan field into one.
template <int N>
struct XNatInOp {
  static constexpr bool kPre = false, kPost = false, kNatIn = true;
  const float2* in;
  float2* out;
  __device__ void coords(unsigned item, int& o, int& c0, int& c) const {
    tile_coords<N>(item, o, c0);
    c = 0;
  }
  __device__ const float2* src(int) const { return in; }
  __device__ float2* dst(int) const { return out; }
};
template <int N>
struct XNatOutOp {
  static constexpr bool kPre = false, kPost = false, kNatOut = true;
  const float2* in;
  float2* out;
  __device__ void coords(unsigned item, int& o, int& c0, int& c) const {
    tile_coords<N>(item, o, c0);
    c = 0;
  }
  __device__ const float2* src(int) const { return in; }
  __device__ float2* dst(int) const { return out; }
};

// Item order of the passes that write several output fields from one input
// tile: groups of `grp` consecutive tiles, and within a group all tiles of
// output 0, then all of output 1, ...; a group's input tiles stay in L2
// while its outputs are produced.
template <int N>
__device__ __forceinline__ void group_order(unsigned item, unsigned nc, unsigned grp, unsigned& t, int& c) {
  constexpr unsigned tiles = TileCfg<N>::TILES;
  const unsigned span = grp * nc;
  const unsigned g = item / span, r = item - g * span;
  const unsigned gs = min(grp, tiles - g * grp);  // the last group may be short
  c = (int)(r / gs);
  t = g * grp + (r - (unsigned)c * gs);
}

// Order of a cube of per-cell factors over |kx|, |ky|, kz <= N/2 (K = N/2 + 1
// each), `planes` of them: the columns kz < N/2 as [p][|ky|][kz / 8][|kx|][8], so
// that a warp's factors of a value index are 4 rows of 8 consecutive floats on
// 32-byte boundaries, then the columns kz = N/2 as [p][|ky|][|kx|].  (With that
// column padded to a block of its own a cube took 1.4 % more at N = 1024, 21 %
// at 64, which a plan's memory limit may not have.)
struct CubeMap {
  int K, planes;
  __host__ __device__ __forceinline__ int64_t at(int p, int ay, int kz, int ax) const {
    const int NB = (K - 1) / 8;
    const int64_t row = (int64_t)p * K + ay;
    return kz < K - 1 ? ((row * NB + kz / 8) * K + ax) * 8 + kz % 8 : ((int64_t)planes * K * NB * 8 + row) * K + ax;
  }
  // the cell of index i < K^3 of a one-plane cube
  __host__ __device__ __forceinline__ void cell(int64_t i, int& ax, int& ay, int& kz) const {
    const int NB = (K - 1) / 8;
    const int64_t blocks = (int64_t)K * NB * K * 8;
    if (i < blocks) {
      const int64_t r = i / 8, s = r / K;
      ax = (int)(r % K), kz = (int)(s % NB) * 8 + (int)(i % 8), ay = (int)(s / NB);
    } else {
      ax = (int)((i - blocks) % K), kz = K - 1, ay = (int)((i - blocks) / K);
    }
  }
};

// A thread's factors f[i] at kx of line value i, |ky| = ay and column kz of
// plane p; zero on the padding columns.
template <int N>
__device__ __forceinline__ void cube_load(float* f, const float* __restrict__ cube, int planes, int p, int ay, int kz,
                                          int t) {
  using C = TileCfg<N>;
  const float* q = cube + CubeMap{N / 2 + 1, planes}.at(p, ay, min(kz, N / 2), 0);
  auto load = [&](auto step) {
#pragma unroll
    for (int i = 0; i < C::R1; ++i) {
      // value i < R1 / 2 has kx = t + T i < N / 2, the others |kx| = N - n
      const int n = tile_n<N>(t, i);
      f[i] = __ldg(q + (i < C::R1 / 2 ? n : N - n) * decltype(step)::value);
    }
  };
  if (kz < N / 2) {
    load(std::integral_constant<int, 8>{});
  } else {
    load(std::integral_constant<int, 1>{});
    if (kz > N / 2) {
#pragma unroll
      for (int i = 0; i < C::R1; ++i) f[i] = 0.f;
    }
  }
}

// First modal pass: phi tile times q_p(k) (zero on the cut, DC and padding
// columns), inverse x FFT, into field dst0 + p, for the modes p = mode.s[c] that
// the products read.  The factors come from the plan's
// filter cube (qcube_build); they load together with the tile.
template <int N>
struct XinvOp {
  static constexpr bool kPre = true, kPost = false;
  const float2* phi;
  float2* work;
  int64_t fs;
  int nin;
  Slots mode;
  unsigned grp;
  int dst0, planes;
  const float* qcube;
  __device__ void coords(unsigned item, int& o, int& c0, int& c) const {
    unsigned t;
    group_order<N>(item, (unsigned)nin, grp, t, c);
    tile_coords<N>(t, o, c0);
  }
  __device__ const float2* src(int) const { return phi; }
  __device__ float2* dst(int c) const { return work + (int64_t)(dst0 + mode.s[c]) * fs; }
  __device__ void pre(float2* v, int o, int kz, int c, int t) const {
    using C = TileCfg<N>;
    float f[C::R1];
    cube_load<N>(f, qcube, planes, mode.s[c], o <= N / 2 ? o : N - o, kz, t);
#pragma unroll
    for (int i = 0; i < C::R1; ++i) v[i] = cscale(v[i], f[i]);
  }
};

template <int N>
struct XinvNatOp : XinvOp<N> {  // phi in the caller's natural order
  static constexpr bool kNatIn = true;
};
// The transposed chain's passes from T, which carries rho_0 Fnl / N^3 (w the
// weights of the half spectrum): rho_r = q_r rho_0 but for r = 3, which takes G
// itself on the kept cells, where q_3 > 0.
template <int N>
struct XinvGradOp : XinvOp<N> {
  const float2* G;
  float fnl_n3;
  __device__ const float2* src(int c) const { return this->mode.s[c] == 3 ? G : this->phi; }
  __device__ void pre(float2* v, int o, int kz, int c, int t) const {
    using C = TileCfg<N>;
    float f[C::R1];
    cube_load<N>(f, this->qcube, this->planes, this->mode.s[c], o <= N / 2 ? o : N - o, kz, t);
    const bool one = this->mode.s[c] == 3;
    const float s = fnl_n3 / half_weight(kz, N);
#pragma unroll
    for (int i = 0; i < C::R1; ++i) v[i] = cscale(v[i], !one ? f[i] : f[i] > 0.f ? s : 0.f);
  }
};

// 2LPT x passes.  The spectral factors of main.c:1180-1368 are products of
// one factor per axis, except T/(D Beta), which the transfer cube brings (laid
// out as the filter cube, so phi needs no scaled copy), and 1/k^2 of psi2,
// which the forward x pass of the source applies (XfwdInvK2Op); so an x pass
// writes one field per distinct x factor and a fan-out y pass (YFanOp) and
// the c2r rows (ZFac) apply the rest.  KIND 0, Hessians d_ab = -k_a k_b T/(D
// Beta) phi: x factors -kF^2 kx^2, -kF^2 kx, -kF^2 (3 outputs).  KIND 1,
// displacements i k_a smth on T/(D Beta) phi (psi1, outputs 0 and 1) and on
// -S/k^2 (psi2, 2 and 3), smth = [sinc_x sinc_y sinc_z]^-2: x factors
// i kF kx / sinc_x^2 and i / sinc_x^2.  Items in group_order over the outputs.
// Bound by the fields' bytes.  A scaled copy of phi and two passes for the
// displacements took 13.7 ms at 1024^3 and 1.72 at 512^3; these two passes take
// 11.4 and 1.30, and 16.3 and 1.83 where the factor is read by |n|^2 (a
// gather: neighbouring kz lie 2 kz + 1 entries apart).
template <int N, int KIND>
struct LptXOp {
  static constexpr bool kPre = true, kPost = false;
  static constexpr int NC = KIND == 0 ? 3 : 4;
  const float2* phi;
  const float2* s;  // psi2's input
  float2* work;
  int64_t fs;
  int out[4];
  unsigned grp;
  float kF;
  const float* isinc2;
  const float* tcube;  // one plane; null: twb by |n|^2
  const float* twb;
  __device__ void coords(unsigned item, int& o, int& c0, int& c) const {
    unsigned t;
    group_order<N>(item, NC, grp, t, c);
    tile_coords<N>(t, o, c0);
  }
  __device__ const float2* src(int c) const { return KIND == 1 && c >= 2 ? s : phi; }
  __device__ float2* dst(int c) const { return work + (int64_t)out[c] * fs; }
  __device__ void pre(float2* v, int o, int kz, int c, int t) const {
    using C = TileCfg<N>;
    const int ay = o <= N / 2 ? o : N - o;
    const bool psi2 = KIND == 1 && c >= 2;
    float f[C::R1];
    if (psi2 || kz > N / 2) {
#pragma unroll
      for (int i = 0; i < C::R1; ++i) f[i] = kz <= N / 2 ? 1.f : 0.f;
    } else if (tcube) {
      cube_load<N>(f, tcube, 1, 0, ay, kz, t);
    } else {
      const int b = ay * ay + kz * kz;
#pragma unroll
      for (int i = 0; i < C::R1; ++i) {
        const int n = tile_n<N>(t, i), ax = i < C::R1 / 2 ? n : N - n;
        f[i] = __ldg(twb + b + ax * ax);
      }
    }
#pragma unroll
    for (int i = 0; i < C::R1; ++i) {
      const int n = tile_n<N>(t, i);
      const float kx = (float)(i < C::R1 / 2 ? n : n - N);
      if (KIND == 0) {
        f[i] *= c == 0 ? -kF * kF * kx * kx : c == 1 ? -kF * kF * kx : -kF * kF;
        v[i] = make_float2(v[i].x * f[i], v[i].y * f[i]);
      } else {
        const float is2 = __ldg(isinc2 + n);
        f[i] *= (c & 1) == 0 ? kF * kx * is2 : is2;
        v[i] = make_float2(-f[i] * v[i].y, f[i] * v[i].x);
      }
    }
  }
};
template <int N>
struct LptXNatOp : LptXOp<N, 0> {  // phi in the caller's natural order
  static constexpr bool kNatIn = true;
};

// Inverse y pass fanning fields out: item (tile, c), c < NC: field in[c]
// times the y factor type[c] (axis_table, axis_poly), inverse y FFT, into out[c].
// Outputs never alias an input that another item still reads (an in-place
// output reads only its own input).
template <int N>
struct YFanOp {
  static constexpr bool kPre = true, kPost = false;
  static constexpr int NC = 6;
  float2* work;
  int64_t fs;
  int in[NC], out[NC], type[NC];
  unsigned grp;
  float kF;
  const float* isinc2;
  __device__ void coords(unsigned item, int& o, int& c0, int& c) const {
    unsigned t;
    group_order<N>(item, NC, grp, t, c);
    tile_coords<N>(t, o, c0);
  }
  __device__ const float2* src(int c) const { return work + (int64_t)in[c] * fs; }
  __device__ float2* dst(int c) const { return work + (int64_t)out[c] * fs; }
  __device__ void pre(float2* v, int, int, int c, int t) const {
    using C = TileCfg<N>;
    // (a branch and a load per value left the loads one after another: 15.7
    // vs 9.9 ms for the displacements at 1024^3)
    const int ty = type[c];
    float f[C::R1];
#pragma unroll
    for (int i = 0; i < C::R1; ++i) f[i] = axis_table(ty, isinc2, tile_n<N>(t, i));
#pragma unroll
    for (int i = 0; i < C::R1; ++i) {
      const float k = (float)(i < C::R1 / 2 ? tile_n<N>(t, i) : tile_n<N>(t, i) - N);
      v[i] = cscale(v[i], axis_poly(ty, k, kF) * f[i]);
    }
  }
};

// Forward x pass of the 2LPT source in place, then S <- -S / (kF^2 |k|^2)
// (0 at k = 0): the non-separable part of psi2 = -i k_a / k^2 S smth
// (main.c:1356-1363).
template <int N>
struct XfwdInvK2Op {
  static constexpr bool kPre = false, kPost = true;
  float2* f;
  float kF;
  __device__ void coords(unsigned item, int& o, int& c0, int& c) const {
    tile_coords<N>(item, o, c0);
    c = 0;
  }
  __device__ const float2* src(int) const { return f; }
  __device__ float2* dst(int) const { return f; }
  __device__ void post(float2* v, int o, int kz, int, int t) const {
    using C = TileCfg<N>;
    const int ky = sidx(o, N);
#pragma unroll
    for (int b = 0; b < C::G; ++b)
#pragma unroll
      for (int r = 0; r < C::R2; ++r) {
        const int i = tile_out_i<N>(b, r), n = tile_n<N>(t, i);
        const int kx = i < C::R1 / 2 ? n : n - N;
        const int n2 = kx * kx + ky * ky + kz * kz;
        const float g = n2 ? -1.f / (kF * kF * (float)n2) : 0.f;
        v[b * C::R2 + r] = cscale(v[b * C::R2 + r], g);
      }
  }
};

// keep_cell with the cells on the sphere's boundary, which take FP64, looked up in
// the filter cube: q_0 is 1 inside the cut and 0 outside.  (Unrolled over the
// values the FP64 code made k_xacc slower: 512^3, three slots, 0.96 ms against 0.78;
// 64^3 and 32^3, 2 to 4 us.)
template <int N>
__device__ __forceinline__ bool keep_cube(const Grid& g, const float* __restrict__ qcube, int planes, int kx, int ky,
                                          int kz) {
  if (!g.sphere) return abs(kx) <= g.kcut && abs(ky) <= g.kcut && kz <= g.kcut;
  const int n2 = kx * kx + ky * ky + kz * kz;
  if (n2 != g.nsq_bnd) return n2 < g.nsq_bnd;
  return __ldg(qcube + CubeMap{N / 2 + 1, planes}.at(0, abs(ky), kz, abs(kx))) > 0.f;
}
// The same for a thread's line, bit i value i, the lookups out of line: with 32
// values keep_cube at each spills (512^3, 11 slots: 2.01 ms against 1.88), with 16 the
// mask does (256^3, a potential with 19 slots: 2255 us against 2245).
template <int N>
__device__ __forceinline__ unsigned keep_mask(const Grid& g, const float* __restrict__ qcube, int planes, int t, int ky,
                                              int kz) {
  using C = TileCfg<N>;
  auto kx = [&](int i) { return i < C::R1 / 2 ? tile_n<N>(t, i) : tile_n<N>(t, i) - N; };
  unsigned m = 0;
  if (!g.sphere) {
    if (abs(ky) > g.kcut || kz > g.kcut) return 0;
#pragma unroll
    for (int i = 0; i < C::R1; ++i) m |= (abs(kx(i)) <= g.kcut ? 1u : 0u) << i;
    return m;
  }
  const int b = g.nsq_bnd - ky * ky - kz * kz;
  bool edge = false;
#pragma unroll
  for (int i = 0; i < C::R1; ++i) {
    const int k2 = kx(i) * kx(i);
    m |= (k2 < b ? 1u : 0u) << i;
    edge |= k2 == b;
  }
  if (edge) {
#pragma unroll 1
    for (int i = 0; i < C::R1; ++i)
      if (kx(i) * kx(i) == b && keep_cube<N>(g, qcube, planes, kx(i), ky, kz)) m |= 1u << i;
  }
  return m;
}

// Last modal step: forward x pass of every active slot and the accumulation,
// phi <- phi + fnl_n3 sum_r rho_r(k) g_r(k), DC = 0 (main.c:825-867,
// 1101-1126).  rho_r = q_r k^(ns - 4) for every r (main.c:580-637, 833-860), so
// the sum takes the filter cube's factors and then rho_0 = k^(ns - 4), both
// rounded once from 64 bits; rho_3 = 1, so r = 3 comes last and takes neither.
// (k^(ns - 4) as an FP32 power of |k|^2 was up to 1.7e-6 off.)  One
// block per tile walks the slots: the tile of the next slot comes in through
// shared memory (from N = 256 on) while one is transformed, the compensated
// sums (two_sum2) stay in registers -- the transformed slots never go back to
// memory, where a forward x pass and a pointwise accumulation moved them
// three more times.  Cut cells keep phi.
//
// GRAD: the last step of the transposed chain (chain.cuh) instead.
//
// What bounds it: instruction issue of the 8 (N >= 512) to 16 warps that
// 32 values, their sums and compensations leave room for.  Against the forward
// x pass and the specialised pointwise accumulation: 0.39 -> 0.23 ms (256^3, 12
// slots), 0.71 -> 0.33 (256^3, 19), 3.39 -> 1.88 (512^3, 11), 48.1 -> 35.3
// (1024^3, 19).
template <int N>
struct XaccArgs {
  Grid g;
  float2* phi;
  const float2* work;
  int64_t fs;
  int nr, nw;  // active r; the first nw of them are weighted (all but r = 3)
  Slots slot;  // the active r: field and cube plane
  int planes;
  const float* qcube;
  const float* rho0;  // per |k|^2
  float fnl_n3;
  // gradient form (k_xacc<N, true>): gw = amp (phi + w sum) in natural order,
  // w = 1 on the kz = 0 and N/2 planes, else 2
  const float* amp;
  float2* gw;
};
template <int N>
struct XaccCfg {
  using C = TileCfg<N>;
  static constexpr bool kStaged = N >= 256;
  // the weights, too: 512^3 with 11 slots 1.91 -> 1.88 ms; at 256^3, where more warps
  // hide a thread's own gather, a potential with 19 slots 2251 against 2243 us
  static constexpr bool kStagedW = kStaged && C::R1 == 32;
  static constexpr int K = N / 2 + 1;
  static constexpr size_t QROWS = (size_t)K * C::W;  // floats of a plane's block of columns
  static constexpr size_t SMEM = C::SMEM + (kStaged ? sizeof(float2) * N * C::W + 2 * sizeof(float) * QROWS : 0);
  static constexpr int MINB = C::R1 == 32 ? 256 / C::THREADS : C::R1 == 16 ? 512 / C::THREADS : 8;
};
template <int N, bool GRAD>
__global__ void __launch_bounds__(TileCfg<N>::THREADS, XaccCfg<N>::MINB)
    k_xacc(const __grid_constant__ XaccArgs<N> a, const float2* __restrict__ tw2) {
  using C = TileCfg<N>;
  using X = XaccCfg<N>;
  extern __shared__ float2 ex[];
  const int w = threadIdx.x % C::W, t = threadIdx.x / C::W;
  int o, c0;
  tile_coords<N>(blockIdx.x, o, c0);
  const int64_t base = TileMap<N, 0>(o, c0, t, w).base;
  const int ay = o <= N / 2 ? o : N - o;
  // a block of eight columns, or (last) the column kz = N/2 alone: the sums of
  // the padding columns beside it are not stored
  const bool last = c0 == N / 2;
  const int qw = last ? 0 : w;
  auto qplane = [&](int s) { return a.qcube + CubeMap{X::K, a.planes}.at(a.slot.s[s], ay, c0, 0); };
  float2* stage = ex + C::SMEM / sizeof(float2);
  float* qs = reinterpret_cast<float*>(stage + N * C::W);  // two buffers
  const int kz = c0 + w, ky = sidx(o, N);
  // rho_0 is taken into the sums behind the last weighted slot
  const bool weighted = !GRAD && a.nw > 0;
  auto issue = [&](int s) {
    if (s < a.nr) tile_stage_load<N, 0>(stage, a.work + (int64_t)a.slot.s[s] * a.fs, o, c0);
    float* d = qs + (s & 1) * X::QROWS;
    if (GRAD || s < a.nw) {
      const float* q = qplane(s);
      if (last)
        for (int i = threadIdx.x; i < X::K; i += C::THREADS) cp_async4(d + C::W * i, q + i);
      else
        for (int i = threadIdx.x; i < (int)X::QROWS / 4; i += C::THREADS) cp_async16(d + 4 * i, q + 4 * i);
    } else if (X::kStagedW && weighted) {
      // s = nw, r = 3 or none: the buffer takes the tile's weights, a gather per
      // |kx| and column while the slot before is transformed
      const int b = ky * ky;
      for (int i = threadIdx.x; i < (int)X::QROWS; i += C::THREADS) {
        const int ax = i / C::W, z = c0 + i % C::W;
        cp_async4(d + i, a.rho0 + (z <= N / 2 ? ax * ax + b + z * z : 0));
      }
    }
    cp_async_commit();
  };
  float2 sum[C::R1], cmp[C::R1];
#pragma unroll
  for (int i = 0; i < C::R1; ++i) sum[i] = cmp[i] = make_float2(0.f, 0.f);
  if constexpr (X::kStaged) issue(0);
  auto weight = [&](int t0, int i) {
    const int n = tile_n<N>(t0, i), ax = i < C::R1 / 2 ? n : N - n;
    if constexpr (X::kStagedW) return qs[(a.nw & 1) * X::QROWS + ax * C::W + w];
    else return kz <= N / 2 ? __ldg(a.rho0 + (ax * ax + ky * ky + kz * kz)) : 0.f;
  };
#pragma unroll 1
  for (int s = 0;; ++s) {
    if constexpr (X::kStaged)
      if (s < a.nr || (X::kStagedW && weighted)) {
        cp_async_wait<0>();
        __syncthreads();
      }
    if (weighted && s == a.nw) {
      // the sums so far, as the exact products' leading and trailing parts
      constexpr int H = 8 < C::R1 ? 8 : C::R1;  // values whose loads go out together
      int tt = t;
      asm volatile("" : "+r"(tt));  // keeps the indices out of the loop over slots (they would spill)
#pragma unroll
      for (int h = 0; h < C::R1; h += H) {
        float f[H];
#pragma unroll
        for (int j = 0; j < H; ++j) f[j] = weight(tt, h + j);
#pragma unroll
        for (int j = 0; j < H; ++j) {
          const int i = h + j;
          const float2 u = cscale(sum[i], f[j]);
          cmp[i] = make_float2(fmaf(cmp[i].x, f[j], fmaf(sum[i].x, f[j], -u.x)),
                               fmaf(cmp[i].y, f[j], fmaf(sum[i].y, f[j], -u.y)));
          sum[i] = u;
        }
      }
    }
    if (s == a.nr) break;
    float2 v[C::R1];
    const float* q;
    if constexpr (X::kStaged) {
#pragma unroll
      for (int r = 0; r < C::R1; ++r) v[r] = stage[tile_n<N>(t, r) * C::W + w];
      __syncthreads();  // the stage is free, and the exchange of the slot before has been read
      if (s + 1 < a.nr || (X::kStagedW && weighted && s + 1 == a.nw)) issue(s + 1);
      q = qs + (s & 1) * X::QROWS + qw;
    } else {
      const float2* src = a.work + (int64_t)a.slot.s[s] * a.fs + base;
#pragma unroll
      for (int r = 0; r < C::R1; ++r) v[r] = src[TileMap<N, 0>::off(C::T * r)];
      if (s) __syncthreads();  // the exchange has been read
      q = qplane(s) + qw;
    }
    tile_fft2<N, -1>(v, ex, t, w, tw2);
#pragma unroll
    for (int b = 0; b < C::G; ++b)
#pragma unroll
      for (int r = 0; r < C::R2; ++r) {
        const int i = tile_out_i<N>(b, r), n = tile_n<N>(t, i);
        const int ax = i < C::R1 / 2 ? n : N - n;
        const float f = !GRAD && s >= a.nw ? 1.f : q[X::kStaged || !last ? ax * C::W : ax];
        two_sum2(sum[i], cmp[i], cscale(v[b * C::R2 + r], f));
      }
  }
  if (kz > N / 2) return;
  float2* phi = a.phi + base;
  float2 u[C::R1];  // all loads first: behind one another's stores they cost 9 ms at 1024^3
#pragma unroll
  for (int i = 0; i < C::R1; ++i) u[i] = phi[TileMap<N, 0>::off(C::T * i)];
  constexpr bool kMask = !GRAD && C::R1 == 32;
  const unsigned keep = kMask ? keep_mask<N>(a.g, a.qcube, a.planes, t, ky, kz) : 0u;
#pragma unroll
  for (int i = 0; i < C::R1; ++i) {
    const int n = tile_n<N>(t, i);
    const int kx = i < C::R1 / 2 ? n : n - N;
    const float2 d = add2(sum[i], cmp[i]);
    if constexpr (GRAD) {
      const float h = half_weight(kz, N), m = gauss_amp(a.g, a.amp, n, o, kx, ky, kz);
      a.gw[NatMap<N>::base(o, c0, n, w)] = make_float2(m * fmaf(h, d.x, u[i].x), m * fmaf(h, d.y, u[i].y));
      continue;
    }
    float2 r = make_float2(fmaf(a.fnl_n3, d.x, u[i].x), fmaf(a.fnl_n3, d.y, u[i].y));
    if (kMask ? !(keep >> i & 1u) : !keep_cube<N>(a.g, a.qcube, a.planes, kx, ky, kz)) r = u[i];
    if (kx == 0 && ky == 0 && kz == 0) r = make_float2(0.f, 0.f);
    phi[TileMap<N, 0>::off(C::T * i)] = r;
  }
}

// The same with a single active r (Local templates): nothing to accumulate,
// so a pass of its own with the plain passes' occupancy.  ONE: r = 3, rho = 1.
template <int N, bool ONE>
struct XaddOp {
  static constexpr bool kPre = false, kPost = true;
  Grid g;
  float2* phi;
  const float2* slot;
  const float* rho;  // per |k|^2
  float fnl_n3;
  __device__ void coords(unsigned item, int& o, int& c0, int& c) const {
    tile_coords<N>(item, o, c0);
    c = 0;
  }
  __device__ const float2* src(int) const { return slot; }
  __device__ float2* dst(int) const { return phi; }
  __device__ void post(float2* v, int o, int kz, int, int t) const {
    using C = TileCfg<N>;
    const int ky = sidx(o, N);
    const float2* ph = phi + TileMap<N, 0>(o, kz, t, 0).base;
    constexpr int H = 8 < C::R1 ? 8 : C::R1;  // values whose loads go out together
#pragma unroll
    for (int h = 0; h < C::R1; h += H) {
      float2 u[H];
      float f[H];
#pragma unroll
      for (int j = 0; j < H; ++j) {
        const int i = h + j, n = tile_n<N>(t, i), kx = i < C::R1 / 2 ? n : n - N;
        u[j] = ph[TileMap<N, 0>::off(C::T * i)];
        f[j] = ONE ? 1.f : __ldg(rho + (kz <= N / 2 ? kx * kx + ky * ky + kz * kz : 0));
      }
#pragma unroll
      for (int j = 0; j < H; ++j) {
        const int i = h + j, n = tile_n<N>(t, i);
        const int kx = i < C::R1 / 2 ? n : n - N;
        float2& x = v[(i % C::G) * C::R2 + i / C::G];  // tile_out_i
        float2 r = make_float2(fmaf(fnl_n3, x.x * f[j], u[j].x), fmaf(fnl_n3, x.y * f[j], u[j].y));
        if (kz > N / 2 || !keep_cell(g, kx, ky, kz)) r = u[j];
        if (kx == 0 && ky == 0 && kz == 0) r = make_float2(0.f, 0.f);
        x = r;
      }
    }
  }
};
