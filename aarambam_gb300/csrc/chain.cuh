// The differentiable chain (included by fused.cu): white noise w -> amp w ->
// modal potential -> 2LPT displacement field, and its transpose in one go, in
// the plan's row order from the first pass to the last one.
//
// Transposes on half spectra: adjoint.cu.  With X_a = r2c(gdisp_a) and the
// cell factors of spectral.cuh, both displacement fields see X_a through D =
// sum_a k_a X_a alone, the six Hessians' gradients are summed along the axes
// the forward fan-out split them on, rho_r = q_r k^(ns - 4) makes the products'
// gradients filter passes of one field, and the last forward x pass sums over
// the modes (k_xacc): 2 M + 13 transforms with no copies between row orders
// and no pass per component over the spectra.  Against the chain composed
// of aar_c2r, aar_r2c and aar_adj_*: 256^3, 10 modes, field and gradients 15.4
// -> 7.3 ms; 64^3, where some 240 launches waited for the host, 2.7 -> 0.46 ms.
#pragma once
// (included inside namespace aar)

// x, y, kz of half-spectrum element i of the plan's rows (K = N/2 + 1 per row)
// and its offset in a field
template <int N>
__device__ __forceinline__ int64_t spec_cell(int64_t i, int HP, int& x, int& y, int& kz) {
  constexpr int K = N / 2 + 1;
  const int64_t row = i / K;
  kz = (int)(i - row * K);
  row_xy(row, N, kXB, x, y);
  return row * HP + kz;
}
template <int N>
__device__ __forceinline__ int64_t nat_cell(int x, int y, int kz) {
  return ((int64_t)x * N + y) * (N / 2 + 1) + kz;
}

// Gaussian potential amp w, into the plan's spectrum and the caller's.
template <int N>
__global__ void __launch_bounds__(256) k_chain_gauss(Grid g, const float* __restrict__ amp,
                                                     const float2* __restrict__ w, float2* phik, float2* phig) {
  constexpr int64_t total = (int64_t)N * N * (N / 2 + 1);
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
    int x, y, kz;
    const int64_t e = spec_cell<N>(i, g.HP, x, y, kz), n = nat_cell<N>(x, y, kz);
    const float2 r = cscale(w[n], gauss_amp(g, amp, x, y, sidx(x, N), sidx(y, N), kz));
    phik[e] = r;
    phig[n] = r;
  }
}

// Displacement psi1 - c psi2 from the plan's six real fields, natural order.
template <int N>
__global__ void __launch_bounds__(256) k_chain_disp(const float* __restrict__ work, int64_t fsr, int HP, float c,
                                                    float* __restrict__ disp) {
  constexpr int64_t n3 = (int64_t)N * N * N;
  const int a = blockIdx.y;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n3; i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t row = i / N;
    const int z = (int)(i - row * N);
    int x, y;
    row_xy(row, N, kXB, x, y);
    const float* f = work + row * 2 * HP + z;
    disp[a * n3 + ((int64_t)x * N + y) * N + z] = f[a * fsr] + c * f[(a + 3) * fsr];
  }
}

// D = sum_a k_a X_a of the displacement gradients X_a (fields 0..2 of X):
//   G = conj(F1) w X summed = -i kF T/(D Beta) smth w D          (psi1)
//   T = c conj(F2) X summed =  i c smth / (kF k^2) D (0 at k = 0) (psi2's
// source, over the 1/w of the c2r that takes it to real space).
template <int N>
__global__ void __launch_bounds__(256) k_chain_div(LptArgs a, const float2* __restrict__ X, int64_t fs, float c,
                                                   float2* __restrict__ G, float2* __restrict__ T) {
  constexpr int64_t total = (int64_t)N * N * (N / 2 + 1);
  const float kF = a.m.g.kF;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
    int x, y, kz;
    const int64_t e = spec_cell<N>(i, a.m.g.HP, x, y, kz);
    const int kx = sidx(x, N), ky = sidx(y, N), n2 = kx * kx + ky * ky + kz * kz;
    const float2 X0 = X[e], X1 = X[fs + e], X2 = X[2 * fs + e];
    const float fx = (float)kx, fy = (float)ky, fz = (float)kz;
    const float2 D = make_float2(fx * X0.x + fy * X1.x + fz * X2.x, fx * X0.y + fy * X1.y + fz * X2.y);
    const float smth = __ldg(a.isinc2 + x) * __ldg(a.isinc2 + y) * __ldg(a.isinc2 + kz);
    const float g = kF * __ldg(a.twb + n2) * smth * half_weight(kz, N);
    const float s = n2 ? c * smth / (kF * (float)n2) : 0.f;
    G[e] = make_float2(g * D.y, -g * D.x);
    T[e] = make_float2(-s * D.y, s * D.x);
  }
}

// Transpose of the 2LPT source rows: lines 0..5 the Hessians d00 d01 d02 d11
// d12 d22 (z factors as SourceRowOp), line 6 the source gradient g; the six
// gradients over the Hessians' lines and fields, their z factors again on the
// way out.
struct SourceAdjRowOp {
  static constexpr bool kPairs = true;
  static constexpr bool kZfac = true, kZfacOut = true;
  int src_slot;
  float kF;
  const float* isinc2;
  __device__ ZFac zfac(int l) const { return ZFac{l == 2 || l == 4 ? 1 : l == 5 ? 2 : 0, kF, isinc2}; }
  __device__ int nin() const { return 7; }
  __device__ int nlines() const { return 7; }
  __device__ int in_slot(int l) const { return l == 6 ? src_slot : l; }
  __device__ int in_line(int l) const { return l; }
  __device__ int nout() const { return 6; }
  __device__ int out_line(int l) const { return l; }
  __device__ int out_slot(int l) const { return l; }
  template <int K>
  __device__ void combine(float2* sm, const int* pos, int LS) const {
#pragma unroll
    for (int i = 0; i < K; ++i) {
      float2 d[7];
#pragma unroll
      for (int c = 0; c < 7; ++c) d[c] = sm[c * LS + pos[i]];
      const float2 g = d[6], m = make_float2(-2.f * g.x, -2.f * g.y);
      sm[0 * LS + pos[i]] = make_float2(g.x * (d[3].x + d[5].x), g.y * (d[3].y + d[5].y));
      sm[1 * LS + pos[i]] = make_float2(m.x * d[1].x, m.y * d[1].y);
      sm[2 * LS + pos[i]] = make_float2(m.x * d[2].x, m.y * d[2].y);
      sm[3 * LS + pos[i]] = make_float2(g.x * (d[0].x + d[5].x), g.y * (d[0].y + d[5].y));
      sm[4 * LS + pos[i]] = make_float2(m.x * d[4].x, m.y * d[4].y);
      sm[5 * LS + pos[i]] = make_float2(g.x * (d[0].x + d[3].x), g.y * (d[0].y + d[3].y));
    }
  }
};
constexpr int kSevenThreads = 224;
template <int N>
__global__ void __launch_bounds__(kSevenThreads, two_stage_r1(N) == 32 ? 2 : 4)
    k_rows_source_adj(const __grid_constant__ SourceAdjRowOp op, float2* work, int64_t fs, int HP, int64_t nrows,
                      const float2* __restrict__ tw2) {
  rows_pairs<N, SourceAdjRowOp, kSevenThreads>(op, work, fs, HP, nrows, tw2, 32 / PairCfg<N>::T);
}

// Forward y pass of the Hessian gradients in place with their y factors:
// field c gets the polynomial of type ty.s[c].
template <int N>
struct YAdjOp {
  static constexpr bool kPre = false, kPost = true;
  float2* base;
  int64_t fs;
  Slots ty;
  __device__ void coords(unsigned item, int& o, int& c0, int& c) const {
    c = (int)(item / TileCfg<N>::TILES);
    tile_coords<N>(item - c * TileCfg<N>::TILES, o, c0);
  }
  __device__ const float2* src(int c) const { return base + (int64_t)c * fs; }
  __device__ float2* dst(int c) const { return base + (int64_t)c * fs; }
  __device__ void post(float2* v, int, int, int c, int t) const {
    using C = TileCfg<N>;
    const int type = ty.s[c];
#pragma unroll
    for (int b = 0; b < C::G; ++b)
#pragma unroll
      for (int r = 0; r < C::R2; ++r) {
        const int i = tile_out_i<N>(b, r), n = tile_n<N>(t, i);
        const float k = (float)(i < C::R1 / 2 ? n : n - N);
        v[b * C::R2 + r] = cscale(v[b * C::R2 + r], axis_poly(type, k, 1.f));
      }
  }
};

// Forward x pass of sums of fields: item (tile, c), the n[c] fields from
// first[c] on into first[c].
template <int N>
struct XSumOp {
  static constexpr bool kPre = true, kPost = false;
  float2* base;
  int64_t fs;
  int first[3], n[3];
  __device__ void coords(unsigned item, int& o, int& c0, int& c) const {
    c = (int)(item / TileCfg<N>::TILES);
    tile_coords<N>(item - c * TileCfg<N>::TILES, o, c0);
  }
  __device__ const float2* src(int c) const { return base + (int64_t)first[c] * fs; }
  __device__ float2* dst(int c) const { return base + (int64_t)first[c] * fs; }
  __device__ void pre(float2* v, int o, int kz, int c, int t) const {
    using C = TileCfg<N>;
    const float2* f = src(c) + TileMap<N, 0>(o, kz, t, 0).base;
    for (int j = 1; j < n[c]; ++j) {
      f += fs;
#pragma unroll
      for (int r = 0; r < C::R1; ++r) v[r] = cadd(v[r], f[TileMap<N, 0>::off(C::T * r)]);
    }
  }
};

// G -= w kF^2 T/(D Beta) (kx^2 P + kx Q + R), the Hessians' gradients P, Q, R
// (fields 0, 1, 3 of X), and T = rho_0 Fnl / N^3 G / w, rho_0 = k^(ns - 4): what
// the filters q_r take to the gradients of the products g_r (XinvGradOp).
template <int N>
__global__ void __launch_bounds__(256) k_chain_hess(LptArgs a, const float2* __restrict__ X, int64_t fs,
                                                    const float* __restrict__ rho0, float fnl_n3,
                                                    float2* __restrict__ G, float2* __restrict__ T) {
  constexpr int64_t total = (int64_t)N * N * (N / 2 + 1);
  const float kF = a.m.g.kF;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
    int x, y, kz;
    const int64_t e = spec_cell<N>(i, a.m.g.HP, x, y, kz);
    const int kx = sidx(x, N), ky = sidx(y, N), n2 = kx * kx + ky * ky + kz * kz;
    const float fx = (float)kx, w = half_weight(kz, N), f = -kF * kF * __ldg(a.twb + n2) * w;
    const float2 P = X[e], Q = X[fs + e], R = X[3 * fs + e];
    float2 g = G[e];
    g.x = fmaf(f, fmaf(fx, fmaf(fx, P.x, Q.x), R.x), g.x);
    g.y = fmaf(f, fmaf(fx, fmaf(fx, P.y, Q.y), R.y), g.y);
    G[e] = g;
    const float s = fnl_n3 * __ldg(rho0 + n2) / w;  // 0 at k = 0
    T[e] = cscale(g, s);
  }
}

// Transposes of the modal products on real fields in the plan's row order: f_p
// (fields 0..M-1, replaced by their gradients gf_p) and the gradients of g_r
// (fields M..2M-1):
//   gf_p     = sum_r gg_r sum_q c_pqr f_q       (groups (p, r) of entries (c, q))
//   G(p,q,r) = sum_x gg_r f_p f_q  for p <= q <= r, and (0, 2, 1), FP64 per block
// Two kernels, G first (gf goes over f): the sums hold 128 registers of partial
// sums a thread, the gradients a few but wait on one load after another.
// k_chain_sums: a block walks chunks of kChainChunk positions staged in shared
// memory; a thread takes a pair (p, q) and RB values of r over its share of the
// chunk, four positions per load in four FP32 partial sums, so f_p f_q is
// formed once for RB sums and the lanes of a warp, which are pairs, read the
// same gg_r.  k_chain_gf: two positions per thread, its own column of shared
// memory.  256^3, 10 modes: 1.12 + 1.08 ms; one kernel with a triple per thread
// (three loads per product) and an FP64 fold of every chunk took 2.86.
constexpr int kChainThreads = 128, kChainChunk = 256, kChainLd = kChainChunk + 4;
struct AdjEntry {
  float c;
  int q;
};
struct AdjGroup {  // entries [begin, end) of one (p, r); p ascending
  int p, r, begin, end;
};
// the index of the sorted triple (p, q, q) among all in (p, q, r) order, r
// fastest; the counter-term product (0, 2, 1) follows the last
__host__ __device__ __forceinline__ int chain_triple(int p, int q, int M) {
  // triples with a smaller p, then pairs (p, q') with q' < q
  int k = 0;
  for (int a = 0; a < p; ++a) k += (M - a) * (M - a + 1) / 2;
  for (int b = p; b < q; ++b) k += M - b;
  return k;
}
constexpr int chain_ntrip(int M) { return M * (M + 1) * (M + 2) / 6 + 1; }
template <int N>
__global__ void __launch_bounds__(kChainThreads) k_chain_gf(float* work, int64_t fsr, int HP, int M,
                                                            const AdjEntry* __restrict__ ent, int nent,
                                                            const AdjGroup* __restrict__ grp, int ngrp) {
  extern __shared__ float2 shc[];
  float2* sf = shc + threadIdx.x;                     // [M][kChainThreads]
  float2* sg = sf + M * kChainThreads;                // [M][kChainThreads]
  AdjEntry* se = reinterpret_cast<AdjEntry*>(shc + 2 * M * kChainThreads);  // [nent]
  AdjGroup* sp = reinterpret_cast<AdjGroup*>(se + (nent + 1) / 2 * 2);      // [ngrp]
  for (int k = threadIdx.x; k < nent; k += kChainThreads) se[k] = ent[k];
  for (int k = threadIdx.x; k < ngrp; k += kChainThreads) sp[k] = grp[k];
  __syncthreads();
  constexpr int64_t n2 = (int64_t)N * N * N / 2;
  const int64_t fs2 = fsr / 2;
  for (int64_t i = (int64_t)blockIdx.x * kChainThreads + threadIdx.x; i < n2; i += (int64_t)gridDim.x * kChainThreads) {
    const int64_t row = i / (N / 2);
    float2* p = reinterpret_cast<float2*>(work) + row * HP + (i - row * (N / 2));
    for (int m = 0; m < M; ++m) {
      sf[m * kChainThreads] = p[m * fs2];
      sg[m * kChainThreads] = p[(M + m) * fs2];
    }
    int k = 0;
    for (int m = 0; m < M; ++m) {
      float2 g = make_float2(0.f, 0.f);
      for (; k < ngrp && sp[k].p == m; ++k) {
        const AdjGroup gr = sp[k];
        const float2 r = sg[gr.r * kChainThreads];
        float2 h = make_float2(0.f, 0.f);
#pragma unroll 4
        for (int e = gr.begin; e < gr.end; ++e) {
          const AdjEntry en = se[e];
          const float2 f = sf[en.q * kChainThreads];
          h.x = fmaf(en.c, f.x, h.x);
          h.y = fmaf(en.c, f.y, h.y);
        }
        g.x = fmaf(r.x, h.x, g.x);
        g.y = fmaf(r.y, h.y, g.y);
      }
      p[m * fs2] = g;
    }
  }
}

template <int N, int RB>
__global__ void __launch_bounds__(kChainThreads) k_chain_sums(const float* __restrict__ work, int64_t fsr, int HP, int M,
                                                              int share, double* gsum) {
  extern __shared__ double shd[];
  const int ntrip = chain_ntrip(M);
  double* acc = shd;  // [share][ntrip]
  float* sf = reinterpret_cast<float*>(shd + (share * ntrip + 1) / 2 * 2);  // [M][kChainLd]
  float* sg = sf + M * kChainLd;                                            // [M][kChainLd]
  const int t = threadIdx.x;
  for (int k = t; k < share * ntrip; k += kChainThreads) acc[k] = 0.0;
  constexpr int64_t n3 = (int64_t)N * N * N;
  static_assert(n3 % kChainChunk == 0);
  const int npair = M * (M + 1) / 2, nitem = npair * ((M + RB - 1) / RB);
  const int lanes = kChainThreads / share, mine = t / lanes;  // this thread's share of a chunk
  const int u0 = mine * (kChainChunk / 4) / share, u1 = (mine + 1) * (kChainChunk / 4) / share;
  float4 s[RB];
  auto clear = [&] {
#pragma unroll
    for (int j = 0; j < RB; ++j) s[j] = make_float4(0.f, 0.f, 0.f, 0.f);
  };
  // item: pair in the order (0,0) (0,1) (1,1) (0,2) .. (q slow, pp <= q), then
  // blocks of r
  auto decode = [&](int it, int& pp, int& q, int& r0) {
    const int pair = it % npair;
    r0 = it / npair * RB;
    q = (int)((sqrtf(8.f * pair + 1.f) - 1.f) * 0.5f);
    while ((q + 1) * (q + 2) / 2 <= pair) ++q;
    while (q * (q + 1) / 2 > pair) --q;
    pp = pair - q * (q + 1) / 2;
  };
  auto sums = [&](int pp, int q, int r0) {
    const float4* a = reinterpret_cast<const float4*>(sf + pp * kChainLd);
    const float4* b = reinterpret_cast<const float4*>(sf + q * kChainLd);
    const float4* c = reinterpret_cast<const float4*>(sg + r0 * kChainLd);
#pragma unroll 1
    for (int u = u0; u < u1; ++u) {
      const float4 A = a[u], B = b[u];
      const float4 ab = make_float4(A.x * B.x, A.y * B.y, A.z * B.z, A.w * B.w);
#pragma unroll
      for (int j = 0; j < RB; ++j) {
        const float4 R = c[(r0 + j < M ? j : 0) * (kChainLd / 4) + u];  // past the last r: not stored
        s[j].x = fmaf(ab.x, R.x, s[j].x);
        s[j].y = fmaf(ab.y, R.y, s[j].y);
        s[j].z = fmaf(ab.z, R.z, s[j].z);
        s[j].w = fmaf(ab.w, R.w, s[j].w);
      }
    }
  };
  auto fold = [&](int pp, int q, int r0) {
    const int base = mine * ntrip + chain_triple(pp, q, M);
#pragma unroll
    for (int j = 0; j < RB; ++j) {
      const int r = r0 + j;
      const float v = (s[j].x + s[j].y) + (s[j].z + s[j].w);
      if (r < M && r >= q) acc[base + r - q] += (double)v;
      else if (r == 1 && pp == 0 && q == 2) acc[mine * ntrip + ntrip - 1] += (double)v;
    }
    clear();
  };
  // one item per thread: its partial sums run over kFold chunks (at most 128
  // terms each) before they are folded into FP64 -- the FP64 adds of every
  // chunk were most of the kernel's time
  const int it0 = t - mine * lanes;
  const bool one = nitem <= lanes;
  const int kFold = share * 2;
  int pp = 0, q = 0, r0 = 0, pend = 0;
  if (it0 < nitem) decode(it0, pp, q, r0);
  clear();
  for (int64_t x0 = (int64_t)blockIdx.x * kChainChunk; x0 < n3; x0 += (int64_t)gridDim.x * kChainChunk) {
    const int64_t x = x0 + 2 * t, row = x / N;
    const float2* p = reinterpret_cast<const float2*>(work + row * 2 * HP + (x - row * N));
    const int64_t fs2 = fsr / 2;
    __syncthreads();  // the chunk before has been read
    for (int m = 0; m < M; ++m) {
      *reinterpret_cast<float2*>(sf + m * kChainLd + 2 * t) = p[m * fs2];
      *reinterpret_cast<float2*>(sg + m * kChainLd + 2 * t) = p[(M + m) * fs2];
    }
    __syncthreads();
    if (one) {
      if (it0 >= nitem) continue;
      sums(pp, q, r0);
      if (++pend == kFold) fold(pp, q, r0), pend = 0;
    } else {
      for (int it = it0; it < nitem; it += lanes) {
        int ip, iq, ir;
        decode(it, ip, iq, ir);
        sums(ip, iq, ir);
        fold(ip, iq, ir);
      }
    }
  }
  if (one && it0 < nitem && pend) fold(pp, q, r0);
  __syncthreads();
  for (int k = t; k < ntrip; k += kChainThreads) {
    double v = acc[k];
    for (int j = 1; j < share; ++j) v += acc[j * ntrip + k];
    atomicAdd(gsum + k, v);
  }
}

// alpha's gradient [M][M][M] from the sums: sorted triples at [p][q][r], the
// counter-terms' G(0,1,2) - G(0,2,1) (the last sum) added to [1][1][1].
__global__ void k_chain_galpha(const double* __restrict__ gsum, int M, int counter, double* galpha) {
  for (int i = threadIdx.x; i < M * M * M; i += blockDim.x) {
    const int r = i % M, q = i / M % M, p = i / M / M;
    double g = 0.0;
    if (p <= q && q <= r) {
      g = gsum[chain_triple(p, q, M) + r - q];
      if (counter && p == 1 && r == 1) g += gsum[chain_triple(0, 1, M) + 1] - gsum[chain_ntrip(M) - 1];
    }
    galpha[i] = g;
  }
}
