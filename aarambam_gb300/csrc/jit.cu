// Run-time specialised modal row kernel.
//
// The generic row kernel (fused.cu, ModalRowOp) walks its term list at run
// time: in factored order a term costs a shared-memory load at each of two
// positions, its address and the loop.  Here the kernel is generated for the plan's term structure
// and compiled with NVRTC for sm_103a: a thread loads the M values f_p of
// its positions into registers once and a term is a multiply-add per component with
// compile-time register indices; the coefficients sit in the module's
// __constant__ memory, so a new alpha table with the same nonzero pattern
// (same terms) only rewrites them.  The FFT and row code are the same
// headers the library is built from (fft.cuh, rows.cuh, embedded at build
// time).  If NVRTC or the module load fails, the plan keeps the generic
// kernel and records why.
#include <cuda_runtime.h>
#include <nvrtc.h>
#include <stdint.h>

#include <algorithm>
#include <string>
#include <vector>

#include "aar_internal.cuh"
#include "rows.cuh"
#include "jit_embed.h"  // kEmbedFft, kEmbedRows (generated by build.py)
#include "spectral.cuh"

namespace aar {

struct JitState {
  cudaLibrary_t lib = nullptr;
  cudaKernel_t kern = nullptr;
  float* coef = nullptr;  // the module's __constant__ coefficients
  std::string key;        // N, M and the term structure the module was made for
  size_t smem = 0;
  int nterms = 0;
  int threads = 0;        // block size the module was compiled for
  int pr = 0;             // row pairs per block (rows_pairs), 0: rows_fold, one row per block
};

static std::string gen_source(int N, int M, int minb, int threads, int pr, int pairs, const TermList& tl,
                              const std::vector<Term>& terms) {
  std::string s = "struct JitRowOp {\n";
  s += "  static constexpr bool kPairs = " + std::string(pairs ? "true" : "false") + ";\n";
  s += "  static constexpr bool kZfac = false;\n";
  // maps of the inputs and outputs to field slots and lines: the identity
  // where it is one, else constant memory (a switch in the loops over lines
  // cost the 512^3 rows 5.8 -> 7.2 ms)
  std::string consts;
  auto map = [&](const char* name, int n, auto&& value) {
    bool id = true;
    std::string v;
    for (int i = 0; i < n; ++i) {
      id = id && value(i) == i;
      v += (i ? "," : "") + std::to_string(value(i));
    }
    if (!id) consts += std::string("__constant__ int k_") + name + "[] = {" + v + "};\n";
    s += std::string("  __device__ int ") + name + "(int l) const { return " +
         (id ? "l" : std::string("k_") + name + "[l]") + "; }\n";
  };
  const int nin = tl.nin;
  s += "  __device__ int nlines() const { return " + std::to_string(tl.nlines) + "; }\n";
  s += "  __device__ int nin() const { return " + std::to_string(nin) + "; }\n";
  map("in_slot", nin, [&](int i) { return tl.in_mode[i]; });
  map("in_line", nin, [&](int i) { return tl.line[tl.in_mode[i]]; });
  s += "  __device__ int nout() const { return " + std::to_string(tl.nr) + "; }\n";
  map("out_slot", tl.nr, [&](int i) { return tl.r_of_slot[i]; });
  map("out_line", tl.nr, [&](int i) { return tl.line[tl.r_of_slot[i]]; });
  s += "  template <int K>\n  __device__ __forceinline__ void combine(float2* sm, const int* pos, int LS) const {\n";
  s += "    float2 f[" + std::to_string(nin) + "][K];\n";
  for (int p = 0; p < nin; ++p)
    s += "#pragma unroll\n    for (int i = 0; i < K; ++i) f[" + std::to_string(p) + "][i] = sm[" +
         std::to_string(tl.line[tl.in_mode[p]]) + " * LS + pos[i]];\n";
  int in_of[kMaxModes] = {};  // f index of a mode
  for (int i = 0; i < nin; ++i) in_of[tl.in_mode[i]] = i;
  // one block per output slot (the counter-term f0 f2 -> g1 with its own
  // target r), its terms in factored order.
  for (int sl = 0; sl < tl.nr; ++sl) {
    const int r = tl.r_of_slot[sl];
    s += "    {\n      float2 a[K];\n#pragma unroll\n      for (int i = 0; i < K; ++i) a[i] = make_float2(0.f, 0.f);\n";
    std::vector<int> own;
    for (size_t t = 0; t < terms.size(); ++t)
      if (terms[t].r == r) own.push_back((int)t);
    std::vector<TermF> fac;
    factor_terms(terms.data(), own, M, fac);
    bool first = true;
    for (const TermF& t : fac) {
      const std::string c = "kCoef[" + std::to_string(t.t) + "]", fo = "f[" + std::to_string(in_of[t.o]) + "][i]";
      if (first)
        s += "      {\n      float2 h[K];\n#pragma unroll\n      for (int i = 0; i < K; ++i) h[i] = make_float2(" + c + " * " + fo +
             ".x, " + c + " * " + fo + ".y);\n";
      else
        s += "#pragma unroll\n      for (int i = 0; i < K; ++i) { h[i].x = fmaf(" + c + ", " + fo + ".x, h[i].x); h[i].y = fmaf(" + c +
             ", " + fo + ".y, h[i].y); }\n";
      first = t.end;
      if (!t.end) continue;
      const std::string fF = "f[" + std::to_string(in_of[t.F]) + "][i]";
      s += "#pragma unroll\n      for (int i = 0; i < K; ++i) { a[i].x = fmaf(" + fF + ".x, h[i].x, a[i].x); a[i].y = fmaf(" + fF +
           ".y, h[i].y, a[i].y); }\n      }\n";
    }
    s += "#pragma unroll\n      for (int i = 0; i < K; ++i) sm[" + std::to_string(tl.line[r]) + " * LS + pos[i]] = a[i];\n    }\n";
  }
  s += "  }\n};\n}  // namespace aar\n";
  // kCoef at global scope: its symbol name is not mangled (cudaLibraryGetGlobal)
  s = "#include \"rows.cuh\"\n__constant__ float kCoef[" + std::to_string(terms.empty() ? 1 : terms.size()) +
      "];\nnamespace aar {\n" + consts + s;
  s += "extern \"C\" __global__ void __launch_bounds__(" + std::to_string(threads) + ", " + std::to_string(minb) +
       ") aar_modal_rows_jit(float2* work, long long fs, int HP, long long nrows, const float2* __restrict__ twN, "
       "const float2* __restrict__ twH, const float2* __restrict__ tw2) {\n";
  const std::string targs = std::to_string(N) + ", aar::JitRowOp, " + std::to_string(threads);
  if (pr)
    s += "  aar::rows_pairs<" + targs + ">(aar::JitRowOp{}, work, fs, HP, nrows, tw2, " + std::to_string(pr) + ");\n}\n";
  else
    s += "  aar::rows_fold<" + targs + ">(aar::JitRowOp{}, work, fs, HP, twN, twH);\n}\n";
  return s;
}

static void jit_release(JitState* j) {
  if (!j) return;
  if (j->lib) cudaLibraryUnload(j->lib);
  delete j;
}

void jit_free(Plan* p) {
  jit_release((JitState*)p->jit);
  p->jit = nullptr;
}

// Blocks of the specialised kernel: what the plan asks for (jit_minb,
// jit_threads), else by its lines.
struct RowShape {
  int minb, threads, pr;
  size_t smem;
};
static RowShape row_shape(const Plan* p, const TermList& tl) {
  const int N = p->N;
  RowShape s{};
  if (rows_use_pairs(N, tl.nlines)) {
    // a line per T threads: as many row pairs as fill 192 threads within 72
    // KB, one or more rounds of at most 512 threads where a pair has more lines
    const int R1 = two_stage_r1(N), T = N / R1, m = std::max(tl.nin, tl.nr);
    const size_t pair = sizeof(float2) * (size_t)tl.nlines * (N + T);
    s.pr = std::max(1, (p->jit_threads > 0 ? p->jit_threads : 192) / (m * T));
    while (s.pr > 1 && s.pr * pair > 72 * 1024) --s.pr;
    const int want = s.pr * m * T, rounds = (want + 511) / 512;
    s.threads = p->jit_threads > 0 ? p->jit_threads : ((want + rounds - 1) / rounds + 31) / 32 * 32;
    s.minb = p->jit_minb > 0 ? p->jit_minb : std::max(1, 65536 / (R1 == 32 ? 112 : 64) / s.threads);
    s.minb = std::min(s.minb, 65536 / 64 / s.threads);
    s.smem = s.pr * pair;
  } else {
    s.minb = p->jit_minb > 0 ? p->jit_minb : 2;
    // 320 threads (ten warps) where they take the input lines in fewer rounds
    // than eight warps (measured at 1024^3, 20 modes: 362 vs 372 ms per step);
    // the autotuner may choose otherwise
    s.threads = p->jit_threads > 0 ? p->jit_threads : (tl.nin + 9) / 10 < (tl.nin + 7) / 8 ? 320 : kRowThreads;
    s.smem = sizeof(float2) * ((size_t)tl.nlines * FoldCfg<1024>::LS + FoldCfg<1024>::LT);
  }
  return s;
}

bool jit_row_shape(const Plan* p, int& minb, int& threads) {
  const RowShape s = row_shape(p, *(const TermList*)p->host_terms.data());
  minb = s.minb;
  threads = s.threads;
  return s.pr > 0;
}

// Build (or reuse) the specialised kernel for the plan's current term list.
// Returns AAR_OK with p->jit set, or AAR_OK with p->jit == nullptr and the
// reason in p->jit_status when the generic kernel stays in use.
int jit_prepare(Plan* p) {
  const bool want = p->jit_mode == 2 || (p->jit_mode == 1 && p->N >= 256);
  if (!want || p->prm.precision != AAR_FUSED_FP32 || p->nr_active == 0) {
    jit_free(p);
    p->jit_status = want ? "no modal terms" : "off";
    return AAR_OK;
  }
  const TermList& tl = *(const TermList*)p->host_terms.data();
  const Term* ft = (const Term*)(p->host_terms.data() + sizeof(TermList));
  std::vector<Term> terms(ft, ft + tl.nterms);
  const int N = p->N, M = p->M;
  const RowShape rs = row_shape(p, tl);
  const int minb = rs.minb, threads = rs.threads, pr = rs.pr;
  const size_t smem = rs.smem;
  const int regcap = 65536 / (threads * minb);
  const int pairs = 2 * 2 * tl.nin + 16 <= regcap * 3 / 4;  // f values of two positions fit the register budget
  std::string key = std::to_string(N) + ":" + std::to_string(M) + ":" + std::to_string(minb) + ":" +
                    std::to_string(threads) + ":" + std::to_string(pr) + ":" + std::to_string(pairs) + ":";
  for (const Term& t : terms) key += std::to_string(t.p) + "," + std::to_string(t.q) + "," + std::to_string(t.r) + ";";
  std::vector<float> coef(terms.size());
  for (size_t i = 0; i < terms.size(); ++i) coef[i] = terms[i].c;
  JitState* j = (JitState*)p->jit;
  if (!j || j->key != key) {
    jit_free(p);
    const std::string src = gen_source(N, M, minb, threads, pr, pairs, tl, terms);
    nvrtcProgram prog;
    const char* hdrs[2] = {kEmbedFft, kEmbedRows};
    const char* names[2] = {"fft.cuh", "rows.cuh"};
    if (nvrtcCreateProgram(&prog, src.c_str(), "aar_modal_rows_jit.cu", 2, hdrs, names) != NVRTC_SUCCESS) {
      p->jit_status = "nvrtcCreateProgram failed";
      return AAR_OK;
    }
    const char* opts[] = {"--gpu-architecture=sm_103a", "-std=c++20", "-lineinfo", "-default-device"};
    nvrtcResult cr = nvrtcCompileProgram(prog, 4, opts);
    if (cr != NVRTC_SUCCESS) {
      size_t n = 0;
      nvrtcGetProgramLogSize(prog, &n);
      std::string log(n, '\0');
      if (n) nvrtcGetProgramLog(prog, &log[0]);
      nvrtcDestroyProgram(&prog);
      p->jit_status = "NVRTC: " + log.substr(0, 2000);
      return AAR_OK;
    }
    size_t nbin = 0;
    nvrtcGetCUBINSize(prog, &nbin);
    std::vector<char> bin(nbin);
    nvrtcGetCUBIN(prog, bin.data());
    nvrtcDestroyProgram(&prog);
    j = new JitState();
    if (cudaLibraryLoadData(&j->lib, bin.data(), nullptr, nullptr, 0, nullptr, nullptr, 0) != cudaSuccess ||
        cudaLibraryGetKernel(&j->kern, j->lib, "aar_modal_rows_jit") != cudaSuccess) {
      cudaGetLastError();
      jit_release(j);
      p->jit_status = "module load failed";
      return AAR_OK;
    }
    size_t csize = 0;
    if (cudaLibraryGetGlobal((void**)&j->coef, &csize, j->lib, "kCoef") != cudaSuccess) {
      cudaGetLastError();
      jit_release(j);
      p->jit_status = "coefficient symbol missing";
      return AAR_OK;
    }
    j->key = key;
    j->nterms = (int)terms.size();
    j->threads = threads;
    j->pr = pr;
    p->jit = j;
  }
  j->smem = smem;
  if (cudaFuncSetAttribute((const void*)j->kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)j->smem) !=
      cudaSuccess) {
    cudaGetLastError();
    jit_free(p);
    p->jit_status = "shared-memory attribute refused";
    return AAR_OK;
  }
  if (int rc_ = upload(p, j->coef, coef.data(), sizeof(float) * coef.size())) return rc_;
  p->jit_status = "on";
  return AAR_OK;
}

int jit_modal_rows(Plan* p, float2* work, int64_t fs, cudaStream_t st, int64_t nrows) {
  JitState* j = (JitState*)p->jit;
  if (nrows < 0) nrows = (int64_t)p->N * p->N;
  long long fsl = fs, nr = nrows;
  int hp = p->HP;
  void* args[] = {&work, &fsl, &hp, &nr, &p->d_twN, &p->d_twH, &p->d_tw2};
  const int64_t rows = j->pr ? 2 * j->pr : 1;  // of a block
  {
    ProfScope ps_(p, "modal_rows", st);
    AAR_CUDA_TRY(p, cudaLaunchKernel((const void*)j->kern, dim3((unsigned)((nrows + rows - 1) / rows)),
                                     dim3(j->threads), args, j->smem, st));
  }
  p->last_launches += 1;
  return AAR_OK;
}

}  // namespace aar
