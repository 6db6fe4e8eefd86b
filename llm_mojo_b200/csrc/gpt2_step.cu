// One forward or backward micro-step of GPT-2 (bf16, fp32 storage with TF32 products, block-scaled FP8 or NVFP4 sites) as ONE host call:
// the launch sequence of models/gpt2.py (reference: train_gpt2.mojo:3050-3848 forward, :3948-5056 backward) issued from native code
// over the same kernels, buffers and scratch.
//
// What it is for: a layer is 7 launches forward and 17 backward, and issuing one from Python (tensor views, pointer reads, a ctypes
// call) takes 15 - 20 us of host time, more than the kernels of a small batch run: sampling with d12 at 64 positions spent 1.75 ms
// per token on 0.64 ms of kernels.  From here a launch costs 2 - 3 us: that token takes
// 0.74 ms (d24 at 776 positions 3.36 -> 2.24), a d6 training step of 2 x 128 tokens 2.75 -> 1.36; steps whose kernels outlast the
// Python loop (d12 from 4 x 1024 on) keep their time.
// Nothing is kept between calls: every pointer comes with the call.
#include "common.cuh"
using namespace llmb;

// entry points of the other files of this library
LLMB_API int llmb_encoder_fwd(void* out, const int* tok, const void* wte, const void* wpe, int B, int T, int C, int V, int dtype, cudaStream_t st);
LLMB_API int llmb_encoder_bwd(float* dwte, float* dwpe, const void* dout, const int* tok, void* scratch, long long scratch_bytes, int B, int T,
                              int C, int V, int vocab_bits, int dtype, cudaStream_t st);
LLMB_API int llmb_gelu_fwd(void* out, const void* inp, long long n, int dtype, cudaStream_t st);
LLMB_API int llmb_dbias_launches(int rows);
LLMB_API int llmb_dbias(float* dbias, const void* dout, float* scratch, long long scratch_bytes, int rows, int OC, int dtype, cudaStream_t st);
LLMB_API int llmb_layernorm_fwd(void* out, float* mean, float* rstd, void* resid_out, const void* inp1, const void* inp2, const void* w,
                                const void* b, int rows, int C, int dtype, cudaStream_t st);
LLMB_API int llmb_layernorm_bwd(void* dres, float* dw, float* db, float* scratch, long long scratch_bytes, const void* dout, const void* inp,
                                const void* w, const float* mean, const float* rstd, int rows, int C, int accumulate, int dtype, cudaStream_t st);
LLMB_API int llmb_gemm(void* D, const void* A, const void* B, const void* bias, void* aux, const float* alpha, int M, int N, int K, long long lda,
                       long long ldb, long long ldd, long long ldaux, int a_mn, int b_mn, int kind, int a_fmt, int b_fmt, int epi, int splits,
                       int* status, cudaStream_t st);
LLMB_API void llmb_gemm_set_colsum(float* colsum);
LLMB_API int llmb_gemm_dw_splits(int kind, int M, int N, int K, int splits);
LLMB_API int llmb_attention_fwd(void* out, float* lse, const void* qkv, int B, int T, int NH, int* status, cudaStream_t st);
LLMB_API int llmb_attention_bwd_fused(void* dqkv, float* dbias, float* stats, float* dq_acc, const void* dout, const void* qkv, const void* out,
                                      const float* lse, int B, int T, int NH, int* status, cudaStream_t st);
LLMB_API int llmb_attention_f32_fwd(float* out, float* lse, const float* qkv, int B, int T, int NH, cudaStream_t st);
LLMB_API int llmb_attention_f32_bwd(float* dqkv, float* D, const float* dout, const float* qkv, const float* out, const float* lse, int B, int T,
                                    int NH, int split, cudaStream_t st);
LLMB_API int llmb_fp8_block_quant(void* q, void* sf, const void* x, int rows, int cols, int gran, int fmt, int transpose, cudaStream_t st);
LLMB_API int llmb_fp8_block_quant_dual(void* q0, void* sf0, void* q1, void* sf1, const void* x, int rows, int cols, int fmt, cudaStream_t st);
LLMB_API int llmb_gemm_mxfp8(void* D, const void* A, const void* B, const void* sfa, const void* sfb, const void* bias, void* aux,
                             const float* alpha, int M, int N, int K, int a_fmt, int b_fmt, long long ldd, long long ldaux, int epi, int splits,
                             int* status, cudaStream_t st);
LLMB_API int llmb_nvfp4_operand_ws_floats();
LLMB_API int llmb_nvfp4_operand(void* q0, void* sf0, void* q1, void* sf1, float* ws, const void* x, int rows, int cols, int block16, int rht,
                                int sr, unsigned long long seed, unsigned long long stream0, unsigned long long stream1, long long step,
                                const float* alpha_other0, float factor0, const float* alpha_other1, float factor1, cudaStream_t st);
LLMB_API int llmb_gemm_nvfp4(void* D, const void* A, const void* B, const void* sfa, const void* sfb, const void* bias, void* aux,
                             const float* alpha, int M, int N, int K, long long ldd, long long ldaux, int epi, int splits, int* status,
                             cudaStream_t st);
LLMB_API int llmb_fused_classifier(void* logits, float* losses, const int* targets, float dloss, int rows, int V, int Vp, int write_dlogits,
                                   int dtype, int* status, cudaStream_t st);
LLMB_API int llmb_ce_pass1(float* stats, const void* tile, const int* targets, int rows, int ld, int col0, int width, int V, int first, int dtype,
                           cudaStream_t st);
LLMB_API int llmb_ce_loss(float* losses, const float* stats, int rows, cudaStream_t st);
LLMB_API int llmb_ce_pass2(void* tile, const float* stats, const int* targets, int rows, int ld, int col0, int width, int V, float dloss, int dtype,
                           cudaStream_t st);

namespace {
enum { EPI_NONE = 0, EPI_BIAS = 1, EPI_BIAS_GELU = 2, EPI_DGELU = 3, EPI_ACC_F32 = 4, EPI_BIAS_RESID = 5, EPI_STORE_F32 = 6 };

// acc += scale * sum(x), one CTA: 16-byte loads, eight in flight per thread.  It replaces a sum, a product and an addition (three
// launches, 9 us of them the sum of 16384 losses on one SM).
__global__ void __launch_bounds__(1024) loss_accumulate_kernel(float* __restrict__ acc, const float* __restrict__ x, int n, float scale) {
  pdl_trigger();
  pdl_wait();
  __shared__ float red[32];
  float s[4] = {0.f, 0.f, 0.f, 0.f};
  const bool vec = (reinterpret_cast<uintptr_t>(x) & 15) == 0;
  const int nv = vec ? n / 4 : 0;
  int i = threadIdx.x;
  for (; i + 7 * 1024 < nv; i += 8 * 1024) {
    float4 t[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) t[k] = reinterpret_cast<const float4*>(x)[i + k * 1024];
#pragma unroll
    for (int k = 0; k < 8; ++k) { s[0] += t[k].x; s[1] += t[k].y; s[2] += t[k].z; s[3] += t[k].w; }
  }
  for (; i < nv; i += 1024) { const float4 t = reinterpret_cast<const float4*>(x)[i]; s[0] += t.x; s[1] += t.y; s[2] += t.z; s[3] += t.w; }
  for (int j = nv * 4 + threadIdx.x; j < n; j += 1024) s[j & 3] += x[j];
  const float w = warp_sum((s[0] + s[1]) + (s[2] + s[3]));
  if (threadIdx.x % 32 == 0) red[threadIdx.x / 32] = w;
  __syncthreads();
  if (threadIdx.x < 32) {
    const float t = warp_sum(red[threadIdx.x]);
    if (threadIdx.x == 0) *acc += t * scale;
  }
}
}  // namespace

LLMB_API int llmb_loss_accumulate(float* acc, const float* losses, int n, float scale, cudaStream_t st) {
  if (n <= 0) return LLMB_ERR_BAD_ARG;
  return launch_pdl(loss_accumulate_kernel, 1, 1024, 0, st, acc, losses, n, scale);
}

// Mirrored by ops/step.py.  Pointers are in the order of the enums below; of the storage type unless noted.
enum { P_WTE, P_WPE, P_LN1W, P_LN1B, P_QKVW, P_QKVB, P_ATTW, P_ATTB, P_LN2W, P_LN2B, P_FCW, P_FCB, P_PROJW, P_PROJB, P_LNFW, P_LNFB, P_COUNT };
enum { A_ENCODED, A_LN1, A_LN1_MEAN, A_LN1_RSTD, A_QKV, A_ATTY, A_LSE, A_RES2, A_LN2, A_LN2_MEAN, A_LN2_RSTD, A_FCH, A_GELU, A_RES3, A_LNF,
       A_LNF_MEAN, A_LNF_RSTD, A_LOSSES, A_DRES, A_DL, A_DL4, A_LOGITS, A_CE_STATS, A_COUNT };
struct Gpt2Step {
  const void* p[P_COUNT];
  float* g[P_COUNT];             // fp32 gradients (backward only)
  void* a[A_COUNT];              // means, rstds, lse, losses and ce_stats fp32; A_LOGITS: [rows, Vp], or one vocabulary tile [rows, tile_width]
  const int* tokens; const int* targets;                      // targets: null = logits only
  float* loss_acc; int* status;
  void* s_encoder; float* s_ln; float* s_dbias; float* s_stats; float* s_dq;      // scratch (backward only)
  long long s_encoder_bytes, s_ln_bytes, s_dbias_bytes;
  float dloss;
  int B, T, L, C, NH, V, Vp;
  int recompute;                 // 1: one GELU buffer for all layers, recomputed in the backward pass
  int tile_width;                // > 0: LM head in vocabulary tiles of this many columns
  int fc_colsum;                 // the dGELU GEMM takes the fc bias gradient in its epilogue
  int splits_qkv, splits_att, splits_fc, splits_proj, splits_head, splits_head_last;   // split-K factors of the weight gradients
  int vocab_bits;
  int launches;                  // out: launches issued
  int dtype;                     // storage: LLMB_BF16 or LLMB_F32 (products on the TF32 path)
  int lowp;                      // 0: none; LP_FP8B: the four linear layers of every block; LP_FP4: the MLP of layers [fp4_first, fp4_end)
  int fp4_first, fp4_end, fp4_rht, fp4_sr;
  int lp_splits_qkv, lp_splits_att, lp_splits_fc, lp_splits_proj;
  unsigned long long seed; long long micro;                   // stochastic rounding
  unsigned char* s_lowp;         // scratch, llmb_gpt2_lowp_scratch_bytes()
  unsigned char* kept;           // FP8B: the layer inputs as operands of the weight gradients, from forward to backward (null in the backward
                                 // pass: quantised again); llmb_gpt2_lowp_kept_bytes()
  int first;                     // backward: the gradients start from zero (see Step::begin_gradients)
  int T_max;                     // rows of wpe
};
enum { LP_FP8B = 2, LP_FP4 = 3 };
enum { S_QKV, S_ATT, S_FC, S_PROJ };

namespace {
size_t up16(size_t n) { return (n + 15) / 16 * 16; }
size_t sf8_bytes(size_t rows, size_t cols) { return rows / 128 * (cols / 128) * 512; }
// One NVFP4 operand in a buffer: workspace, then bytes and scale atoms of the orientations asked for
struct Op4 {
  float* ws; unsigned char *q0 = nullptr, *sf0 = nullptr, *q1 = nullptr, *sf1 = nullptr; unsigned char* end;
  Op4(unsigned char* at, size_t rows, size_t cols, bool row, bool col) : ws(reinterpret_cast<float*>(at)) {
    at += up16((size_t)llmb_nvfp4_operand_ws_floats() * 4);
    if (row) { q0 = at; sf0 = at += up16(rows * cols / 2); at += (rows + 127) / 128 * ((cols + 63) / 64) * 512; }
    if (col) { q1 = at; sf1 = at += up16(rows * cols / 2); at += (cols + 127) / 128 * ((rows + 63) / 64) * 512; }
    end = at;
  }
};

struct Step {
  const Gpt2Step& s; cudaStream_t st; int launches = 0, rc = 0;
  const int rows, C, dt, kind; const size_t esz;
  Step(const Gpt2Step& s_, cudaStream_t st_)
      : s(s_), st(st_), rows(s_.B * s_.T), C(s_.C), dt(s_.dtype), kind(s_.dtype == LLMB_F32 ? 1 : 0), esz(s_.dtype == LLMB_F32 ? 4 : 2) {}

  const char* p(int i, int l, size_t per) const { return reinterpret_cast<const char*>(s.p[i]) + l * per * esz; }
  float* g(int i, int l, size_t per) const { return s.g[i] + l * per; }
  char* a(int i, int l = 0, size_t per = 0) const { return reinterpret_cast<char*>(s.a[i]) + l * per * esz; }
  float* f(int i, int l = 0) const { return reinterpret_cast<float*>(s.a[i]) + l * (size_t)rows; }
  bool ok(int code, int n = 1) { if (rc == 0) { rc = code; launches += n; } return rc == 0; }
  int mode(int site, int l) const {
    return s.lowp == LP_FP4 ? (site >= S_FC && l >= s.fp4_first && l < s.fp4_end ? LP_FP4 : 0) : s.lowp;
  }
  // the kept copy of one site's input: bytes [K, rows], then its scale atoms
  unsigned char* kept(int site, int l) const {
    // qkv, attproj and fc have C columns, fcproj 4 C.  With recomputed GELU fcproj's input exists for one layer at a time: the last
    // layer's copy is kept, the others are made again from the recomputed values.
    if (!s.kept || (s.recompute && site == S_PROJ && l < s.L - 1)) return nullptr;
    const size_t one = (size_t)rows * C + sf8_bytes(rows, C), per = s.recompute ? 3 : 7;
    return s.kept + (per * l + site) * one;
  }

  // D[rows, N] = inp[rows, K] W[N, K]^T with the epilogue
  bool linear(void* out, const void* inp, const void* w, const void* bias, void* aux, int N, int K, int epi, long long ldd = 0) {
    return ok(llmb_gemm(out, inp, w, bias, aux, nullptr, rows, N, K, K, K, ldd ? ldd : N, N, 0, 0, kind, 0, 0, epi, 1, s.status, st));
  }
  bool site(int st_, int l, void* out, const void* inp, const void* w, const void* bias, void* aux, int N, int K, int epi) {
    if (mode(st_, l) == LP_FP8B) {
      unsigned char *q = s.s_lowp, *sf = q + (size_t)rows * K, *wq = sf + sf8_bytes(rows, K), *wsf = wq + (size_t)N * K, *kq = kept(st_, l);
      return ok(kq ? llmb_fp8_block_quant_dual(q, sf, kq, kq + (size_t)rows * K, inp, rows, K, 0, st)
                   : llmb_fp8_block_quant(q, sf, inp, rows, K, 0, 0, 0, st)) &&
             ok(llmb_fp8_block_quant(wq, wsf, w, N, K, 2, 0, 0, st)) &&
             ok(llmb_gemm_mxfp8(out, q, wq, sf, wsf, bias, aux, nullptr, rows, N, K, 0, 0, N, aux ? N : 0, epi, 1, s.status, st));
    }
    if (mode(st_, l) == LP_FP4) {
      const Op4 x(s.s_lowp, rows, K, true, false), ww(x.end, N, K, true, false);
      return ok(llmb_nvfp4_operand(x.q0, x.sf0, nullptr, nullptr, x.ws, inp, rows, K, 0, 0, 0, 0, 0, 0, 0, nullptr, 1.f, nullptr, 1.f, st), 2) &&
             ok(llmb_nvfp4_operand(ww.q0, ww.sf0, nullptr, nullptr, ww.ws, w, N, K, 1, 0, 0, 0, 0, 0, 0, x.ws, 1.f, nullptr, 1.f, st), 2) &&
             ok(llmb_gemm_nvfp4(out, x.q0, ww.q0, x.sf0, ww.sf0, bias, aux, ww.ws + 2, rows, N, K, N, aux ? N : 0, epi, 1, s.status, st));
    }
    return linear(out, inp, w, bias, aux, N, K, epi);
  }
  // dinp[rows, K] = dout[rows, N] W[N, K] (times GELU' of aux, or plus aux), then dW[N, K] += dout^T inp
  bool linear_bwd(void* dinp, float* dw, const void* dout, const void* inp, const void* w, void* aux, int N, int K, int epi, int splits,
                  bool store, float* colsum = nullptr, long long ldo = 0) {
    const long long lo = ldo ? ldo : N;
    if (colsum) llmb_gemm_set_colsum(colsum);
    return ok(llmb_gemm(dinp, dout, w, nullptr, aux, nullptr, rows, K, N, lo, K, K, aux ? K : 0, 0, 1, kind, 0, 0, epi, 1, s.status, st)) &&
           ok(llmb_gemm(dw, dout, inp, nullptr, nullptr, nullptr, N, K, rows, lo, K, K, 0, 1, 1, kind, 0, 0, store ? EPI_STORE_F32 : EPI_ACC_F32, splits,
                        s.status, st));
  }
  // A micro-step that starts the accumulation leaves out the zero fill and the read of every gradient that ONE kernel writes as a whole
  // (weights whose contraction is not split: the widest ones, where these bytes count); what is added to in parts - split weights,
  // biases, LayerNorms, positions - is filled here.
  // d36 fp8b, B 4, T 1024: 36.07 -> 35.63 ms a step, d48 NVFP4 61.63 -> 60.73; d12, where the layers' weights are split, unchanged.
  bool store_qkv = false, store_att = false, store_fc = false, store_proj = false, store_head = false;
  bool begin_gradients() {
    if (!s.first) return true;
    const size_t cc = (size_t)C * C, LC = (size_t)s.L * C;
    // one rule for a tensor of all layers: every layer's product must be in one part
    auto one = [&](int st_, int N, int K, int splits, int lp_splits) {
      bool plain = false, lp = false;
      for (int l = 0; l < s.L; ++l) (mode(st_, l) ? lp : plain) = true;
      return (!plain || llmb_gemm_dw_splits(kind, N, K, rows, splits) == 1) && (!lp || lp_splits == 1);
    };
    store_qkv = one(S_QKV, 3 * C, C, s.splits_qkv, s.lp_splits_qkv);
    store_att = one(S_ATT, C, C, s.splits_att, s.lp_splits_att);
    store_fc = one(S_FC, 4 * C, C, s.splits_fc, s.lp_splits_fc);
    store_proj = one(S_PROJ, C, 4 * C, s.splits_proj, s.lp_splits_proj);
    const int tile = s.tile_width > 0 ? s.tile_width : s.Vp, rest = s.Vp - (s.Vp - 1) / tile * tile;
    store_head = llmb_gemm_dw_splits(kind, tile, C, rows, s.splits_head) == 1 && llmb_gemm_dw_splits(kind, rest, C, rows, s.splits_head_last) == 1;
    const size_t n[P_COUNT] = {store_head ? 0 : (size_t)s.Vp * C, (size_t)s.T_max * C, LC, LC, store_qkv ? 0 : 3 * cc * s.L, 3 * LC, store_att ? 0 : cc * s.L, LC,
                               LC, LC, store_fc ? 0 : 4 * cc * s.L, 4 * LC, store_proj ? 0 : 4 * cc * s.L, LC, (size_t)C, (size_t)C};
    float *from = nullptr, *to = nullptr;                 // neighbours in memory are filled together
    for (int i = 0; i <= P_COUNT; ++i) {
      if (i < P_COUNT && n[i] && s.g[i] == to) { to += n[i]; continue; }
      if (i < P_COUNT && !n[i]) continue;
      if (from != to && !ok((int)cudaMemsetAsync(from, 0, (to - from) * sizeof(float), st), 0)) return false;
      if (i < P_COUNT) { from = s.g[i]; to = from + n[i]; }
    }
    return true;
  }
  bool site_bwd(int st_, int l, void* dinp, float* dw, const void* dout, const void* inp, const void* w, void* aux, int N, int K, int epi,
                int splits, int lp_splits, bool store, float* colsum = nullptr) {
    const int acc = store ? EPI_STORE_F32 : EPI_ACC_F32;
    if (mode(st_, l) == LP_FP8B) {
      const size_t nd = (size_t)rows * N, sd_n = sf8_bytes(rows, N);
      unsigned char *qd = s.s_lowp, *sd = qd + nd, *qdt = sd + sd_n, *sdt = qdt + nd, *wq = sdt + sd_n, *wsf = wq + (size_t)N * K;
      unsigned char* qx = kept(st_, l);
      if (!(ok(llmb_fp8_block_quant_dual(qd, sd, qdt, sdt, dout, rows, N, 1, st)) && ok(llmb_fp8_block_quant(wq, wsf, w, N, K, 2, 0, 1, st)) &&
            ok(llmb_gemm_mxfp8(dinp, qd, wq, sd, wsf, nullptr, aux, nullptr, rows, K, N, 1, 0, K, aux ? K : 0, epi, 1, s.status, st)))) return false;
      if (!qx) {
        qx = wsf + sf8_bytes(N, K);
        if (!ok(llmb_fp8_block_quant(qx, qx + (size_t)rows * K, inp, rows, K, 1, 0, 1, st))) return false;
      }
      return ok(llmb_gemm_mxfp8(dw, qdt, qx, sdt, qx + (size_t)rows * K, nullptr, nullptr, nullptr, N, K, rows, 1, 0, K, 0, acc, lp_splits, s.status, st));
    }
    if (mode(st_, l) == LP_FP4) {
      const Op4 d(s.s_lowp, rows, N, true, true), ww(d.end, N, K, false, true), x(ww.end, rows, K, false, true);
      return ok(llmb_nvfp4_operand(d.q0, d.sf0, d.q1, d.sf1, d.ws, dout, rows, N, 0, s.fp4_rht, s.fp4_sr, s.seed, FP4_STREAM + 2, FP4_STREAM + 3, s.micro,
                                   nullptr, 1.f, nullptr, 1.f, st), 2) &&
             ok(llmb_nvfp4_operand(nullptr, nullptr, ww.q1, ww.sf1, ww.ws, w, N, K, 1, 0, 0, 0, 0, 0, 0, nullptr, 1.f, d.ws, 1.f, st), 2) &&
             ok(llmb_gemm_nvfp4(dinp, d.q0, ww.q1, d.sf0, ww.sf1, nullptr, aux, ww.ws + 3, rows, K, N, K, aux ? K : 0, epi, 1, s.status, st)) &&
             ok(llmb_nvfp4_operand(nullptr, nullptr, x.q1, x.sf1, x.ws, inp, rows, K, 0, s.fp4_rht, 0, 0, 0, 0, 0, nullptr, 1.f, d.ws + 1,
                                   s.fp4_rht ? 1.f / 16.f : 1.f, st), 2) &&
             ok(llmb_gemm_nvfp4(dw, d.q1, x.q1, d.sf1, x.sf1, nullptr, nullptr, x.ws + 3, N, K, rows, K, 0, acc, lp_splits, s.status, st));
    }
    return linear_bwd(dinp, dw, dout, inp, w, aux, N, K, epi, splits, store, colsum);
  }
  static constexpr unsigned long long FP4_STREAM = 16;    // NVFP4_SR_STREAM of ops/lowp.py
  bool attention(int l, size_t rc1, size_t lse) {
    char *o = a(A_ATTY, l, rc1), *qkv = a(A_QKV, l, 3 * rc1);
    float* ls = reinterpret_cast<float*>(s.a[A_LSE]) + l * lse;
    return ok(dt == LLMB_BF16 ? llmb_attention_fwd(o, ls, qkv, s.B, s.T, s.NH, s.status, st)
                              : llmb_attention_f32_fwd(reinterpret_cast<float*>(o), ls, reinterpret_cast<float*>(qkv), s.B, s.T, s.NH, st));
  }
  // dqkv and the gradient of the qkv bias
  bool attention_bwd(void* dqkv, int l, size_t rc1, size_t lse) {
    const char *o = a(A_ATTY, l, rc1), *qkv = a(A_QKV, l, 3 * rc1);
    const float* ls = reinterpret_cast<float*>(s.a[A_LSE]) + l * lse;
    float* db = g(P_QKVB, l, 3 * C);
    if (dt == LLMB_BF16) return ok(llmb_attention_bwd_fused(dqkv, db, s.s_stats, s.s_dq, s.a[A_DL], qkv, o, ls, s.B, s.T, s.NH, s.status, st), 3);
    return ok(llmb_attention_f32_bwd(reinterpret_cast<float*>(dqkv), s.s_stats, reinterpret_cast<float*>(s.a[A_DL]), reinterpret_cast<const float*>(qkv),
                                     reinterpret_cast<const float*>(o), ls, s.B, s.T, s.NH, 0, st), 2) && bias_grad(db, dqkv, 3 * C);
  }
  bool bias_grad(float* db, const void* dout, int N) { return ok(llmb_dbias(db, dout, s.s_dbias, s.s_dbias_bytes, rows, N, dt, st), llmb_dbias_launches(rows)); }
  bool ln_bwd(float* dw, float* db, const void* inp, const void* w, const float* mean, const float* rstd, int accumulate) {
    return ok(llmb_layernorm_bwd(s.a[A_DRES], dw, db, s.s_ln, s.s_ln_bytes, s.a[A_DL], inp, w, mean, rstd, rows, C, accumulate, dt, st), 2);
  }

  void forward() {
    const size_t rc1 = (size_t)rows * C, cc = (size_t)C * C, lse = (size_t)s.B * s.NH * s.T;
    if (!ok(llmb_encoder_fwd(a(A_ENCODED), s.tokens, s.p[P_WTE], s.p[P_WPE], s.B, s.T, C, s.Vp, dt, st))) return;
    for (int l = 0; l < s.L && !rc; ++l) {
      void* x = l == 0 ? a(A_ENCODED) : a(A_RES3, l - 1, rc1);
      void* act = a(A_GELU, s.recompute ? 0 : l, 4 * rc1);
      ok(llmb_layernorm_fwd(a(A_LN1, l, rc1), f(A_LN1_MEAN, l), f(A_LN1_RSTD, l), nullptr, x, nullptr, p(P_LN1W, l, C), p(P_LN1B, l, C), rows, C, dt, st)) &&
      site(S_QKV, l, a(A_QKV, l, 3 * rc1), a(A_LN1, l, rc1), p(P_QKVW, l, 3 * cc), p(P_QKVB, l, 3 * C), nullptr, 3 * C, C, EPI_BIAS) &&
      attention(l, rc1, lse) &&
      site(S_ATT, l, a(A_RES2, l, rc1), a(A_ATTY, l, rc1), p(P_ATTW, l, cc), p(P_ATTB, l, C), x, C, C, EPI_BIAS_RESID) &&
      ok(llmb_layernorm_fwd(a(A_LN2, l, rc1), f(A_LN2_MEAN, l), f(A_LN2_RSTD, l), nullptr, a(A_RES2, l, rc1), nullptr, p(P_LN2W, l, C), p(P_LN2B, l, C), rows, C, dt, st)) &&
      site(S_FC, l, act, a(A_LN2, l, rc1), p(P_FCW, l, 4 * cc), p(P_FCB, l, 4 * C), a(A_FCH, l, 4 * rc1), 4 * C, C, EPI_BIAS_GELU) &&
      site(S_PROJ, l, a(A_RES3, l, rc1), act, p(P_PROJW, l, 4 * cc), p(P_PROJB, l, C), a(A_RES2, l, rc1), C, 4 * C, EPI_BIAS_RESID);
    }
    if (rc || !ok(llmb_layernorm_fwd(a(A_LNF), f(A_LNF_MEAN), f(A_LNF_RSTD), nullptr, a(A_RES3, s.L - 1, rc1), nullptr, s.p[P_LNFW], s.p[P_LNFB], rows, C, dt, st))) return;
    if (s.tile_width > 0) {
      for (int c0 = 0; c0 < s.Vp && !rc; c0 += s.tile_width) {
        const int w = s.Vp - c0 < s.tile_width ? s.Vp - c0 : s.tile_width;
        linear(a(A_LOGITS), a(A_LNF), p(P_WTE, c0, C), nullptr, nullptr, w, C, EPI_NONE, s.tile_width) &&
        ok(llmb_ce_pass1(f(A_CE_STATS), a(A_LOGITS), s.targets, rows, s.tile_width, c0, w, s.V, c0 == 0, dt, st));
      }
      if (rc || !ok(llmb_ce_loss(f(A_LOSSES), f(A_CE_STATS), rows, st))) return;
    } else {
      if (!linear(a(A_LOGITS), a(A_LNF), s.p[P_WTE], nullptr, nullptr, s.Vp, C, EPI_NONE) || !s.targets) return;
      if (!ok(llmb_fused_classifier(a(A_LOGITS), f(A_LOSSES), s.targets, s.dloss, rows, s.V, s.Vp, 1, dt, s.status, st))) return;
    }
    ok(llmb_loss_accumulate(s.loss_acc, f(A_LOSSES), rows, s.dloss, st));
  }

  void backward() {
    const size_t rc1 = (size_t)rows * C, cc = (size_t)C * C, lse = (size_t)s.B * s.NH * s.T;
    if (!begin_gradients()) return;
    void *dres = s.a[A_DRES], *dl = s.a[A_DL], *dl4 = s.a[A_DL4], *dqkv = s.a[A_DL4];
    if (s.tile_width > 0) {                               // every logits tile again, as dlogits, consumed at once
      for (int c0 = 0; c0 < s.Vp && !rc; c0 += s.tile_width) {
        const bool last = s.Vp - c0 <= s.tile_width;
        const int w = last ? s.Vp - c0 : s.tile_width;
        linear(a(A_LOGITS), a(A_LNF), p(P_WTE, c0, C), nullptr, nullptr, w, C, EPI_NONE, s.tile_width) &&
        ok(llmb_ce_pass2(a(A_LOGITS), f(A_CE_STATS), s.targets, rows, s.tile_width, c0, w, s.V, s.dloss, dt, st)) &&
        linear_bwd(dl, g(P_WTE, c0, C), a(A_LOGITS), a(A_LNF), p(P_WTE, c0, C), c0 ? dl : nullptr, w, C, c0 ? EPI_BIAS_RESID : EPI_NONE,
                   last ? s.splits_head_last : s.splits_head, store_head, nullptr, s.tile_width);
      }
    } else {
      linear_bwd(dl, s.g[P_WTE], a(A_LOGITS), a(A_LNF), s.p[P_WTE], nullptr, s.Vp, C, EPI_NONE, s.splits_head, store_head);
    }
    if (rc || !ln_bwd(s.g[P_LNFW], s.g[P_LNFB], a(A_RES3, s.L - 1, rc1), s.p[P_LNFW], f(A_LNF_MEAN), f(A_LNF_RSTD), 0)) return;
    for (int l = s.L - 1; l >= 0 && !rc; --l) {
      const void* x = l == 0 ? a(A_ENCODED) : a(A_RES3, l - 1, rc1);
      void* act = a(A_GELU, s.recompute ? 0 : l, 4 * rc1);
      if (s.recompute && !ok(llmb_gelu_fwd(act, a(A_FCH, l, 4 * rc1), 4 * (long long)rc1, dt, st))) return;
      float* dfcb = g(P_FCB, l, 4 * C);
      const bool fused = s.fc_colsum && mode(S_PROJ, l) == 0;               // the dGELU GEMM takes the fc bias gradient
      site_bwd(S_PROJ, l, dl4, g(P_PROJW, l, 4 * cc), dres, act, p(P_PROJW, l, 4 * cc), a(A_FCH, l, 4 * rc1), C, 4 * C, EPI_DGELU, s.splits_proj,
               s.lp_splits_proj, store_proj, fused ? dfcb : nullptr) &&
      (fused || bias_grad(dfcb, dl4, 4 * C)) &&
      bias_grad(g(P_PROJB, l, C), dres, C) &&
      site_bwd(S_FC, l, dl, g(P_FCW, l, 4 * cc), dl4, a(A_LN2, l, rc1), p(P_FCW, l, 4 * cc), nullptr, 4 * C, C, EPI_NONE, s.splits_fc, s.lp_splits_fc, store_fc) &&
      ln_bwd(g(P_LN2W, l, C), g(P_LN2B, l, C), a(A_RES2, l, rc1), p(P_LN2W, l, C), f(A_LN2_MEAN, l), f(A_LN2_RSTD, l), 1) &&
      site_bwd(S_ATT, l, dl, g(P_ATTW, l, cc), dres, a(A_ATTY, l, rc1), p(P_ATTW, l, cc), nullptr, C, C, EPI_NONE, s.splits_att, s.lp_splits_att, store_att) &&
      bias_grad(g(P_ATTB, l, C), dres, C) &&
      attention_bwd(dqkv, l, rc1, lse) &&
      site_bwd(S_QKV, l, dl, g(P_QKVW, l, 3 * cc), dqkv, a(A_LN1, l, rc1), p(P_QKVW, l, 3 * cc), nullptr, 3 * C, C, EPI_NONE, s.splits_qkv, s.lp_splits_qkv, store_qkv) &&
      ln_bwd(g(P_LN1W, l, C), g(P_LN1B, l, C), x, p(P_LN1W, l, C), f(A_LN1_MEAN, l), f(A_LN1_RSTD, l), 1);
    }
    if (!rc) ok(llmb_encoder_bwd(s.g[P_WTE], s.g[P_WPE], dres, s.tokens, s.s_encoder, s.s_encoder_bytes, s.B, s.T, C, s.Vp, s.vocab_bits, dt, st), 4);
  }
};
}  // namespace

LLMB_API int llmb_abi() { return LLMB_ABI; }
LLMB_API int llmb_gpt2_step_bytes() { return (int)sizeof(Gpt2Step); }
// the largest site, backward: both orientations of the output gradient, the weight and the input
LLMB_API long long llmb_gpt2_lowp_scratch_bytes(const Gpt2Step* s) {
  const size_t rows = (size_t)s->B * s->T, C = s->C;
  if (s->lowp == LP_FP8B) return (long long)(3 * (rows * 4 * C + sf8_bytes(rows, 4 * C)) + 4 * C * C + sf8_bytes(4 * C, C));
  if (s->lowp == LP_FP4) {
    const Op4 d(nullptr, rows, 4 * C, true, true), w(d.end, 4 * C, C, true, true), x(w.end, rows, 4 * C, true, true);
    return (long long)reinterpret_cast<uintptr_t>(x.end);
  }
  return 0;
}
LLMB_API long long llmb_gpt2_lowp_kept_bytes(const Gpt2Step* s) {
  const size_t rows = (size_t)s->B * s->T, C = s->C;
  return s->lowp == LP_FP8B ? (long long)((s->recompute ? 3 * s->L + 4 : 7 * s->L) * (rows * C + sf8_bytes(rows, C))) : 0;
}
// Both return 0 or the code of the first entry point that failed; nothing after it is launched.
LLMB_API int llmb_gpt2_forward(Gpt2Step* s, cudaStream_t st) {
  Step x(*s, st);
  x.forward();
  s->launches = x.launches;
  return x.rc;
}
LLMB_API int llmb_gpt2_backward(Gpt2Step* s, cudaStream_t st) {
  Step x(*s, st);
  x.backward();
  s->launches = x.launches;
  return x.rc;
}
