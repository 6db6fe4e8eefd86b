// Persistent, warp-specialised tcgen05 GEMM for sm_100a:  D[M,N] = epilogue(A[M,K] · B[N,K]^T).
//
// Covers every linear-layer GEMM of the trainer (reference call sites: llmm/matmul.mojo:463-696
// forward + bias / bias+GELU epilogues, :2789-2938 dinp with the dGELU epilogue, :3231-3509 dW
// with beta=1 accumulate, :3671-3908 LM head; all of them cuBLASLt calls in the reference).
//
// Design: warp-specialised kernels in which a TMA producer streams 128-byte-swizzled operand tiles through a shared-memory ring
// (cp.async.bulk.tensor, no multicast), one elected lane issues tcgen05.mma into TMEM accumulators, and epilogue warps read a
// finished accumulator back, apply bias / GELU / dGELU / residual / fp32 accumulate and store through TMA.  Operands may be K-major or
// MN-major (the UMMA descriptor and the TMA box change, not the data), which is how dinp (B = W as stored) and dW (A = dout^T,
// B = inp^T as stored) run without any transposes.  Split-K work units add into the (fp32) gradient buffer.
//
// gemm_pair_kernel (gemm_pair.cuh: two CTAs per 256 x 256 tile with cta_group::2 MMAs, persistent, 8 epilogue warps, optional
// all-gather of A from peer GPUs and optional column sums of the result) runs what fills the chip with such tiles; gemm_small.cu runs the
// rest on 128-row tiles; pick_tile() chooses.  gemm_scaled.cu has the block-scaled operands (NVFP4, MXFP8).
#include <math.h>
#include "gemm_pair.cuh"

namespace {
int g_dbg_mn_lbo = -1, g_dbg_mn_sbo = -1;   // test hooks: override the MN-major descriptor strides
thread_local float* g_pending_colsum = nullptr;   // armed by llmb_gemm_set_colsum, consumed by the calling thread's next llmb_gemm
thread_local GatherArgs g_pending_gather{};   // armed by llmb_gemm_set_gather, consumed (and cleared) by the calling thread's next llmb_gemm
thread_local bool g_pending_pair = false;     // armed by llmb_gemm_set_pair, consumed the same way
thread_local PullArgs g_pending_pull{};       // armed by llmb_gemm_set_pull, consumed (and cleared) the same way
// LLMB_GEMM_PAIR=0 / llmb_gemm_set_pair_mode(0): 128 x 128 tiles on single CTAs wherever the layout allows (a comparator)
int g_pair_mode = -1;
bool pair_mode() {
  if (g_pair_mode < 0) { const char* e = getenv("LLMB_GEMM_PAIR"); g_pair_mode = (e && e[0] == '0') ? 0 : 1; }
  return g_pair_mode == 1;
}

// Tile configuration of one problem: bn = 256 is the CTA-pair kernel, 64 / 128 the kernel of gemm_small.cu with cl CTAs per tile.
struct Tile { int bn, cl, splits; };
thread_local int g_force_bn = 0, g_force_cl = 1;          // test hook (llmb_gemm_force_tile): 0 = the rule decides

// The configuration with the smallest estimated time, in microseconds on a B200 from linear fits over M = 64 ... 5439, K and N =
// 384 ... 5120 (the small kernel must win by 5 %): a fixed part (launch, set-up, epilogue) plus a cost per
// 128-byte k-block, bounded by what one SM can fetch (24 / 32 KB per k-block) in the small kernel and by the 256-row MMAs in the pair
// kernel; MN-major operands cost more per k-block; more CTAs than SMs run side by side at the cost of each other's k-blocks; a
// further round of pair tiles costs its epilogue if that is longer than its k-loop.  Clusters only while they fit in one round:
// beyond it they are 1.5 - 4 times slower than one CTA per tile.
// The constants were fitted to kernels whose epilogues took longer and whose loads of MN-major operands did cost more, which those of today
// no longer do.  With the kernels as they are the choice is 1.9 % slower than the best configuration on average over 19 sizes, at worst 44 % (TF32 M
// 1024, C 768, N 3072 with GELU, 31.8 against 22.0 us; M 8192, C 384 C x C input gradient 7.2 / 5.9).  A new fit (0.7 %, 15 %) was not kept: forward
// passes of one row at C 384 with 656 and more tokens became 3 - 9 % slower.  Now, us, launches from a graph, pair / 128 x 128 / best 64-column
// form: bias + residual, M 64, K 3072, N 768 19.8 / 15.8 / (4 CTAs) 7.7, M 776, K 1024, N 1024 10.9 / 8.7 / (1) 7.4, M 776, K 1600, N 1600 14.2 / 11.7 /
// (1) 12.4; bias + GELU, M 4096, K 768, N 3072 21.4 / 30.9 / (1) 45.5; the rule takes the fastest of the three each time.
// splits: parts of K in the pair kernel; most: the most that this kernel's CTAs may cut it into.
Tile pick_tile(int kind, int epi, int M, int N, int kb_total, int splits, int most, int a_mn, int b_mn) {
  if (g_force_bn) return {kind == KIND_F8F6F4 && g_force_bn == 64 ? 128 : g_force_bn, g_force_cl, splits};
  if (!pair_mode()) return {128, 1, splits};
  const bool aux = epi == EPI_BIAS_GELU || epi == EPI_DGELU || epi == EPI_BIAS_RESID, acc = epi == EPI_ACC_F32;
  const int sms = sm_count();
  const float mn = a_mn ? 1.8f : b_mn ? 1.4f : 1.0f, f32 = kind == KIND_TF32 ? 2.0f : 0.0f;
  const long long pt = (long long)ceil_div(M, 256) * ceil_div(N, 256) * splits;
  const int rounds = (int)((pt + sms / 2 - 1) / (sms / 2));
  const float pair_kb = 0.285f * ceil_div(kb_total, splits) * (a_mn ? 1.4f : b_mn ? 1.12f : 1.0f);
  const float pair_epi = aux ? 6.0f + f32 : 4.8f;
  float best = 0.95f * ((aux ? 9.3f : acc ? 8.0f : 6.7f) + f32 + pair_kb + (rounds - 1) * (pair_kb > pair_epi ? pair_kb : pair_epi));
  Tile t{256, 1, splits};
  for (int bn = 64; bn <= 128; bn += 64) {
    if (bn == 64 && kind == KIND_F8F6F4) continue;        // an fp8 row of an MN-major operand is 128 columns
    const long long tiles = (long long)ceil_div(M, BM) * ceil_div(N, bn);
    for (int cl = 1; cl <= (bn == 64 ? 4 : 2); cl *= 2) {
      if (cl > 1 && (acc || kind == KIND_TF32 || tiles * cl > sms || cl > kb_total)) break;
      int sp = 1;
      if (acc)                                            // one round of CTAs, at least four k-blocks each, no more parts than allowed
        while (sp < most && tiles * (sp + 1) <= sms && kb_total / (sp + 1) >= 4) ++sp;
      const float per_sm = (float)(tiles * cl * sp) / sms;
      // one to two CTAs per SM and operands stored along K: the second CTA of an SM overlaps the first one's epilogue, and the kernels
      // before and after overlap the short tail.  M 776, us, pair / 128 x 128: K 1024, N 3072 (168 CTAs) 11.4 / 10.7, N 4096 with GELU
      // (224) 13.5 / 12.5; K 1600, N 4800 (266) 20.1 / 14.9.  Not with an auxiliary input: bias + residual, M 4096, N 768 (192), K 768
      // 11.0 / 16.1, K 3072 21.9 / 33.9; dGELU, M 776, K 1024, N 3072 (168) 12.2 / 17.2, N 4096 (224) 12.5 / 17.5 (a backward product,
      // whose weights lie along N, is out by that already).
      const bool beside = per_sm > 1.f && per_sm <= 2.f && !a_mn && !b_mn && epi != EPI_BIAS_RESID && epi != EPI_DGELU;
      const float w = per_sm <= 1.f ? 1.f : beside ? per_sm : 0.5f * (per_sm + ceilf(per_sm));
      const float fixed = (cl == 1 ? (bn == 64 ? 4.2f : 5.0f) : cl == 2 ? 5.6f : 6.2f) + (aux ? (bn == 64 ? 0.3f : 1.2f) : 0.f) + f32;
      const float est = fixed + w * ceil_div(kb_total, cl * sp) * 0.24f * mn + (w - 1.f) * (!aux ? 0.7f : beside ? 1.0f : 3.0f) * (bn / 64);
      if (est < best) { best = est; t = {bn, cl, sp}; }
    }
  }
  return t;
}

// The caller's `splits` (see llmb_gemm): makes it the parts of the pair kernel, 1 ... kb_total, and returns the most parts for other tiles.
// Why a caller may leave those to the rule: the parts that fill 74 CTA pairs are too few for 128-row tiles at small row counts.  A layer's
// four weight gradients, us, held to them / left to the rule: C 384, 777 rows 36.0 / 24.4, C 512, 960 rows 42.1 / 28.6, C 768, 960
// rows 45.9 / 42.7; from 1024 rows on the two differ by less than 3 us.
int parts(int& splits, int kb_total) {
  const bool rule = splits < 0;
  if (rule) splits = splits < -kb_total ? kb_total : -splits;
  splits = splits < 1 ? 1 : splits > kb_total ? kb_total : splits;
  return rule ? 16 : splits;
}

template <int KIND>
int gemm_dispatch(void* D, const void* A, const void* B, const void* bias, void* aux, const float* alpha, int M, int N,
                  int K, long long lda, long long ldb, long long ldd, long long ldaux, int a_mn, int b_mn, int a_fmt,
                  int b_fmt, int epi, int splits, int* status, cudaStream_t st) {
  constexpr int ESZ = KindTraits<KIND>::ESZ;
  constexpr int ROW_ELEMS = ROW_BYTES / ESZ;          // elements per swizzled row
  constexpr int BKE = ROW_ELEMS;                      // K elements per stage
  constexpr int MMA_K = 32 / ESZ;
  if (M <= 0 || N <= 0 || K <= 0) return LLMB_ERR_BAD_ARG;
  if ((lda * ESZ) % 16 || (ldb * ESZ) % 16 || N % 8) return LLMB_ERR_BAD_ARG;
  if ((reinterpret_cast<uintptr_t>(A) | reinterpret_cast<uintptr_t>(B) | reinterpret_cast<uintptr_t>(D)) & 15) return LLMB_ERR_BAD_ARG;

  GemmParams p;
  p.g = g_pending_gather;
  g_pending_gather.W = 0;
  p.pull = g_pending_pull;
  g_pending_pull.nseg = 0; g_pending_pull.nwait = 0;
  p.colsum = g_pending_colsum;
  g_pending_colsum = nullptr;
  const bool keep_pair = g_pending_pair;
  g_pending_pair = false;
  if ((p.pull.nseg > 0 || p.pull.nwait > 0) && p.g.W > 1) return LLMB_ERR_BAD_ARG;
  if (p.colsum && !(epi == EPI_DGELU && (KIND == KIND_F16 || KIND == KIND_F8F6F4))) return LLMB_ERR_BAD_ARG;   // bf16 output, TMA epilogue
  if (p.g.W > 1) {
    // gathered A: K-major bf16 rows, CTA-pair kernel, whole 256-row tiles per chunk, no split-K
    if (a_mn || KIND != KIND_F16 || p.g.tiles_per_chunk <= 0 || M != p.g.W * p.g.tiles_per_chunk * 2 * BM || epi == EPI_ACC_F32)
      return LLMB_ERR_BAD_ARG;
  }
  // outputs (and auxiliary tensors) travel by TMA when their layout allows a tensor map
  const bool needs_aux = epi == EPI_BIAS_GELU || epi == EPI_DGELU || epi == EPI_BIAS_RESID;
  const bool out_f32 = KIND == KIND_TF32 || epi == EPI_ACC_F32 || epi == EPI_STORE_F32;
  const int osz = out_f32 ? 4 : 2;
  static int tma_epi_on = -1;
  if (tma_epi_on < 0) { const char* e = getenv("LLMB_GEMM_TMA_EPI"); tma_epi_on = (e && e[0] == '0') ? 0 : 1; }
  CUtensorMap ta, tb, td, taux;
  p.tma_epi = 0;
  const bool tma_layout = tma_epi_on && (ldd * osz) % 16 == 0 && (!needs_aux || (aux && (reinterpret_cast<uintptr_t>(aux) & 15) == 0 && (ldaux * osz) % 16 == 0));
  const bool reg_layout = register_epilogue_takes(epi, KIND == KIND_TF32, M, bias, aux, ldd, ldaux);
  if (!tma_layout && !reg_layout) return LLMB_ERR_BAD_ARG;
  if (tma_layout) {
    const CUtensorMapDataType odt = out_f32 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
    const uint32_t box_cols = out_f32 ? 32 : 64;
    int ok = make_tmap_2d(&td, D, odt, osz, (uint64_t)M, (uint64_t)N, (uint64_t)ldd, 32, box_cols) == 0;
    if (ok && needs_aux) ok = make_tmap_2d(&taux, aux, odt, osz, (uint64_t)M, (uint64_t)N, (uint64_t)ldaux, 32, box_cols) == 0;
    p.tma_epi = ok;
  }
  if (!p.tma_epi && !reg_layout) return LLMB_ERR_BAD_ARG;
  if (p.colsum && !p.tma_epi) return LLMB_ERR_BAD_ARG;    // the column sums are taken in the TMA epilogue only
  const int kb_total = ceil_div(K, BKE);
  const int most = parts(splits, kb_total);
  if (epi != EPI_ACC_F32) splits = 1;
  Tile tile{256, 1, splits};
  if (p.tma_epi && !keep_pair && p.g.W <= 1 && p.pull.nseg == 0 && p.pull.nwait == 0) tile = pick_tile(KIND, epi, M, N, kb_total, splits, most, a_mn, b_mn);
  while (tile.cl > 1 && tile.cl > kb_total) tile.cl >>= 1;
  splits = tile.splits;
  const bool pair = tile.bn == 256;
  // weight gradients of fp32 operands: vector reductions from registers; adding boxes by TMA took the LM head's from 263 to 299 us
  // (2048 x 768 x 50304) and left the layers' as they were
  if (pair && KIND == KIND_TF32 && epi == EPI_ACC_F32) p.tma_epi = 0;
  const int b_rows = pair ? 128 : tile.bn;                // rows of B per load (in the pair kernel each CTA fetches half of the tile)

  int rc;
  // K-major: global [MN rows, K cols], box [tile rows, ROW_ELEMS]; MN-major: global [K rows, MN cols], box [BKE, ROW_ELEMS]
  const bool base32 = (KIND == KIND_TF32);            // fp32 operands stored MN-major need the 32-byte-base swizzle
  const CUtensorMapSwizzle mn_swz = base32 ? CU_TENSOR_MAP_SWIZZLE_128B_ATOM_32B : CU_TENSOR_MAP_SWIZZLE_128B;
  rc = a_mn ? make_tmap_2d(&ta, A, KindTraits<KIND>::DT, ESZ, (uint64_t)K, (uint64_t)M, (uint64_t)lda, BKE, ROW_ELEMS, mn_swz)
            : make_tmap_2d(&ta, A, KindTraits<KIND>::DT, ESZ, (uint64_t)M, (uint64_t)K, (uint64_t)lda, BM, ROW_ELEMS);
  if (rc) return 1000 + rc;
  int a_3d = 0, b_3d = 0;
  static int use3d = -1;
  if (use3d < 0) { const char* e = getenv("LLMB_GEMM_3D"); use3d = (e && e[0] == '0') ? 0 : 1; }
  // MN-major tiles as one 3-D box: (elements of one 128-byte row, k rows, row-chunks) - one TMA request per operand and stage
  if (a_mn && use3d && M % ROW_ELEMS == 0) {
    CUtensorMap t3;
    if (make_tmap_3d(&t3, A, KindTraits<KIND>::DT, ESZ, ROW_ELEMS, (uint64_t)K, (uint64_t)(M / ROW_ELEMS), (uint64_t)lda, ROW_ELEMS,
                     ROW_ELEMS, BKE, BM / ROW_ELEMS, mn_swz) == 0) { ta = t3; a_3d = 1; }
  }
  rc = b_mn ? make_tmap_2d(&tb, B, KindTraits<KIND>::DT, ESZ, (uint64_t)K, (uint64_t)N, (uint64_t)ldb, BKE, ROW_ELEMS, mn_swz)
            : make_tmap_2d(&tb, B, KindTraits<KIND>::DT, ESZ, (uint64_t)N, (uint64_t)K, (uint64_t)ldb, b_rows, ROW_ELEMS);
  if (rc) return 1000 + rc;

  if (b_mn && use3d && N % ROW_ELEMS == 0) {
    CUtensorMap t3;
    if (make_tmap_3d(&t3, B, KindTraits<KIND>::DT, ESZ, ROW_ELEMS, (uint64_t)K, (uint64_t)(N / ROW_ELEMS), (uint64_t)ldb, ROW_ELEMS,
                     ROW_ELEMS, BKE, b_rows / ROW_ELEMS, mn_swz) == 0) { tb = t3; b_3d = 1; }
  }
  if (!p.tma_epi) td = ta;                                // placeholders
  if (!p.tma_epi || !needs_aux) taux = ta;
  p.a_3d = a_3d; p.b_3d = b_3d;
  p.D = D; p.bias = bias; p.aux = aux; p.alpha = alpha;
  p.M = M; p.N = N; p.K = K; p.ldd = ldd; p.ldaux = ldaux;
  p.a_mn = a_mn; p.b_mn = b_mn;
  const uint32_t mn_lbo = g_dbg_mn_lbo >= 0 ? (uint32_t)g_dbg_mn_lbo : (uint32_t)(BKE * ROW_BYTES);
  const uint32_t mn_sbo = g_dbg_mn_sbo >= 0 ? (uint32_t)g_dbg_mn_sbo : (base32 ? 512u : 1024u);
  p.a_layout = (a_mn && base32) ? 1u : 2u;
  p.b_layout = (b_mn && base32) ? 1u : 2u;
  p.a_lbo = a_mn ? mn_lbo : 16; p.a_sbo = a_mn ? mn_sbo : 1024; p.a_kstep = a_mn ? MMA_K * ROW_BYTES : 32;
  p.b_lbo = b_mn ? mn_lbo : 16; p.b_sbo = b_mn ? mn_sbo : 1024; p.b_kstep = b_mn ? MMA_K * ROW_BYTES : 32;
  p.idesc = make_idesc((uint32_t)a_fmt, (uint32_t)b_fmt, (uint32_t)a_mn, (uint32_t)b_mn, pair ? 2 * BM : BM, (uint32_t)tile.bn);
  p.m_tiles = ceil_div(M, BM); p.n_tiles = ceil_div(N, tile.bn);
  p.kb_total = kb_total;
  p.kb_per_split = ceil_div(kb_total, splits);
  p.splits = pair ? ceil_div(kb_total, p.kb_per_split) : splits;
  p.status = status;
  p.io_f32 = (KIND == KIND_TF32) ? 1 : 0;
  p.bias_vec = (reinterpret_cast<uintptr_t>(bias) & 15) == 0;
  if (!pair) return llmb_gemm_small_launch(KIND, epi, tile.bn, tile.cl, ta, tb, td, taux, p, st);

  return launch_pair_epi<KIND>(epi, ta, tb, td, taux, ScaleMaps<KIND>{}, p, st);
}
}  // namespace

// D[M,N] = epi(alpha * A·B^T).  a_mn/b_mn = 1 when the operand is stored [K, M] / [K, N].
// kind: 0 bf16, 1 tf32 (fp32 storage), 2 fp8 (a_fmt/b_fmt: 0 e4m3, 1 e5m2).  D is bf16 except for the
// fp32 epilogues (4 = accumulate with red.add; 6 = plain fp32 store).  splits: the most parts that K may be cut into by an accumulating
// product.  Parts are added in the order in which they finish, so with one part the result is the same on every run.  splits < 0: -splits
// parts on CTA pairs, and as many as fill the chip (up to 16) where the tile rule takes other tiles.
// `status` is a device int the kernel sets to LLMB_ERR_TIMEOUT if a bounded wait expires.
LLMB_API int llmb_gemm(void* D, const void* A, const void* B, const void* bias, void* aux, const float* alpha, int M,
                       int N, int K, long long lda, long long ldb, long long ldd, long long ldaux, int a_mn, int b_mn,
                       int kind, int a_fmt, int b_fmt, int epi, int splits, int* status, cudaStream_t st) {
  switch (kind) {
    case 0: return gemm_dispatch<KIND_F16>(D, A, B, bias, aux, alpha, M, N, K, lda, ldb, ldd, ldaux, a_mn, b_mn, FMT_BF16, FMT_BF16, epi, splits, status, st);
    case 1: return gemm_dispatch<KIND_TF32>(D, A, B, bias, aux, alpha, M, N, K, lda, ldb, ldd, ldaux, a_mn, b_mn, FMT_TF32, FMT_TF32, epi, splits, status, st);
    case 2: return gemm_dispatch<KIND_F8F6F4>(D, A, B, bias, aux, alpha, M, N, K, lda, ldb, ldd, ldaux, a_mn, b_mn, a_fmt, b_fmt, epi, splits, status, st);
  }
  return LLMB_ERR_BAD_ARG;
}

// How many parts of the contraction an accumulating llmb_gemm (epilogue 4, both operands stored [K, *]) of this size is cut into: with
// one part the result may as well be stored (epilogue 6) where nothing has to be added to.
LLMB_API int llmb_gemm_dw_splits(int kind, int M, int N, int K, int splits) {
  const int kb = ceil_div(K, kind == 0 ? 64 : 32);
  const int most = parts(splits, kb);
  return pick_tile(kind == 0 ? KIND_F16 : KIND_TF32, EPI_ACC_F32, M, N, kb, splits, most, 1, 1).splits;
}

// Arms the calling thread's NEXT llmb_gemm call to gather its A matrix from W ranks (see GatherArgs): A must be the
// local [W*n, K] buffer, n a multiple of 256; peer_src[r] = address of chunk r in rank r's buffer; flags = this
// rank's flag words; counts = 16 local counters that the caller zeroes (stream-ordered) before the GEMM.
LLMB_API void llmb_gemm_set_gather(void* const* peer_src, void* local, const void* flags, unsigned* counts, long long chunk_bytes,
                                   unsigned seq, int W, int me, int rows_per_rank) {
  GatherArgs g{};
  for (int r = 0; r < W && r < 8; ++r) g.peer_src[r] = peer_src[r];
  g.local = local; g.flags = flags; g.counts = counts; g.chunk_vecs = chunk_bytes / 16;
  g.seq = seq; g.target = (unsigned)((g.chunk_vecs + 2047) / 2048); g.W = W; g.me = me; g.tiles_per_chunk = rows_per_rank / (2 * BM);
  g_pending_gather = g;
}
// Arms the calling thread's NEXT llmb_gemm call (CTA-pair kernel) with a parameter pull and / or a wait (see PullArgs).
// Segment s copies nbytes[s] bytes (a multiple of 16, both addresses 16-byte aligned) from src[s] (memory of rank
// owner[s], mapped here) to dst[s]; counts = 16 counters zeroed (stream-ordered) before the launch.  wait_counts[i]
// must reach wait_bytes[i] / 32 KB (rounded up) before the GEMM's B operand is read.  seq: parameter sequence number
// every owner must have announced (0 = parameters as loaded, nothing to wait for).
LLMB_API int llmb_gemm_set_pull(const void* const* src, void* const* dst, const long long* nbytes, const int* owner, int nseg,
                                const void* flags, unsigned seq, unsigned* counts, const unsigned* const* wait_counts,
                                const long long* wait_bytes, int nwait, int W) {
  if (nseg < 0 || nseg > 8 || nwait < 0 || nwait > 8) return LLMB_ERR_BAD_ARG;
  PullArgs a{};
  for (int i = 0; i < nseg; ++i) {
    if ((reinterpret_cast<uintptr_t>(src[i]) | reinterpret_cast<uintptr_t>(dst[i]) | (uintptr_t)nbytes[i]) & 15) return LLMB_ERR_BAD_ARG;
    a.src[i] = src[i]; a.dst[i] = dst[i]; a.vecs[i] = nbytes[i] / 16; a.owner[i] = owner[i];
  }
  for (int i = 0; i < nwait; ++i) { a.wait_counts[i] = wait_counts[i]; a.wait_target[i] = (unsigned)((wait_bytes[i] / 16 + 2047) / 2048); }
  a.flags = flags; a.counts = counts; a.seq = seq; a.nseg = nseg; a.nwait = nwait; a.W = W;
  g_pending_pull = a;
  return 0;
}
// Arms the calling thread's NEXT llmb_gemm call (bf16 result, epilogue 3 = dGELU, any tile, TMA epilogue) to add the column
// sums of its result to colsum[N] (fp32, red.add): the bias gradient of the layer that produced the pre-activations.
LLMB_API void llmb_gemm_set_colsum(float* colsum) { g_pending_colsum = colsum; }
// Arms the calling thread's NEXT llmb_gemm call to run as the CTA-pair kernel, whose sums run through K in one chain, as they do where a
// pull is armed: for a product whose result has to be that of an armed one, bit by bit (the tile rule may cut K among four CTAs).
LLMB_API void llmb_gemm_set_pair() { g_pending_pair = true; }
LLMB_API void llmb_gemm_debug_mn_strides(int lbo_bytes, int sbo_bytes) { g_dbg_mn_lbo = lbo_bytes; g_dbg_mn_sbo = sbo_bytes; }
// 0: single-CTA 128x128 tiles, 1: the rule of pick_tile() (default; env LLMB_GEMM_PAIR=0 selects the former)
LLMB_API void llmb_gemm_set_pair_mode(int on) { g_pair_mode = on ? 1 : 0; }
// Test hook: every following llmb_gemm call of the calling thread uses tiles of bn columns (256: CTA pair; 64 / 128: gemm_small.cu with cl = 1, 2 or 4 CTAs
// per tile); bn = 0 gives the choice back to pick_tile().
LLMB_API void llmb_gemm_force_tile(int bn, int cl) { g_force_bn = bn; g_force_cl = cl; }
