// Block-scaled GEMMs on CTA pairs (gemm_pair.cuh):  D[M,N] = epi(alpha * sum_k (A[m,k] sfa[m,k/B]) (B[n,k] sfb[n,k/B])).
// NVFP4: A and B are packed e2m1 (two values per byte, even index in the low nibble), one ue4m3 scale per 16 values
// (`kind::mxf4nvf4.block_scale.scale_vec::4X`, K = 64 per MMA).  MXFP8: e4m3 / e5m2 bytes, one ue8m0 scale per 32 values
// (`kind::mxf8f6f4.block_scale`, K = 32 per MMA).  Both operands K-major.  The scales come in 128-row x 4-block atoms of 512 bytes (byte
// (r % 32) * 16 + (r / 32) * 4 + block), atoms of one row block contiguous along K: the layout the tensor core's scale path wants, so
// a stage's atoms of a row block are one TMA row and go from shared to tensor memory by one tcgen05.cp each.
//
// What bounds these products is the operands' way from L2: 512 cycles of MMAs eat 32 KB per CTA of a 256 x 256 pair tile, 64 bytes a
// cycle and SM of the 68 - 86 there are; a 128 x 256 tile of one CTA needs 96.  The eight products of a layer, us, 128 x 256 tiles on
// single CTAs (whose fp32 results went through registers of four warps) / pairs: MXFP8 M 128, C 1280 98.9 / 88.5, M 4096, C 1280 246 /
// 206, M 8192, C 768 194 / 175; NVFP4 M 128, C 1600 94.4 / 80.2, M 4096, C 1600 234 / 193.  Single ones that stay slower than on single CTAs, for
// the cluster's set-up: MXFP8 dGELU M 2048, K 384, N 1536 7.8 / 8.3, M 1024, K 768, N 3072 8.9 / 9.3; weight gradient 3072 x 768 of 2048 rows 9.3 / 9.9.
#include "gemm_pair.cuh"

namespace {
template <int KIND>
int gemm_block_scaled(void* D, const void* A, const void* B, const void* sfa, const void* sfb, const void* bias, void* aux,
                      const float* alpha, int M, int N, int K, int a_fmt, int b_fmt, long long ldd, long long ldaux, int epi,
                      int splits, int* status, cudaStream_t st) {
  constexpr int EPB = KIND == KIND_MXF8 ? 1 : 2;          // elements per byte
  constexpr int BKE = EPB * ROW_BYTES;                    // K values per stage
  constexpr int SF_WORDS = PairCfg<KIND, EPI_NONE>::SF_A / 8;
  if (M <= 0 || N <= 0 || K <= 0 || K % 32 || N % 8) return LLMB_ERR_BAD_ARG;
  if ((reinterpret_cast<uintptr_t>(A) | reinterpret_cast<uintptr_t>(B) | reinterpret_cast<uintptr_t>(D) |
       reinterpret_cast<uintptr_t>(sfa) | reinterpret_cast<uintptr_t>(sfb)) & 15) return LLMB_ERR_BAD_ARG;
  // outputs (and bf16 auxiliary tensors) travel by TMA when their layout allows a tensor map
  const bool needs_aux = epi == EPI_BIAS_GELU || epi == EPI_DGELU || epi == EPI_BIAS_RESID, out_f32 = epi == EPI_ACC_F32 || epi == EPI_STORE_F32;
  const int osz = out_f32 ? 4 : 2;
  const bool tma_layout = (ldd * osz) % 16 == 0 && (!needs_aux || (aux && (reinterpret_cast<uintptr_t>(aux) & 15) == 0 && (ldaux * 2) % 16 == 0));
  const bool reg_layout = register_epilogue_takes(epi, false, M, bias, aux, ldd, ldaux);
  if (!tma_layout && !reg_layout) return LLMB_ERR_BAD_ARG;
  CUtensorMap ta, tb;
  int rc = make_tmap_2d(&ta, A, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, (uint64_t)M, (uint64_t)(K / EPB), (uint64_t)(K / EPB), BM, ROW_BYTES);
  if (rc) return 1000 + rc;
  rc = make_tmap_2d(&tb, B, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, (uint64_t)N, (uint64_t)(K / EPB), (uint64_t)(K / EPB), 128, ROW_BYTES);
  if (rc) return 1000 + rc;
  // scale atoms: ceil(K / 64) for NVFP4, ceil(K / 128) for MXFP8 along K; row blocks and atoms that do not exist are read as zeros
  const uint64_t words = (uint64_t)ceil_div(K, KIND == KIND_MXF8 ? 128 : 64) * 64;
  ScaleMaps<KIND> sfm;
  rc = make_tmap_2d(&sfm.a, sfa, CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 8, (uint64_t)ceil_div(M, 128), words, words, 1, SF_WORDS, CU_TENSOR_MAP_SWIZZLE_NONE);
  if (rc) return 1000 + rc;
  rc = make_tmap_2d(&sfm.b, sfb, CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 8, (uint64_t)ceil_div(N, 128), words, words, 2, SF_WORDS, CU_TENSOR_MAP_SWIZZLE_NONE);
  if (rc) return 1000 + rc;
  GemmParams p{};
  p.D = D; p.bias = bias; p.aux = aux; p.alpha = alpha;
  p.M = M; p.N = N; p.K = K; p.ldd = ldd; p.ldaux = ldaux;
  p.a_lbo = p.b_lbo = 16; p.a_sbo = p.b_sbo = 1024; p.a_kstep = p.b_kstep = 32; p.a_layout = p.b_layout = 2;
  p.m_tiles = ceil_div(M, BM); p.n_tiles = ceil_div(N, BN);
  p.kb_total = ceil_div(K, BKE);
  if (splits < 1) splits = 1;
  if (splits > p.kb_total) splits = p.kb_total;
  if (epi != EPI_ACC_F32) splits = 1;
  p.kb_per_split = ceil_div(p.kb_total, splits);
  p.splits = ceil_div(p.kb_total, p.kb_per_split);
  p.status = status;
  p.bias_vec = (reinterpret_cast<uintptr_t>(bias) & 15) == 0;
  p.idesc = KIND == KIND_MXF8 ? make_idesc_mxfp8((uint32_t)a_fmt, (uint32_t)b_fmt, 2 * BM, BN) : make_idesc_nvfp4(2 * BM, BN);
  CUtensorMap td = ta, taux = ta;
  if (tma_layout) {
    int ok = make_tmap_2d(&td, D, out_f32 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, osz, (uint64_t)M, (uint64_t)N,
                          (uint64_t)ldd, 32, out_f32 ? 32 : 64) == 0;
    if (ok && needs_aux)
      ok = make_tmap_2d(&taux, aux, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, (uint64_t)M, (uint64_t)N, (uint64_t)ldaux, 32, 64) == 0;
    p.tma_epi = ok;
  }
  if (!p.tma_epi && !reg_layout) return LLMB_ERR_BAD_ARG;
  return launch_pair_epi<KIND>(epi, ta, tb, td, taux, sfm, p, st);
}
}  // namespace

// D[M,N] = epi(alpha * (A sfa)(B sfb)^T) on the NVFP4 tensor path (`kind::mxf4nvf4`, 16-value blocks, ue4m3 scales).
// A [M, K/2] and B [N, K/2]: packed e2m1 bytes as llmb_nvfp4_quantize writes them (K % 32 == 0); sfa / sfb: its
// swizzled scale buffers (llmb_nvfp4_scale_bytes(rows, K, 1) bytes, zero where no block exists).  D is bf16
// except for epi 4 / 6 (fp32 accumulate with split-K / fp32 store); bias and aux are bf16.
LLMB_API int llmb_gemm_nvfp4(void* D, const void* A, const void* B, const void* sfa, const void* sfb, const void* bias, void* aux,
                             const float* alpha, int M, int N, int K, long long ldd, long long ldaux, int epi, int splits,
                             int* status, cudaStream_t st) {
  return gemm_block_scaled<KIND_NVF4>(D, A, B, sfa, sfb, bias, aux, alpha, M, N, K, 0, 0, ldd, ldaux, epi, splits, status, st);
}

// The same product on the MXFP8 tensor path (`kind::mxf8f6f4`): A [M, K] and B [N, K] are e4m3 (fmt 0) or e5m2 (fmt 1) bytes,
// sfa / sfb one ue8m0 scale (byte = biased exponent of a power of two) per row and 32 values of K in the same 128 x 4 atoms,
// ceil(K / 128) atoms per row block.
LLMB_API int llmb_gemm_mxfp8(void* D, const void* A, const void* B, const void* sfa, const void* sfb, const void* bias, void* aux,
                             const float* alpha, int M, int N, int K, int a_fmt, int b_fmt, long long ldd, long long ldaux,
                             int epi, int splits, int* status, cudaStream_t st) {
  return gemm_block_scaled<KIND_MXF8>(D, A, B, sfa, sfb, bias, aux, alpha, M, N, K, a_fmt, b_fmt, ldd, ldaux, epi, splits, status, st);
}
