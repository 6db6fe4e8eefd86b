// GEMM for problems with too few 256 x 256 tiles to fill the chip:  D[M,N] = epilogue(A[M,K] · B[N,K]^T), the operand layouts,
// epilogues and tensor maps of gemm.cu.
//
// What bounds these problems is latency: at M = 64 the CTA-pair kernel spends 0.29 us per 64 values of K on the MMAs of a 256-row
// tile that is mostly padding, on a handful of SMs, after about 9 us of launch, set-up and epilogue.  Here a CTA of four warps owns ONE
// 128 x BN tile (BN = 64 or 128), is not persistent (several fit an SM, so that one's epilogue overlaps another's loads), and up to
// four CTAs of a cluster share the contraction of a tile: each accumulates its part of K in tensor memory, sends every 32-row band
// to the CTA that owns it through distributed shared memory, and the owner adds the parts in rank order (the result does not depend
// on timing) and runs the epilogue.  Weight gradients (fp32 accumulate) split K over blockIdx.y and add by TMA instead.
// A cluster's CTAs wait for one another, so none may be kept from starting by tensor memory that others hold: the bands' buffers leave
// room for at most three CTAs of a cluster launch per SM, and 3 x 128 columns fit the 512.
//   warp 0  TMA producer, warp 1  MMA issuer; then all four warps drain the accumulator (warp = TMEM lane quarter).
// gemm.cu's pick_tile() decides when this kernel runs, with the measurements.
#include "gemm_common.cuh"

namespace {
constexpr int SM_THREADS = 128;
constexpr int SM_MAX_STAGES = 12;
constexpr int SM_TAIL = 512;                             // barriers, TMEM slot, abort flag

// shared memory besides the operand ring: auxiliary-input boxes, bands received from the other CTAs of the cluster
template <int KIND, int EPI, int BN_, int CL> struct SmallCfg {
  static constexpr bool AUX_IN = EPI == EPI_DGELU || EPI == EPI_BIAS_RESID;
  static constexpr bool TWO_OUT = EPI == EPI_BIAS_GELU;
  static constexpr bool F32_OUT = EPI == EPI_ACC_F32 || EPI == EPI_STORE_F32;
  static constexpr bool F32_IO = KIND == KIND_TF32 && !F32_OUT;
  static constexpr int BOXES = BN_ / ((F32_IO || F32_OUT) ? 32 : 64);      // output boxes per warp
  static constexpr int STAGE = A_STAGE + BN_ * ROW_BYTES;
  static constexpr int AUX_BYTES = AUX_IN ? 4 * BOXES * SLAB_BYTES : 0;
  static constexpr int RECV_BYTES = CL > 1 ? 4 * 32 * BN_ * 4 : 0;         // (4 / CL bands) x CL sources x 32 rows x BN fp32
  static constexpr int OUT_BYTES = AUX_IN ? 0 : 4 * BOXES * SLAB_BYTES * (TWO_OUT ? 2 : 1);   // aliases the ring
};

template <int KIND, int EPI, int BN_, int CL>
__global__ void __launch_bounds__(SM_THREADS)
gemm_small_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                  const __grid_constant__ CUtensorMap tmD, const __grid_constant__ CUtensorMap tmAux, const GemmParams p, int stages) {
  using Cfg = SmallCfg<KIND, EPI, BN_, CL>;
  constexpr int BKE = KindTraits<KIND>::BKE;
  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  unsigned char* aux_s = smem + stages * Cfg::STAGE;
  unsigned char* recv_s = aux_s + Cfg::AUX_BYTES;
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(recv_s + Cfg::RECV_BYTES);
  uint64_t* empty_bar = full_bar + SM_MAX_STAGES;
  uint64_t* tfull_bar = empty_bar + SM_MAX_STAGES;
  uint64_t* aux_bar = tfull_bar + 1;                     // [4] one per warp
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(aux_bar + 4);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  const int rank = CL > 1 ? (int)cluster_ctarank() : 0;
  const int tile = blockIdx.x / CL;
  const int m_blk = tile % p.m_tiles, n_blk = tile / p.m_tiles;
  const int m0 = m_blk * BM, n0 = n_blk * BN_;
  const int part = CL > 1 ? rank : blockIdx.y, parts = CL > 1 ? CL : gridDim.y;     // parts <= kb_total
  const int kb0 = (int)((long long)part * p.kb_total / parts), kb1 = (int)((long long)(part + 1) * p.kb_total / parts);

  if (threadIdx.x == 0) {
    for (int s = 0; s < stages; ++s) { mbar_init(&full_bar[s], 1); mbar_init(&empty_bar[s], 1); }
    mbar_init(tfull_bar, 1);
    for (int w = 0; w < 4; ++w) mbar_init(&aux_bar[w], 1);
    *abort_flag = 0;
    fence_barrier_init();
    prefetch_tmap(&tmA); prefetch_tmap(&tmB); prefetch_tmap(&tmD);
    if (Cfg::AUX_IN || Cfg::TWO_OUT) prefetch_tmap(&tmAux);
  }
  if (warp == 1) tmem_alloc<BN_>(tmem_slot);
  if (CL > 1) asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");   // the peers run before anything is sent to them
  fence_before_sync();
  __syncthreads();
  fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  pdl_trigger();
  // While the kernel before this one drains: B (weights, as a rule) into L2.  A hint only, so it may run before the wait; if that kernel
  // writes B, the loads below still read what it wrote.
  if (warp == 0 && m_blk == 0 && elect_one()) {
    for (int kb = kb0; kb < kb1 && kb < kb0 + 16; ++kb) {
      const int k0 = kb * BKE;
      if (!p.b_mn) tma_prefetch_l2_2d(&tmB, k0, n0);
      else if (p.b_3d) tma_prefetch_l2_3d(&tmB, 0, k0, n0 / BKE);
    }
  }
  __syncwarp();
  pdl_wait();

  // the 32-row band this warp runs the epilogue of: its own quarter, or one of the 4 / CL bands that this CTA collects
  constexpr int NB = 4 / CL;
  const bool owner = CL == 1 || warp < NB;
  const int band = CL == 1 ? warp : rank * NB + warp;
  const int row0 = m0 + band * 32;
  unsigned char* aux_w = aux_s + warp * Cfg::BOXES * SLAB_BYTES;
  constexpr int BOX_COLS = BN_ / Cfg::BOXES;
  if (Cfg::AUX_IN && owner && row0 < p.M && lane == 0) {
    int nbox = 0;
    for (int b = 0; b < Cfg::BOXES; ++b) nbox += n0 + b * BOX_COLS < p.N;
    mbar_expect_tx(&aux_bar[warp], nbox * SLAB_BYTES);
    for (int b = 0; b < nbox; ++b) tma_load_2d(aux_w + b * SLAB_BYTES, &tmAux, &aux_bar[warp], n0 + b * BOX_COLS, row0);
  }
  __syncwarp();

  if (warp == 0) {
    int stage = 0; uint32_t phase = 0;
    bool ok = true;
    for (int kb = kb0; kb < kb1; ++kb) {
      if (kb - kb0 >= stages && !mbar_wait(&empty_bar[stage], phase ^ 1)) { ok = false; break; }
      unsigned char* sa = smem + stage * Cfg::STAGE;
      unsigned char* sb = sa + A_STAGE;
      const int k0 = kb * BKE;
      if (elect_one()) {
        mbar_expect_tx(&full_bar[stage], Cfg::STAGE);
        if (!p.a_mn) tma_load_2d(sa, &tmA, &full_bar[stage], k0, m0);
        else if (p.a_3d) tma_load_3d(sa, &tmA, &full_bar[stage], 0, k0, m0 / BKE);
        else for (int c = 0; c < BM / BKE; ++c) tma_load_2d(sa + c * BKE * ROW_BYTES, &tmA, &full_bar[stage], m0 + c * BKE, k0);
        if (!p.b_mn) tma_load_2d(sb, &tmB, &full_bar[stage], k0, n0);
        else if (p.b_3d) tma_load_3d(sb, &tmB, &full_bar[stage], 0, k0, n0 / BKE);
        else for (int c = 0; c < BN_ / BKE; ++c) tma_load_2d(sb + c * BKE * ROW_BYTES, &tmB, &full_bar[stage], n0 + c * BKE, k0);
      }
      __syncwarp();
      if (++stage == stages) { stage = 0; phase ^= 1; }
    }
    if (!ok && lane == 0) { *abort_flag = 1; atomicExch(p.status, LLMB_ERR_TIMEOUT); }
  } else if (warp == 1) {
    int stage = 0; uint32_t phase = 0;
    const uint64_t adesc0 = make_smem_desc(smem_u32(smem), p.a_lbo, p.a_sbo, p.a_layout);
    const uint64_t bdesc0 = make_smem_desc(smem_u32(smem) + A_STAGE, p.b_lbo, p.b_sbo, p.b_layout);
    const uint64_t a_inc = (uint64_t)(p.a_kstep >> 4), b_inc = (uint64_t)(p.b_kstep >> 4);
    const uint32_t idesc = p.idesc;
    bool ok = true;
    for (int kb = kb0; kb < kb1; ++kb) {
      if (!mbar_wait(&full_bar[stage], phase)) { ok = false; break; }
      fence_after_sync();
      const uint64_t adesc = adesc0 + (uint64_t)(stage * (Cfg::STAGE >> 4)), bdesc = bdesc0 + (uint64_t)(stage * (Cfg::STAGE >> 4));
      if (elect_one()) {
        umma_ss<KIND>(tmem_base, adesc, bdesc, idesc, kb > kb0 ? 1u : 0u);
#pragma unroll
        for (int k = 1; k < 4; ++k) umma_ss<KIND>(tmem_base, adesc + k * a_inc, bdesc + k * b_inc, idesc, 1u);
        umma_commit(&empty_bar[stage]);
      }
      __syncwarp();
      if (++stage == stages) { stage = 0; phase ^= 1; }
    }
    if (ok) { if (elect_one()) umma_commit(tfull_bar); }
    else if (lane == 0) { *abort_flag = 1; atomicExch(p.status, LLMB_ERR_TIMEOUT); }
    __syncwarp();
  }
  __syncwarp();
  bool ok = mbar_wait(tfull_bar, 0);
  __syncwarp();                                          // converged for the .aligned instructions below
  if (!ok && lane == 0) { *abort_flag = 1; atomicExch(p.status, LLMB_ERR_TIMEOUT); }
  __syncwarp();
  fence_after_sync();
  const uint32_t tacc = tmem_base + ((uint32_t)(warp * 32) << 16);

  if (CL > 1) {
    // every band goes to its owner: [band][source][64-column slab][16 column groups][32 rows][4] fp32
    asm volatile("barrier.cluster.wait.aligned;" ::: "memory");
    const uint32_t dst = mapa_u32(smem_u32(recv_s), (uint32_t)(warp / NB)) + (uint32_t)(((warp % NB) * CL + rank) * (32 * BN_ * 4));
#pragma unroll 1
    for (int sl = 0; sl < BN_ / 64; ++sl) {
      uint32_t r0[32], r1[32];
      tmem_ld32(tacc + sl * 64, r0);
      tmem_ld32(tacc + sl * 64 + 32, r1);
      tmem_wait_ld();
#pragma unroll
      for (int c = 0; c < 16; ++c) {
        const uint32_t (&r)[32] = c < 8 ? r0 : r1;
        asm volatile("st.shared::cluster.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(dst + sl * 8192 + c * 512 + lane * 16), "r"(r[(c & 7) * 4]),
                     "r"(r[(c & 7) * 4 + 1]), "r"(r[(c & 7) * 4 + 2]), "r"(r[(c & 7) * 4 + 3]) : "memory");
      }
    }
    cluster_sync_all();
  }

  if (ok && owner && row0 < p.M) {
    const float alpha = p.alpha ? *p.alpha : 1.0f;
    unsigned char* out_w = Cfg::AUX_IN ? aux_w : smem + warp * Cfg::BOXES * SLAB_BYTES * (Cfg::TWO_OUT ? 2 : 1);   // the ring is idle by now
    if (Cfg::AUX_IN && !mbar_wait(&aux_bar[warp], 0)) { ok = false; if (lane == 0) atomicExch(p.status, LLMB_ERR_TIMEOUT); }
#pragma unroll 1
    for (int sl = 0; sl < BN_ / 64 && ok; ++sl) {
      const int col0 = n0 + sl * 64;
      if (col0 >= p.N) break;                              // warp-uniform
      uint32_t r0[32], r1[32];
      if (CL == 1) {
        tmem_ld32(tacc + sl * 64, r0);
        tmem_ld32(tacc + sl * 64 + 32, r1);
        tmem_wait_ld();
      } else {
        const unsigned char* src = recv_s + warp * CL * (32 * BN_ * 4) + sl * 8192 + lane * 16;
#pragma unroll
        for (int c = 0; c < 16; ++c) {
          float4 v = *reinterpret_cast<const float4*>(src + c * 512);
#pragma unroll
          for (int s = 1; s < CL; ++s) {
            const float4 w = *reinterpret_cast<const float4*>(src + s * (32 * BN_ * 4) + c * 512);
            v.x += w.x; v.y += w.y; v.z += w.z; v.w += w.w;
          }
          uint32_t (&r)[32] = c < 8 ? r0 : r1;
          r[(c & 7) * 4] = __float_as_uint(v.x); r[(c & 7) * 4 + 1] = __float_as_uint(v.y);
          r[(c & 7) * 4 + 2] = __float_as_uint(v.z); r[(c & 7) * 4 + 3] = __float_as_uint(v.w);
        }
      }
      if (Cfg::F32_OUT || Cfg::F32_IO) {
        // two boxes of 32 fp32 columns
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          unsigned char* box = out_w + (sl * 2 + h) * SLAB_BYTES * (Cfg::TWO_OUT ? 2 : 1);
          if (col0 + h * 32 >= p.N) break;
          epi_box_f32<EPI>(p, h ? r1 : r0, box, box + SLAB_BYTES, col0 + h * 32, alpha, lane);
          fence_proxy_async();
          __syncwarp();
          if (lane == 0) {
            if (EPI == EPI_ACC_F32) tma_reduce_add_2d(&tmD, box, col0 + h * 32, row0);
            else if (Cfg::TWO_OUT) { tma_store_2d(&tmAux, box, col0 + h * 32, row0); tma_store_2d(&tmD, box + SLAB_BYTES, col0 + h * 32, row0); }
            else tma_store_2d(&tmD, box, col0 + h * 32, row0);
            bulk_commit();
          }
        }
        continue;
      }
      unsigned char* box = out_w + sl * SLAB_BYTES * (Cfg::TWO_OUT ? 2 : 1);
      epi_slab_bf16<EPI>(p, r0, r1, box, col0, alpha, lane);
      fence_proxy_async();
      __syncwarp();
      if (EPI == EPI_DGELU && p.colsum) epi_slab_colsum(p, box, row0, col0, lane);
      if (lane == 0) {
        if (Cfg::TWO_OUT) { tma_store_2d(&tmAux, box, col0, row0); tma_store_2d(&tmD, box + SLAB_BYTES, col0, row0); }
        else tma_store_2d(&tmD, box, col0, row0);
        bulk_commit();
      }
    }
    if (lane == 0) bulk_wait_read<0>();                    // shared memory must outlive the stores' reads of it
    __syncwarp();
  }
  fence_before_sync();
  __syncthreads();
  if (warp == 1) { fence_after_sync(); tmem_dealloc<BN_>(tmem_base); }
}

template <int KIND, int EPI, int BN_, int CL>
int launch_small(const CUtensorMap& ta, const CUtensorMap& tb, const CUtensorMap& td, const CUtensorMap& taux, const GemmParams& p,
                 cudaStream_t st) {
  using Cfg = SmallCfg<KIND, EPI, BN_, CL>;
  auto kern = gemm_small_kernel<KIND, EPI, BN_, CL>;
  constexpr int FIXED = Cfg::AUX_BYTES + Cfg::RECV_BYTES + SM_TAIL + 1024;
  const long long ctas = (long long)p.m_tiles * p.n_tiles * CL * p.splits;
  // one CTA per SM: as deep a ring as fits; more CTAs than SMs: half the shared memory each, so that two run side by side
  // (where half leaves fewer than three stages beside the fixed part, one CTA takes it all)
  static_assert(FIXED + 3 * Cfg::STAGE <= 227 * 1024, "at least three stages fit");
  int stages = (113 * 1024 - FIXED) / Cfg::STAGE;
  if (ctas <= sm_count() || stages < 3) stages = (227 * 1024 - FIXED) / Cfg::STAGE;
  const int kbs = ceil_div(p.kb_total, CL > 1 ? CL : p.splits);
  if (stages > kbs) stages = kbs;
  if (stages > SM_MAX_STAGES) stages = SM_MAX_STAGES;
  constexpr int NEED = (Cfg::OUT_BYTES + Cfg::STAGE - 1) / Cfg::STAGE;   // the output boxes alias the ring
  static_assert(FIXED + NEED * Cfg::STAGE <= 227 * 1024, "output boxes fit");
  if (stages < NEED) stages = NEED;
  if (stages < 1 || p.kb_total < CL) return LLMB_ERR_BAD_ARG;            // every CTA of a cluster has a part of K
  const int smem = stages * Cfg::STAGE + FIXED;
  static bool attr_done = false;
  if (!attr_done) {
    const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
    if (e != cudaSuccess) return (int)e;
    attr_done = true;
  }
  return launch_pdl_cluster(CL, kern, dim3(p.m_tiles * p.n_tiles * CL, CL > 1 ? 1 : p.splits), SM_THREADS, smem, st, ta, tb, td, taux, p, stages);
}

template <int KIND, int EPI>
int pick(int bn, int cl, const CUtensorMap& ta, const CUtensorMap& tb, const CUtensorMap& td, const CUtensorMap& taux, const GemmParams& p,
         cudaStream_t st) {
  constexpr bool CLUSTERS = KIND != KIND_TF32 && EPI != EPI_ACC_F32;
  if (bn == 64 && KIND != KIND_F8F6F4) {
    if (CLUSTERS && cl == 4) return launch_small<KIND, EPI, KIND == KIND_F8F6F4 ? 128 : 64, CLUSTERS ? 4 : 1>(ta, tb, td, taux, p, st);
    if (CLUSTERS && cl == 2) return launch_small<KIND, EPI, KIND == KIND_F8F6F4 ? 128 : 64, CLUSTERS ? 2 : 1>(ta, tb, td, taux, p, st);
    return launch_small<KIND, EPI, KIND == KIND_F8F6F4 ? 128 : 64, 1>(ta, tb, td, taux, p, st);
  }
  if (CLUSTERS && cl == 2) return launch_small<KIND, EPI, 128, CLUSTERS ? 2 : 1>(ta, tb, td, taux, p, st);
  return launch_small<KIND, EPI, 128, 1>(ta, tb, td, taux, p, st);
}

template <int KIND>
int pick_epi(int epi, int bn, int cl, const CUtensorMap& ta, const CUtensorMap& tb, const CUtensorMap& td, const CUtensorMap& taux,
             const GemmParams& p, cudaStream_t st) {
  switch (epi) {
    case EPI_NONE: return pick<KIND, EPI_NONE>(bn, cl, ta, tb, td, taux, p, st);
    case EPI_BIAS: return pick<KIND, EPI_BIAS>(bn, cl, ta, tb, td, taux, p, st);
    case EPI_BIAS_GELU: return pick<KIND, EPI_BIAS_GELU>(bn, cl, ta, tb, td, taux, p, st);
    case EPI_DGELU: return pick<KIND, EPI_DGELU>(bn, cl, ta, tb, td, taux, p, st);
    case EPI_ACC_F32: return pick<KIND, EPI_ACC_F32>(bn, cl, ta, tb, td, taux, p, st);
    case EPI_BIAS_RESID: return pick<KIND, EPI_BIAS_RESID>(bn, cl, ta, tb, td, taux, p, st);
    case EPI_STORE_F32: return pick<KIND, EPI_STORE_F32>(bn, cl, ta, tb, td, taux, p, st);
  }
  return LLMB_ERR_BAD_ARG;
}
}  // namespace

int llmb_gemm_small_launch(int kind, int epi, int bn, int cl, const CUtensorMap& ta, const CUtensorMap& tb, const CUtensorMap& td,
                           const CUtensorMap& taux, const GemmParams& p, cudaStream_t st) {
  switch (kind) {
    case KIND_F16: return pick_epi<KIND_F16>(epi, bn, cl, ta, tb, td, taux, p, st);
    case KIND_TF32: return pick_epi<KIND_TF32>(epi, bn, cl, ta, tb, td, taux, p, st);
    case KIND_F8F6F4: return pick_epi<KIND_F8F6F4>(epi, bn, cl, ta, tb, td, taux, p, st);
  }
  return LLMB_ERR_BAD_ARG;
}
