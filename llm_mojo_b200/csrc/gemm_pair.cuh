// The CTA-pair GEMM kernel and its launch; gemm.cu instantiates it for bf16, TF32 and fp8 operands, gemm_scaled.cu for block-scaled ones.
#pragma once
#include "gemm_common.cuh"

namespace {
// CTA-pair GEMM kernel: a cluster of two CTAs computes a 256 x 256 tile with cta_group::2 MMAs.  Each
// CTA stages its own 128 rows of A and its own 128-row half of B (half the B traffic per SM, and
// a ring of 32 KB stages instead of 48 KB ones), the leader issues the MMAs, and both
// CTAs drain their 128 x 256 accumulator halves.  No load is multicast: every CTA fetches only
// the tiles it owns; the peer's TMA completions are reported to the leader's mbarrier.
constexpr int B2_STAGE = 128 * ROW_BYTES;             // 16 KB: this CTA's half of the B tile
constexpr int STAGE2_BYTES = A_STAGE + B2_STAGE;      // 32 KB
constexpr int SMEM2_TAIL = 512;                        // barriers, TMEM slot, abort flag
// TMA producer, MMA issuer, 8 epilogue warps, 2 gather copier warps.
//
// What a tile's epilogue costs its warps beside the arithmetic, and what was done about it (cycles per tile and warp at K = 768, where a tile's
// MMAs take 6144; clock traces): the hand-back of the accumulator released at cluster scope, which waited for every store and reduction in
// flight (1200 - 2500; relaxed now, see mbar_arrive_cluster); five integer divisions for the tile's place (500); the bias from L2 (700 a
// slab in which its loads took turns; the four of 32 columns go out together now); with an auxiliary input one box per warp, whose load,
// work and store took turns (two boxes now, each loaded again as soon as it has left); column sums before the store of the box (after it now).  Sixteen epilogue warps hid some of
// that behind one another, at 96 registers and with four of them contending for a scheduler; with it gone eight are faster with two outputs,
// nearly as fast with an auxiliary input, and one form serves both.  C 768, N 3072, us, before / 16 / 8 warps: bias + GELU, M 16384 81.6 / 79.0 / 71.0, M
// 65536 324 / 304 - 313 / 265 - 275; dGELU + column sums, M 16384 85.0 / 76.5 / 78.4.  What bounds a tile now is what it moves: 390 KB of operands and 128 KB of auxiliary input and results per CTA at the 60 - 70
// bytes a cycle that an SM gets when all of them load.
constexpr int EPI_WARPS = 8;
constexpr int PAIR_THREADS = 32 * (4 + EPI_WARPS);
//
// Block-scaled operands (KIND_MXF8: e4m3 / e5m2 bytes, one ue8m0 scale per 32 values; KIND_NVF4: packed e2m1, one ue4m3 scale per 16), both
// K-major: a stage's 128-byte rows hold 128 / 256 values of K and come with their scales, in the atoms of 512 bytes that gemm_scaled.cu
// describes: those of this CTA's 128 rows of A (SF_A bytes) and those of all 256 rows of B, of which either CTA needs every one.  The
// leader copies a stage's atoms to both CTAs' tensor memory (tcgen05.cp.cta_group::2) just ahead of the MMAs that use them.  Those 48
// columns leave no room for two 256-column accumulators, so the two OVERLAP in one 64-column slab: accumulator 0 = [0, 256), accumulator 1
// = [192, 448), scales from 448.  The epilogue of a tile reads that slab first and says so (`tover`); the next tile's MMAs start when
// it is read and the tile before has been drained completely (`tempty`).
template <int KIND, int EPI> struct PairCfg {
  static constexpr bool SCALED = KIND == KIND_MXF8 || KIND == KIND_NVF4;
  static constexpr int SF_A = KIND == KIND_NVF4 ? 2048 : KIND == KIND_MXF8 ? 512 : 0;     // scales of 128 rows x one stage
  static constexpr int STAGES = EpiCfg<EPI>::STAGES - (SCALED ? 1 : 0);
  static constexpr int SMEM = STAGES * (STAGE2_BYTES + 3 * SF_A) + 4 * EpiCfg<EPI>::WARP_STAGE + 1024 + SMEM2_TAIL;
  static constexpr uint32_t ACC1_COL = SCALED ? 192 : BN;
};
constexpr uint32_t SFA_COL = 448, SFB_COL = 464;
// the tensor maps of the scales: [row blocks of 128][atoms along K * 64] 8-byte words, boxes of one / two row blocks and one stage
template <int KIND> struct ScaleMaps {};
template <> struct ScaleMaps<KIND_MXF8> { CUtensorMap a, b; };
template <> struct ScaleMaps<KIND_NVF4> { CUtensorMap a, b; };
constexpr int FLAG_ROWS_READY = 6;                     // flag kind (layout of comm.cu: flags[kind][8 ranks])
constexpr int FLAG_PARAM = 3;                          // owners announce the optimizer step their parameter shard holds

template <int KIND, int EPI>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(PAIR_THREADS, 1)
gemm_pair_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                 const __grid_constant__ CUtensorMap tmD, const __grid_constant__ CUtensorMap tmAux, const __grid_constant__ ScaleMaps<KIND> sfm,
                 const GemmParams p) {
  using Cfg = EpiCfg<EPI>;
  using PCfg = PairCfg<KIND, EPI>;
  constexpr bool SCALED = PCfg::SCALED;
  constexpr int NST = PCfg::STAGES, SF_A = PCfg::SF_A;
  constexpr int WSB = Cfg::WARP_STAGE;
  constexpr int BKE = KindTraits<KIND>::BKE;            // elements of a swizzled row: K of a stage, and the columns of an MN-major chunk
  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  unsigned char* epi_stage = smem + NST * STAGE2_BYTES;
  unsigned char* sf_stage = epi_stage + 4 * WSB;       // [NST][A rows][B rows 0..127][B rows 128..255]
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(sf_stage + NST * 3 * SF_A);
  uint64_t* empty_bar = full_bar + NST;
  uint64_t* tfull_bar = empty_bar + NST;
  uint64_t* tempty_bar = tfull_bar + 2;
  uint64_t* aux_bar = tempty_bar + 2;                   // [8 warps][2 boxes]: auxiliary-input tiles landed
  uint64_t* tover_bar = aux_bar + 16;                   // [2] block-scaled: the columns shared with the other accumulator are read
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tover_bar + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  const uint32_t cta = cluster_ctarank();              // 0 = leader
  const bool leader = cta == 0;

  if (threadIdx.x == 0) {
    for (int s = 0; s < NST; ++s) { mbar_init(&full_bar[s], 1); mbar_init(&empty_bar[s], 1); }
    for (int a = 0; a < 2; ++a) { mbar_init(&tfull_bar[a], 1); mbar_init(&tempty_bar[a], 2 * EPI_WARPS); mbar_init(&tover_bar[a], 8); }
    for (int a = 0; a < 16; ++a) mbar_init(&aux_bar[a], 1);
    *abort_flag = 0;
    fence_barrier_init();
    prefetch_tmap(&tmA); prefetch_tmap(&tmB);
    if constexpr (SCALED) { prefetch_tmap(&sfm.a); prefetch_tmap(&sfm.b); }
    if (p.tma_epi) { prefetch_tmap(&tmD); prefetch_tmap(&tmAux); }
  }
  if (warp == 1) tmem_alloc_pair<512>(tmem_slot);
  fence_before_sync();
  __syncthreads();
  cluster_sync_all();                                   // both CTAs' barriers exist before any remote signal
  fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  if (p.g.W <= 1 && p.pull.nseg == 0 && p.pull.nwait == 0) pdl_trigger();   // else this kernel waits for other GPUs or streams

  const int m_tiles = ceil_div(p.M, 2 * BM);            // cluster tiles of 256 rows
  const int tiles_per_split = m_tiles * p.n_tiles;
  const int total_units = tiles_per_split * p.splits;
  const int cluster_id = blockIdx.x >> 1, num_clusters = gridDim.x >> 1;
  constexpr int BAND2 = 8;

  // n / d for 0 <= n < 2^24, given 1 / d: five integer divisions a tile cost each role about 500 cycles
  auto div = [](int n, int d, float inv) {
    int q = __float2int_rz(__int2float_rn(n) * inv);
    const int r = n - q * d;
    if (r < 0) --q; else if (r >= d) ++q;
    return q;
  };
  const int band_sz = BAND2 * p.n_tiles, last_band = m_tiles % BAND2;
  const float inv_band = 1.0f / (float)band_sz, inv_last = 1.0f / (float)max(last_band, 1), inv_tiles = 1.0f / (float)tiles_per_split;
  auto unit_k = [&](int split, int& kb0, int& kb1) { kb0 = split * p.kb_per_split; kb1 = min(p.kb_total, kb0 + p.kb_per_split); };
  auto unit_split = [&](int unit) { return p.splits > 1 ? div(unit, tiles_per_split, inv_tiles) : 0; };
  auto unit_coords = [&](int unit, int& m_blk, int& n_blk, int& kb0, int& kb1) {
    const int split = unit_split(unit), t = unit - split * tiles_per_split;
    const int b = div(t, band_sz, inv_band), r = t - b * band_sz;
    const bool full = (b + 1) * BAND2 <= m_tiles;
    n_blk = full ? r / BAND2 : div(r, last_band, inv_last);
    m_blk = b * BAND2 + r - n_blk * (full ? BAND2 : last_band);
    if (p.g.W > 1) m_blk = (m_blk + p.g.me * p.g.tiles_per_chunk) % m_tiles;   // the local chunk's tiles come first
    unit_k(split, kb0, kb1);
  };

  // While the kernel before this one drains: the first ring of B (a forward or input-gradient GEMM's weights) into L2, once per column
  // of tiles.  A hint only, so it may run before the wait; if that kernel writes B, the loads below still read what it wrote.
  if (warp == 0 && cluster_id < total_units && p.pull.nwait == 0) {
    int m_blk, n_blk, kb0, kb1; unit_coords(cluster_id, m_blk, n_blk, kb0, kb1);
    const int n0 = n_blk * BN + (int)cta * 128;
    if (m_blk % BAND2 == 0 && elect_one())
      for (int kb = kb0; kb < kb1 && kb < kb0 + NST; ++kb) {
        if (!p.b_mn) tma_prefetch_l2_2d(&tmB, kb * BKE, n0);
        else if (p.b_3d) tma_prefetch_l2_3d(&tmB, 0, kb * BKE, n0 / BKE);
      }
    __syncwarp();
  }
  pdl_wait();

  if (warp == 0) {
    // ------------------------------------------------------------ TMA producer (both CTAs)
    // warp-uniform loop, one elected lane issues (same reasoning as for the MMA issuer below).
    // The loop, not TMA, can be what paces an MN-major operand: the four MMAs of a k-block take 512 cycles, the barrier round trips of a
    // turn about 300, and a chunk index m0 / (k-block size) with a divisor known at run time only cost 155 more per operand and turn
    // (690 cycles in all for a weight gradient; 380 as it is now).  Hence BKE.  M 65536, C 768: weight gradients of a layer 891 -> 636
    // us, input gradients 917 -> 730; M 4096, C 768: 82.8 -> 69.0, 82.0 -> 77.4.
    {
      int stage = 0; uint32_t phase = 0;
      const uint32_t lead_full0 = mapa_u32(smem_u32(&full_bar[0]), 0);
      bool ok = true;
      int landed = -1;
      // B operand pulled from peers (by this kernel's copier warps or by an earlier kernel's): all of it must have landed
      for (int w = 0; w < p.pull.nwait && ok; ++w) {
        unsigned spins = 0;
        while ((int)(ld_acquire_gpu(p.pull.wait_counts[w]) - p.pull.wait_target[w]) < 0) {
          if (++spins > (1u << 24)) { ok = false; break; }
          __nanosleep(100);
        }
      }
      if (p.pull.nwait) fence_proxy_async_all();          // the copiers' generic-proxy stores before this warp's TMA reads
      if (!ok && lane == 0) { *abort_flag = 1; atomicExch(p.status, LLMB_ERR_TIMEOUT); }
      for (int unit = cluster_id; unit < total_units && ok && !*abort_flag; unit += num_clusters) {
        int m_blk, n_blk, kb0, kb1; unit_coords(unit, m_blk, n_blk, kb0, kb1);
        const int m0 = m_blk * 2 * BM + (int)cta * BM, n0 = n_blk * BN + (int)cta * 128;
        if (p.g.W > 1) {                                 // gathered A: this tile's chunk must have landed in local memory
          const int chunk = m_blk / p.g.tiles_per_chunk;
          if (chunk != p.g.me && chunk != landed) {
            unsigned spins = 0;
            while ((int)(ld_acquire_gpu(&p.g.counts[chunk]) - p.g.target) < 0) {
              if (++spins > (1u << 24)) { ok = false; break; }
              __nanosleep(100);
            }
            if (!ok) break;
            fence_proxy_async_all();                      // the copiers' generic-proxy stores before this warp's TMA reads
            landed = chunk;
          }
        }
        for (int kb = kb0; kb < kb1; ++kb) {
          if (!mbar_wait(&empty_bar[stage], phase ^ 1)) { ok = false; break; }
          unsigned char* sa = smem + stage * STAGE2_BYTES;
          unsigned char* sb = sa + A_STAGE;
          const uint32_t lead_full = lead_full0 + stage * 8;
          const int k0 = kb * BKE;
          if (elect_one()) {
            if (leader) mbar_expect_tx(&full_bar[stage], 2 * (STAGE2_BYTES + 3 * SF_A));     // bytes of both CTAs
            if constexpr (SCALED) {
              unsigned char* sf = sf_stage + stage * 3 * SF_A;
              tma_load_2d_pair(sf, &sfm.a, lead_full, kb * (SF_A / 8), m_blk * 2 + (int)cta);
              tma_load_2d_pair(sf + SF_A, &sfm.b, lead_full, kb * (SF_A / 8), n_blk * 2);
            }
            if (!p.a_mn) tma_load_2d_pair(sa, &tmA, lead_full, k0, m0);
            else if (p.a_3d) tma_load_3d_pair(sa, &tmA, lead_full, 0, k0, m0 / BKE);
            else {
#pragma unroll
              for (int c = 0; c < BM / BKE; ++c) tma_load_2d_pair(sa + c * BKE * ROW_BYTES, &tmA, lead_full, m0 + c * BKE, k0);
            }
            if (!p.b_mn) tma_load_2d_pair(sb, &tmB, lead_full, k0, n0);
            else if (p.b_3d) tma_load_3d_pair(sb, &tmB, lead_full, 0, k0, n0 / BKE);
            else {
#pragma unroll
              for (int c = 0; c < 128 / BKE; ++c) tma_load_2d_pair(sb + c * BKE * ROW_BYTES, &tmB, lead_full, n0 + c * BKE, k0);
            }
          }
          __syncwarp();
          if (++stage == NST) { stage = 0; phase ^= 1; }
        }
        if (!ok) break;
      }
      if (!ok && lane == 0) { *abort_flag = 1; atomicExch(p.status, LLMB_ERR_TIMEOUT); }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------ MMA issuer (leader CTA only)
    // The whole warp walks the loop (uniform control flow, so descriptors and barrier addresses stay in
    // uniform registers) and one elected lane issues.  Everything that does not change per k-block is
    // computed once: the descriptors of stage 0 (a later stage only adds its byte offset >> 4 to the
    // address field), the per-MMA descriptor increments and the cluster addresses of the barriers.
    if (leader) {
      int stage = 0; uint32_t phase = 0;
      int it = 0;
      const uint64_t adesc0 = make_smem_desc(smem_u32(smem), p.a_lbo, p.a_sbo, p.a_layout);
      const uint64_t bdesc0 = make_smem_desc(smem_u32(smem) + A_STAGE, p.b_lbo, p.b_sbo, p.b_layout);
      const uint64_t a_inc = (uint64_t)(p.a_kstep >> 4), b_inc = (uint64_t)(p.b_kstep >> 4);
      const uint64_t sf0 = SCALED ? make_sf_desc(smem_u32(sf_stage)) : 0;
      const uint32_t idesc = p.idesc;
      const uint32_t eb0 = mapa_u32(smem_u32(&empty_bar[0]), 0), eb1 = mapa_u32(smem_u32(&empty_bar[0]), 1);
      const uint32_t tb0 = mapa_u32(smem_u32(&tfull_bar[0]), 0), tb1 = mapa_u32(smem_u32(&tfull_bar[0]), 1);
      bool ok = true;
      for (int unit = cluster_id; unit < total_units && !*abort_flag; unit += num_clusters, ++it) {
        int kb0, kb1; unit_k(unit_split(unit), kb0, kb1);
        const int acc = it & 1;
        const uint32_t acc_phase = (it >> 1) & 1;
        if (!mbar_wait(&tempty_bar[acc], acc_phase ^ 1)) { ok = false; break; }
        if (SCALED && it > 0 && !mbar_wait(&tover_bar[acc ^ 1], ((it - 1) >> 1) & 1)) { ok = false; break; }
        fence_after_sync();
        const uint32_t d_tmem = tmem_base + acc * PCfg::ACC1_COL;
        for (int kb = kb0; kb < kb1; ++kb) {
          if (!mbar_wait(&full_bar[stage], phase)) { ok = false; break; }
          fence_after_sync();
          const uint64_t adesc = adesc0 + (uint64_t)(stage * (STAGE2_BYTES >> 4));
          const uint64_t bdesc = bdesc0 + (uint64_t)(stage * (STAGE2_BYTES >> 4));
          if (elect_one()) {
            if constexpr (SCALED) {
              // Up to four MMAs (32 bytes of K per row each), the scales of each on their way to tensor memory beside the MMA before it; the
              // copies and MMAs of a thread run in order.  Unrolled: a loop over the copies and then one over the MMAs, with trip counts known
              // at run time, took 930 cycles per NVFP4 k-block where the MMAs take 512, and products of few tiles were slower than the single-CTA
              // kernel before this one.  us, that kernel / the loops / now: NVFP4 4096 x 768 x 3072 9.63 / 10.53 / 8.80, 128 x 1600 x 6400
              // 14.4 / 15.3 / 11.5, 8192 x 1600 x 6400 55.2 / 54.0 / 39.5; MXFP8 128 x 1280 x 5120 with residual 21.1 / 19.9 / 18.4.
              constexpr int VALS = KIND == KIND_NVF4 ? 64 : 32, ATOMS = SF_A / 512;
              const int nk = min(4, (p.K - kb * 4 * VALS + VALS - 1) / VALS);
              const uint32_t sfa_t = tmem_base + SFA_COL, sfb_t = tmem_base + SFB_COL;
              const uint64_t sfa = sf0 + (uint64_t)(stage * (3 * SF_A >> 4)), sfb = sfa + (uint64_t)(SF_A >> 4);
              auto scales = [&](int k) {
                tmem_cp_sf_pair(sfa_t + 4 * k, sfa + (uint64_t)(k * 32));
                tmem_cp_sf_pair(sfb_t + 8 * k, sfb + (uint64_t)(k * 32));
                tmem_cp_sf_pair(sfb_t + 8 * k + 4, sfb + (uint64_t)((SF_A >> 4) + k * 32));
              };
              scales(0);
#pragma unroll
              for (int k = 0; k < 4; ++k) {
                if (k + 1 < ATOMS && k + 1 < nk) scales(k + 1);
                if (k >= nk) continue;
                const uint32_t acc_in = kb > kb0 || k > 0 ? 1u : 0u;
                if constexpr (KIND == KIND_NVF4)
                  umma_nvfp4_pair(d_tmem, adesc + k * a_inc, bdesc + k * b_inc, idesc, sfa_t + 4 * k, sfb_t + 8 * k, acc_in);
                else                                        // byte k of the atom's columns: in the descriptor and in the addresses
                  umma_mxfp8_pair(d_tmem, adesc + k * a_inc, bdesc + k * b_inc, idesc | ((uint32_t)k << 29) | ((uint32_t)k << 4),
                                  sfa_t | ((uint32_t)k << 30), sfb_t | ((uint32_t)k << 30), acc_in);
              }
            } else {
              umma_ss_pair<KIND>(d_tmem, adesc, bdesc, idesc, kb > kb0 ? 1u : 0u);
#pragma unroll
              for (int k = 1; k < 4; ++k) umma_ss_pair<KIND>(d_tmem, adesc + k * a_inc, bdesc + k * b_inc, idesc, 1u);
            }
            umma_commit_pair(eb0 + stage * 8);            // stage free in both CTAs once these MMAs have read it
            umma_commit_pair(eb1 + stage * 8);
          }
          __syncwarp();
          if (++stage == NST) { stage = 0; phase ^= 1; }
        }
        if (!ok) break;
        if (elect_one()) {
          umma_commit_pair(tb0 + acc * 8);
          umma_commit_pair(tb1 + acc * 8);
        }
        __syncwarp();
      }
      if (!ok && lane == 0) { *abort_flag = 1; atomicExch(p.status, LLMB_ERR_TIMEOUT); }
    }
  } else if (warp >= 2 + EPI_WARPS) {
    // ------------------------------------------------------------ gather copiers (the last two warps, both CTAs)
    if (p.g.W > 1) {
      // Slices of 32 KB are handed out by ticket, so the copy completes with whatever CTAs are resident.
      constexpr long long SLICE = 2048;                  // 16-byte vectors
      bool ok = true;
      for (int step = 1; step < p.g.W && ok; ++step) {
        const int r = (p.g.me + step) % p.g.W;
        // rank r has announced that its chunk is complete (bounded wait, one lane polls)
        if (lane == 0) {
          const unsigned* f = reinterpret_cast<const unsigned*>(p.g.flags) + FLAG_ROWS_READY * 8 + r;
          unsigned spins = 0;
          while ((int)(ld_acquire_sys(f) - p.g.seq) < 0) {
            if (++spins > (1u << 24)) { ok = false; break; }
            __nanosleep(200);
          }
        }
        ok = __shfl_sync(0xffffffffu, ok, 0);
        if (!ok) break;
        const uint4* src = reinterpret_cast<const uint4*>(p.g.peer_src[r]);
        uint4* dst = reinterpret_cast<uint4*>(p.g.local) + (long long)r * p.g.chunk_vecs;
        for (;;) {
          unsigned ticket = 0;
          if (lane == 0) ticket = atomicAdd(&p.g.counts[8 + r], 1u);
          ticket = __shfl_sync(0xffffffffu, ticket, 0);
          if (ticket >= p.g.target) break;
          const long long v0 = (long long)ticket * SLICE;
          const long long v1 = v0 + SLICE < p.g.chunk_vecs ? v0 + SLICE : p.g.chunk_vecs;
          long long v = v0 + lane;
          for (; v + 7 * 32 < v1; v += 8 * 32) {         // eight peer loads in flight per thread
            uint4 t[8];
#pragma unroll
            for (int k = 0; k < 8; ++k) t[k] = ld_nc_v4(src + v + k * 32);
#pragma unroll
            for (int k = 0; k < 8; ++k) dst[v + k * 32] = t[k];
          }
          for (; v < v1; v += 32) dst[v] = ld_nc_v4(src + v);
          __threadfence();
          __syncwarp();
          if (lane == 0) atomicAdd(&p.g.counts[r], 1u);
        }
      }
      if (!ok && lane == 0) { *abort_flag = 1; atomicExch(p.status, LLMB_ERR_TIMEOUT); }
    } else if (p.pull.nseg > 0) {
      // ZeRO-3 parameter pull: same ticketed 32 KB slices, one list of segments instead of one chunk per rank
      constexpr long long SLICE = 2048;                  // 16-byte vectors
      bool ok = true;
      for (int sgm = 0; sgm < p.pull.nseg && ok; ++sgm) {
        if (p.pull.seq && lane == 0) {                    // the owner's shard holds this step's parameters
          const unsigned* f = reinterpret_cast<const unsigned*>(p.pull.flags) + FLAG_PARAM * 8 + p.pull.owner[sgm];
          unsigned spins = 0;
          while ((int)(ld_acquire_sys(f) - p.pull.seq) < 0) {
            if (++spins > (1u << 24)) { ok = false; break; }
            __nanosleep(200);
          }
        }
        ok = __shfl_sync(0xffffffffu, ok, 0);
        if (!ok) break;
        const uint4* src = reinterpret_cast<const uint4*>(p.pull.src[sgm]);
        uint4* dst = reinterpret_cast<uint4*>(p.pull.dst[sgm]);
        const long long nvec = p.pull.vecs[sgm];
        const unsigned target = (unsigned)((nvec + SLICE - 1) / SLICE);
        for (;;) {
          unsigned ticket = 0;
          if (lane == 0) ticket = atomicAdd(&p.pull.counts[8 + sgm], 1u);
          ticket = __shfl_sync(0xffffffffu, ticket, 0);
          if (ticket >= target) break;
          const long long v0 = (long long)ticket * SLICE;
          const long long v1 = v0 + SLICE < nvec ? v0 + SLICE : nvec;
          long long v = v0 + lane;
          for (; v + 7 * 32 < v1; v += 8 * 32) {         // eight loads in flight per thread
            uint4 t[8];
#pragma unroll
            for (int k = 0; k < 8; ++k) t[k] = ld_nc_v4(src + v + k * 32);
#pragma unroll
            for (int k = 0; k < 8; ++k) dst[v + k * 32] = t[k];
          }
          for (; v < v1; v += 32) dst[v] = ld_nc_v4(src + v);
          __threadfence();
          __syncwarp();
          if (lane == 0) atomicAdd(&p.pull.counts[sgm], 1u);
        }
      }
      if (!ok && lane == 0) { *abort_flag = 1; atomicExch(p.status, LLMB_ERR_TIMEOUT); }
    }
  } else {
    // ------------------------------------------------------------ epilogue (warps 2..9, both CTAs)
    // Eight warps: warp % 4 selects the 32-row band (the TMEM lane quarter a warp may read), (warp - 2) / 4 the
    // 128-column half of the tile, i.e. two 64-column slabs per warp and tile.  The register epilogue (fp32
    // outputs, layouts without a tensor map) keeps four working warps with all four slabs of a band each.
    // An fp32-storage problem (tf32) moves its 128 columns as four 32-column boxes through the same buffers.
    constexpr bool F32_IO = KIND == KIND_TF32 && !Cfg::F32_OUT, AUX = Cfg::AUX_IN;
    constexpr int NBOX = F32_IO ? 4 : 2, BOXC = F32_IO ? 32 : 64;
    const int q = warp & 3, e = warp - 2, hcol = e >> 2;
    const bool tma_epi = p.tma_epi;                       // warp-uniform
    unsigned char* wstage = epi_stage + e * (tma_epi ? WSB / 2 : WSB);
    uint64_t* abar = aux_bar + e * 2;
    const int band_off = (int)cta * BM + q * 32;
    uint32_t aux_phase = 0, aux_pending = 0;              // per-slab-buffer phase bits / loads in flight (warp-uniform)
    // auxiliary-input tiles of a work unit: one box per slab that lies inside the matrix (ls < NBOX), in buffer ls & 1
    auto slab_valid = [&](int row0, int n0, int ls) { return row0 < p.M && n0 + hcol * 128 + ls * BOXC < p.N; };
    auto aux_issue = [&](int row0, int n0, int ls) {      // all lanes keep the books, lane 0 issues
      if (!slab_valid(row0, n0, ls)) return;
      const int b = ls & 1;
      aux_pending |= 1u << b;
      if (lane == 0) {
        mbar_expect_tx(&abar[b], SLAB_BYTES);
        tma_load_2d(wstage + b * SLAB_BYTES, &tmAux, &abar[b], n0 + hcol * 128 + ls * BOXC, row0);
      }
    };
    if (AUX && tma_epi && cluster_id < total_units) {
      int m_blk, n_blk, kb0, kb1; unit_coords(cluster_id, m_blk, n_blk, kb0, kb1);
      for (int ls = 0; ls < 2; ++ls) aux_issue(m_blk * 2 * BM + band_off, n_blk * BN, ls);
    }
    const uint32_t te0 = mapa_u32(smem_u32(&tempty_bar[0]), 0), to0 = mapa_u32(smem_u32(&tover_bar[0]), 0);
    const float alpha = p.alpha ? *p.alpha : 1.0f;
    int it = 0;
    for (int unit = cluster_id; unit < total_units && !*abort_flag; unit += num_clusters, ++it) {
      int m_blk, n_blk, kb0, kb1; unit_coords(unit, m_blk, n_blk, kb0, kb1);
      const int acc = it & 1;
      const uint32_t acc_phase = (it >> 1) & 1;
      if (!mbar_wait(&tfull_bar[acc], acc_phase)) { *abort_flag = 1; atomicExch(p.status, LLMB_ERR_TIMEOUT); break; }
      fence_after_sync();
      const int n0 = n_blk * BN;
      const int row0 = m_blk * 2 * BM + band_off;
      const uint32_t tacc = tmem_base + ((uint32_t)(q * 32) << 16) + acc * PCfg::ACC1_COL;
      if (!tma_epi) {
        if (e < 4) epilogue_warp<EPI>(p, tacc, wstage, row0, n0, alpha, lane);
        if (SCALED && e < 4) {
          fence_before_sync();
          __syncwarp();
          if (lane == 0) mbar_arrive_cluster(to0 + acc * 8);
        }
      } else {
        const int nunit = unit + num_clusters;
        const bool has_next = AUX && nunit < total_units;
        int nrow0 = 0, nn0 = 0;
        if (has_next) { int mb, nb, k0, k1; unit_coords(nunit, mb, nb, k0, k1); nrow0 = mb * 2 * BM + band_off; nn0 = nb * BN; }
        bool ok = true;
        // block-scaled: the slab shared with the other accumulator goes first, the last of accumulator 0 and the first of accumulator 1
        const bool over = SCALED && hcol == (acc ? 0 : 1);
        const int flip = SCALED && hcol == 1 && acc == 0 ? 1 : 0;
#pragma unroll 1
        for (int i = 0; i < NBOX; ++i) {
          const int ls = i ^ flip;
          const bool valid = slab_valid(row0, n0, ls);     // warp-uniform
          if (!SCALED && !valid) break;
          const int col0 = n0 + hcol * 128 + ls * BOXC;
          uint32_t r0[32], r1[32];
          if (valid) {
            tmem_ld32(tacc + hcol * 128 + ls * BOXC, r0);
            if (!F32_IO) tmem_ld32(tacc + hcol * 128 + ls * BOXC + 32, r1);
            tmem_wait_ld();
          }
          if (SCALED) {
            if (i == 0 && over) {
              fence_before_sync();
              __syncwarp();
              if (lane == 0) mbar_arrive_cluster(to0 + acc * 8);
            }
            if (!valid) continue;
          }
          unsigned char* buf;
          if (Cfg::F32_OUT) {
            // fp32 accumulate / store: the slab leaves as two boxes of 32 rows x 32 fp32 columns (128-byte rows, swizzled), which
            // the TMA engine adds into (split-K partial sums, gradient accumulation) or writes to the output; the warp goes on
            // to its next slab at once instead of waiting on 64 vector reductions per lane.
            buf = wstage;
            if (lane == 0) bulk_wait_read<0>();           // the previous slab's boxes have been read
            __syncwarp();
            unsigned char* myrow = buf + lane * 128;
#pragma unroll
            for (int c = 0; c < 8; ++c) {
              const int sw = (c ^ (lane & 7)) << 4;
              *reinterpret_cast<float4*>(myrow + sw) = make_float4(__uint_as_float(r0[4 * c]) * alpha, __uint_as_float(r0[4 * c + 1]) * alpha,
                                                                   __uint_as_float(r0[4 * c + 2]) * alpha, __uint_as_float(r0[4 * c + 3]) * alpha);
              *reinterpret_cast<float4*>(myrow + SLAB_BYTES + sw) = make_float4(__uint_as_float(r1[4 * c]) * alpha, __uint_as_float(r1[4 * c + 1]) * alpha,
                                                                                __uint_as_float(r1[4 * c + 2]) * alpha, __uint_as_float(r1[4 * c + 3]) * alpha);
            }
            fence_proxy_async();
            __syncwarp();
            if (lane == 0) {
              if (EPI == EPI_ACC_F32) {
                tma_reduce_add_2d(&tmD, buf, col0, row0);
                if (col0 + 32 < p.N) tma_reduce_add_2d(&tmD, buf + SLAB_BYTES, col0 + 32, row0);
              } else {
                tma_store_2d(&tmD, buf, col0, row0);
                if (col0 + 32 < p.N) tma_store_2d(&tmD, buf + SLAB_BYTES, col0 + 32, row0);
              }
              bulk_commit();
            }
            continue;
          }
          if (AUX) {
            const int b = ls & 1;
            buf = wstage + b * SLAB_BYTES;
            if (!mbar_wait(&abar[b], (aux_phase >> b) & 1)) { ok = false; break; }
            aux_phase ^= 1u << b; aux_pending &= ~(1u << b);
          } else {
            buf = wstage;
            // the previous slab's stores have read the buffer
            if (lane == 0) { if (Cfg::TWO_OUT && !F32_IO) bulk_wait_read<1>(); else bulk_wait_read<0>(); }
            __syncwarp();
          }
          if (F32_IO) {
            epi_box_f32<EPI>(p, r0, buf, buf + SLAB_BYTES, col0, alpha, lane);
            fence_proxy_async();
            __syncwarp();
            if (lane == 0) {
              if (Cfg::TWO_OUT) { tma_store_2d(&tmAux, buf, col0, row0); tma_store_2d(&tmD, buf + SLAB_BYTES, col0, row0); }
              else tma_store_2d(&tmD, buf, col0, row0);
              bulk_commit();
            }
            if (AUX && ls + 2 < NBOX && slab_valid(row0, n0, ls + 2)) {   // this buffer's next box, once the store has read it
              if (lane == 0) bulk_wait_read<0>();
              __syncwarp();
              aux_issue(row0, n0, ls + 2);
            }
            continue;
          }
          if (Cfg::TWO_OUT) {
            uint4 pre[8];
            epi_half_pre<0>(p, r0, buf, col0, alpha, lane, pre);
            epi_half_pre<1>(p, r1, buf, col0, alpha, lane, pre);
            fence_proxy_async();
            __syncwarp();
            if (lane == 0) { tma_store_2d(&tmAux, buf, col0, row0); bulk_commit(); }
            epi_slab_gelu(pre);
            if (lane == 0) bulk_wait_read<1>();   // the previous slab's activations have left
            __syncwarp();
            epi_slab_store(pre, buf + SLAB_BYTES, lane);
            fence_proxy_async();
            __syncwarp();
            if (lane == 0) { tma_store_2d(&tmD, buf + SLAB_BYTES, col0, row0); bulk_commit(); }
            continue;
          }
          epi_slab_bf16<EPI>(p, r0, r1, buf, col0, alpha, lane);
          fence_proxy_async();
          __syncwarp();
          if (lane == 0) { tma_store_2d(&tmD, buf, col0, row0); bulk_commit(); }
          if (EPI == EPI_DGELU && p.colsum) { epi_slab_colsum(p, buf, row0, col0, lane); __syncwarp(); }
        }
        if (!ok) { *abort_flag = 1; atomicExch(p.status, LLMB_ERR_TIMEOUT); break; }
        if (AUX && has_next) {                            // refill each buffer once its store has been read
          // (a unit at the right edge may have stored its last slab from buffer 0: then both stores must have been read)
          if (lane == 0) { if (slab_valid(row0, n0, NBOX - 1) && !flip) bulk_wait_read<1>(); else bulk_wait_read<0>(); }
          __syncwarp();
          aux_issue(nrow0, nn0, 0);
          if (lane == 0) bulk_wait_read<0>();
          __syncwarp();
          aux_issue(nrow0, nn0, 1);
        }
      }
      fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(te0 + acc * 8);   // the leader owns the accumulator hand-back
    }
    if (tma_epi) {
      // nothing of this CTA's shared memory may still be a source or a destination of a copy at exit
      for (int ls = 0; ls < 2; ++ls)
        if (aux_pending & (1u << ls)) (void)mbar_wait(&abar[ls], (aux_phase >> ls) & 1);
      if (lane == 0) bulk_wait_read<0>();
      __syncwarp();
    }
  }

  fence_before_sync();
  __syncthreads();
  cluster_sync_all();                                   // the peer may still be signalling / reading this CTA's smem
  if (warp == 1) { fence_after_sync(); tmem_dealloc_pair<512>(tmem_base); }
}

template <int KIND, int EPI>
int launch_pair(const CUtensorMap& ta, const CUtensorMap& tb, const CUtensorMap& td, const CUtensorMap& taux,
                const ScaleMaps<KIND>& sfm, const GemmParams& p, int grid, cudaStream_t st) {
  static bool attr_done = false;
  constexpr int SMEM = PairCfg<KIND, EPI>::SMEM;
  static_assert(SMEM <= 227 * 1024, "shared memory of a CTA");
  if (!attr_done) {
    cudaError_t e = cudaFuncSetAttribute(gemm_pair_kernel<KIND, EPI>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM);
    if (e != cudaSuccess) return (int)e;
    attr_done = true;
  }
  return launch_pdl(gemm_pair_kernel<KIND, EPI>, grid, PAIR_THREADS, SMEM, st, ta, tb, td, taux, sfm, p);
}
// ... by the epilogue's number, on as many pairs as there are work units (256 x 256 tiles x parts of K), at most one per two SMs
template <int KIND>
int launch_pair_epi(int epi, const CUtensorMap& ta, const CUtensorMap& tb, const CUtensorMap& td, const CUtensorMap& taux, const ScaleMaps<KIND>& sfm,
                    const GemmParams& p, cudaStream_t st) {
  const long long units = (long long)ceil_div(p.M, 2 * BM) * p.n_tiles * p.splits;
  const int most = sm_count() / 2, grid = 2 * (int)(units < most ? units : most);
  switch (epi) {
    case EPI_NONE: return launch_pair<KIND, EPI_NONE>(ta, tb, td, taux, sfm, p, grid, st);
    case EPI_BIAS: return launch_pair<KIND, EPI_BIAS>(ta, tb, td, taux, sfm, p, grid, st);
    case EPI_BIAS_GELU: return launch_pair<KIND, EPI_BIAS_GELU>(ta, tb, td, taux, sfm, p, grid, st);
    case EPI_DGELU: return launch_pair<KIND, EPI_DGELU>(ta, tb, td, taux, sfm, p, grid, st);
    case EPI_ACC_F32: return launch_pair<KIND, EPI_ACC_F32>(ta, tb, td, taux, sfm, p, grid, st);
    case EPI_BIAS_RESID: return launch_pair<KIND, EPI_BIAS_RESID>(ta, tb, td, taux, sfm, p, grid, st);
    case EPI_STORE_F32: return launch_pair<KIND, EPI_STORE_F32>(ta, tb, td, taux, sfm, p, grid, st);
  }
  return LLMB_ERR_BAD_ARG;
}
}  // namespace
