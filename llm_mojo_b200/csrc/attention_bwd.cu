// Causal flash attention backward for head size 64 on tcgen05 + TMEM: one fused persistent kernel.
//
// Reference behaviour: llmm/attention.mojo:4692-5030 / :5033-5276 (backward via dP, the row dot D = sum(dO * O), dS,
// and the dQ / dK / dV products over stored [T,T] probabilities).  Here nothing of size T x T reaches HBM and the
// scores are recomputed ONCE: a CTA owns a 128-key tile (K and V resident in shared memory, dK and dV accumulating
// in TMEM) and walks the 128-row query blocks i that can see it.  Per block, with lanes = keys, columns = queries:
//   S^T  = K Q_i^T - lse / a    (tensor core, fp32 in TMEM)
//   dP^T = V dO_i^T - D         (tensor core, fp32 in TMEM)
//   P^T  = 2^(S^T * a)          compute warps; packed bf16 into its own TMEM columns
//   dS^T = P^T * dP^T           compute warps; bf16 into a swizzled shared-memory tile [keys, queries]
//   dV  += P^T dO_i         (A operand read from TMEM, dO_i as an MN-major shared-memory operand)
//   dK  += dS^T Q_i         (A K-major from that tile)
//   dQ_i partial = dS K     (A MN-major from the SAME tile, B = the resident K tile as an MN-major operand)
// A block is one chain - scores, compute warps, products - and the next block's scores are made beside it: as soon as the compute warps
// hold S^T(n) and dP^T(n) in registers, those of n+1 are issued.  What the chain was spent on, and how that was cut (cycles per block of
// about 6000, from clock traces of the roles):
//   * -lse and -D differ from column to column, so every thread needed all of them: 32 vector loads a thread, 2000 cycles of the shared-memory
//     pipe.  The tensor core adds them now, as one more K = 16 step of each score product: ones times rows that hold the values in
//     three bf16 parts (24 bits, all of an fp32 value; attn_bwd3_prep_kernel writes them).  Each product reads its own statistic only:
//     a shared row whose other half meets zeros would carry an infinity or NaN from one product into the other (0 * inf).
//   * two phases of the compute warps (P^T, then dS^T) with twelve barrier round trips of 170 - 250 cycles: one phase with two waits.
//   * one issuing warp, whose round trips came on top of 34 MMAs: one for the scores, one for the products.
//   * reductions of the dQ partials in the way of the compute warps' stores: see there.
//   * dK / dV stores that the dQ warpgroup waited for: warp 15 issues them.
// Whole backward pass, us, before / now: B 64, T 1024, 12 heads 743 / 570 - 602; B 4 83 / 61; B 7, T 777 101 / 75; B 6, T 2048, 16 heads 339 / 238 - 247.
// What bounds a block now (3200 cycles): the chain of 64 exponentials a thread at two warps per scheduler (1600), stores and barriers,
// products (1700, beside them), TMEM loads.
// The dQ partials of the key tiles are summed in an fp32 buffer by vector reductions (`red.global.add.v4.f32`, 16
// per thread and block, laid out so that a warp's 32 lanes hit 512 consecutive bytes); a small second kernel scales
// and rounds that buffer into the dQ part of dqkv and leaves it zeroed for the next call.  dK and dV are produced
// by exactly one CTA each in a fixed order and leave through a staging tile as TMA stores.
//
// Roles of the 512 threads:
//   warps 0..7          compute: one thread per key row and 64 of the block's queries
//   warps 8..11         dQ warpgroup: TMEM -> reductions per block, and the dK / dV epilogue per tile
//   warp 12             TMA producer: K, V per tile (two buffers), Q_i, dO_i and the row statistics per block (ring),
//                       and L2 prefetches of the CTA's next tile
//   warps 13, 14        MMA issuers of the scores / of the products
//   warp 15             dK and dV of a tile from the staging tile to memory
// TMEM columns (512): S^T 0..127 | dP^T 128..255 | dV 256..319 | dK 320..383 | dQ 384..447 | P^T 448..511.
// Every wait is bounded; a wait that runs out sets the status word and the role leaves its loop.
#include <type_traits>
#include "attention_common.cuh"

namespace {
constexpr int B3_NS = 3;                                   // ring depth in blocks: Q_i and dO_i, 16 KB each
constexpr int B3_THREADS = 512;
constexpr int B3_COL = TILE * 16;                          // 128 rows of 8 bf16: a column of core matrices of 8 rows x 16 bytes (no swizzle)
constexpr int B3_EXT = 2 * B3_COL;                         // the statistics of a block: a column of -lse / scale, one of -D
// A pause after every second reduction.  __nanosleep counts in steps: 90 and 120 ns give the same time, 150 falls into the next step, and eight of
// those with the reductions' own 1400 cycles outlast a block of 3200.  Whole backward, 12 heads, us, none / 45 / 90 / 120 / 150 ns: B 64, T 1024 620 / 611 /
// 602 / 604 / 652; B 4 65.5 / 61.9 / 60.5 / 60.5 / 67.9; B 7, T 777 81.6 / 77.4 / 75.2 / 75.2 / 84.7; B 2, T 1024 35.2 / 33.5 / 32.8 / 32.8 / 36.7.
constexpr unsigned B3_PACE_NS = 90;
constexpr int B3_SMEM = 4 * T128 /*K,V x2*/ + B3_NS * (2 * T128 + B3_EXT) + 2 * T128 /*dS^T*/ + T128 /*epilogue staging*/ + 2 * B3_COL + 256 /*barriers*/ +
                        1024 /*alignment*/;
static_assert(B3_SMEM <= 227 * 1024, "shared memory of a CTA");
constexpr uint32_t IDESC_TS_MN = make_idesc(FMT_BF16, FMT_BF16, 0, 1, 128, 64);     // A K-major (TMEM or smem), B stored [K rows, 64]
constexpr uint32_t IDESC_MN_MN = make_idesc(FMT_BF16, FMT_BF16, 1, 1, 128, 64);     // A stored [K rows, 128], B stored [K rows, 64]

#define B3_FAIL() do { atomicExch(p.status, LLMB_ERR_TIMEOUT); failed = true; } while (0)

struct B3Params {
  const uint4* stats;    // per (batch, head, 128-row tile): the column of -lse / scale, then that of -D, 16 bytes a row
  float* dq_acc;         // per (batch, head, tile): [16 column groups][128 rows][4] fp32, zero on entry
  float* dbias;          // optional fp32 [3C]
  int B, T, NH, C;
  float scale_log2, scale;
  int* status;
};

// D = rowsum(dO * O) and the statistics of every row as operands of the score products (see above): three bf16 parts, 24 bits, all of an fp32
// value.  Eight threads per row, 16 bytes of dO and O each, so that a warp reads four whole 128-byte rows per instruction.
__device__ __forceinline__ uint4 parts3(float v) {
  const __nv_bfloat16 hi = __float2bfloat16_rn(v);
  const float h = __bfloat162float(hi), r1 = isinf(h) ? 0.f : v - h;                // (an infinite value is its first part)
  const __nv_bfloat16 mid = __float2bfloat16_rn(r1), lo = __float2bfloat16_rn(r1 - __bfloat162float(mid));
  return make_uint4((uint32_t)__bfloat16_as_ushort(hi) | (uint32_t)__bfloat16_as_ushort(mid) << 16, __bfloat16_as_ushort(lo), 0u, 0u);
}
__global__ void attn_bwd3_prep_kernel(uint4* __restrict__ stats, const float* __restrict__ lse, const __nv_bfloat16* __restrict__ dout,
                                      const __nv_bfloat16* __restrict__ out, int B, int T, int NH, int C, float inv_scale_log2) {
  pdl_trigger();
  pdl_wait();
  const int n_t = ceil_div(T, TILE), Tp = n_t * TILE;
  const long long idx = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 3;   // (b * NH + h) * Tp + t
  const int part = threadIdx.x & 7;
  if (idx >= (long long)B * NH * Tp) return;                                       // whole groups of eight leave together
  const int t = (int)(idx % Tp); const long long bh = idx / Tp;
  const int h = (int)(bh % NH), b = (int)(bh / NH);
  float s = 0.f;
  if (t < T) {
    const long long bt = (long long)b * T + t;
    Pack<__nv_bfloat16> x, y;
    x.load(dout + bt * C + h * HS + part * 8); y.load(out + bt * C + h * HS + part * 8);
#pragma unroll
    for (int k = 0; k < 8; ++k) s += x.v[k] * y.v[k];
  }
  s += __shfl_xor_sync(0xffffffffu, s, 1); s += __shfl_xor_sync(0xffffffffu, s, 2); s += __shfl_xor_sync(0xffffffffu, s, 4);
  uint4* st = stats + idx / TILE * (2 * TILE) + idx % TILE;
  if (part == 0) st[0] = parts3(t < T ? -lse[bh * T + t] * inv_scale_log2 : -1e6f);     // rows beyond T: 2^(-1e6 scale) = 0
  if (part == 1) st[TILE] = parts3(-s);
}

struct Tile3 { int w, t, g, bh, tile; bool sub, done; };    // work item, tiles / blocks consumed so far, current tile
// Work item w = (batch, head) w / n_pairs and the key tiles x = w % n_pairs (n_t - x blocks) and n_t - 1 - x (x + 1
// blocks): n_t + 1 blocks whatever x.  Neighbouring CTAs work on the same (batch, head), so its Q and dO are read
// from HBM once.
__device__ __forceinline__ void tile3_seek(Tile3& c, int n_t, int n_items) {
  const int n_pairs = (n_t + 1) / 2;
  for (;;) {
    if (c.w >= n_items) { c.done = true; return; }
    const int x = c.w % n_pairs;
    c.bh = c.w / n_pairs;
    if (!c.sub) { c.tile = x; return; }
    if (n_t - 1 - x != x) { c.tile = n_t - 1 - x; return; }
    c.w += gridDim.x; c.sub = false;
  }
}
struct Blk3 { Tile3 c; int ib, nbt, n; };                   // block within the tile, blocks of the tile, blocks so far
__device__ __forceinline__ Blk3 blk3_begin(int n_t, int n_items) {
  Blk3 it;
  it.c = Tile3{(int)blockIdx.x, 0, 0, 0, 0, false, false};
  tile3_seek(it.c, n_t, n_items);
  it.ib = 0; it.n = 0; it.nbt = it.c.done ? 0 : n_t - it.c.tile;
  return it;
}
__device__ __forceinline__ void tile3_next(Tile3& c, int nbt, int n_t, int n_items) {
  c.t += 1; c.g += nbt;
  if (!c.sub) c.sub = true; else { c.sub = false; c.w += gridDim.x; }
  tile3_seek(c, n_t, n_items);
}
__device__ __forceinline__ void blk3_next(Blk3& it, int n_t, int n_items) {
  ++it.n;
  if (++it.ib == it.nbt) {
    tile3_next(it.c, it.nbt, n_t, n_items);
    it.ib = 0; it.nbt = it.c.done ? 0 : n_t - it.c.tile;
  }
}

__device__ __forceinline__ void umma_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
               "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
               ::"r"(tmem_d), "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void red_add_v4(float* addr, float a, float b, float c, float d) {
  asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(addr), "f"(a), "f"(b), "f"(c), "f"(d) : "memory");
}

__global__ void __launch_bounds__(B3_THREADS, 1) attn_bwd3_kernel(const __grid_constant__ CUtensorMap tmQKV,
                                                                  const __grid_constant__ CUtensorMap tmDO,
                                                                  const __grid_constant__ CUtensorMap tmOUT, const B3Params p) {
  extern __shared__ unsigned char smem_raw[];
  unsigned char* sm = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  unsigned char* sKV = sm;                                  // buffer kb: K at kb*2*T128, V at +T128
  unsigned char* sST = sKV + 4 * T128;                      // ring: stage s holds Q_i at s*2*T128, dO_i at +T128
  unsigned char* sDS = sST + B3_NS * 2 * T128;              // dS^T: queries 0..63 at +0, 64..127 at +T128 ([128 keys][64] each)
  unsigned char* sEXT = sDS + 2 * T128;                     // per stage: the block's statistics, two columns
  unsigned char* sEP = sEXT + B3_NS * B3_EXT;               // staging tile of the dK / dV epilogue ([128 keys][64] bf16, swizzled)
  unsigned char* sONE = sEP + T128;                         // a column of rows 1 1 1 0 0 0 0 0, then one of zeros: the second half of K on either side
  uint64_t* bars = reinterpret_cast<uint64_t*>(sONE + 2 * B3_COL);
  uint64_t* kv_full = bars;                                 // [2]
  uint64_t* kv_empty = kv_full + 2;                         // [2] the tile's last reads of K and V are complete
  uint64_t* st_full = kv_empty + 2;                         // [NS]
  uint64_t* st_empty = st_full + B3_NS;                     // [NS] the block's reads of Q and dO are complete 
  uint64_t* s_full = st_empty + B3_NS;                      // S^T and dP^T of a block are in TMEM
  uint64_t* s_free = s_full + 1;                            // ... and in the compute warps' registers (8 warps)
  uint64_t* p_full = s_free + 1;                            // P^T is in TMEM and dS^T in shared memory (8 warps), the block before's dQ has left TMEM (4 warps)
  uint64_t* ds_free = p_full + 1;                           // dV has read P^T, dK and dQ have read dS^T
  uint64_t* dq_full = ds_free + 1;                          // the block's dQ partial is in TMEM
  uint64_t* acc_full = dq_full + 1;                         // dK and dV of a tile are complete 
  uint64_t* acc_free = acc_full + 1;                        // ... and have left TMEM (4 warps)
  uint64_t* ep_ready = acc_free + 1;                        // the staging tile is written (4 warps)
  uint64_t* ep_free = ep_ready + 1;                         // ... and its TMA stores have read it
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(ep_free + 1);

  const int tid = threadIdx.x, warp = tid / 32, lane = tid % 32;
  const int n_t = ceil_div(p.T, TILE);
  const int n_items = ((n_t + 1) / 2) * p.B * p.NH;

  if (tid == 0) {
    for (int i = 0; i < 2; ++i) { mbar_init(&kv_full[i], 1); mbar_init(&kv_empty[i], 1); }
    for (int i = 0; i < B3_NS; ++i) { mbar_init(&st_full[i], 1); mbar_init(&st_empty[i], 1); }
    mbar_init(s_full, 1); mbar_init(s_free, 8); mbar_init(p_full, 12); mbar_init(ds_free, 1);
    mbar_init(dq_full, 1); mbar_init(acc_full, 1); mbar_init(acc_free, 4); mbar_init(ep_ready, 4); mbar_init(ep_free, 1);
    fence_barrier_init();
    prefetch_tmap(&tmQKV); prefetch_tmap(&tmDO); prefetch_tmap(&tmOUT);
  }
  if (tid < 2 * TILE) {
    *reinterpret_cast<uint4*>(sONE + tid * 16) = tid < TILE ? make_uint4(0x3f803f80u, 0x3f80u, 0u, 0u) : make_uint4(0u, 0u, 0u, 0u);
    fence_proxy_async();
  }
  if (warp == 13) tmem_alloc<512>(tmem_slot);
  fence_before_sync();
  __syncthreads();
  fence_after_sync();
  const uint32_t tmem = *tmem_slot;
  const uint32_t tS = tmem, tDP = tmem + 128, tDV = tmem + 256, tDK = tmem + 320, tDQ = tmem + 384, tP = tmem + 448;
  bool failed = false;
  pdl_trigger();
  pdl_wait();

  // Registers move from the dQ warpgroup and the producer / issuer warpgroup to the two compute warpgroups:
  // 128 x (2 x 176 + 2 x 80) = 65536 = the registers of the launch (512 x 128).
  if (warp >= 12) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 80;");
    if (warp == 12) {
      // ------------------------------------------------------------ TMA producer
      Tile3 c{(int)blockIdx.x, 0, 0, 0, 0, false, false};
      for (tile3_seek(c, n_t, n_items); !c.done && !failed;) {
        const int b = c.bh / p.NH, h = c.bh % p.NH, kb = c.t & 1, nbt = n_t - c.tile;
        const int colQ = h * HS, colK = p.C + h * HS, colV = 2 * p.C + h * HS;
        if (c.t >= 2 && !mbar_wait_sleep(&kv_empty[kb], ((c.t >> 1) + 1) & 1)) { B3_FAIL(); break; }
        if (elect_one()) {
          mbar_expect_tx(&kv_full[kb], 2 * T128);
          load128(sKV + kb * 2 * T128, &tmQKV, &kv_full[kb], colK, c.tile * TILE, b);
          load128(sKV + kb * 2 * T128 + T128, &tmQKV, &kv_full[kb], colV, c.tile * TILE, b);
        }
        __syncwarp();
        // While this tile's blocks are loaded, the operands of the CTA's NEXT tile are pulled into L2, a few boxes per
        // block, so that its loads find them there.
        Tile3 nx = c;
        tile3_next(nx, nbt, n_t, n_items);
        const int nxb = nx.bh / p.NH, nxh = nx.bh % p.NH, nx0 = nx.tile * TILE;
        const int pf_per = nx.done ? 0 : ceil_div(2 + 2 * (n_t - nx.tile), nbt);     // prefetch steps (64 rows) per block of this tile
        int pf = nx0 - 128;                                                          // next row to prefetch; the first two steps take K and V
        for (int ib = 0; ib < nbt; ++ib) {
          const int n = c.g + ib, st = n % B3_NS, i = c.tile + ib;
          if (n >= B3_NS && !mbar_wait_sleep(&st_empty[st], ((n / B3_NS) + 1) & 1)) { B3_FAIL(); break; }
          if (elect_one()) {
            unsigned char* stg = sST + st * 2 * T128;
            mbar_expect_tx(&st_full[st], 2 * T128 + B3_EXT);
            load128(stg, &tmQKV, &st_full[st], colQ, i * TILE, b);
            load128(stg + T128, &tmDO, &st_full[st], colQ, i * TILE, b);
            bulk_load_1d(sEXT + st * B3_EXT, p.stats + ((size_t)c.bh * n_t + i) * (2 * TILE), B3_EXT, &st_full[st]);
            for (int k = 0; k < pf_per; ++k) {
              const int r = pf + 64 * k;
              if (r < nx0) {
                tma_prefetch_l2_3d(&tmQKV, p.C + nxh * HS, r + 128, nxb);
                tma_prefetch_l2_3d(&tmQKV, 2 * p.C + nxh * HS, r + 128, nxb);
              } else if (r < n_t * TILE) {
                tma_prefetch_l2_3d(&tmQKV, nxh * HS, r, nxb);
                tma_prefetch_l2_3d(&tmDO, nxh * HS, r, nxb);
              }
            }
          }
          pf += 64 * pf_per;
          __syncwarp();
        }
        if (failed) break;
        tile3_next(c, nbt, n_t, n_items);
      }
    } else if (warp < 15) {
      // ------------------------------------------------------------ MMA issuers: warp 13 S^T and dP^T of block n + 1 as soon as the compute
      // warps hold those of n in registers, warp 14 dV, dK and dQ of n when P^T and dS^T are written.
      const uint64_t k_kk0 = make_smem_desc(smem_u32(sKV), 16, 1024);                 // K / V as K-major A operands
      const uint64_t k_mn0 = make_smem_desc(smem_u32(sKV), 8192, 1024);               // K as an MN-major B operand
      const uint64_t q_kk0 = make_smem_desc(smem_u32(sST), 16, 1024);                 // Q_i / dO_i as K-major B operands
      const uint64_t q_mn0 = make_smem_desc(smem_u32(sST), 8192, 1024);               // Q_i / dO_i as MN-major B operands
      const uint64_t ds_kk = make_smem_desc(smem_u32(sDS), 16, 1024);                 // dS^T as a K-major A operand (K = queries)
      const uint64_t ds_mn = make_smem_desc(smem_u32(sDS), T128, 1024);               // dS^T as an MN-major A operand (M = queries)
      // the statistics' step: ones / a statistic in the first eight values of K, zeros (the same column) in the others
      const uint64_t one0 = make_smem_desc(smem_u32(sONE), B3_COL, 128, 0);
      auto stat_desc = [&](int st, int col) {
        const uint32_t at = smem_u32(sEXT) + st * B3_EXT + col * B3_COL;
        return make_smem_desc(at, smem_u32(sONE) + B3_COL - at, 128, 0);
      };
      // a block in one word: 4 * (tiles before its tile) + 2 * (last of its tile) + (first of its tile), -1 when there is none left
      auto info = [](const Blk3& b) { return b.c.done ? -1 : b.c.t * 4 + (b.ib + 1 == b.nbt ? 2 : 0) + (b.ib == 0 ? 1 : 0); };
      auto scores = [&](int n, int what) {                                            // S^T and dP^T of block n
        const int st = n % B3_NS, t = what >> 2, kb = t & 1;
        if ((what & 1) && !mbar_wait(&kv_full[kb], (t >> 1) & 1)) { B3_FAIL(); return; }
        if (!mbar_wait(&st_full[st], (n / B3_NS) & 1)) { B3_FAIL(); return; }
        if (n >= 1 && !mbar_wait(s_free, (n - 1) & 1)) { B3_FAIL(); return; }
        fence_after_sync();
        const uint64_t kd = k_kk0 + (uint64_t)((kb * 2 * T128) >> 4), qd = q_kk0 + (uint64_t)((st * 2 * T128) >> 4);
        const uint64_t nlse = stat_desc(st, 0), nd = stat_desc(st, 1);
        if (elect_one()) {
          umma_ss<KIND_F16>(tS, one0, nlse, IDESC_S_128x128, 0u);                      // -lse / scale in every row
#pragma unroll
          for (int ks = 0; ks < HS / 16; ++ks) umma_ss<KIND_F16>(tS, kd + 2 * ks, qd + 2 * ks, IDESC_S_128x128, 1u);
          umma_ss<KIND_F16>(tDP, one0, nd, IDESC_S_128x128, 0u);                       // -D
#pragma unroll
          for (int ks = 0; ks < HS / 16; ++ks) umma_ss<KIND_F16>(tDP, kd + (T128 >> 4) + 2 * ks, qd + (T128 >> 4) + 2 * ks, IDESC_S_128x128, 1u);
          umma_commit(s_full);
        }
        __syncwarp();
      };
      auto products = [&](int n, int what) {                                          // dV += P^T dO, dK += dS^T Q, dQ = dS K of block n
        const int st = n % B3_NS, t = what >> 2, kb = t & 1;
        const bool first = what & 1, last = what & 2;
        if (!mbar_wait(p_full, n & 1)) { B3_FAIL(); return; }
        if (first && t >= 1 && !mbar_wait(acc_free, (t - 1) & 1)) { B3_FAIL(); return; }
        fence_after_sync();
        const uint64_t q_mn = q_mn0 + (uint64_t)((st * 2 * T128) >> 4), do_mn = q_mn + (T128 >> 4);
        const uint64_t kmn = k_mn0 + (uint64_t)((kb * 2 * T128) >> 4);
        if (elect_one()) {
#pragma unroll
          for (int ks = 0; ks < TILE / 16; ++ks) umma_ts(tDV, tP + ks * 8, do_mn + 128 * ks, IDESC_TS_MN, (ks > 0 || !first) ? 1u : 0u);
#pragma unroll
          for (int ks = 0; ks < TILE / 16; ++ks)
            umma_ss<KIND_F16>(tDK, ds_kk + (ks < 4 ? 2 * ks : (T128 >> 4) + 2 * (ks - 4)), q_mn + 128 * ks, IDESC_TS_MN, (ks > 0 || !first) ? 1u : 0u);
#pragma unroll
          for (int ks = 0; ks < TILE / 16; ++ks) umma_ss<KIND_F16>(tDQ, ds_mn + 128 * ks, kmn + 128 * ks, IDESC_MN_MN, ks > 0 ? 1u : 0u);
          umma_commit(dq_full);
          umma_commit(ds_free);
          umma_commit(&st_empty[st]);
          if (last) { umma_commit(acc_full); umma_commit(&kv_empty[kb]); }
        }
        __syncwarp();
      };
      for (Blk3 it = blk3_begin(n_t, n_items); !it.c.done && !failed; blk3_next(it, n_t, n_items)) {
        if (warp == 13) scores(it.n, info(it)); else products(it.n, info(it));
      }
    } else {
      // ------------------------------------------------------------ warp 15: dV, then dK of every tile from the staging tile to memory
      Tile3 c{(int)blockIdx.x, 0, 0, 0, 0, false, false};
      for (tile3_seek(c, n_t, n_items); !c.done && !failed; tile3_next(c, n_t - c.tile, n_t, n_items)) {
        const int b = c.bh / p.NH, h = c.bh % p.NH, k0 = c.tile * TILE;
        for (int mat = 0; mat < 2 && !failed; ++mat) {
          if (!mbar_wait_sleep(ep_ready, mat)) { B3_FAIL(); break; }                   // two phases a tile
          if (elect_one()) {
            const int col = (mat ? 1 : 2) * p.C + h * HS;
            tma_store_3d(&tmOUT, sEP, col, k0, b);
            tma_store_3d(&tmOUT, sEP + T64, col, k0 + 64, b);
            bulk_commit();
            bulk_wait_read<0>();
            mbar_arrive(ep_free);
          }
          __syncwarp();
        }
      }
    }
  } else if (warp >= 8) {
    // ---------------------------------------------------------------- dQ warpgroup: one thread per query row (dQ) / key row (dK, dV)
    asm volatile("setmaxnreg.dec.sync.aligned.u32 80;");
    const int row = (warp & 3) * 32 + lane;
    const uint32_t lane_addr = (uint32_t)((warp & 3) * 32) << 16;
    int ne = 0;                                             // staging tiles written so far
    if (lane == 0) mbar_arrive(p_full);                     // nothing to drain before the first block's dQ
    for (Blk3 it = blk3_begin(n_t, n_items); !it.c.done && !failed; blk3_next(it, n_t, n_items)) {
      const int n = it.n, i = it.c.tile + it.ib;
      if (!mbar_wait_sleep(dq_full, n & 1)) { B3_FAIL(); break; }
      fence_after_sync();
      float* dst = p.dq_acc + ((size_t)it.c.bh * n_t + i) * (TILE * HS) + row * 4;
      uint32_t r0[32], r1[32];
      tmem_ld32(tDQ + lane_addr, r0); tmem_ld32(tDQ + lane_addr + 32, r1);
      tmem_wait_ld();
      fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(p_full);
      // Sixteen reductions at a stretch keep the load / store pipe busy for 1400 cycles, and the commit that starts them also lets the compute
      // warps store dS^T(n+1), which then took 1000 cycles instead of 250.  So they go out two at a time, with a pause, inside a tile.
#pragma unroll
      for (int c = 0; c < 16; ++c) {
        const uint32_t (&r)[32] = c < 8 ? r0 : r1;
        red_add_v4(dst + c * (TILE * 4), __uint_as_float(r[4 * (c & 7)]), __uint_as_float(r[4 * (c & 7) + 1]), __uint_as_float(r[4 * (c & 7) + 2]),
                   __uint_as_float(r[4 * (c & 7) + 3]));
        if (c % 2 == 1 && it.ib + 1 < it.nbt) __nanosleep(B3_PACE_NS);
      }
      if (it.ib + 1 < it.nbt) continue;
      // The tile's dV and dK: rounded rows go through a swizzled staging tile and leave as TMA stores that warp 15 issues (whole 128-byte
      // rows; rows beyond T are clipped by the tensor map).  Per-thread stores of 16 bytes at a row stride of 3C would keep this
      // warpgroup busy for longer than a whole block takes.
      if (!mbar_wait_sleep(acc_full, it.c.t & 1)) { B3_FAIL(); break; }
      fence_after_sync();
      const int h = it.c.bh % p.NH, kj = it.c.tile * TILE + row;
#pragma unroll 1
      for (int mat = 0; mat < 2; ++mat) {                   // 0: dV, 1: dK
        const float sc = mat ? p.scale : 1.0f;              // dS^T was stored without the 1/sqrt(HS) factor
#pragma unroll 1
        for (int half = 0; half < 2; ++half) {
          uint32_t r[32];
          tmem_ld32((mat ? tDK : tDV) + lane_addr + half * 32, r);
          tmem_wait_ld();
          if (mat == 1 && half == 1) {
            fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive(acc_free);
          }
          float v[32];
#pragma unroll
          for (int x = 0; x < 32; ++x) v[x] = kj < p.T ? __uint_as_float(r[x]) * sc : 0.f;
          uint4 q[4];
#pragma unroll
          for (int j = 0; j < 4; ++j)
            q[j] = make_uint4(pack_bf16x2(v[8 * j], v[8 * j + 1]), pack_bf16x2(v[8 * j + 2], v[8 * j + 3]),
                                         pack_bf16x2(v[8 * j + 4], v[8 * j + 5]), pack_bf16x2(v[8 * j + 6], v[8 * j + 7]));
          if (p.dbias) {                                    // qkv bias gradient, dK and dV parts: column sums of this warp's 32 rows
            const float cs = warp_colsum32(v, lane);
            atomicAdd(p.dbias + (mat ? 1 : 2) * p.C + h * HS + half * 32 + lane, cs);
          }
          if (half == 0 && ne >= 1 && !mbar_wait_sleep(ep_free, (ne - 1) & 1)) { B3_FAIL(); break; }   // the stores before have read the tile
#pragma unroll
          for (int j = 0; j < 4; ++j) *reinterpret_cast<uint4*>(sEP + sw128(row, half * 4 + j)) = q[j];
        }
        if (failed) break;
        fence_proxy_async();
        __syncwarp();
        if (lane == 0) mbar_arrive(ep_ready);
        ++ne;
      }
    }
  } else {
    // ------------------------------------------------------------------ compute warpgroup hq: one thread per key row, query columns hq*64 .. +63
    asm volatile("setmaxnreg.inc.sync.aligned.u32 176;");
    const int hq = warp >> 2;
    const int row = (warp & 3) * 32 + lane;
    const uint32_t lane_addr = (uint32_t)((warp & 3) * 32) << 16;
    const uint32_t tSh = tS + lane_addr + hq * 64, tDPh = tDP + lane_addr + hq * 64, tPh = tP + lane_addr + hq * 32;
    const float2 sc2 = make_float2(p.scale_log2, p.scale_log2);
    for (Blk3 it = blk3_begin(n_t, n_items); !it.c.done && !failed; blk3_next(it, n_t, n_items)) {
      const int n = it.n;
      if (!mbar_wait_sleep(s_full, n & 1)) { B3_FAIL(); break; }
      fence_after_sync();
      uint32_t s[64], d[64];
      {
        uint32_t (&s0)[32] = *reinterpret_cast<uint32_t (*)[32]>(&s[0]);
        uint32_t (&s1)[32] = *reinterpret_cast<uint32_t (*)[32]>(&s[32]);
        uint32_t (&d0)[32] = *reinterpret_cast<uint32_t (*)[32]>(&d[0]);
        uint32_t (&d1)[32] = *reinterpret_cast<uint32_t (*)[32]>(&d[32]);
        tmem_ld32(tSh, s0); tmem_ld32(tDPh, d0); tmem_ld32(tSh + 32, s1); tmem_ld32(tDPh + 32, d1);
      }
      tmem_wait_ld();
      fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(s_free);              // the scores of block n+1 may be issued now
      uint32_t pk[32], dk[32];
      {
        auto work = [&](auto diag) {
          const int lim = row - hq * 64;                    // diagonal block: local query columns x < lim see nothing of this key
          auto exps = [&](int c) {
#pragma unroll
            for (int k = 0; k < 8; k += 2) {
              const float2 t = __fmul2_rn(make_float2(__uint_as_float(s[8 * c + k]), __uint_as_float(s[8 * c + k + 1])), sc2);
              float e0 = ex2_approx(t.x), e1 = ex2_approx(t.y);
              if (decltype(diag)::value) { e0 = 8 * c + k < lim ? 0.f : e0; e1 = 8 * c + k + 1 < lim ? 0.f : e1; }
              s[8 * c + k] = __float_as_uint(e0); s[8 * c + k + 1] = __float_as_uint(e1);
            }
          };
          exps(0);
#pragma unroll
          for (int c = 0; c < 8; ++c) {                     // a chunk's products beside the next chunk's exponentials
            if (c + 1 < 8) exps(c + 1);
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              const float2 e = make_float2(__uint_as_float(s[8 * c + 2 * k]), __uint_as_float(s[8 * c + 2 * k + 1]));
              const float2 r = __fmul2_rn(e, make_float2(__uint_as_float(d[8 * c + 2 * k]), __uint_as_float(d[8 * c + 2 * k + 1])));
              pk[4 * c + k] = pack_bf16x2(e.x, e.y); dk[4 * c + k] = pack_bf16x2(r.x, r.y);
            }
          }
        };
        if (it.ib == 0) work(std::true_type{}); else work(std::false_type{});
#pragma unroll
        for (int j = 0; j < 32; ++j) asm volatile("" : "+r"(pk[j]), "+r"(dk[j]));        // packed before the wait, not after it
      }
      if (n >= 1 && !mbar_wait_sleep(ds_free, (n - 1) & 1)) { B3_FAIL(); break; }   // the products of block n-1 have read P^T and dS^T
#pragma unroll
      for (int j = 0; j < 8; ++j)
        *reinterpret_cast<uint4*>(sDS + hq * T128 + sw128(row, j)) = make_uint4(dk[4 * j], dk[4 * j + 1], dk[4 * j + 2], dk[4 * j + 3]);
      fence_after_sync();
      tmem_st32(tPh, pk);
      fence_proxy_async();
      tmem_wait_st();
      fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(p_full);
    }
  }
  fence_before_sync();
  __syncthreads();
  if (warp == 13) { fence_after_sync(); tmem_dealloc<512>(tmem); }
}

// dq_acc -> the dQ part of dqkv (scaled, rounded), the buffer zeroed again, and optionally the dQ part of the bias gradient.
// One block of 128 threads per (batch, head, tile): thread r reads row r (a warp reads 512 consecutive bytes per load), the
// rounded rows cross a swizzled shared-memory tile, and every warp then writes four whole 128-byte rows per instruction.
__global__ void __launch_bounds__(128) attn_bwd3_dq_kernel(__nv_bfloat16* __restrict__ dqkv, float* __restrict__ dbias, float* __restrict__ dq_acc,
                                                           int T, int NH, int C, float scale) {
  pdl_trigger();
  pdl_wait();
  __shared__ float part[4][HS];
  __shared__ __align__(16) unsigned char tile_s[TILE * ROWB];
  const int n_t = ceil_div(T, TILE);
  const int tile = blockIdx.x % n_t, bh = blockIdx.x / n_t, h = bh % NH, b = bh / NH;
  const int r = threadIdx.x, lane = r % 32, warp = r / 32;
  float* src = dq_acc + (size_t)blockIdx.x * (TILE * HS) + r * 4;
#pragma unroll 1
  for (int half = 0; half < 2; ++half) {
    float v[32];
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      const float4 x = *reinterpret_cast<const float4*>(src + (half * 8 + c) * (TILE * 4));
      v[4 * c] = x.x * scale; v[4 * c + 1] = x.y * scale; v[4 * c + 2] = x.z * scale; v[4 * c + 3] = x.w * scale;
    }
#pragma unroll
    for (int j8 = 0; j8 < 4; ++j8) {
      uint4 u;
      u.x = pack_bf16x2(v[j8 * 8 + 0], v[j8 * 8 + 1]); u.y = pack_bf16x2(v[j8 * 8 + 2], v[j8 * 8 + 3]);
      u.z = pack_bf16x2(v[j8 * 8 + 4], v[j8 * 8 + 5]); u.w = pack_bf16x2(v[j8 * 8 + 6], v[j8 * 8 + 7]);
      *reinterpret_cast<uint4*>(tile_s + sw128(r, half * 4 + j8)) = u;
    }
    if (dbias) {                                            // rows beyond T hold zeros: their dS was zero
      const float cs = warp_colsum32(v, lane);
      part[warp][half * 32 + lane] = cs;
    }
  }
  __syncthreads();
  const int chunk = r & 7;
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    const int row = k * 16 + (r >> 3), qi = tile * TILE + row;
    if (qi < T)
      *reinterpret_cast<uint4*>(dqkv + ((size_t)b * T + qi) * (3 * (size_t)C) + h * HS + chunk * 8) =
          *reinterpret_cast<const uint4*>(tile_s + sw128(row, chunk));
  }
  // Zeroed only now, when every load above has returned its data: a store to an address whose load is still in flight
  // waits for it, and the kernel then runs at a quarter of the memory bandwidth.
#pragma unroll
  for (int c = 0; c < 16; ++c) *reinterpret_cast<float4*>(src + c * (TILE * 4)) = make_float4(0.f, 0.f, 0.f, 0.f);
  if (dbias && r < HS) atomicAdd(dbias + h * HS + r, part[0][r] + part[1][r] + part[2][r] + part[3][r]);
}
}  // namespace

// Sizes (in floats) of the two scratch buffers of llmb_attention_bwd_fused.
LLMB_API long long llmb_attention_bwd_fused_stats_floats(int B, int T, int NH) { return (long long)B * NH * ceil_div(T, TILE) * (B3_EXT / 4); }
LLMB_API long long llmb_attention_bwd_fused_acc_floats(int B, int T, int NH) { return (long long)B * NH * ceil_div(T, TILE) * (TILE * HS); }

// dqkv [B,T,3C] bf16 (fully overwritten) from dout [B,T,C], qkv [B,T,3C], out [B,T,C] (bf16) and the forward's lse [B,NH,T]
// (log2 domain); C = NH*64.  `stats` (..._stats_floats elements) and `dq_acc` (..._acc_floats): fp32 scratch, 16-byte aligned; `dq_acc` must be
// ZERO on entry and is zero again when the call has completed without an error in the status word.  dbias (optional, fp32 [3C]) +=
// column sums of dqkv, by atomic adds.
LLMB_API int llmb_attention_bwd_fused(void* dqkv, float* dbias, float* stats, float* dq_acc, const void* dout, const void* qkv, const void* out,
                                      const float* lse, int B, int T, int NH, int* status, cudaStream_t st) {
  const int C = NH * HS;
  CUtensorMap tq, td;
  int rc = make_qkv_map(&tq, qkv, B, T, 3 * C); if (rc) return 1000 + rc;
  rc = make_qkv_map(&td, dout, B, T, C); if (rc) return 1000 + rc;
  CUtensorMap to;
  rc = make_qkv_map(&to, dqkv, B, T, 3 * C); if (rc) return 1000 + rc;
  if (reinterpret_cast<uintptr_t>(stats) & 15) return LLMB_ERR_BAD_ARG;
  B3Params p{}; p.stats = (const uint4*)stats; p.dq_acc = dq_acc; p.dbias = dbias;
  p.B = B; p.T = T; p.NH = NH; p.C = C; p.scale = 0.125f; p.scale_log2 = 0.125f * 1.4426950408889634f; p.status = status;
  static bool attr = false;
  if (!attr) {
    cudaError_t e = cudaFuncSetAttribute(attn_bwd3_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, B3_SMEM); if (e) return (int)e;
    attr = true;
  }
  const int n_t = ceil_div(T, TILE);
  const long long rows = (long long)B * NH * n_t * TILE;
  launch_pdl(attn_bwd3_prep_kernel, (unsigned)ceil_div_ll(rows * 8, 256), 256, 0, st, (uint4*)stats, lse, (const __nv_bfloat16*)dout, (const __nv_bfloat16*)out, B, T, NH, C,
             1.0f / p.scale_log2);
  const long long n_items = (long long)((n_t + 1) / 2) * B * NH;
  const int grid = (int)(n_items < sm_count() ? n_items : sm_count());          // persistent: one CTA per SM
  launch_pdl(attn_bwd3_kernel, grid, B3_THREADS, B3_SMEM, st, tq, td, to, p);
  launch_pdl(attn_bwd3_dq_kernel, (unsigned)(B * NH * n_t), 128, 0, st, (__nv_bfloat16*)dqkv, dbias, dq_acc, T, NH, C, p.scale);
  return (int)cudaGetLastError();
}
