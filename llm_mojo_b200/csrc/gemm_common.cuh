// Parts shared by the GEMM kernels: parameters, epilogue arithmetic and staging.
#pragma once
#include <stdlib.h>
#include "tc05.cuh"
using namespace llmb;
using namespace tc05;

namespace lgemm {
__device__ __forceinline__ unsigned ld_acquire_gpu(const unsigned* p) {
  unsigned v; asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory"); return v;
}
__device__ __forceinline__ unsigned ld_acquire_sys(const unsigned* p) {
  unsigned v; asm volatile("ld.acquire.sys.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory"); return v;
}
__device__ __forceinline__ uint4 ld_nc_v4(const uint4* p) {     // streaming 16-byte load (peer memory: read once)
  uint4 v; asm volatile("ld.global.cg.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p) : "memory"); return v;
}
__device__ __forceinline__ void fence_proxy_async_all() { asm volatile("fence.proxy.async;" ::: "memory"); }
constexpr int BM = 128, BN = 256;
constexpr int ROW_BYTES = 128;                       // one swizzled row
constexpr int A_STAGE = BM * ROW_BYTES;              // 16 KB
constexpr int BAND = 16;                             // m-tiles per rasterisation band

enum { EPI_NONE = 0, EPI_BIAS = 1, EPI_BIAS_GELU = 2, EPI_DGELU = 3, EPI_ACC_F32 = 4, EPI_BIAS_RESID = 5, EPI_STORE_F32 = 6 };

// All-gather fused into the GEMM: the A matrix [W*n, K] is the concatenation of W row chunks, chunk r produced by
// rank r.  Every rank holds a full-size local buffer whose own chunk is already in place; two copier warps per
// CTA pull the other chunks out of the peers' buffers (plain 16-byte peer loads over NVLink, each byte crosses
// once) into the local buffer WHILE the tile loop runs, starting with the tiles of the local chunk and taking the
// remote chunks in ring order.  A chunk's tiles are fetched (TMA, local memory) once every CTA's copiers have
// counted it complete.
struct GatherArgs {
  const void* peer_src[8];     // [r]: start of chunk r inside rank r's buffer
  void* local;                 // start of this rank's [W*n, K] buffer
  const void* flags;           // this rank's flag words: peers announce "my chunk is written" (kind ROWS_READY)
  unsigned* counts;            // [16] local counters, zeroed before the launch: [r] = slices of chunk r copied, [8 + r] = slice tickets
  long long chunk_vecs;        // 16-byte vectors per chunk
  unsigned seq, target;        // announce sequence number to wait for; slices per chunk (counts[r] == target: chunk landed)
  int W, me, tiles_per_chunk;  // W = 0: no gather
};

// Parameter pull fused into a GEMM (ZeRO-3): the kernel's copier warps copy up to 8 segments of weights out of their
// owners' parameter shards (plain 16-byte loads over NVLink, or local memory for the rank's own part) into this
// rank's layer window while the tensor-core tile loop of the SAME kernel runs.  The segments may belong to the B
// operand of this GEMM (then its TMA producer waits for them) or to the operand of a later GEMM of the layer, which
// only checks the counters: every weight then arrives under the math of a tile loop.  Owners announce "my shard
// holds the parameters of optimizer step seq" at flag kind PARAM; all waits are bounded.
struct PullArgs {
  const void* src[8];          // segment source (peer or local shard memory), 16-byte aligned
  void* dst[8];                // segment destination inside the local window
  long long vecs[8];           // 16-byte vectors per segment
  const void* flags;           // this rank's flag words
  unsigned* counts;            // [16] zeroed before the launch: [s] = slices of segment s landed, [8 + s] = slice tickets
  const unsigned* wait_counts[8];   // counters this GEMM's B operand depends on ...
  unsigned wait_target[8];          // ... and the value each must reach
  unsigned seq;                // parameter sequence number the owners must have announced (0: none yet, no wait)
  int owner[8];
  int nseg, nwait, W;          // nseg = 0: nothing to pull; nwait = 0: nothing to wait for
};

struct GemmParams {
  GatherArgs g;
  PullArgs pull;
  void* D; const void* bias; void* aux; const float* alpha;
  int M, N, K;                 // K in elements
  long long ldd, ldaux;
  int a_mn, b_mn;              // operand majorness (0 = K-major)
  int a_3d, b_3d;              // MN-major operand fetched with ONE 3-D box (chunk, k, chunk index) per stage
  uint32_t a_lbo, a_sbo, a_kstep, b_lbo, b_sbo, b_kstep;   // bytes
  uint32_t a_layout, b_layout; // UMMA layout type: 2 = SWIZZLE_128B, 1 = SWIZZLE_128B with 32-byte base (fp32 MN-major)
  uint32_t idesc;
  int m_tiles, n_tiles, splits, kb_per_split, kb_total;
  int io_f32;                  // 1: D, bias and aux are fp32 (tf32 kind); 0: bf16
  int tma_epi;                 // 1: bf16 outputs leave (and auxiliary inputs arrive) by TMA; 0: register/shared-memory epilogue
  int bias_vec;                // bias pointer is 16-byte aligned (vector loads)
  float* colsum;               // EPI_DGELU, TMA epilogue: colsum[n] += sum over rows of the (bf16) result, i.e. the bias gradient of the layer below
  int* status;
};

// ------------------------------------------------------------------------------------------------
// Coalesced epilogue.  tcgen05.ld hands each thread one accumulator ROW; stored directly, a warp
// would touch 32 different rows per instruction.  Instead every 64-column slab of the warp's
// 32 x 256 block goes through an 8 KB shared-memory transpose (XOR-swizzled 16-byte chunks, conflict
// free in both directions) so that 8 consecutive lanes cover 64 contiguous bytes of one output row
// and all global traffic of the epilogue (output, bias, GELU aux, residual) is sector-aligned.
constexpr int EPI_STAGE_BYTES = 32 * 256;             // per epilogue warp: 32 rows x 64 fp32

template <int EPI>
__device__ __forceinline__ void epi4(const GemmParams& p, float (&v)[4], int row, int col, float alpha) {
#pragma unroll
  for (int k = 0; k < 4; ++k) v[k] *= alpha;
  if (EPI == EPI_BIAS || EPI == EPI_BIAS_GELU || EPI == EPI_BIAS_RESID) {
    if (p.bias && p.io_f32) {
      const float4 b = *reinterpret_cast<const float4*>(reinterpret_cast<const float*>(p.bias) + col);
      v[0] += b.x; v[1] += b.y; v[2] += b.z; v[3] += b.w;
    } else if (p.bias) {
      const uint2 braw = *reinterpret_cast<const uint2*>(reinterpret_cast<const __nv_bfloat16*>(p.bias) + col);
      const __nv_bfloat162* bh = reinterpret_cast<const __nv_bfloat162*>(&braw);
      const float2 b0 = __bfloat1622float2(bh[0]), b1 = __bfloat1622float2(bh[1]);
      v[0] += b0.x; v[1] += b0.y; v[2] += b1.x; v[3] += b1.y;
    }
  }
  if (EPI == EPI_ACC_F32 || EPI == EPI_STORE_F32) {
    float* dp = reinterpret_cast<float*>(p.D) + (size_t)row * p.ldd + col;
    if (EPI == EPI_ACC_F32)
      asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(dp), "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3]) : "memory");
    else
      *reinterpret_cast<float4*>(dp) = make_float4(v[0], v[1], v[2], v[3]);
    return;
  }
  if (p.io_f32) {                                       // fp32 storage (tf32 tensor path)
    float* dp = reinterpret_cast<float*>(p.D) + (size_t)row * p.ldd + col;
    float* ap = reinterpret_cast<float*>(p.aux) + (size_t)row * p.ldaux + col;
    if (EPI == EPI_BIAS_GELU) {
      *reinterpret_cast<float4*>(ap) = make_float4(v[0], v[1], v[2], v[3]);
#pragma unroll
      for (int k = 0; k < 4; ++k) v[k] = gelu_f(v[k]);
    } else if (EPI == EPI_DGELU) {
      const float4 x = *reinterpret_cast<const float4*>(ap);
      v[0] *= gelu_grad_f(x.x); v[1] *= gelu_grad_f(x.y); v[2] *= gelu_grad_f(x.z); v[3] *= gelu_grad_f(x.w);
    } else if (EPI == EPI_BIAS_RESID) {
      const float4 x = *reinterpret_cast<const float4*>(ap);
      v[0] += x.x; v[1] += x.y; v[2] += x.z; v[3] += x.w;
    }
    *reinterpret_cast<float4*>(dp) = make_float4(v[0], v[1], v[2], v[3]);
    return;
  }
  __nv_bfloat16* dp = reinterpret_cast<__nv_bfloat16*>(p.D) + (size_t)row * p.ldd + col;
  __nv_bfloat16* ap = reinterpret_cast<__nv_bfloat16*>(p.aux) + (size_t)row * p.ldaux + col;
  auto pack4 = [](const float (&x)[4]) {
    uint2 u; __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&u);
    h[0] = __floats2bfloat162_rn(x[0], x[1]); h[1] = __floats2bfloat162_rn(x[2], x[3]);
    return u;
  };
  auto unpack4 = [](uint2 u, float (&x)[4]) {
    const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&u);
    const float2 a = __bfloat1622float2(h[0]), b = __bfloat1622float2(h[1]);
    x[0] = a.x; x[1] = a.y; x[2] = b.x; x[3] = b.y;
  };
  if (EPI == EPI_BIAS_GELU) {
    const uint2 pre = pack4(v);
    *reinterpret_cast<uint2*>(ap) = pre;               // pre-GELU activations (bf16)
    float x[4]; unpack4(pre, x);
#pragma unroll
    for (int k = 0; k < 4; ++k) v[k] = gelu_f(x[k]);
  } else if (EPI == EPI_DGELU) {
    float x[4]; unpack4(*reinterpret_cast<const uint2*>(ap), x);
#pragma unroll
    for (int k = 0; k < 4; ++k) v[k] *= gelu_grad_f(x[k]);
  } else if (EPI == EPI_BIAS_RESID) {
    float x[4]; unpack4(*reinterpret_cast<const uint2*>(ap), x);
#pragma unroll
    for (int k = 0; k < 4; ++k) v[k] += x[k];
  }
  const uint2 o = pack4(v);
  *reinterpret_cast<uint2*>(dp) = o;
}

// What epi4's 16-byte (fp32) and 8-byte (bf16) accesses need of a layout that has no tensor map; D is 16-byte aligned and N % 8 == 0 in any
// case, and the pitch of a single row is not used.  A dispatch that would fall back to it with anything else refuses the call.
inline bool register_epilogue_takes(int epi, bool io_f32, int M, const void* bias, const void* aux, long long ldd, long long ldaux) {
  const bool needs_aux = epi == EPI_BIAS_GELU || epi == EPI_DGELU || epi == EPI_BIAS_RESID;
  const bool needs_bias = epi == EPI_BIAS || epi == EPI_BIAS_GELU || epi == EPI_BIAS_RESID;
  const uintptr_t mask = io_f32 ? 15 : 7;
  return (M == 1 || ldd % 4 == 0) && (!needs_aux || (aux && (reinterpret_cast<uintptr_t>(aux) & mask) == 0 && (M == 1 || ldaux % 4 == 0))) &&
         (!needs_bias || (reinterpret_cast<uintptr_t>(bias) & mask) == 0);
}

// One epilogue warp drains its 32 rows x NCOLS columns of accumulator `tacc` (TMEM address incl. lane quarter).
template <int EPI, int NCOLS = BN>
__device__ __forceinline__ void epilogue_warp(const GemmParams& p, uint32_t tacc, unsigned char* stage, int row_base, int n0,
                                              float alpha, int lane) {
  const int rsub = lane >> 3, cl = lane & 7;
#pragma unroll 1
  for (int s = 0; s < NCOLS / 64; ++s) {
    if (n0 + s * 64 >= p.N) break;                      // warp-uniform
    uint32_t r0[32], r1[32];
    tmem_ld32(tacc + s * 64, r0);
    tmem_ld32(tacc + s * 64 + 32, r1);
    tmem_wait_ld();
    unsigned char* myrow = stage + lane * 256;
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      *reinterpret_cast<uint4*>(myrow + ((c ^ (lane & 15)) << 4)) = make_uint4(r0[4 * c], r0[4 * c + 1], r0[4 * c + 2], r0[4 * c + 3]);
      *reinterpret_cast<uint4*>(myrow + (((c + 8) ^ (lane & 15)) << 4)) = make_uint4(r1[4 * c], r1[4 * c + 1], r1[4 * c + 2], r1[4 * c + 3]);
    }
    __syncwarp();
#pragma unroll
    for (int it = 0; it < 8; ++it) {
      const int rr = it * 4 + rsub;
      const int row = row_base + rr;
      const unsigned char* src = stage + rr * 256;
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        const int chunk = cl + half * 8;
        const float4 f = *reinterpret_cast<const float4*>(src + ((chunk ^ (rr & 15)) << 4));
        const int col = n0 + s * 64 + chunk * 4;
        if (row < p.M && col < p.N) {
          float v[4] = {f.x, f.y, f.z, f.w};
          epi4<EPI>(p, v, row, col, alpha);
        }
      }
    }
    __syncwarp();
  }
}

// ------------------------------------------------------------------------------------------------
// Epilogue through TMA.  A warp moves its part of the accumulator in boxes of 32 rows x 128 bytes (4 KB, 128-byte swizzle):
// 64 columns of bf16 or 32 of fp32.
//   * tcgen05.ld gives each lane one row of a box; bias, GELU, dGELU and the residual add happen in registers in that layout;
//   * the auxiliary INPUT (residual stream, pre-GELU activations) arrives by TMA in the buffer that the result is then written to in
//     place.  In the CTA-pair kernel a warp has two boxes (bf16: its two 64-column slabs of a tile; fp32 storage: four 32-column ones in
//     turn); a box is filled again, with the next tile's input, once the store of its last result has read it;
//   * results leave by TMA stores (fp32 accumulate: by TMA additions), so no lane ever waits on global memory and every global access
//     of the epilogue is a full 128-byte row segment; out-of-range rows and columns are clipped by the tensor maps.
// Epilogues with an auxiliary input or a second output (BIAS_GELU stores the pre-activation too) and the fp32 outputs get 64 KB of
// boxes and a 5-deep operand ring in the CTA-pair kernel; the others 32 KB and a 6-deep ring.
template <int EPI> struct EpiCfg {
  static constexpr bool AUX_IN = EPI == EPI_DGELU || EPI == EPI_BIAS_RESID;
  static constexpr bool TWO_OUT = EPI == EPI_BIAS_GELU;
  static constexpr bool F32_OUT = EPI == EPI_ACC_F32 || EPI == EPI_STORE_F32;
  static constexpr int STAGES = (F32_OUT || AUX_IN || TWO_OUT) ? 5 : 6;
  static constexpr int WARP_STAGE = STAGES == 5 ? 16384 : 8192;     // staging bytes per warp of the 4-warp register epilogue (half that per warp of 8 in the TMA epilogues)
};
constexpr int SLAB_BYTES = 32 * 128;

__device__ __forceinline__ uint4 pack8(const float (&x)[8]) {
  uint4 u; __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&u);
#pragma unroll
  for (int i = 0; i < 4; ++i) h[i] = __floats2bfloat162_rn(x[2 * i], x[2 * i + 1]);
  return u;
}
__device__ __forceinline__ void unpack8(const uint4& u, float (&x)[8]) {
  const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&u);
#pragma unroll
  for (int i = 0; i < 4; ++i) { const float2 f = __bfloat1622float2(h[i]); x[2 * i] = f.x; x[2 * i + 1] = f.y; }
}

// Eight bias values from column `col` on (N is a multiple of 8; columns beyond it, which no store writes, read the last ones).
__device__ __forceinline__ uint4 bias8(const GemmParams& p, const __nv_bfloat16* bias, int col) {
  bias += min(col, p.N - 8);
  if (p.bias_vec) return __ldg(reinterpret_cast<const uint4*>(bias));
  const unsigned short* h = reinterpret_cast<const unsigned short*>(bias);
  uint4 u;
  u.x = __ldg(h) | (uint32_t)__ldg(h + 1) << 16; u.y = __ldg(h + 2) | (uint32_t)__ldg(h + 3) << 16;
  u.z = __ldg(h + 4) | (uint32_t)__ldg(h + 5) << 16; u.w = __ldg(h + 6) | (uint32_t)__ldg(h + 7) << 16;
  return u;
}
// alpha * accumulator + bias of 32 columns (this lane's row)
template <bool BIAS>
__device__ __forceinline__ void epi_affine32(const GemmParams& p, const uint32_t (&r)[32], int col0, float alpha, float (&v)[32]) {
  const __nv_bfloat16* bias = reinterpret_cast<const __nv_bfloat16*>(p.bias);
  if (BIAS && bias) {
    uint4 bq[4];
#pragma unroll
    for (int c = 0; c < 4; ++c) bq[c] = bias8(p, bias, col0 + c * 8);
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      float b[8]; unpack8(bq[c], b);
#pragma unroll
      for (int j = 0; j < 8; j += 2) {
        const float2 y = __ffma2_rn(make_float2(__uint_as_float(r[c * 8 + j]), __uint_as_float(r[c * 8 + j + 1])), make_float2(alpha, alpha), make_float2(b[j], b[j + 1]));
        v[c * 8 + j] = y.x; v[c * 8 + j + 1] = y.y;
      }
    }
  } else {
#pragma unroll
    for (int j = 0; j < 32; j += 2) {
      const float2 y = __fmul2_rn(make_float2(__uint_as_float(r[j]), __uint_as_float(r[j + 1])), make_float2(alpha, alpha));
      v[j] = y.x; v[j + 1] = y.y;
    }
  }
}

// Half a slab (this lane's row, 32 columns: chunks 4 * H .. 4 * H + 3) from registers to the swizzled staging buffer.  With an
// auxiliary input the buffer holds it on entry and the result replaces it.
template <int EPI, int H>
__device__ __forceinline__ void epi_half_bf16(const GemmParams& p, const uint32_t (&r)[32], unsigned char* buf, int col0, float alpha, int lane) {
  unsigned char* myrow = buf + lane * 128;
  float v[32];
  epi_affine32<EPI == EPI_BIAS || EPI == EPI_BIAS_RESID>(p, r, col0 + H * 32, alpha, v);
#pragma unroll
  for (int c4 = 0; c4 < 4; ++c4) {
    const int c = H * 4 + c4;
    unsigned char* slot = myrow + ((c ^ (lane & 7)) << 4);
    float o[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) o[j] = v[c4 * 8 + j];
    if (EPI == EPI_DGELU || EPI == EPI_BIAS_RESID) {
      float x[8]; unpack8(*reinterpret_cast<const uint4*>(slot), x);
#pragma unroll
      for (int j = 0; j < 8; j += 2) {
        const float2 xx = make_float2(x[j], x[j + 1]), vv = make_float2(o[j], o[j + 1]);
        const float2 y = (EPI == EPI_DGELU) ? __fmul2_rn(vv, gelu_grad_fast2(xx)) : __fadd2_rn(vv, xx);
        o[j] = y.x; o[j + 1] = y.y;
      }
    }
    *reinterpret_cast<uint4*>(slot) = pack8(o);
  }
}
// Column sums of a 32 x 64 slab as stored (bf16), added to colsum.  Lane l reads 16-byte chunk l % 8 (eight columns) of the rows l / 8 + 4 i out of
// the swizzled box (the 8 lanes of a row read its 128 bytes); the four partial sums of a column meet in two exchanges that leave every
// lane two columns.
__device__ __forceinline__ void epi_slab_colsum(const GemmParams& p, const unsigned char* buf, int row0, int col0, int lane) {
  const int nrows = min(32, p.M - row0), c = lane & 7, g = lane >> 3;
  float2 s[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) s[k] = make_float2(0.f, 0.f);
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int r = g + 4 * i;
    uint4 u = *reinterpret_cast<const uint4*>(buf + r * 128 + ((c ^ (r & 7)) << 4));
    if (r >= nrows) u = make_uint4(0u, 0u, 0u, 0u);
    const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
    for (int k = 0; k < 4; ++k) s[k] = __fadd2_rn(s[k], make_float2(__uint_as_float(w[k] << 16), __uint_as_float(w[k] & 0xffff0000u)));
  }
  auto swap = [&](float2 give, float2 keep, int mask) {
    return __fadd2_rn(keep, make_float2(__shfl_xor_sync(0xffffffffu, give.x, mask), __shfl_xor_sync(0xffffffffu, give.y, mask)));
  };
  const bool hi = g & 2, odd = g & 1;
  const float2 t0 = swap(hi ? s[0] : s[2], hi ? s[2] : s[0], 16), t1 = swap(hi ? s[1] : s[3], hi ? s[3] : s[1], 16);
  const float2 t = swap(odd ? t0 : t1, odd ? t1 : t0, 8);
  const int col = col0 + c * 8 + (hi ? 4 : 0) + (odd ? 2 : 0);
  if (col < p.N) {
    asm volatile("red.global.add.f32 [%0], %1;" ::"l"(p.colsum + col), "f"(t.x) : "memory");
    asm volatile("red.global.add.f32 [%0], %1;" ::"l"(p.colsum + col + 1), "f"(t.y) : "memory");
  }
}

// The bias + GELU epilogue in two steps, so that the pre-activation box can leave by TMA while the GELU of the same slab is computed: first
// alpha, bias and the bf16 pre-activations of half a slab, kept in registers as well ...
template <int H>
__device__ __forceinline__ void epi_half_pre(const GemmParams& p, const uint32_t (&r)[32], unsigned char* buf, int col0, float alpha, int lane, uint4 (&pre)[8]) {
  unsigned char* myrow = buf + lane * 128;
  float v[32];
  epi_affine32<true>(p, r, col0 + H * 32, alpha, v);
#pragma unroll
  for (int c4 = 0; c4 < 4; ++c4) {
    const int c = H * 4 + c4;
    float o[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) o[j] = v[c4 * 8 + j];
    pre[c] = pack8(o);
    *reinterpret_cast<uint4*>(myrow + ((c ^ (lane & 7)) << 4)) = pre[c];
  }
}
// ... then the GELU of those bf16 values, in place, ...
__device__ __forceinline__ void epi_slab_gelu(uint4 (&pre)[8]) {
#pragma unroll
  for (int c = 0; c < 8; ++c) {
    float x[8]; unpack8(pre[c], x);
#pragma unroll
    for (int j = 0; j < 8; j += 2) {
      const float2 y = gelu_fast2(make_float2(x[j], x[j + 1]));
      x[j] = y.x; x[j + 1] = y.y;
    }
    pre[c] = pack8(x);
  }
}
// ... and to a box.
__device__ __forceinline__ void epi_slab_store(const uint4 (&v)[8], unsigned char* buf, int lane) {
  unsigned char* myrow = buf + lane * 128;
#pragma unroll
  for (int c = 0; c < 8; ++c) *reinterpret_cast<uint4*>(myrow + ((c ^ (lane & 7)) << 4)) = v[c];
}


// A whole slab; BIAS_GELU writes the pre-activation to `buf` and the activation to `buf + SLAB_BYTES`.
template <int EPI>
__device__ __forceinline__ void epi_slab_bf16(const GemmParams& p, const uint32_t (&r0)[32], const uint32_t (&r1)[32],
                                              unsigned char* buf, int col0, float alpha, int lane) {
  if (EPI == EPI_BIAS_GELU) {
    uint4 pre[8];
    epi_half_pre<0>(p, r0, buf, col0, alpha, lane, pre);
    epi_half_pre<1>(p, r1, buf, col0, alpha, lane, pre);
    epi_slab_gelu(pre);
    epi_slab_store(pre, buf + SLAB_BYTES, lane);
    return;
  }
  epi_half_bf16<EPI, 0>(p, r0, buf, col0, alpha, lane);
  epi_half_bf16<EPI, 1>(p, r1, buf, col0, alpha, lane);
}

// fp32 storage (tf32 kind): one box of 32 rows x 32 columns (this lane's row) from registers to the swizzled staging box; with an
// auxiliary input the box holds it on entry, BIAS_GELU writes the activation to `act` and the pre-activation to `buf`.
template <int EPI>
__device__ __forceinline__ void epi_box_f32(const GemmParams& p, const uint32_t (&r)[32], unsigned char* buf, unsigned char* act, int col0,
                                            float alpha, int lane) {
  const float* bias = reinterpret_cast<const float*>(p.bias);
#pragma unroll
  for (int c = 0; c < 8; ++c) {
    const int col = col0 + c * 4;
    float4 v = make_float4(__uint_as_float(r[4 * c]) * alpha, __uint_as_float(r[4 * c + 1]) * alpha, __uint_as_float(r[4 * c + 2]) * alpha,
                           __uint_as_float(r[4 * c + 3]) * alpha);
    if ((EPI == EPI_BIAS || EPI == EPI_BIAS_GELU || EPI == EPI_BIAS_RESID) && bias && col < p.N) {
      float4 b;
      if (p.bias_vec) b = __ldg(reinterpret_cast<const float4*>(bias + col));
      else b = make_float4(bias[col], bias[col + 1], bias[col + 2], bias[col + 3]);
      v.x += b.x; v.y += b.y; v.z += b.z; v.w += b.w;
    }
    const int off = lane * 128 + ((c ^ (lane & 7)) << 4);
    if (EPI == EPI_BIAS_GELU) {
      *reinterpret_cast<float4*>(buf + off) = v;
      v = make_float4(gelu_f(v.x), gelu_f(v.y), gelu_f(v.z), gelu_f(v.w));
      *reinterpret_cast<float4*>(act + off) = v;
      continue;
    }
    if (EPI == EPI_DGELU || EPI == EPI_BIAS_RESID) {
      const float4 x = *reinterpret_cast<const float4*>(buf + off);
      if (EPI == EPI_DGELU) { v.x *= gelu_grad_f(x.x); v.y *= gelu_grad_f(x.y); v.z *= gelu_grad_f(x.z); v.w *= gelu_grad_f(x.w); }
      else { v.x += x.x; v.y += x.y; v.z += x.z; v.w += x.w; }
    }
    *reinterpret_cast<float4*>(buf + off) = v;
  }
}

template <int KIND> struct KindTraits;
template <> struct KindTraits<KIND_F16> { static constexpr int ESZ = 2, BKE = ROW_BYTES / ESZ; static constexpr CUtensorMapDataType DT = CU_TENSOR_MAP_DATA_TYPE_BFLOAT16; };
template <> struct KindTraits<KIND_TF32> { static constexpr int ESZ = 4, BKE = ROW_BYTES / ESZ; static constexpr CUtensorMapDataType DT = CU_TENSOR_MAP_DATA_TYPE_FLOAT32; };
template <> struct KindTraits<KIND_F8F6F4> { static constexpr int ESZ = 1, BKE = ROW_BYTES / ESZ; static constexpr CUtensorMapDataType DT = CU_TENSOR_MAP_DATA_TYPE_UINT8; };
template <> struct KindTraits<KIND_MXF8> { static constexpr int ESZ = 1, BKE = ROW_BYTES; static constexpr CUtensorMapDataType DT = CU_TENSOR_MAP_DATA_TYPE_UINT8; };
template <> struct KindTraits<KIND_NVF4> { static constexpr int ESZ = 1, BKE = ROW_BYTES; static constexpr CUtensorMapDataType DT = CU_TENSOR_MAP_DATA_TYPE_UINT8; };
}  // namespace lgemm
using namespace lgemm;

// gemm_small.cu: 128 x bn tiles, one per CTA, `cl` CTAs sharing the contraction of a tile (see there)
int llmb_gemm_small_launch(int kind, int epi, int bn, int cl, const CUtensorMap& ta, const CUtensorMap& tb, const CUtensorMap& td,
                           const CUtensorMap& taux, const GemmParams& p, cudaStream_t st);
