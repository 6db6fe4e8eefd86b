// Causal flash attention for fp32 storage and head size 64, forward and backward, in fp32 arithmetic on the FMA pipe.
//
// Reference behaviour: llmm/attention.mojo:1748-1945 (forward), :4692-5276 (backward).  The bf16 kernels (attention_fwd.cu,
// attention_bwd.cu) run on the tensor core; the fp32 path keeps its scores, probabilities and sums in fp32, which the tensor core's
// TF32 products would not, and the FMA pipe bounds it: 64 x 64 x 64 products per pair of tiles, two forward and five backward.
//
// Every operand tile is 64 rows x 64 columns of fp32 in shared memory, row-major at a pitch of 68 words, and a CTA of 128 threads holds
// a 64 x 64 product as 8 x 4 values per thread: thread (ty, tx) = (tid / 16, tid % 16) has rows ty * 8 + i.  Three forms of product
// cover all seven uses without a transposed copy; each reads shared memory in 16-byte pieces, four steps of the contraction at a time
// (16 wavefronts per 128 FMAs of a warp):
//   nt: sum_k A[i][k] B[j][k]   S = Q K^T, dP = dO V^T            columns j * 16 + tx (rows of B 68 words apart: no bank conflicts)
//   nn: sum_k A[i][k] B[k][j]   O += P V, dQ = dS K               columns tx * 4 + j
//   tn: sum_k A[k][i] B[k][j]   dV += P^T dO, dK += dS^T Q        columns tx * 4 + j
// Forward: a CTA per 64 query rows walks the key tiles up to its own (longest rows first).  Backward: a CTA per 64 keys walks the
// query tiles from its own on, recomputes P once, keeps dK and dV in registers and adds its part of dQ to the zeroed output by
// vector reductions; the row dots D = sum(dO * O) come from a small kernel before it.  The parts of dQ arrive in any order, so its last
// bits differ from run to run; the split form leaves dQ to a kernel of its own, a CTA per 64 query rows that walks the key tiles in
// order and recomputes P and dP (seven products instead of five), and is the same on every run.
// Measured (us, with the library in brackets; its backward included a second forward): forward B 8, T 64, 6 heads 9.2 (25.6), B 2, T 512, 12
// heads 82 (64), B 4, T 512 97 (76), B 8, T 1024 351 (359), B 2, T 2048, 16 heads 455 (500); backward 27 (189), 162 (237), 164 (314), 891
// (1487), 1158 (1982).  The library's forward is ahead at two to six tiles per SM: there the longest CTA, eight tiles one after the other
// with one warp per scheduler, is the whole time.  Split backward: 208 at B 4, T 512, 1607 at B 2, T 2048.
// Relative error against 64 bits, unit normal inputs: 1.7e-7 and 2.8e-7 (library 4.3e-7 and 6.6e-7): scores in four partial sums, tile sums
// before running sums.  At B 8, T 1024 the SMs are 75 % (forward) and 67 % (backward) busy, L1 62 %, with 19 % and 12 % of the warp slots taken.
#include "common.cuh"
using namespace llmb;

namespace {
constexpr int FT = 64;                                    // tile: rows, keys and head size
constexpr int FP = 68;                                    // pitch in words
constexpr int TILE_WORDS = FT * FP;
constexpr int F32_THREADS = 128;
constexpr float SCALE = 0.125f, SCALE_LOG2 = 0.125f * 1.4426950408889634f;

__device__ __forceinline__ float4 lds4(const float* p) { return *reinterpret_cast<const float4*>(p); }

// rows r0 .. r0 + 63 of a [.., pitch] matrix (64 columns at src) to shared memory; rows from `rows` on read as zero
__device__ __forceinline__ void load_tile(float* dst, const float* src, long long pitch, int r0, int rows) {
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int id = threadIdx.x + i * F32_THREADS, r = id / 16, c = (id % 16) * 4;
    const float4 v = r0 + r < rows ? *reinterpret_cast<const float4*>(src + (long long)(r0 + r) * pitch + c) : make_float4(0.f, 0.f, 0.f, 0.f);
    *reinterpret_cast<float4*>(dst + r * FP + c) = v;
  }
}
// the same, asynchronously (one group per call; rows beyond the end are zero-filled)
__device__ __forceinline__ void load_tile_async(float* dst, const float* src, long long pitch, int r0, int rows) {
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int id = threadIdx.x + i * F32_THREADS, r = id / 16, c = (id % 16) * 4;
    const bool in = r0 + r < rows;
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst + r * FP + c);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(in ? src + (long long)(r0 + r) * pitch + c : src), "r"(in ? 16 : 0) : "memory");
  }
  asm volatile("cp.async.commit_group;" ::: "memory");
}
template <int N> __device__ __forceinline__ void async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }
__device__ __forceinline__ void add(float (&a)[8][4], const float (&b)[8][4]) {
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) a[i][j] += b[i][j];
}
__device__ __forceinline__ void zero(float (&a)[8][4]) {
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) a[i][j] = 0.f;
}
// (in four partial sums of 16 terms: a score's rounding error is what the exponential magnifies)
__device__ __forceinline__ void mm_nt(float (&acc)[8][4], const float* A, const float* B, int ty, int tx) {
  zero(acc);
#pragma unroll 1
  for (int k0 = 0; k0 < FT; k0 += 16) {
    float c[8][4];
#pragma unroll
    for (int k = k0; k < k0 + 16; k += 4) {
      float4 b[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) b[j] = lds4(B + (j * 16 + tx) * FP + k);
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const float4 a = lds4(A + (ty * 8 + i) * FP + k);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          c[i][j] = k == k0 ? a.x * b[j].x : fmaf(a.x, b[j].x, c[i][j]);
          c[i][j] = fmaf(a.y, b[j].y, c[i][j]); c[i][j] = fmaf(a.z, b[j].z, c[i][j]); c[i][j] = fmaf(a.w, b[j].w, c[i][j]);
        }
      }
    }
    add(acc, c);
  }
}
__device__ __forceinline__ void mm_nn(float (&acc)[8][4], const float* A, const float* B, int ty, int tx) {
  zero(acc);
#pragma unroll 2
  for (int k = 0; k < FT; k += 4) {
    float4 b[4];
#pragma unroll
    for (int kk = 0; kk < 4; ++kk) b[kk] = lds4(B + (k + kk) * FP + tx * 4);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const float4 a = lds4(A + (ty * 8 + i) * FP + k);
      const float av[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
      for (int kk = 0; kk < 4; ++kk) {
        acc[i][0] = fmaf(av[kk], b[kk].x, acc[i][0]); acc[i][1] = fmaf(av[kk], b[kk].y, acc[i][1]);
        acc[i][2] = fmaf(av[kk], b[kk].z, acc[i][2]); acc[i][3] = fmaf(av[kk], b[kk].w, acc[i][3]);
      }
    }
  }
}
__device__ __forceinline__ void mm_tn(float (&acc)[8][4], const float* A, const float* B, int ty, int tx) {
  zero(acc);
#pragma unroll 4
  for (int k = 0; k < FT; ++k) {
    const float4 a0 = lds4(A + k * FP + ty * 8), a1 = lds4(A + k * FP + ty * 8 + 4), b = lds4(B + k * FP + tx * 4);
    const float av[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      acc[i][0] = fmaf(av[i], b.x, acc[i][0]); acc[i][1] = fmaf(av[i], b.y, acc[i][1]);
      acc[i][2] = fmaf(av[i], b.z, acc[i][2]); acc[i][3] = fmaf(av[i], b.w, acc[i][3]);
    }
  }
}

__global__ void __launch_bounds__(F32_THREADS, 3) attn_f32_fwd_kernel(float* __restrict__ out, float* __restrict__ lse, const float* __restrict__ qkv,
                                                                   int T, int NH, int n_t) {
  extern __shared__ __align__(16) float smf[];
  float *sQ = smf, *sK = sQ + TILE_WORDS, *sV = sK + TILE_WORDS, *sP = sV + TILE_WORDS;
  pdl_trigger();
  pdl_wait();
  const int BH = gridDim.x / n_t, qt = n_t - 1 - (int)(blockIdx.x / BH), bh = blockIdx.x % BH;      // longest rows first
  const int b = bh / NH, h = bh % NH, C = NH * FT;
  const long long pitch = 3LL * C;
  const float* base = qkv + (long long)b * T * pitch + h * FT;
  const int ty = threadIdx.x / 16, tx = threadIdx.x % 16, q0 = qt * FT;
  load_tile_async(sK, base + C, pitch, 0, T);
  load_tile_async(sV, base + 2 * C, pitch, 0, T);
  load_tile(sQ, base, pitch, q0, T);
  float o[8][4], m[8], l[8];
  zero(o);
#pragma unroll
  for (int i = 0; i < 8; ++i) { m[i] = -INFINITY; l[i] = 0.f; }
  for (int kt = 0; kt <= qt; ++kt) {
    float s[8][4];
    async_wait<1>();                                      // this tile's K (V, the newer group, may still be on its way)
    __syncthreads();
    mm_nt(s, sQ, sK, ty, tx);
    __syncthreads();
    if (kt < qt) load_tile_async(sK, base + C, pitch, (kt + 1) * FT, T);     // the next K travels during the exponentials and P V
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      float mx = -INFINITY;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        s[i][j] *= SCALE_LOG2;
        if (kt == qt && j * 16 + tx > ty * 8 + i) s[i][j] = -INFINITY;      // keys after the query (and so all beyond T of a real row)
        mx = fmaxf(mx, s[i][j]);
      }
#pragma unroll
      for (int w = 8; w > 0; w >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, w));
      const float mn = fmaxf(m[i], mx), alpha = exp2f(m[i] - mn);            // the first key of a row is never masked: mn is finite
      m[i] = mn;
      float sum = 0.f;
#pragma unroll
      for (int j = 0; j < 4; ++j) { const float p = exp2f(s[i][j] - mn); sum += p; sP[(ty * 8 + i) * FP + j * 16 + tx] = p; }
#pragma unroll
      for (int w = 8; w > 0; w >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, w);
      l[i] = l[i] * alpha + sum;
#pragma unroll
      for (int j = 0; j < 4; ++j) o[i][j] *= alpha;
    }
    if (kt < qt) async_wait<1>(); else async_wait<0>();   // this tile's V
    __syncthreads();                                      // (a warp's rows of P are written and read by that warp only)
    mm_nn(s, sP, sV, ty, tx);
    add(o, s);
    __syncthreads();
    if (kt < qt) load_tile_async(sV, base + 2 * C, pitch, (kt + 1) * FT, T);
  }
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int q = q0 + ty * 8 + i;
    if (q >= T) continue;
    const float inv = 1.0f / l[i];
    *reinterpret_cast<float4*>(out + ((long long)b * T + q) * C + h * FT + tx * 4) = make_float4(o[i][0] * inv, o[i][1] * inv, o[i][2] * inv, o[i][3] * inv);
    if (tx == 0 && lse) lse[(long long)bh * T + q] = m[i] + log2f(l[i]);
  }
}

// D[bh][q] = sum over the head of dO * O: sixteen threads per row
__global__ void __launch_bounds__(256) attn_f32_dot_kernel(float* __restrict__ D, const float* __restrict__ dout, const float* __restrict__ out, int T,
                                                           int NH, long long rows) {
  pdl_trigger();
  pdl_wait();
  const long long r = ((long long)blockIdx.x * blockDim.x + threadIdx.x) / 16;        // (b, q, h): consecutive in memory
  const int l = threadIdx.x % 16;
  float s = 0.f;
  if (r < rows) {
    const float4 a = *reinterpret_cast<const float4*>(dout + r * FT + l * 4), c = *reinterpret_cast<const float4*>(out + r * FT + l * 4);
    s = fmaf(a.x, c.x, fmaf(a.y, c.y, fmaf(a.z, c.z, a.w * c.w)));
  }
#pragma unroll
  for (int w = 8; w > 0; w >>= 1) s += __shfl_xor_sync(0xffffffffu, s, w);
  if (r < rows && l == 0) {
    const int h = (int)(r % NH);
    const long long bq = r / NH, b = bq / T, q = bq % T;
    D[(b * NH + h) * T + q] = s;
  }
}

// DQ: parts of dQ are added to dqkv, where it must be zero on entry; otherwise dQ is left alone.
template <bool DQ>
__global__ void __launch_bounds__(F32_THREADS, 2) attn_f32_bwd_kernel(float* __restrict__ dqkv, const float* __restrict__ dout, const float* __restrict__ qkv,
                                                                   const float* __restrict__ lse, const float* __restrict__ D, int T, int NH, int n_t) {
  extern __shared__ __align__(16) float smf[];
  float *sK = smf, *sV = sK + TILE_WORDS, *sQ = sV + TILE_WORDS, *sO = sQ + TILE_WORDS, *sP = sO + TILE_WORDS, *sS = sP + TILE_WORDS;
  pdl_trigger();
  pdl_wait();
  const int BH = gridDim.x / n_t, kt = (int)(blockIdx.x / BH), bh = blockIdx.x % BH;                // the longest walks first
  const int b = bh / NH, h = bh % NH, C = NH * FT;
  const long long pitch = 3LL * C;
  const float* base = qkv + (long long)b * T * pitch + h * FT;
  const float* dob = dout + (long long)b * T * C + h * FT;
  const int ty = threadIdx.x / 16, tx = threadIdx.x % 16, k0 = kt * FT;
  load_tile(sK, base + C, pitch, k0, T);
  load_tile(sV, base + 2 * C, pitch, k0, T);
  float dk[8][4], dv[8][4];
  zero(dk); zero(dv);
  for (int qt = kt; qt < n_t; ++qt) {
    const int q0 = qt * FT;
    __syncthreads();                                      // the previous tile's products have read sQ, sO, sP and sS
    load_tile(sQ, base, pitch, q0, T);
    load_tile(sO, dob, C, q0, T);
    __syncthreads();
    float acc[8][4];
    mm_nt(acc, sQ, sK, ty, tx);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int q = q0 + ty * 8 + i;
      const float ls = q < T ? lse[(long long)bh * T + q] : INFINITY;        // rows beyond T: p = 0
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const bool seen = qt > kt || j * 16 + tx <= ty * 8 + i;
        sP[(ty * 8 + i) * FP + j * 16 + tx] = seen ? exp2f(acc[i][j] * SCALE_LOG2 - ls) : 0.f;
      }
    }
    mm_nt(acc, sO, sV, ty, tx);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int q = q0 + ty * 8 + i;
      const float d = q < T ? D[(long long)bh * T + q] : 0.f;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int at = (ty * 8 + i) * FP + j * 16 + tx;   // (the thread's own element of P)
        sS[at] = sP[at] * (acc[i][j] - d);
      }
    }
    __syncthreads();
    mm_tn(acc, sP, sO, ty, tx);                           // tile sums first, then the running sums: shorter chains of additions
    add(dv, acc);
    mm_tn(acc, sS, sQ, ty, tx);
    add(dk, acc);
    if (!DQ) continue;
    mm_nn(acc, sS, sK, ty, tx);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int q = q0 + ty * 8 + i;
      if (q < T)
        asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(dqkv + ((long long)b * T + q) * pitch + h * FT + tx * 4),
                     "f"(acc[i][0] * SCALE), "f"(acc[i][1] * SCALE), "f"(acc[i][2] * SCALE), "f"(acc[i][3] * SCALE) : "memory");
    }
  }
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int k = k0 + ty * 8 + i;
    if (k >= T) continue;
    float* dst = dqkv + ((long long)b * T + k) * pitch + h * FT + tx * 4;
    *reinterpret_cast<float4*>(dst + C) = make_float4(dk[i][0] * SCALE, dk[i][1] * SCALE, dk[i][2] * SCALE, dk[i][3] * SCALE);
    *reinterpret_cast<float4*>(dst + 2 * C) = make_float4(dv[i][0], dv[i][1], dv[i][2], dv[i][3]);
  }
}

// dQ of 64 query rows, the key tiles in order.
__global__ void __launch_bounds__(F32_THREADS, 2) attn_f32_dq_kernel(float* __restrict__ dqkv, const float* __restrict__ dout, const float* __restrict__ qkv,
                                                                  const float* __restrict__ lse, const float* __restrict__ D, int T, int NH, int n_t) {
  extern __shared__ __align__(16) float smf[];
  float *sQ = smf, *sO = sQ + TILE_WORDS, *sK = sO + TILE_WORDS, *sV = sK + TILE_WORDS, *sS = sV + TILE_WORDS;
  pdl_trigger();
  pdl_wait();
  const int BH = gridDim.x / n_t, qt = n_t - 1 - (int)(blockIdx.x / BH), bh = blockIdx.x % BH;      // the longest walks first
  const int b = bh / NH, h = bh % NH, C = NH * FT;
  const long long pitch = 3LL * C;
  const float* base = qkv + (long long)b * T * pitch + h * FT;
  const int ty = threadIdx.x / 16, tx = threadIdx.x % 16, q0 = qt * FT;
  load_tile(sQ, base, pitch, q0, T);
  load_tile(sO, dout + (long long)b * T * C + h * FT, C, q0, T);
  float dq[8][4], ls[8], d[8];
  zero(dq);
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int q = q0 + ty * 8 + i;
    ls[i] = q < T ? lse[(long long)bh * T + q] : INFINITY;                   // rows beyond T: p = 0
    d[i] = q < T ? D[(long long)bh * T + q] : 0.f;
  }
  for (int kt = 0; kt <= qt; ++kt) {
    __syncthreads();                                      // the previous tile's products have read sK, sV and sS
    load_tile(sK, base + C, pitch, kt * FT, T);
    load_tile(sV, base + 2 * C, pitch, kt * FT, T);
    __syncthreads();
    float p[8][4], acc[8][4];
    mm_nt(p, sQ, sK, ty, tx);
    mm_nt(acc, sO, sV, ty, tx);
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const bool seen = kt < qt || j * 16 + tx <= ty * 8 + i;
        sS[(ty * 8 + i) * FP + j * 16 + tx] = seen ? exp2f(p[i][j] * SCALE_LOG2 - ls[i]) * (acc[i][j] - d[i]) : 0.f;
      }
    __syncwarp();                                         // (a warp's rows of dS are written and read by that warp only)
    mm_nn(acc, sS, sK, ty, tx);
    add(dq, acc);
  }
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int q = q0 + ty * 8 + i;
    if (q < T)
      *reinterpret_cast<float4*>(dqkv + ((long long)b * T + q) * pitch + h * FT + tx * 4) =
          make_float4(dq[i][0] * SCALE, dq[i][1] * SCALE, dq[i][2] * SCALE, dq[i][3] * SCALE);
  }
}

constexpr int FWD_SMEM = 4 * TILE_WORDS * 4, BWD_SMEM = 6 * TILE_WORDS * 4, DQ_SMEM = 5 * TILE_WORDS * 4;
bool bad(const void* a, const void* b, const void* c) { return (reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(b) | reinterpret_cast<uintptr_t>(c)) & 15; }
}  // namespace

// out [B,T,C], lse [B,NH,T] (log2 domain, may be null), qkv [B,T,3C], all contiguous fp32; C = NH * 64.
LLMB_API int llmb_attention_f32_fwd(float* out, float* lse, const float* qkv, int B, int T, int NH, cudaStream_t st) {
  const long long n_t = ceil_div(T, FT), grid = n_t * B * NH;
  if (B <= 0 || T <= 0 || NH <= 0 || grid > 0x7fffffffLL || bad(out, qkv, nullptr)) return LLMB_ERR_BAD_ARG;
  const cudaError_t e = cudaFuncSetAttribute(attn_f32_fwd_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, FWD_SMEM);
  if (e != cudaSuccess) return (int)e;
  return launch_pdl(attn_f32_fwd_kernel, (unsigned)grid, F32_THREADS, FWD_SMEM, st, out, lse, qkv, T, NH, (int)n_t);
}
// dqkv [B,T,3C] (overwritten) from dout and out [B,T,C], qkv and the forward's lse; D: scratch of B * NH * T floats.  split: dQ by a
// kernel of its own, the same on every run (one launch more: three kernels).
LLMB_API int llmb_attention_f32_bwd(float* dqkv, float* D, const float* dout, const float* qkv, const float* out, const float* lse, int B, int T,
                                    int NH, int split, cudaStream_t st) {
  const long long n_t = ceil_div(T, FT), grid = n_t * B * NH, rows = (long long)B * T * NH, dots = ceil_div_ll(rows * 16, 256);
  if (B <= 0 || T <= 0 || NH <= 0 || grid > 0x7fffffffLL || dots > 0x7fffffffLL || bad(dqkv, dout, qkv) || bad(out, nullptr, nullptr)) return LLMB_ERR_BAD_ARG;
  auto kern = split ? attn_f32_bwd_kernel<false> : attn_f32_bwd_kernel<true>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, BWD_SMEM);
  if (e == cudaSuccess && split) e = cudaFuncSetAttribute(attn_f32_dq_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, DQ_SMEM);
  const size_t row = (size_t)NH * FT * sizeof(float);
  if (e == cudaSuccess && !split) e = cudaMemset2DAsync(dqkv, 3 * row, 0, row, (size_t)B * T, st);
  if (e != cudaSuccess) return (int)e;
  int rc = launch_pdl(attn_f32_dot_kernel, (unsigned)dots, 256, 0, st, D, dout, out, T, NH, rows);
  if (rc) return rc;
  rc = launch_pdl(kern, (unsigned)grid, F32_THREADS, BWD_SMEM, st, dqkv, dout, qkv, lse, D, T, NH, (int)n_t);
  if (rc || !split) return rc;
  return launch_pdl(attn_f32_dq_kernel, (unsigned)grid, F32_THREADS, DQ_SMEM, st, dqkv, dout, qkv, lse, D, T, NH, (int)n_t);
}
