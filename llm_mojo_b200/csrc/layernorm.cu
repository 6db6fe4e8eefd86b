// LayerNorm forward (optionally fused with the residual add that precedes it) and backward
// with the residual-gradient accumulate and dgamma/dbeta reduction.
//
// Reference behaviour: llmm/layernorm.mojo:197-331 (fwd, mean/rstd saved fp32), :651-1096 (fused
// residual fwd), :1582-1895 (bwd with register-accumulated dgamma/dbeta partials + finalize),
// :2426-2614 (fused residual bwd).  B200 design: one warp per row, the row lives in registers
// (single HBM read), 16-byte accesses; backward is a persistent grid whose CTAs write one
// dgamma/dbeta partial row each into scratch, summed in fixed order by a finalize kernel so
// the result does not depend on scheduling.
#include "common.cuh"
using namespace llmb;

namespace {
constexpr int LN_MAX_VEC = 16;  // 16-byte vectors per lane: C <= 32*16*8 = 4096 for bf16
constexpr float LN_EPS = 1e-5f;
constexpr int LN_BWD_ROWS = 3;    // rows a group of the backward kernel has in flight

template <typename T, bool RESID, int PER_LANE>
__global__ void __launch_bounds__(256) ln_fwd_kernel(T* __restrict__ out, float* __restrict__ mean_o, float* __restrict__ rstd_o,
                                                    T* __restrict__ resid_out, const T* __restrict__ inp1,
                                                    const T* __restrict__ inp2, const T* __restrict__ w,
                                                    const T* __restrict__ b, int rows, int C) {
  pdl_trigger();
  pdl_wait();
  constexpr int N = Pack<T>::N;
  const int lane = threadIdx.x % 32, wid = threadIdx.x / 32;
  const int nvec = C / N;                       // vectors per row
  constexpr int per_lane = PER_LANE;            // 16-byte vectors per lane: the row lives in registers
  int row = blockIdx.x * (blockDim.x / 32) + wid;
  if (row >= rows) return;
  float x[PER_LANE][N];
  float sum = 0.f;
#pragma unroll
  for (int i = 0; i < PER_LANE; ++i) {
    if (i < per_lane) {
      int vc = i * 32 + lane;
      if (vc < nvec) {
        Pack<T> p; p.load(inp1 + (size_t)row * C + vc * N);
        if (RESID) {
          Pack<T> q; q.load(inp2 + (size_t)row * C + vc * N);
#pragma unroll
          for (int k = 0; k < N; ++k) p.v[k] = to_f<T>(from_f<T>(p.v[k] + q.v[k]));  // round like the stored residual
          p.store(resid_out + (size_t)row * C + vc * N);
        }
#pragma unroll
        for (int k = 0; k < N; ++k) { x[i][k] = p.v[k]; sum += p.v[k]; }
      } else {
#pragma unroll
        for (int k = 0; k < N; ++k) x[i][k] = 0.f;
      }
    }
  }
  float mean = warp_sum(sum) / C;
  float var = 0.f;
#pragma unroll
  for (int i = 0; i < PER_LANE; ++i) {
    if (i < per_lane) {
      int vc = i * 32 + lane;
      if (vc < nvec) {
#pragma unroll
        for (int k = 0; k < N; ++k) { float d = x[i][k] - mean; var += d * d; }
      }
    }
  }
  float rstd = rsqrtf(warp_sum(var) / C + LN_EPS);
  if (lane == 0) { if (mean_o) mean_o[row] = mean; if (rstd_o) rstd_o[row] = rstd; }
#pragma unroll
  for (int i = 0; i < PER_LANE; ++i) {
    if (i < per_lane) {
      int vc = i * 32 + lane;
      if (vc < nvec) {
        Pack<T> ww, bb, o; ww.load(w + vc * N); bb.load(b + vc * N);
#pragma unroll
        for (int k = 0; k < N; ++k) o.v[k] = (x[i][k] - mean) * rstd * ww.v[k] + bb.v[k];
        o.store(out + (size_t)row * C + vc * N);
      }
    }
  }
}

// Backward.  dres[row] (+)= LN'(dout[row]); partial dgamma / dbeta of every CTA into scratch.
//
// Bound by memory: three row reads and one row write.  A row belongs to a GROUP of ceil(C / N) threads rounded up to a warp, one
// 16-byte vector per thread, so that a thread's dgamma / dbeta sums are 2 N registers whatever C is (with a warp per row they are
// 2 C / 32 and leave one CTA of 256 threads per SM at C = 1280).  A group takes ROWS rows at a time: all their loads are in flight
// before the first use, and their 2 ROWS dot products share one exchange through shared memory.  Several groups fill a CTA (one
// CTA per SM), meet only at named barriers of their own, and add their sums up in group order at the end, which leaves
// 148 partial rows for the finalize kernel instead of 296.
// Measured on a B200, both kernels of a call, warp-per-row form -> this one: 4096 x 1280 25.2 -> 15.5 us, 8192 x 1280 32.1 -> 21.4,
// 4096 x 1600 31.8 -> 18.5, 12288 x 1024 34.9 -> 23.5, 4096 x 768 14.5 -> 12.8, 65536 x 768 82.9 -> 81.8 (403 MB: 4.9 TB/s).
// ROWS = 2 is within 1 us of 3 up to 12288 rows and 9 % slower at 65536; 4 spills and is 10 - 30 % slower everywhere.
// SUMOUT: the column sums of the values written to dres are a third partial (the bias gradient of the linear layer whose output
// gradient dres is), taken from the values as stored (after rounding to T).
template <typename T, int ROWS, bool ACCUM, bool SUMOUT>
__global__ void __launch_bounds__(640) ln_bwd_kernel(T* __restrict__ dres, float* __restrict__ partial, const T* __restrict__ dout,
                                                    const T* __restrict__ inp, const T* __restrict__ w,
                                                    const float* __restrict__ mean_i, const float* __restrict__ rstd_i, int rows,
                                                    int C, int gthreads, int groups) {
  pdl_trigger();
  pdl_wait();
  constexpr int N = Pack<T>::N;
  constexpr int NS = SUMOUT ? 3 : 2;
  extern __shared__ float sm[];                        // [NS][C] column sums
  __shared__ float2 xch[2][20][ROWS];                  // [parity][warp of the CTA][row]
  const int group = threadIdx.x / gthreads, t = threadIdx.x - group * gthreads;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, gwarps = gthreads >> 5, gw0 = group * gwarps;
  const int nvec = C / N;
  const bool act = t < nvec;
  float dg[N], db[N], ds[SUMOUT ? N : 1];
#pragma unroll
  for (int k = 0; k < N; ++k) { dg[k] = 0.f; db[k] = 0.f; if (SUMOUT) ds[k] = 0.f; }
  uint4 wr = make_uint4(0, 0, 0, 0);                   // gamma of this thread's channels (raw: unpacked where it is used)
  if (act) wr = *reinterpret_cast<const uint4*>(w + t * N);
  const float inv_c = 1.f / C;
  int par = 0;
  const int stride = gridDim.x * groups * ROWS;
  for (int row0 = (group * gridDim.x + blockIdx.x) * ROWS; row0 < rows; row0 += stride, par ^= 1) {
    uint4 xr[ROWS], dr[ROWS], ar[ROWS];
#pragma unroll
    for (int r = 0; r < ROWS; ++r) {
      const int row = row0 + r;
      if (row < rows) {
        if (act) {
          const size_t o = (size_t)row * C + t * N;
          xr[r] = *reinterpret_cast<const uint4*>(inp + o);
          dr[r] = *reinterpret_cast<const uint4*>(dout + o);
          if (ACCUM) ar[r] = *reinterpret_cast<const uint4*>(dres + o);
        }
      }
      if (row >= rows || !act) { xr[r] = make_uint4(0, 0, 0, 0); dr[r] = make_uint4(0, 0, 0, 0); }
    }
    float s1[ROWS], s2[ROWS];
#pragma unroll
    for (int r = 0; r < ROWS; ++r) {
      Pack<T> x, d, ww; x.load(reinterpret_cast<const T*>(&xr[r])); d.load(reinterpret_cast<const T*>(&dr[r]));
      ww.load(reinterpret_cast<const T*>(&wr));
      const int row = min(row0 + r, rows - 1);
      const float mean = mean_i[row], rstd = rstd_i[row];
      s1[r] = 0.f; s2[r] = 0.f;
#pragma unroll
      for (int k = 0; k < N; ++k) {
        const float n_ = (x.v[k] - mean) * rstd;
        const float dn_ = d.v[k] * ww.v[k];
        s1[r] += dn_; s2[r] += dn_ * n_;
        dg[k] += d.v[k] * n_; db[k] += d.v[k];
      }
    }
#pragma unroll
    for (int r = 0; r < ROWS; ++r) { s1[r] = warp_sum(s1[r]); s2[r] = warp_sum(s2[r]); }
    if (gwarps > 1) {                                  // alternating buffers: one barrier per exchange
      if (lane == 0) {
#pragma unroll
        for (int r = 0; r < ROWS; ++r) xch[par][wid][r] = make_float2(s1[r], s2[r]);
      }
      asm volatile("bar.sync %0, %1;" ::"r"(group + 1), "r"(gthreads) : "memory");
#pragma unroll
      for (int r = 0; r < ROWS; ++r) { s1[r] = 0.f; s2[r] = 0.f; }
      for (int j = 0; j < gwarps; ++j) {
#pragma unroll
        for (int r = 0; r < ROWS; ++r) { const float2 v = xch[par][gw0 + j][r]; s1[r] += v.x; s2[r] += v.y; }
      }
    }
    if (act) {
#pragma unroll
      for (int r = 0; r < ROWS; ++r) {
        const int row = row0 + r;
        if (row >= rows) break;
        // opaque to the compiler: otherwise it keeps the unpacked values of the first pass (64 registers) across the exchange
        asm volatile("" : "+r"(xr[r].x), "+r"(xr[r].y), "+r"(xr[r].z), "+r"(xr[r].w), "+r"(dr[r].x), "+r"(dr[r].y), "+r"(dr[r].z), "+r"(dr[r].w));
        asm volatile("" : "+r"(wr.x), "+r"(wr.y), "+r"(wr.z), "+r"(wr.w));
        const float mean = mean_i[row], rstd = rstd_i[row];
        Pack<T> ww; ww.load(reinterpret_cast<const T*>(&wr));
        Pack<T> x, d, o; x.load(reinterpret_cast<const T*>(&xr[r])); d.load(reinterpret_cast<const T*>(&dr[r]));
        if (ACCUM) o.load(reinterpret_cast<const T*>(&ar[r]));
        const float m1 = s1[r] * inv_c, m2 = s2[r] * inv_c;
#pragma unroll
        for (int k = 0; k < N; ++k) {
          const float n_ = (x.v[k] - mean) * rstd;
          const float g = (d.v[k] * ww.v[k] - m1 - n_ * m2) * rstd;
          o.v[k] = ACCUM ? o.v[k] + g : g;
          if (SUMOUT) ds[k] += round_to<T>(o.v[k]);
        }
        o.store(dres + (size_t)row * C + t * N);
      }
    }
  }
  // the groups of the CTA in fixed order
  for (int g = 0; g < groups; ++g) {
    if (group == g && act) {
#pragma unroll
      for (int k = 0; k < N; ++k) {
        const int c = t * N + k;
        if (g == 0) { sm[c] = dg[k]; sm[C + c] = db[k]; if (SUMOUT) sm[2 * C + c] = ds[k]; }
        else { sm[c] += dg[k]; sm[C + c] += db[k]; if (SUMOUT) sm[2 * C + c] += ds[k]; }
      }
    }
    __syncthreads();
  }
  for (int c = threadIdx.x; c < NS * C; c += blockDim.x) partial[(size_t)blockIdx.x * NS * C + c] = sm[c];
}

// dw[c] += sum_i partial[i][c], db[c] += sum_i partial[i][C + c] over the per-CTA partial rows.  A block of
// 32 x 32 threads owns 32 adjacent columns of the partial matrix: 32 row groups walk the rows in parallel (coalesced
// 128-byte reads, at most five dependent steps for 148 rows) and are combined in fixed order through shared memory.
__global__ void __launch_bounds__(1024) ln_bwd_final_kernel(float* __restrict__ dw, float* __restrict__ db, float* __restrict__ dsum,
                                                           const float* __restrict__ partial, int C, int nblocks) {
  pdl_trigger();
  pdl_wait();
  __shared__ float red[32][33];
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  const int c = blockIdx.x * 32 + tx;
  const int NS = dsum ? 3 : 2;                           // dsum: third partial = column sums of the stored dres
  float s = 0.f;
  if (c < NS * C) {
#pragma unroll 5
    for (int i = ty; i < nblocks; i += 32) s += partial[(size_t)i * NS * C + c];
  }
  red[ty][tx] = s;
  __syncthreads();
  const float v = warp_sum(red[tx][ty]);                 // warp ty adds up column ty
  const int cc = blockIdx.x * 32 + ty;
  if (tx == 0 && cc < NS * C) {
    if (cc < C) dw[cc] += v; else if (cc < 2 * C) db[cc - C] += v; else dsum[cc - 2 * C] += v;
  }
}

template <typename T, int PER_LANE>
int ln_fwd_launch_n(void* out, float* mean, float* rstd, void* resid_out, const void* inp1, const void* inp2,
                    const void* w, const void* b, int rows, int C, cudaStream_t st) {
  int grid = ceil_div(rows, 8);
  if (inp2)
    launch_pdl(ln_fwd_kernel<T, true, PER_LANE>, grid, 256, 0, st, (T*)out, mean, rstd, (T*)resid_out, (const T*)inp1, (const T*)inp2, (const T*)w, (const T*)b, rows, C);
  else
    launch_pdl(ln_fwd_kernel<T, false, PER_LANE>, grid, 256, 0, st, (T*)out, mean, rstd, nullptr, (const T*)inp1, nullptr, (const T*)w, (const T*)b, rows, C);
  return (int)cudaGetLastError();
}

template <typename T>
int ln_fwd_launch(void* out, float* mean, float* rstd, void* resid_out, const void* inp1, const void* inp2,
                  const void* w, const void* b, int rows, int C, cudaStream_t st) {
  constexpr int N = Pack<T>::N;
  if (C % N || C / N > 32 * LN_MAX_VEC) return LLMB_ERR_BAD_ARG;
  const int per = ceil_div(C / N, 32);
#define LNF(P) return ln_fwd_launch_n<T, P>(out, mean, rstd, resid_out, inp1, inp2, w, b, rows, C, st)
  if (per <= 1) LNF(1); if (per <= 2) LNF(2); if (per <= 3) LNF(3); if (per <= 4) LNF(4); if (per <= 5) LNF(5);
  if (per <= 6) LNF(6); if (per <= 7) LNF(7); if (per <= 8) LNF(8); if (per <= 10) LNF(10); if (per <= 12) LNF(12);
  if (per <= 13) LNF(13); LNF(16);
#undef LNF
}

// Threads per row group, groups per CTA and CTAs of the backward kernel: as many groups as fill 640 threads (96 registers each),
// but no more than there are chunks of rows for (every group costs a step of the final combination).
struct LnBwdPlan { int gthreads, groups, grid; };
inline LnBwdPlan ln_bwd_plan(int rows, int C, int elems_per_vec) {
  LnBwdPlan p;
  p.gthreads = ceil_div(ceil_div(C, elems_per_vec), 32) * 32;
  const int chunks = ceil_div(rows, LN_BWD_ROWS);
  p.grid = chunks < sm_count() ? chunks : sm_count();
  p.groups = 640 / p.gthreads;
  if (p.groups > ceil_div(chunks, p.grid)) p.groups = ceil_div(chunks, p.grid);
  if (p.groups < 1) p.groups = 1;
  if (p.groups > 15) p.groups = 15;                      // named barriers 1 .. 15
  return p;
}

template <typename T>
int ln_bwd_launch(void* dres, float* partial, const void* dout, const void* inp, const void* w, const float* mean, const float* rstd,
                  int rows, int C, int accumulate, bool sumout, cudaStream_t st) {
  constexpr int N = Pack<T>::N;
  if (C % N || C / N > 512) return LLMB_ERR_BAD_ARG;
  const LnBwdPlan p = ln_bwd_plan(rows, C, N);
  const size_t smem = (size_t)(sumout ? 3 : 2) * C * sizeof(float);
  auto kern = sumout ? (accumulate ? ln_bwd_kernel<T, LN_BWD_ROWS, true, true> : ln_bwd_kernel<T, LN_BWD_ROWS, false, true>)
                     : (accumulate ? ln_bwd_kernel<T, LN_BWD_ROWS, true, false> : ln_bwd_kernel<T, LN_BWD_ROWS, false, false>);
  if (smem > 40 * 1024) {
    const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return (int)e;
  }
  launch_pdl(kern, p.grid, p.gthreads * p.groups, smem, st, (T*)dres, partial, (const T*)dout, (const T*)inp, (const T*)w, mean, rstd, rows, C,
                                                    p.gthreads, p.groups);
  return (int)cudaGetLastError();
}
}  // namespace

LLMB_API int llmb_layernorm_fwd(void* out, float* mean, float* rstd, void* resid_out, const void* inp1,
                                const void* inp2, const void* w, const void* b, int rows, int C, int dtype,
                                cudaStream_t st) {
  return dtype == LLMB_BF16 ? ln_fwd_launch<__nv_bfloat16>(out, mean, rstd, resid_out, inp1, inp2, w, b, rows, C, st)
                            : ln_fwd_launch<float>(out, mean, rstd, resid_out, inp1, inp2, w, b, rows, C, st);
}

LLMB_API long long llmb_layernorm_bwd_scratch_bytes(int rows, int C) {
  const int need = ceil_div(rows, LN_BWD_ROWS);
  return (long long)(need < sm_count() ? need : sm_count()) * 3 * C * sizeof(float);      // room for the optional column-sum partial
}

// dres (+)= LN-backward(dout); dw += ..., db += ...  (dw/db fp32).  accumulate=1 adds into dres.
LLMB_API int llmb_layernorm_bwd_colsum(void* dres, float* dw, float* db, float* dsum, float* scratch, long long scratch_bytes,
                                       const void* dout, const void* inp, const void* w, const float* mean,
                                       const float* rstd, int rows, int C, int accumulate, int dtype, cudaStream_t st);
LLMB_API int llmb_layernorm_bwd(void* dres, float* dw, float* db, float* scratch, long long scratch_bytes,
                                const void* dout, const void* inp, const void* w, const float* mean,
                                const float* rstd, int rows, int C, int accumulate, int dtype, cudaStream_t st) {
  return llmb_layernorm_bwd_colsum(dres, dw, db, nullptr, scratch, scratch_bytes, dout, inp, w, mean, rstd, rows, C, accumulate, dtype, st);
}
// As llmb_layernorm_bwd; with dsum != nullptr additionally dsum[c] += sum over rows of the values written to dres[:, c]
// (fp32 [C]): the bias gradient of the linear layer whose output gradient dres is, without another pass over dres.
LLMB_API int llmb_layernorm_bwd_colsum(void* dres, float* dw, float* db, float* dsum, float* scratch, long long scratch_bytes,
                                       const void* dout, const void* inp, const void* w, const float* mean,
                                       const float* rstd, int rows, int C, int accumulate, int dtype, cudaStream_t st) {
  const bool sumout = dsum != nullptr;
  if (rows <= 0 || C <= 0) return LLMB_ERR_BAD_ARG;       // (before the plan divides by them)
  const int grid = ln_bwd_plan(rows, C, 8).grid;
  if (scratch_bytes < (long long)grid * (sumout ? 3 : 2) * C * (long long)sizeof(float)) return LLMB_ERR_BAD_ARG;
  const int rc = dtype == LLMB_BF16 ? ln_bwd_launch<__nv_bfloat16>(dres, scratch, dout, inp, w, mean, rstd, rows, C, accumulate, sumout, st)
                                    : ln_bwd_launch<float>(dres, scratch, dout, inp, w, mean, rstd, rows, C, accumulate, sumout, st);
  if (rc) return rc;
  launch_pdl(ln_bwd_final_kernel, ceil_div((sumout ? 3 : 2) * C, 32), 1024, 0, st, dw, db, dsum, scratch, C, grid);
  return (int)cudaGetLastError();
}
