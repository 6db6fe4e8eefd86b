// Fused softmax + cross-entropy + in-place dlogits over the padded vocabulary, plus the
// generic row softmax used by sampling.
//
// Reference behaviour: llmm/fused_classifier.mojo:186-279, :311-370 (per row: max, sum exp,
// loss, dlogits = (p - 1[y])·dloss written over the logits, padded tail [V, Vp) zeroed);
// llmm/softmax.mojo:172-304.  B200 design: the whole row (Vp·2 B ≈ 100 KB for GPT-2) is staged once
// in shared memory so HBM sees exactly one read and one write.  bf16 rows stream through a persistent
// CTA per SM: the bulk-copy engine loads row r+1 into one buffer and stores row r-1 out of it while the
// 1024 threads make their three passes (max, exponentials + sum, scale) over row r in the other.
#include "tc05.cuh"
using namespace llmb;
using namespace tc05;

namespace {
template <typename T>
__global__ void __launch_bounds__(1024) classifier_kernel(T* __restrict__ logits, float* __restrict__ losses,
                                                         const int* __restrict__ targets, float dloss, int V, int Vp,
                                                         int write_dlogits) {
  pdl_trigger();
  pdl_wait();
  constexpr int N = Pack<T>::N;
  extern __shared__ __align__(16) unsigned char smraw[];
  T* row_s = reinterpret_cast<T*>(smraw);
  __shared__ float red[32];
  __shared__ float bcast[2];
  const int row = blockIdx.x;
  T* g = logits + (size_t)row * Vp;
  const int nvec = Vp / N;
  const int tid = threadIdx.x, lane = tid % 32, wid = tid / 32, nw = blockDim.x / 32;
  float mx = -INFINITY;
  for (int v = tid; v < nvec; v += blockDim.x) {
    uint4 raw = *reinterpret_cast<const uint4*>(g + v * N);
    *reinterpret_cast<uint4*>(row_s + v * N) = raw;
    Pack<T> p; p.load(row_s + v * N);
#pragma unroll
    for (int k = 0; k < N; ++k) if (v * N + k < V) mx = fmaxf(mx, p.v[k]);
  }
  mx = warp_max(mx);
  if (lane == 0) red[wid] = mx;
  __syncthreads();
  if (wid == 0) { float m = lane < nw ? red[lane] : -INFINITY; m = warp_max(m); if (lane == 0) bcast[0] = m; }
  __syncthreads();
  mx = bcast[0];
  const float L2E = 1.4426950408889634f;
  // second pass: e = 2^((x - max)·log2e) once per element; the row buffer is overwritten with e (in the
  // storage dtype) so that the third pass is a multiply, not another exponential
  const int tgt_raw = targets[row];
  const int tgt = llmb_in_range(tgt_raw, V, LLMB_SITE_CLASSIFIER_TARGET) ? tgt_raw : 0;   // checked build: a bad target is recorded and clamped
  const float x_tgt = to_f<T>(row_s[tgt]);            // read before the buffer is overwritten
  __syncthreads();
  float sum = 0.f;
  for (int v = tid; v < nvec; v += blockDim.x) {
    Pack<T> p; p.load(row_s + v * N);
#pragma unroll
    for (int k = 0; k < N; ++k) {
      const float e = (v * N + k < V) ? exp2f((p.v[k] - mx) * L2E) : 0.f;
      sum += e;
      p.v[k] = e;
    }
    if (write_dlogits) p.store(row_s + v * N);
  }
  sum = warp_sum(sum);
  if (lane == 0) red[wid] = sum;
  __syncthreads();
  if (wid == 0) { float s = lane < nw ? red[lane] : 0.f; s = warp_sum(s); if (lane == 0) bcast[1] = s; }
  __syncthreads();
  sum = bcast[1];
  if (tid == 0 && losses) losses[row] = -(x_tgt - mx - logf(sum));
  if (!write_dlogits) return;
  const float inv = dloss / sum;
  for (int v = tid; v < nvec; v += blockDim.x) {
    Pack<T> p; p.load(row_s + v * N);
#pragma unroll
    for (int k = 0; k < N; ++k) {
      const int i = v * N + k;
      p.v[k] = p.v[k] * inv - (i == tgt ? dloss : 0.f);      // padded columns hold e = 0
    }
    p.store(g + v * N);
  }
}

// Persistent streaming variant for bf16 rows (two row buffers fit in shared memory).
__device__ __forceinline__ float ex2_fast(float x) { float y; asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x)); return y; }
__device__ __forceinline__ void bulk_store_1d(void* gdst, const void* ssrc, uint32_t bytes) {
  asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;"
               ::"l"(reinterpret_cast<uint64_t>(gdst)), "r"(smem_u32(ssrc)), "r"(bytes) : "memory");
}

__global__ void __launch_bounds__(1024, 1) classifier_stream_kernel(__nv_bfloat16* __restrict__ logits, float* __restrict__ losses,
                                                                   const int* __restrict__ targets, float dloss, int rows, int V,
                                                                   int Vp, int write_dlogits, int buf_bytes, int* status) {
  pdl_trigger();
  pdl_wait();
  using T = __nv_bfloat16;
  constexpr int N = 8;
  extern __shared__ __align__(128) unsigned char smraw[];
  __shared__ uint64_t full[2];
  __shared__ float red[32];
  __shared__ float bcast[2];
  __shared__ int fail_s;
  const int tid = threadIdx.x, lane = tid % 32, wid = tid / 32, nw = blockDim.x / 32;
  const uint32_t row_bytes = (uint32_t)Vp * 2;
  const int nvec = Vp / N;
  if (tid == 0) { mbar_init(&full[0], 1); mbar_init(&full[1], 1); fail_s = 0; fence_barrier_init(); }
  __syncthreads();
  int r = blockIdx.x;
  if (tid == 0 && r < rows) {
    mbar_expect_tx(&full[0], row_bytes);
    bulk_load_1d(smraw, logits + (size_t)r * Vp, row_bytes, &full[0]);
  }
  const float L2E = 1.4426950408889634f;
  for (int it = 0; r < rows; r += gridDim.x, ++it) {
    const int b = it & 1;
    T* row_s = reinterpret_cast<T*>(smraw + (size_t)b * buf_bytes);
    const int rn = r + gridDim.x;
    if (tid == 0 && rn < rows) {
      bulk_wait_read<0>();                  // the store of the previous row has finished reading the other buffer
      mbar_expect_tx(&full[b ^ 1], row_bytes);
      bulk_load_1d(smraw + (size_t)(b ^ 1) * buf_bytes, logits + (size_t)rn * Vp, row_bytes, &full[b ^ 1]);
    }
    if (!mbar_wait(&full[b], (it >> 1) & 1)) { atomicExch(status, LLMB_ERR_TIMEOUT); fail_s = 1; }
    __syncthreads();
    if (fail_s) break;
    // Vectors that lie wholly inside the real vocabulary [0, V) need no per-element bound checks; the one
    // vector that straddles V and the padded ones after it are handled by a second, checked loop.
    const int nfull = V / N;                 // vectors entirely below V
    // pass 1: row maximum over the real vocabulary
    float mx = -INFINITY;
    for (int v = tid; v < nfull; v += blockDim.x) {
      Pack<T> p; p.load(row_s + v * N);
#pragma unroll
      for (int k = 0; k < N; ++k) mx = fmaxf(mx, p.v[k]);
    }
    for (int v = nfull + tid; v < nvec; v += blockDim.x) {
      Pack<T> p; p.load(row_s + v * N);
#pragma unroll
      for (int k = 0; k < N; ++k) if (v * N + k < V) mx = fmaxf(mx, p.v[k]);
    }
    mx = warp_max(mx);
    if (lane == 0) red[wid] = mx;
    __syncthreads();
    if (wid == 0) { float m = lane < nw ? red[lane] : -INFINITY; m = warp_max(m); if (lane == 0) bcast[0] = m; }
    __syncthreads();
    mx = bcast[0];
    const int tgt_raw = targets[r];
  const int tgt = llmb_in_range(tgt_raw, V, LLMB_SITE_CLASSIFIER_TARGET) ? tgt_raw : 0;   // checked build: a bad target is recorded and clamped
    const float x_tgt = __bfloat162float(row_s[tgt]);     // read before the buffer is overwritten
    __syncthreads();
    // pass 2: e = 2^((x - max) log2 e), once per element, written back over the row
    float sum = 0.f;
    const float mb = mx * L2E;
    for (int v = tid; v < nfull; v += blockDim.x) {
      Pack<T> p; p.load(row_s + v * N);
#pragma unroll
      for (int k = 0; k < N; ++k) { p.v[k] = ex2_fast(fmaf(p.v[k], L2E, -mb)); sum += p.v[k]; }
      if (write_dlogits) p.store(row_s + v * N);
    }
    for (int v = nfull + tid; v < nvec; v += blockDim.x) {
      Pack<T> p; p.load(row_s + v * N);
#pragma unroll
      for (int k = 0; k < N; ++k) { p.v[k] = (v * N + k < V) ? ex2_fast(fmaf(p.v[k], L2E, -mb)) : 0.f; sum += p.v[k]; }
      if (write_dlogits) p.store(row_s + v * N);
    }
    sum = warp_sum(sum);
    if (lane == 0) red[wid] = sum;
    __syncthreads();
    if (wid == 0) { float s = lane < nw ? red[lane] : 0.f; s = warp_sum(s); if (lane == 0) bcast[1] = s; }
    __syncthreads();
    sum = bcast[1];
    if (tid == 0 && losses) losses[r] = -(x_tgt - mx - logf(sum));
    if (write_dlogits) {
      // pass 3: dlogits = (e / sum - 1[target]) dloss in place (padded columns hold e = 0); the target column is
      // corrected afterwards by the one thread that owns it; then one bulk store of the row
      const float inv = dloss / sum;
      for (int v = tid; v < nvec; v += blockDim.x) {
        Pack<T> p; p.load(row_s + v * N);
#pragma unroll
        for (int k = 0; k < N; ++k) p.v[k] *= inv;
        p.store(row_s + v * N);
      }
      __syncthreads();
      if (tid == 0) {
        const float e_t = ex2_fast(fmaf(x_tgt, L2E, -mb));
        row_s[tgt] = __float2bfloat16(__bfloat162float(__float2bfloat16(e_t)) * inv - dloss);
      }
      fence_proxy_async();
      __syncthreads();
      if (tid == 0) { bulk_store_1d(logits + (size_t)r * Vp, row_s, row_bytes); bulk_commit(); }
    } else {
      __syncthreads();                      // everyone is done with the buffer before it is reloaded
    }
  }
  if (tid == 0) bulk_wait<0>();             // shared memory must outlive the last store
}

// The same streaming kernel with the row traffic on its own warp.  In the kernel above thread 0 waits for the previous
// row's store to have read its buffer before it may prefetch the next row, and everybody waits for thread 0 at the next
// barrier: the store's read-out is serialised with the row's arithmetic.  Here warps 0..30 (992 threads, named barrier 1)
// only compute; warp 31 moves rows: it stores a buffer once the compute warps hand it over (`done`), waits for that
// store to have read the buffer and refills it with the row after next (`full`).  Per row the steady state is
// max(arithmetic, (arithmetic + store + load) / 2) instead of store + arithmetic.
template <int MAXV>
__global__ void __launch_bounds__(1024, 1) classifier_stream2_kernel(__nv_bfloat16* __restrict__ logits, float* __restrict__ losses,
                                                                     const int* __restrict__ targets, float dloss, int rows, int V,
                                                                     int Vp, int write_dlogits, int buf_bytes, int* status) {
  pdl_trigger();
  pdl_wait();
  using T = __nv_bfloat16;
  constexpr int N = 8;
  constexpr int NC = 992, NCW = 31;                       // compute threads / warps
  extern __shared__ __align__(128) unsigned char smraw[];
  __shared__ uint64_t full[2], done[2];
  __shared__ float red[32], reds[32];
  __shared__ int fail_s;
  const int tid = threadIdx.x, lane = tid % 32, wid = tid / 32;
  const uint32_t row_bytes = (uint32_t)Vp * 2;
  const int nvec = Vp / N;
  if (tid == 0) {
    mbar_init(&full[0], 1); mbar_init(&full[1], 1); mbar_init(&done[0], 1); mbar_init(&done[1], 1);
    fail_s = 0; fence_barrier_init();
  }
  __syncthreads();
  auto csync = [] { asm volatile("bar.sync 1, 992;" ::: "memory"); };

  if (wid == NCW) {
    // ------------------------------------------------------------ row mover (one lane)
    if (lane == 0) {
      for (int j = 0; j < 2; ++j) {
        const long long r = (long long)blockIdx.x + (long long)j * gridDim.x;
        if (r < rows) { mbar_expect_tx(&full[j], row_bytes); bulk_load_1d(smraw + (size_t)j * buf_bytes, logits + (size_t)r * Vp, row_bytes, &full[j]); }
      }
      int it = 0;
      for (int r = blockIdx.x; r < rows; r += gridDim.x, ++it) {
        const int b = it & 1;
        unsigned char* buf = smraw + (size_t)b * buf_bytes;
        if (!mbar_wait(&done[b], (it >> 1) & 1)) { atomicExch(status, LLMB_ERR_TIMEOUT); break; }
        if (write_dlogits) { bulk_store_1d(logits + (size_t)r * Vp, buf, row_bytes); bulk_commit(); }
        const long long rn = (long long)r + 2ll * gridDim.x;
        if (rn < rows) {
          if (write_dlogits) bulk_wait_read<0>();         // the store has read the buffer
          mbar_expect_tx(&full[b], row_bytes);
          bulk_load_1d(buf, logits + (size_t)rn * Vp, row_bytes, &full[b]);
        }
      }
      bulk_wait_read<0>();                                // shared memory must outlive the last store's reads of it
    }
    return;
  }

  // -------------------------------------------------------------- compute warps
  // A thread holds its part of the row (MAXV 16-byte vectors) in registers from the one read of the buffer to the one write:
  // packed bf16 maximum, exponentials packed back into the same registers, scaled by 1 / sum on the way out.  Re-reading the buffer
  // for each pass, with two barriers around every reduction, took 6.5 us a row against the 4.5 us in which an SM's share of the
  // memory bandwidth moves it.  4096 x 50304: 175 -> 162 us, 16384 x 50304: 623 -> 608 us (5.4 TB/s; what is left is the buffers' cycle of
  // load, arithmetic and store: a third buffer does not fit).
  const float L2E = 1.4426950408889634f;
  const int nfull = V / N;                                // vectors entirely below V
  int it = 0;
  for (int r = blockIdx.x; r < rows; r += gridDim.x, ++it) {
    const int b = it & 1;
    T* row_s = reinterpret_cast<T*>(smraw + (size_t)b * buf_bytes);
    if (!mbar_wait(&full[b], (it >> 1) & 1)) { atomicExch(status, LLMB_ERR_TIMEOUT); fail_s = 1; }
    uint4 u[MAXV];
#pragma unroll
    for (int j = 0; j < MAXV; ++j) {
      const int v = tid + j * NC;
      u[j] = v < nvec ? *reinterpret_cast<const uint4*>(row_s + v * N) : make_uint4(0xff80ff80u, 0xff80ff80u, 0xff80ff80u, 0xff80ff80u);
      if (v >= nfull && v < nvec) {                       // padded columns count as -infinity
        unsigned short* h = reinterpret_cast<unsigned short*>(&u[j]);
#pragma unroll
        for (int k = 0; k < N; ++k) if (v * N + k >= V) h[k] = 0xff80u;
      }
    }
    float x_tgt = 0.f;
    int tgt = 0;
    if (tid == 0) {
      tgt = targets[r];
      if (!llmb_in_range(tgt, V, LLMB_SITE_CLASSIFIER_TARGET)) tgt = 0;               // checked build: a bad target is recorded and clamped
      x_tgt = __bfloat162float(row_s[tgt]);
    }
    __nv_bfloat162 m2 = __floats2bfloat162_rn(-INFINITY, -INFINITY);
#pragma unroll
    for (int j = 0; j < MAXV; ++j) {
      const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&u[j]);
      m2 = __hmax2(m2, __hmax2(__hmax2(h[0], h[1]), __hmax2(h[2], h[3])));
    }
    float mx = warp_max(fmaxf(__low2float(m2), __high2float(m2)));
    if (lane == 0) red[wid] = mx;
    csync();
    if (fail_s) break;
    mx = warp_max(lane < NCW ? red[lane] : -INFINITY);
    const float mb = mx * L2E;
    float s0 = 0.f, s1 = 0.f;
#pragma unroll
    for (int j = 0; j < MAXV; ++j) {
      uint32_t* h = reinterpret_cast<uint32_t*>(&u[j]);
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const float e0 = ex2_fast(fmaf(__uint_as_float(h[k] << 16), L2E, -mb)), e1 = ex2_fast(fmaf(__uint_as_float(h[k] & 0xffff0000u), L2E, -mb));
        s0 += e0; s1 += e1;
        const __nv_bfloat162 e = __floats2bfloat162_rn(e0, e1);
        h[k] = *reinterpret_cast<const uint32_t*>(&e);
      }
    }
    float sum = warp_sum(s0 + s1);
    if (lane == 0) reds[wid] = sum;
    csync();
    sum = warp_sum(lane < NCW ? reds[lane] : 0.f);
    if (tid == 0 && losses) losses[r] = -(x_tgt - mx - logf(sum));
    if (write_dlogits) {
      // dlogits = (e / sum - 1[target]) dloss (padded columns hold e = 0); the target column is corrected afterwards by one thread;
      // then the row is handed to the mover
      const float inv = dloss / sum;
#pragma unroll
      for (int j = 0; j < MAXV; ++j) {
        const int v = tid + j * NC;
        uint32_t* h = reinterpret_cast<uint32_t*>(&u[j]);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const __nv_bfloat162 o = __floats2bfloat162_rn(__uint_as_float(h[k] << 16) * inv, __uint_as_float(h[k] & 0xffff0000u) * inv);
          h[k] = *reinterpret_cast<const uint32_t*>(&o);
        }
        if (v < nvec) *reinterpret_cast<uint4*>(row_s + v * N) = u[j];
      }
      fence_proxy_async();                                // these writes, before the mover's bulk store reads them
      csync();
      if (tid == 0) {
        const float e_t = ex2_fast(fmaf(x_tgt, L2E, -mb));
        row_s[tgt] = __float2bfloat16(__bfloat162float(__float2bfloat16(e_t)) * inv - dloss);
        fence_proxy_async();
        mbar_arrive(&done[b]);
      }
    } else {
      csync();                                            // everyone is done with the buffer before it is reloaded
      if (tid == 0) mbar_arrive(&done[b]);
    }
  }
}

// (max, sum of exp(x - max)) of two disjoint sets of values.  fmaxf passes over NaN: a set of nothing but NaN and -infinity has the
// maximum -infinity, and its sum says which (NaN, or 0 where all are -infinity).
__device__ __forceinline__ float2 merge_ms(float2 a, float2 b) {
  const float m = fmaxf(a.x, b.x);
  if (m == -INFINITY) return make_float2(m, a.x + b.x != m ? NAN : a.y + b.y);
  return make_float2(m, a.y * expf(a.x - m) + b.y * expf(b.x - m));
}
// the set of one value
__device__ __forceinline__ float2 single_ms(float x) { return make_float2(x, x == -INFINITY ? 0.f : 1.f); }
// what the exponents of a set are taken relative to: its maximum, if that is finite
__device__ __forceinline__ float base_ms(float m) { return m == -INFINITY ? 0.f : m; }
__device__ __forceinline__ float2 warp_merge_ms(float2 v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = merge_ms(v, make_float2(__shfl_xor_sync(0xffffffffu, v.x, o), __shfl_xor_sync(0xffffffffu, v.y, o)));
  return v;
}

// Row softmax to fp32 with a cluster of CL CTAs per row.  A single row of a 50k vocabulary (one sampling step) is bound by one
// SM's latency and load rate: spread over eight SMs, whose (max, sum) pairs meet through distributed shared memory, each thread
// reads a couple of 16-byte vectors once for the statistics and once (from L1 / L2) for the result.  1 x 50257 bf16, one B200:
// 74 us with one CTA and scalar loads.  From SM_CLUSTER_ROWS rows on one CTA per row fills the chip.
template <typename T, int CL>
__global__ void __launch_bounds__(512) softmax_rows_kernel(float* __restrict__ out, const T* __restrict__ inp, int V, int ld, float inv_temp) {
  pdl_trigger();
  pdl_wait();
  constexpr int N = Pack<T>::N;
  __shared__ float2 red[16];
  __shared__ float2 part[8];                              // written by every CTA of the cluster
  const int tid = threadIdx.x, lane = tid % 32, wid = tid / 32;
  const int row = blockIdx.x / CL, rank = CL > 1 ? (int)cluster_ctarank() : 0;
  const T* g = inp + (size_t)row * ld;
  if (CL > 1) asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");   // the peers have started before anything is written to them
  const bool vec = (reinterpret_cast<uintptr_t>(g) & 15) == 0;
  const int chunk = ceil_div(ceil_div(V, CL), N) * N;     // columns per CTA, a whole number of vectors
  const int c0 = min(rank * chunk, V), c1 = min(c0 + chunk, V);
  float2 ms = make_float2(-INFINITY, 0.f);
  for (int i = c0 + tid * N; i < c1; i += blockDim.x * N) {
    float x[N], m = -INFINITY, sum = 0.f;
    if (vec && i + N <= c1) { Pack<T> p; p.load(g + i);
#pragma unroll
      for (int k = 0; k < N; ++k) x[k] = p.v[k] * inv_temp;
    } else {
#pragma unroll
      for (int k = 0; k < N; ++k) x[k] = i + k < c1 ? to_f<T>(g[i + k]) * inv_temp : -INFINITY;
    }
#pragma unroll
    for (int k = 0; k < N; ++k) m = fmaxf(m, x[k]);
    const float m0 = base_ms(m);
#pragma unroll
    for (int k = 0; k < N; ++k) sum += expf(x[k] - m0);
    ms = merge_ms(ms, make_float2(m, sum));
  }
  ms = warp_merge_ms(ms);
  if (lane == 0) red[wid] = ms;
  __syncthreads();
  if (CL > 1) asm volatile("barrier.cluster.wait.aligned;" ::: "memory");
  if (wid == 0) {
    ms = warp_merge_ms(lane < (int)blockDim.x / 32 ? red[lane] : make_float2(-INFINITY, 0.f));
    if (CL == 1) { if (lane == 0) part[0] = ms; }
    else if (lane < CL) {
      const uint32_t a = mapa_u32(smem_u32(&part[rank]), lane);
      asm volatile("st.shared::cluster.v2.f32 [%0], {%1, %2};" ::"r"(a), "f"(ms.x), "f"(ms.y) : "memory");
    }
  }
  if (CL > 1) cluster_sync_all(); else __syncthreads();
  ms = part[0];
#pragma unroll
  for (int j = 1; j < CL; ++j) ms = merge_ms(ms, part[j]);
  const float inv = 1.f / ms.y;
  for (int i = c0 + tid; i < c1; i += blockDim.x) out[(size_t)row * V + i] = expf(to_f<T>(g[i]) * inv_temp - ms.x) * inv;
}
constexpr int SM_CLUSTER_ROWS = 64;
template <typename T>
int softmax_rows_launch(float* out, const void* inp, int rows, int V, int ld, float inv_temp, cudaStream_t st) {
  if (rows >= SM_CLUSTER_ROWS) {
    return launch_pdl(softmax_rows_kernel<T, 1>, rows, 512, 0, st, out, (const T*)inp, V, ld, inv_temp);
  }
  return launch_pdl_cluster(8, softmax_rows_kernel<T, 8>, rows * 8, 512, 0, st, out, (const T*)inp, V, ld, inv_temp);
}

// dlogits = probs * (dprobs - sum_k dprobs[k] * probs[k]) over the first V columns of a row (one block per row);
// columns V..ld-1 of dlogits are zeroed.  (llmm/softmax.mojo:632, softmax_bwd)
__global__ void softmax_bwd_kernel(float* __restrict__ dlogits, const float* __restrict__ dprobs, const float* __restrict__ probs,
                                   int V, int ld) {
  __shared__ float red[32];
  __shared__ float bc;
  const int row = blockIdx.x, tid = threadIdx.x, lane = tid % 32, wid = tid / 32, nw = blockDim.x / 32;
  const float* dp = dprobs + (size_t)row * ld;
  const float* pr = probs + (size_t)row * ld;
  float dot = 0.f;
  for (int i = tid; i < V; i += blockDim.x) dot = fmaf(dp[i], pr[i], dot);
  dot = warp_sum(dot); if (lane == 0) red[wid] = dot; __syncthreads();
  if (wid == 0) { float t = lane < nw ? red[lane] : 0.f; t = warp_sum(t); if (lane == 0) bc = t; } __syncthreads();
  dot = bc;
  float* out = dlogits + (size_t)row * ld;
  for (int i = tid; i < ld; i += blockDim.x) out[i] = i < V ? pr[i] * (dp[i] - dot) : 0.f;
}

// Unfused cross-entropy over stored probabilities (llmm/crossentropy.mojo:110, :284): loss = -log p[target];
// backward writes only the target slot, dprobs[target] = -dloss / p[target] (the caller zeroes dprobs first).
__global__ void crossentropy_fwd_kernel(float* __restrict__ losses, const float* __restrict__ probs, const int* __restrict__ targets,
                                        int rows, int ld) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < rows) losses[i] = -logf(probs[(size_t)i * ld + targets[i]]);
}
__global__ void crossentropy_bwd_kernel(float* __restrict__ dprobs, const float* __restrict__ dlosses, const float* __restrict__ probs,
                                        const int* __restrict__ targets, int rows, int ld) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < rows) { const size_t o = (size_t)i * ld + targets[i]; dprobs[o] = -dlosses[i] / probs[o]; }
}
}  // namespace

LLMB_API int llmb_softmax_bwd(float* dlogits, const float* dprobs, const float* probs, int rows, int V, int ld, cudaStream_t st) {
  if (rows <= 0 || V <= 0 || ld < V) return LLMB_ERR_BAD_ARG;
  softmax_bwd_kernel<<<rows, 256, 0, st>>>(dlogits, dprobs, probs, V, ld);
  return (int)cudaGetLastError();
}
LLMB_API int llmb_crossentropy_fwd(float* losses, const float* probs, const int* targets, int rows, int ld, cudaStream_t st) {
  if (rows <= 0) return LLMB_ERR_BAD_ARG;
  crossentropy_fwd_kernel<<<ceil_div(rows, 256), 256, 0, st>>>(losses, probs, targets, rows, ld);
  return (int)cudaGetLastError();
}
LLMB_API int llmb_crossentropy_bwd(float* dprobs, const float* dlosses, const float* probs, const int* targets, int rows, int ld,
                                   cudaStream_t st) {
  if (rows <= 0) return LLMB_ERR_BAD_ARG;
  crossentropy_bwd_kernel<<<ceil_div(rows, 256), 256, 0, st>>>(dprobs, dlosses, probs, targets, rows, ld);
  return (int)cudaGetLastError();
}

LLMB_BOUNDS_REPORT_FN(llmb_bounds_report_classifier)

// logits [rows, Vp] are overwritten with dlogits when write_dlogits != 0.
LLMB_API int llmb_fused_classifier(void* logits, float* losses, const int* targets, float dloss, int rows, int V,
                                   int Vp, int write_dlogits, int dtype, int* status, cudaStream_t st) {
  if (dtype == LLMB_BF16) {
    if (Vp % 8) return LLMB_ERR_BAD_ARG;
    static int stream_on = -1;
    if (stream_on < 0) { const char* e = getenv("LLMB_CLASSIFIER_STREAM"); stream_on = (e && e[0] == '0') ? 0 : (e && e[0] == '2') ? 2 : 1; }
    const int buf_bytes = (Vp * 2 + 127) & ~127;
    if (stream_on && status && 2 * buf_bytes <= 224 * 1024 && (reinterpret_cast<uintptr_t>(logits) & 15) == 0) {
      const int grid = rows < sm_count() ? rows : sm_count();
      if (stream_on == 2) {                               // LLMB_CLASSIFIER_STREAM=2: row traffic on thread 0 of the compute block
        cudaFuncSetAttribute(classifier_stream_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 2 * buf_bytes);
        launch_pdl(classifier_stream_kernel, grid, 1024, 2 * buf_bytes, st, (__nv_bfloat16*)logits, losses, targets, dloss, rows, V, Vp,
                                                                   write_dlogits, buf_bytes, status);
      } else {
        auto kern = Vp <= 7 * 992 * 8 ? classifier_stream2_kernel<7> : classifier_stream2_kernel<8>;      // two buffers fit up to Vp = 57344
        cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 2 * buf_bytes);
        launch_pdl(kern, grid, 1024, 2 * buf_bytes, st, (__nv_bfloat16*)logits, losses, targets, dloss, rows, V, Vp,
                                                                    write_dlogits, buf_bytes, status);
      }
      return (int)cudaGetLastError();
    }
    size_t smem = (size_t)Vp * 2;
    if (smem > 200 * 1024) return LLMB_ERR_BAD_ARG;
    cudaFuncSetAttribute(classifier_kernel<__nv_bfloat16>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    launch_pdl(classifier_kernel<__nv_bfloat16>, rows, 1024, smem, st, (__nv_bfloat16*)logits, losses, targets, dloss, V, Vp, write_dlogits);
  } else {
    if (Vp % 4) return LLMB_ERR_BAD_ARG;
    size_t smem = (size_t)Vp * 4;
    if (smem > 220 * 1024) return LLMB_ERR_BAD_ARG;
    cudaFuncSetAttribute(classifier_kernel<float>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    launch_pdl(classifier_kernel<float>, rows, 1024, smem, st, (float*)logits, losses, targets, dloss, V, Vp, write_dlogits);
  }
  return (int)cudaGetLastError();
}

LLMB_API int llmb_softmax_rows(float* out, const void* inp, int rows, int V, int ld, float inv_temp, int dtype,
                               cudaStream_t st) {
  return dtype == LLMB_BF16 ? softmax_rows_launch<__nv_bfloat16>(out, inp, rows, V, ld, inv_temp, st)
                            : softmax_rows_launch<float>(out, inp, rows, V, ld, inv_temp, st);
}

// ---------------------------------------------------------------- chunked cross-entropy
// Two-pass online-softmax CE over vocabulary tiles, so the full [rows, Vp] logits never exist
// (llmm/fused_classifier.mojo:503-841).  stats[row] = {running max, running sum-exp, target logit, -}.
namespace {
// One CTA per row; a thread issues up to four 16-byte loads before it uses the first.  Pass 1 keeps a running (max, sum of exponentials)
// per thread, so the tile is read once (the maximum and the exponentials were separate sweeps of 2-byte loads before).  8192 x 12672, us,
// before -> now: bf16 pass 1 219 -> 79, pass 2 205 -> 88; fp32 244 -> 69 and 229 -> 127.  fp32 tiles are bound by memory (6.0 and 6.5 TB/s),
// bf16 ones (2.6 and 4.7 TB/s) by the arithmetic of expf: 58 and 67 us with ex2.approx of a rounded product, which rounds 20 % more of the
// bf16 dlogits to a neighbour of the 64-bit value (logits of scale 4 and 10: 9.9e-5 and 2.4e-4 of them against 8.2e-5 and 2.0e-4).
template <typename T>
__global__ void __launch_bounds__(256) ce_pass1_kernel(float4* __restrict__ stats, const T* __restrict__ tile, const int* __restrict__ targets,
                                                      int ld, int col0, int width, int V, int first) {
  pdl_trigger();
  pdl_wait();
  constexpr int N = Pack<T>::N, U = 4;
  __shared__ float2 red[8];
  const int row = blockIdx.x, tid = threadIdx.x, lane = tid % 32, wid = tid / 32;
  const T* g = tile + (size_t)row * ld;
  const int valid = min(width, V - col0);           // columns of this tile that are real vocabulary
  const int nvec = (reinterpret_cast<uintptr_t>(g) & 15) == 0 && valid > 0 ? valid / N : 0;
  float2 ms = make_float2(-INFINITY, 0.f);
  for (int v0 = tid; v0 < nvec; v0 += 256 * U) {
    uint4 raw[U];
#pragma unroll
    for (int u = 0; u < U; ++u) if (v0 + u * 256 < nvec) raw[u] = *reinterpret_cast<const uint4*>(g + (size_t)(v0 + u * 256) * N);
    float m = ms.x;
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (v0 + u * 256 < nvec) {
        Pack<T> p; p.load(reinterpret_cast<const T*>(&raw[u]));
#pragma unroll
        for (int k = 0; k < N; ++k) m = fmaxf(m, p.v[k]);
      }
    float s = ms.x == m ? ms.y : ms.y * expf(ms.x - m);
    const float m0 = base_ms(m);
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (v0 + u * 256 < nvec) {
        Pack<T> p; p.load(reinterpret_cast<const T*>(&raw[u]));
#pragma unroll
        for (int k = 0; k < N; ++k) s += expf(p.v[k] - m0);
      }
    ms = make_float2(m, s);
  }
  for (int i = nvec * N + tid; i < valid; i += 256) ms = merge_ms(ms, single_ms(to_f<T>(g[i])));
  ms = warp_merge_ms(ms);
  if (lane == 0) red[wid] = ms;
  __syncthreads();
  if (wid == 0) {
    ms = warp_merge_ms(lane < 8 ? red[lane] : make_float2(-INFINITY, 0.f));
    if (lane == 0) {
      float4 st = first ? make_float4(-INFINITY, 0.f, 0.f, 0.f) : stats[row];
      if (valid > 0) { const float2 n = merge_ms(make_float2(st.x, st.y), ms); st.x = n.x; st.y = n.y; }
      const int tgt = targets[row];
      if (tgt >= col0 && tgt < col0 + valid) st.z = to_f<T>(g[tgt - col0]);
      stats[row] = st;
    }
  }
}
__global__ void ce_loss_kernel(float* __restrict__ losses, const float4* __restrict__ stats, int rows) {
  pdl_trigger();
  pdl_wait();
  int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r < rows) { float4 st = stats[r]; losses[r] = -(st.z - st.x - logf(st.y)); }
}
template <typename T>
__global__ void __launch_bounds__(256) ce_pass2_kernel(T* __restrict__ tile, const float4* __restrict__ stats, const int* __restrict__ targets,
                                                      int ld, int col0, int width, int V, float dloss) {
  pdl_trigger();
  pdl_wait();
  constexpr int N = Pack<T>::N, U = 4;
  const int row = blockIdx.x, tid = threadIdx.x;
  T* g = tile + (size_t)row * ld;
  const float4 st = stats[row];
  const float lse = st.x + logf(st.y);
  const int tgt = targets[row] - col0;
  const int nvec = (reinterpret_cast<uintptr_t>(g) & 15) == 0 ? width / N : 0;
  auto value = [&](float x, int i) { return col0 + i < V ? (expf(x - lse) - (i == tgt ? 1.f : 0.f)) * dloss : 0.f; };
  for (int v0 = tid; v0 < nvec; v0 += 256 * U) {
    uint4 raw[U];
#pragma unroll
    for (int u = 0; u < U; ++u) if (v0 + u * 256 < nvec) raw[u] = *reinterpret_cast<const uint4*>(g + (size_t)(v0 + u * 256) * N);
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int v = v0 + u * 256;
      if (v < nvec) {
        Pack<T> p; p.load(reinterpret_cast<const T*>(&raw[u]));
#pragma unroll
        for (int k = 0; k < N; ++k) p.v[k] = value(p.v[k], v * N + k);
        p.store(g + (size_t)v * N);
      }
    }
  }
  for (int i = nvec * N + tid; i < width; i += 256) g[i] = from_f<T>(value(to_f<T>(g[i]), i));
}
}  // namespace

LLMB_API int llmb_ce_pass1(float* stats, const void* tile, const int* targets, int rows, int ld, int col0, int width, int V,
                           int first, int dtype, cudaStream_t st) {
  if (dtype == LLMB_BF16) launch_pdl(ce_pass1_kernel<__nv_bfloat16>, rows, 256, 0, st, (float4*)stats, (const __nv_bfloat16*)tile, targets, ld, col0, width, V, first);
  else launch_pdl(ce_pass1_kernel<float>, rows, 256, 0, st, (float4*)stats, (const float*)tile, targets, ld, col0, width, V, first);
  return (int)cudaGetLastError();
}
LLMB_API int llmb_ce_loss(float* losses, const float* stats, int rows, cudaStream_t st) {
  launch_pdl(ce_loss_kernel, ceil_div(rows, 256), 256, 0, st, losses, (const float4*)stats, rows);
  return (int)cudaGetLastError();
}
LLMB_API int llmb_ce_pass2(void* tile, const float* stats, const int* targets, int rows, int ld, int col0, int width, int V,
                           float dloss, int dtype, cudaStream_t st) {
  if (dtype == LLMB_BF16) launch_pdl(ce_pass2_kernel<__nv_bfloat16>, rows, 256, 0, st, (__nv_bfloat16*)tile, (const float4*)stats, targets, ld, col0, width, V, dloss);
  else launch_pdl(ce_pass2_kernel<float>, rows, 256, 0, st, (float*)tile, (const float4*)stats, targets, ld, col0, width, V, dloss);
  return (int)cudaGetLastError();
}
