// Row softmax / log-softmax (forward, backward) and fused cross-entropy for sm_100a.
//
// One CTA per row. The row is staged once into shared memory (up to ~200 KB, e.g. a
// 50 304-wide bf16 vocabulary row is 100 KB) so HBM sees one read and one write per element;
// wider rows fall back to re-reading global memory. All statistics are fp32.
//
// The cross-entropy kernel produces the per-row loss and, in the same pass, the gradient
// (softmax - onehot) * scale, optionally in place over the logits. The reference computes
// cross_entropy as log_softmax + one-hot NLL with seven temporaries
// (crates/torsh-nn/src/functional/loss.rs:15-60, crates/torsh-tensor/src/advanced_ops.rs:1045-1090).
#include "common.cuh"
#include "host_util.h"

namespace tb {

constexpr int SM_THREADS = 512;
constexpr int SM_MAX_CACHE_BYTES = 200 * 1024;

template <typename T, bool CACHE>
__device__ __forceinline__ float row_get(const T* g, const T* s, int i) {
  return to_f<T>(CACHE ? s[i] : g[i]);
}

// Loads row into smem (if CACHE) and returns the row maximum over [0, C).
template <typename T, bool CACHE>
__device__ __forceinline__ float load_row_max(const T* __restrict__ xr, T* srow, int C,
                                              float* scratch) {
  constexpr int N = Vec16<T>::N;
  float m = -FLT_MAX;
  const bool vec_ok = ((uintptr_t)xr & 15) == 0;
  const int nvec = vec_ok ? C / N : 0;
  // four 16-byte loads in flight per thread: with one, a 512-thread CTA keeps 8 KB outstanding and two such CTAs per SM
  // cannot cover the memory latency (the kernel then ran at 0.40 of the copy bandwidth)
  int v = threadIdx.x;
  const int bd = blockDim.x;
  for (; v + 3 * bd < nvec; v += 4 * bd) {
    Vec16<T> t[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) t[u].load(xr + (size_t)(v + u * bd) * N);
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      if (CACHE) t[u].store(srow + (v + u * bd) * N);
      float f[N];
      t[u].get(f);
#pragma unroll
      for (int j = 0; j < N; ++j) m = fmaxf(m, f[j]);
    }
  }
  for (; v < nvec; v += bd) {
    Vec16<T> t;
    t.load(xr + (size_t)v * N);
    if (CACHE) t.store(srow + v * N);
    float f[N];
    t.get(f);
#pragma unroll
    for (int j = 0; j < N; ++j) m = fmaxf(m, f[j]);
  }
  for (int i = nvec * N + threadIdx.x; i < C; i += blockDim.x) {
    T e = xr[i];
    if (CACHE) srow[i] = e;
    m = fmaxf(m, to_f<T>(e));
  }
  m = block_max(m, scratch);  // includes the __syncthreads that publishes srow
  return m;
}

template <typename T, bool CACHE, bool LOG>
__global__ void __launch_bounds__(SM_THREADS)
softmax_fwd_kernel(const T* __restrict__ x, T* __restrict__ y, int rows, int C, long ldx, long ldy) {
  extern __shared__ __align__(16) uint8_t smem_raw[];
  __shared__ float scratch[32];
  T* srow = reinterpret_cast<T*>(smem_raw);
  for (int row = blockIdx.x; row < rows; row += gridDim.x) {
    const T* xr = x + (size_t)row * ldx;
    T* yr = y + (size_t)row * ldy;
    float m = load_row_max<T, CACHE>(xr, srow, C, scratch);
    float s = 0.f;
    for (int i = threadIdx.x; i < C; i += blockDim.x) s += __expf(row_get<T, CACHE>(xr, srow, i) - m);
    s = block_sum(s, scratch);
    const float lse = m + __logf(s);
    const float inv = 1.f / s;
    for (int i = threadIdx.x; i < C; i += blockDim.x) {
      float v = row_get<T, CACHE>(xr, srow, i);
      yr[i] = from_f<T>(LOG ? (v - lse) : __expf(v - m) * inv);
    }
    __syncthreads();
  }
}

// softmax:      dx = y * (dy - sum(dy * y));  log_softmax: dx = dy - exp(y) * sum(dy)
template <typename T, bool LOG>
__global__ void __launch_bounds__(SM_THREADS)
softmax_bwd_kernel(const T* __restrict__ dy, const T* __restrict__ y, T* __restrict__ dx, int rows,
                   int C) {
  __shared__ float scratch[32];
  for (int row = blockIdx.x; row < rows; row += gridDim.x) {
    const T* dyr = dy + (size_t)row * C;
    const T* yr = y + (size_t)row * C;
    float s = 0.f;
    for (int i = threadIdx.x; i < C; i += blockDim.x)
      s += LOG ? to_f<T>(dyr[i]) : to_f<T>(dyr[i]) * to_f<T>(yr[i]);
    s = block_sum(s, scratch);
    for (int i = threadIdx.x; i < C; i += blockDim.x) {
      float d = to_f<T>(dyr[i]), yy = to_f<T>(yr[i]);
      dx[(size_t)row * C + i] = from_f<T>(LOG ? (d - __expf(yy) * s) : yy * (d - s));
    }
  }
}

// Fused cross-entropy. logits [rows, ld] with C valid classes (columns C..ld-1 are padding and get
// zero gradient). loss_rows[row] = lse - logit[target] (0 for ignored rows). When dlogits != null
// it receives (softmax - onehot) * scale, `scale` typically 1 / number_of_counted_rows.
template <typename T, bool CACHE>
__global__ void __launch_bounds__(SM_THREADS)
xent_kernel(const T* __restrict__ logits, const long* __restrict__ targets,
            float* __restrict__ loss_rows, float* __restrict__ lse_rows, T* __restrict__ dlogits,
            int rows, int C, long ld, float scale, long ignore_index) {
  extern __shared__ __align__(16) uint8_t smem_raw[];
  __shared__ float scratch[32];
  T* srow = reinterpret_cast<T*>(smem_raw);
  constexpr int N = Vec16<T>::N;
  for (int row = blockIdx.x; row < rows; row += gridDim.x) {
    const T* xr = logits + (size_t)row * ld;
    const long tgt = targets[row];
    const bool ignored = (tgt == ignore_index) || tgt < 0 || tgt >= C;
    if (ignored && tgt != ignore_index && threadIdx.x == 0) report_bad_index();   // a target outside [0, C) that is not the ignore value
    float m = load_row_max<T, CACHE>(xr, srow, C, scratch);
    float s = 0.f;
    {
      // the staged row is read back 16 bytes at a time (the row start is 16-byte aligned in shared memory)
      const int nv = CACHE ? C / N : 0;
      for (int v = threadIdx.x; v < nv; v += blockDim.x) {
        Vec16<T> t;
        t.load(srow + v * N);
        float f[N];
        t.get(f);
#pragma unroll
        for (int j = 0; j < N; ++j) s += __expf(f[j] - m);
      }
      for (int i = nv * N + threadIdx.x; i < C; i += blockDim.x) s += __expf(row_get<T, CACHE>(xr, srow, i) - m);
    }
    s = block_sum(s, scratch);
    const float lse = m + __logf(s);
    if (threadIdx.x == 0) {
      float xt = ignored ? lse : row_get<T, CACHE>(xr, srow, (int)tgt);
      loss_rows[row] = lse - xt;
      if (lse_rows) lse_rows[row] = lse;
    }
    if (!CACHE) __syncthreads();  // the target logit is read before an in-place gradient overwrites it
    if (dlogits) {
      T* dr = dlogits + (size_t)row * ld;
      const float sc = ignored ? 0.f : scale;
      const bool vec_ok = (((uintptr_t)dr & 15) == 0) && CACHE;
      const int nvec = vec_ok ? (int)(ld / N) : 0;
      for (int v = threadIdx.x; v < nvec; v += blockDim.x) {
        float o[N];
#pragma unroll
        for (int j = 0; j < N; ++j) {
          int i = v * N + j;
          float p = (i < C) ? __expf(to_f<T>(srow[i]) - lse) : 0.f;
          if (i == tgt) p -= 1.f;
          o[j] = p * sc;
        }
        Vec16<T> t;
        t.set(o);
        t.store(dr + v * N);
      }
      for (int i = nvec * N + threadIdx.x; i < ld; i += blockDim.x) {
        float p = (i < C) ? __expf(row_get<T, CACHE>(xr, srow, i) - lse) : 0.f;
        if (i == tgt) p -= 1.f;
        dr[i] = from_f<T>(p * sc);
      }
    }
    __syncthreads();
  }
}

// The same for rows of which two fit into shared memory (up to 55 296 bf16 or 27 648 fp32 columns): every thread copies its
// own vectors of the next row (cp.async, no barrier) while it works on the current one, the row maximum and the exponent sum
// meet in ONE block reduction of (maximum, sum) pairs, and nothing but the target's logit is re-read. Staging, sum and gradient of a row one after
// the other, with two CTAs per SM to overlap them, took 242 us at 4096 x 50 304 bf16; this takes 178, against 126 us for
// reading and writing the matrix at the copy rate and about 92 us of exponentials on the special-function units.
__device__ __forceinline__ void xent_cp_async16(void* smem, const void* g) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(smem)), "l"(g) : "memory");
}
__device__ __forceinline__ float2 exp_of_diff(float2 f, float2 minus_m) {   // __expf(f - m), two at a time
  const float2 t = __fmul2_rn(__fadd2_rn(f, minus_m), make_float2(1.4426950408889634f, 1.4426950408889634f));
  return make_float2(exp2f(t.x), exp2f(t.y));
}

// One element, loaded where it stands in the program: a plain load may be moved past a barrier.
__device__ __forceinline__ float load_now(const float* p) { return *(const volatile float*)p; }
__device__ __forceinline__ float load_now(const bf16* p) { return __uint_as_float((uint32_t) * (const volatile unsigned short*)p << 16); }

// dlogits may be logits, so neither is __restrict__: what is read of a row is read before the barrier behind which it is overwritten.
template <typename T, int THREADS>
__global__ void __launch_bounds__(THREADS) xent_ring_kernel(const T* logits, const long* __restrict__ targets,
                                                            float* __restrict__ loss_rows, float* __restrict__ lse_rows,
                                                            T* dlogits, int rows, int C, long ld, float scale,
                                                            long ignore_index) {
  constexpr int N = Vec16<T>::N;
  extern __shared__ __align__(16) uint8_t smem_raw[];
  __shared__ float2 red[2][32];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int nvec = (C + N - 1) / N, nld = (int)(ld / N);   // vectors with valid columns, vectors of the whole row
  auto buf = [&](int b) { return reinterpret_cast<T*>(smem_raw) + (size_t)b * nvec * N; };
  auto request = [&](int row, int b) {
    if (row < rows) {
      const T* xr = logits + (size_t)row * ld;
      for (int v = tid; v < nvec; v += THREADS) xent_cp_async16(buf(b) + v * N, xr + (size_t)v * N);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  request(blockIdx.x, 0);
  int b = 0;
  for (int row = blockIdx.x; row < rows; row += gridDim.x, b ^= 1) {
    request(row + gridDim.x, b ^ 1);
    const long tgt = targets[row];
    const bool ignored = (tgt == ignore_index) || tgt < 0 || tgt >= C;
    if (ignored && tgt != ignore_index && tid == 0) report_bad_index();   // a target outside [0, C) that is not the ignore value
    // the target's logit once more from memory: published from shared memory by the thread that staged it, it cost rows of more
    // than 10 000 columns 5 to 10 %
    const float xt = tid == 0 && !ignored ? load_now(logits + (size_t)row * ld + tgt) : 0.f;
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    const T* srow = buf(b);
    // whole vectors carry no column tests; the last, ragged one is finished by one thread
    const int nfull = C / N;
    const bool tail = nfull < nvec && tid == nfull % THREADS;
    float m = -FLT_MAX;
    for (int v = tid; v < nfull; v += THREADS) {
      Vec16<T> t;
      t.load(srow + v * N);
      float f[N];
      t.get(f);
#pragma unroll
      for (int j = 0; j < N; ++j) m = fmaxf(m, f[j]);
    }
    if (tail)
      for (int i = nfull * N; i < C; ++i) m = fmaxf(m, to_f<T>(srow[i]));
    float2 s2 = make_float2(0.f, 0.f);
    const float2 nm = make_float2(-m, -m);
#pragma unroll 2
    for (int v = tid; v < nfull; v += THREADS) {
      Vec16<T> t;
      t.load(srow + v * N);
      float f[N];
      t.get(f);
#pragma unroll
      for (int j = 0; j < N; j += 2) s2 = __fadd2_rn(s2, exp_of_diff(make_float2(f[j], f[j + 1]), nm));
    }
    if (tail)
      for (int i = nfull * N; i < C; ++i) s2.x += __expf(to_f<T>(srow[i]) - m);
    float s = s2.x + s2.y;
    {
      const float mw = warp_max(m);
      s = warp_sum(s * __expf(m - mw));
      if (lane == 0) red[b][warp] = make_float2(mw, s);   // two sets: the next row's sums do not wait for this row's readers
      __syncthreads();
      const float2 e = lane < THREADS / 32 ? red[b][lane] : make_float2(-FLT_MAX, 0.f);
      m = warp_max(e.x);
      s = warp_sum(e.y * __expf(e.x - m));
    }
    const float lse = m + __logf(s);
    if (tid == 0) {
      loss_rows[row] = lse - (ignored ? lse : xt);
      if (lse_rows) lse_rows[row] = lse;
    }
    if (dlogits) {
      T* dr = dlogits + (size_t)row * ld;
      const float sc = ignored ? 0.f : scale;
      const float2 nl = make_float2(-lse, -lse), sc2 = make_float2(sc, sc);
      const int tvec = ignored ? -1 : (int)(tgt / N), tj = (int)(tgt - (long)tvec * N);
#pragma unroll 2
      for (int v = tid; v < nfull; v += THREADS) {
        Vec16<T> t;
        t.load(srow + v * N);
        float f[N], o[N];
        t.get(f);
#pragma unroll
        for (int j = 0; j < N; j += 2) {
          const float2 pr = exp_of_diff(make_float2(f[j], f[j + 1]), nl);
          o[j] = pr.x;
          o[j + 1] = pr.y;
        }
        if (v == tvec) {
#pragma unroll
          for (int j = 0; j < N; ++j)
            if (j == tj) o[j] -= 1.f;
        }
#pragma unroll
        for (int j = 0; j < N; j += 2) {
          const float2 pr = __fmul2_rn(make_float2(o[j], o[j + 1]), sc2);
          o[j] = pr.x;
          o[j + 1] = pr.y;
        }
        t.set(o);
        t.store(dr + (size_t)v * N);
      }
      // the ragged vector (staged by its thread) and the padding
      for (int v = nfull + (tid - nfull % THREADS + THREADS) % THREADS; v < nld; v += THREADS) {
        float o[N];
#pragma unroll
        for (int j = 0; j < N; ++j) {
          const int i = v * N + j;
          o[j] = i < C ? (__expf(to_f<T>(srow[i]) - lse) - (v == tvec && j == tj ? 1.f : 0.f)) * sc : 0.f;
        }
        Vec16<T> t;
        t.set(o);
        t.store(dr + (size_t)v * N);
      }
    }
  }
}

// One cluster: valid = max(1, rows that are not ignored); loss = sum of the row losses * factor, or / valid when `mean`. The CTAs'
// sums meet in rank order in the first CTA's registers, read through distributed shared memory.
__global__ void __launch_bounds__(1024) xent_mean_kernel(const float* __restrict__ loss_rows, const long* __restrict__ targets,
                                                         int rows, long ignore_index, int mean, float factor,
                                                         float* __restrict__ loss, float* __restrict__ valid) {
  __shared__ float scratch[32];
  __shared__ float2 part;
  float s = 0.f, n = 0.f;
#pragma unroll 4
  for (long i = blockIdx.x * 1024 + threadIdx.x; i < rows; i += gridDim.x * 1024) {
    s += loss_rows[i];
    n += targets[i] != ignore_index ? 1.f : 0.f;
  }
  s = block_sum(s, scratch);
  n = block_sum(n, scratch);
  if (gridDim.x > 1) {   // the grid is one cluster
    if (threadIdx.x == 0) part = make_float2(s, n);
    asm volatile("barrier.cluster.arrive.release.aligned;\n barrier.cluster.wait.acquire.aligned;" ::: "memory");
    if (blockIdx.x == 0 && threadIdx.x == 0) {
      s = n = 0.f;
      for (unsigned r = 0; r < gridDim.x; ++r) {
        float2 v;
        asm volatile("{\n .reg .b32 a;\n mapa.shared::cluster.u32 a, %2, %3;\n ld.shared::cluster.v2.f32 {%0, %1}, [a];\n}"
                     : "=f"(v.x), "=f"(v.y)
                     : "r"((uint32_t)__cvta_generic_to_shared(&part)), "r"(r)
                     : "memory");
        s += v.x;
        n += v.y;
      }
    }
    // no CTA leaves while its sums may still be read
    asm volatile("barrier.cluster.arrive.release.aligned;\n barrier.cluster.wait.acquire.aligned;" ::: "memory");
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    n = fmaxf(n, 1.f);
    *valid = n;
    *loss = mean ? s / n : s * factor;
  }
}

template <typename K>
static int set_smem(K kern, size_t bytes) {
  if (bytes > 48 * 1024) TB_CUDA_CHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
  return 0;
}

template <typename T>
static int softmax_fwd_launch(const void* x, void* y, int rows, int C, long ldx, long ldy, int log,
                              cudaStream_t st) {
  size_t bytes = (size_t)C * sizeof(T);
  bool cache = bytes <= SM_MAX_CACHE_BYTES;
  int grid = rows < sm_count() * 4 ? rows : sm_count() * 4;
  int threads = C >= 4096 ? SM_THREADS : (C >= 1024 ? 256 : 128);
  size_t smem = cache ? ((bytes + 15) / 16 * 16) : 0;
#define TB_SF(CACHE_, LOG_)                                                                        \
  {                                                                                                \
    auto k = softmax_fwd_kernel<T, CACHE_, LOG_>;                                                  \
    if (int r = set_smem(k, smem)) return r;                                                       \
    k<<<grid, threads, smem, st>>>((const T*)x, (T*)y, rows, C, ldx, ldy);                         \
  }
  if (cache) { if (log) TB_SF(true, true) else TB_SF(true, false) }
  else { if (log) TB_SF(false, true) else TB_SF(false, false) }
#undef TB_SF
  TB_CUDA_CHECK(cudaGetLastError());
  return 0;
}

template <typename T>
static int xent_launch(const void* logits, const long* targets, float* loss_rows, float* lse_rows,
                       void* dlogits, int rows, int C, long ld, float scale, long ignore_index,
                       cudaStream_t st) {
  size_t bytes = (size_t)C * sizeof(T);
  const size_t ring = 2 * ((bytes + 15) / 16 * 16);
  const bool aligned = !((uintptr_t)logits & 15) && !((uintptr_t)dlogits & 15) && (ld * sizeof(T)) % 16 == 0;
  if (aligned && ring <= 216 * 1024) {
    // about six vectors a thread; as many CTAs per SM as threads (2048) and shared memory (216 KB) allow
    const int nvec = (int)(bytes / 16), th = nvec >= 3072 ? 1024 : nvec >= 768 ? 512 : nvec >= 192 ? 256 : 128;
    const int fit = (int)((size_t)216 * 1024 / (ring + 1024)), by_thr = 2048 / th;
    const int per_sm = fit < 1 ? 1 : fit < by_thr ? fit : by_thr;
    const int grid = rows < sm_count() * per_sm ? rows : sm_count() * per_sm;
#define TB_XR(TH_)                                                                                                             \
  {                                                                                                                            \
    auto k = xent_ring_kernel<T, TH_>;                                                                                         \
    if (int r = set_smem(k, ring)) return r;                                                                                   \
    k<<<grid, TH_, ring, st>>>((const T*)logits, targets, loss_rows, lse_rows, (T*)dlogits, rows, C, ld, scale, ignore_index); \
  }
    if (th == 1024) TB_XR(1024) else if (th == 512) TB_XR(512) else if (th == 256) TB_XR(256) else TB_XR(128)
#undef TB_XR
    TB_CUDA_CHECK(cudaGetLastError());
    return 0;
  }
  bool cache = bytes <= SM_MAX_CACHE_BYTES;
  int grid = rows < sm_count() * 4 ? rows : sm_count() * 4;
  int threads = C >= 4096 ? SM_THREADS : (C >= 1024 ? 256 : 128);
  size_t smem = cache ? ((bytes + 15) / 16 * 16) : 0;
  if (cache) {
    auto k = xent_kernel<T, true>;
    if (int r = set_smem(k, smem)) return r;
    k<<<grid, threads, smem, st>>>((const T*)logits, targets, loss_rows, lse_rows, (T*)dlogits, rows, C, ld, scale, ignore_index);
  } else {
    auto k = xent_kernel<T, false>;
    k<<<grid, threads, 0, st>>>((const T*)logits, targets, loss_rows, lse_rows, (T*)dlogits, rows, C, ld, scale, ignore_index);
  }
  TB_CUDA_CHECK(cudaGetLastError());
  return 0;
}

}  // namespace tb
using namespace tb;

// dtype: 0 = bf16, 1 = fp32. ldx / ldy are row strides in elements.
TB_EXPORT int tb_softmax_fwd(const void* x, void* y, int rows, int C, long ldx, long ldy, int log,
                             int dtype, cudaStream_t st) {
  TB_ENSURE_DEVICE();
  if (rows <= 0 || C <= 0) return 0;
  return dtype == 0 ? softmax_fwd_launch<bf16>(x, y, rows, C, ldx, ldy, log, st)
                    : softmax_fwd_launch<float>(x, y, rows, C, ldx, ldy, log, st);
}

TB_EXPORT int tb_softmax_bwd(const void* dy, const void* y, void* dx, int rows, int C, int log,
                             int dtype, cudaStream_t st) {
  TB_ENSURE_DEVICE();
  if (rows <= 0 || C <= 0) return 0;
  int grid = rows < sm_count() * 8 ? rows : sm_count() * 8;
  int threads = C >= 4096 ? SM_THREADS : (C >= 1024 ? 256 : 128);
  if (dtype == 0) {
    if (log) softmax_bwd_kernel<bf16, true><<<grid, threads, 0, st>>>((const bf16*)dy, (const bf16*)y, (bf16*)dx, rows, C);
    else softmax_bwd_kernel<bf16, false><<<grid, threads, 0, st>>>((const bf16*)dy, (const bf16*)y, (bf16*)dx, rows, C);
  } else {
    if (log) softmax_bwd_kernel<float, true><<<grid, threads, 0, st>>>((const float*)dy, (const float*)y, (float*)dx, rows, C);
    else softmax_bwd_kernel<float, false><<<grid, threads, 0, st>>>((const float*)dy, (const float*)y, (float*)dx, rows, C);
  }
  TB_CUDA_CHECK(cudaGetLastError());
  return 0;
}

// Fused cross-entropy forward (+ backward when dlogits != null; dlogits may alias logits).
TB_EXPORT int tb_cross_entropy(const void* logits, const long* targets, float* loss_rows,
                               float* lse_rows, void* dlogits, int rows, int C, long ld, float scale,
                               long ignore_index, int dtype, cudaStream_t st) {
  TB_ENSURE_DEVICE();
  if (rows <= 0 || C <= 0) return 0;
  if (ld < C) TB_FAIL(TB_E_ARG, "tb_cross_entropy: ld (%ld) < C (%d)", ld, C);
  return dtype == 0 ? xent_launch<bf16>(logits, targets, loss_rows, lse_rows, dlogits, rows, C, ld, scale, ignore_index, st)
                    : xent_launch<float>(logits, targets, loss_rows, lse_rows, dlogits, rows, C, ld, scale, ignore_index, st);
}

// loss = mean of the row losses over the rows that are not ignored, or (mean = 0) their sum times factor; valid = the number of
// those rows, at least 1.
TB_EXPORT int tb_cross_entropy_mean(const float* loss_rows, const long* targets, int rows, long ignore_index, int mean,
                                    float factor, float* loss, float* valid, cudaStream_t st) {
  TB_ENSURE_DEVICE();
  // One SM takes in about 200 GB/s of the 12 bytes a row: eight as soon as that saves more than starting a cluster costs (one CTA
  // and eight: 16 384 rows 3.2 and 3.8 us, 65 536 5.9 and 4.0, 1 000 000 58 and 12).
  if (rows < 0) rows = 0;
  if (rows < 32768) {
    xent_mean_kernel<<<1, 1024, 0, st>>>(loss_rows, targets, rows, ignore_index, mean, factor, loss, valid);
  } else {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(8);
    cfg.blockDim = dim3(1024);
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 8;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    TB_CUDA_CHECK(cudaLaunchKernelEx(&cfg, xent_mean_kernel, loss_rows, targets, rows, ignore_index, mean, factor, loss, valid));
  }
  TB_CUDA_CHECK(cudaGetLastError());
  return 0;
}

int tb_set_check_word_xent(int* word) {
  TB_CUDA_CHECK(tb::set_check_word_this_tu(word));
  return 0;
}
