// LayerNorm and RMSNorm forward / backward for sm_100a.
//
// Every element is read from HBM exactly once per pass and the row statistics are a mean and then a centred variance, for
// accuracy. Rows of up to 256 vectors of 16 bytes are a warp each in the forward, wider ones a CTA. The backward gives rows of up
// to 8192 elements to teams of warps that copy them ahead through a ring in shared memory, wider ones to a CTA; both keep fp32
// partial sums of d(gamma) / d(beta) in registers over all their rows and leave one partial row per CTA, which a second kernel
// adds up (atomics only where the caller gives no workspace).
//
// Semantics follow the reference layers: LayerNorm eps 1e-5 (biased variance) and
// RMSNorm y = x / sqrt(mean(x^2) + eps) * w with eps 1e-6
// (crates/torsh-nn/src/layers/normalization/layer_group/mod.rs:491-514,539-623).
#include "common.cuh"
#include "host_util.h"

namespace tb {

template <typename T, int VPT, bool RMS>
__global__ void norm_fwd_kernel(const T* __restrict__ x, const T* __restrict__ gamma,
                                const T* __restrict__ beta, T* __restrict__ y,
                                float* __restrict__ mean_out, float* __restrict__ rstd_out, int rows,
                                int H, float eps) {
  constexpr int N = Vec16<T>::N;
  __shared__ float scratch[32];
  const int nvec = H / N;
  Vec16<T> g[VPT], b[VPT];
#pragma unroll
  for (int i = 0; i < VPT; ++i) {
    int v = threadIdx.x + i * blockDim.x;
    if (v < nvec) {
      g[i].load_nc(gamma + v * N);
      if (!RMS && beta) b[i].load_nc(beta + v * N);
    }
  }
  // the next row's vectors are requested before this row's reductions, so their latency hides behind the block sums
  Vec16<T> nxt[VPT];
  if ((int)blockIdx.x < rows) {
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
      int v = threadIdx.x + i * blockDim.x;
      if (v < nvec) nxt[i].load(x + (size_t)blockIdx.x * H + v * N);
    }
  }
  for (int row = blockIdx.x; row < rows; row += gridDim.x) {
    float f[VPT][N];
    float s = 0.f;
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
      int v = threadIdx.x + i * blockDim.x;
      if (v < nvec) {
        nxt[i].get(f[i]);
#pragma unroll
        for (int j = 0; j < N; ++j) s += RMS ? f[i][j] * f[i][j] : f[i][j];
      }
    }
    if (row + (int)gridDim.x < rows) {
#pragma unroll
      for (int i = 0; i < VPT; ++i) {
        int v = threadIdx.x + i * blockDim.x;
        if (v < nvec) nxt[i].load(x + (size_t)(row + gridDim.x) * H + v * N);
      }
    }
    float mean = 0.f, rstd;
    if (RMS) {
      float ms = block_sum(s, scratch) / H;
      rstd = rsqrtf(ms + eps);
    } else {
      mean = block_sum(s, scratch) / H;
      float sq = 0.f;
#pragma unroll
      for (int i = 0; i < VPT; ++i) {
        int v = threadIdx.x + i * blockDim.x;
        if (v < nvec) {
#pragma unroll
          for (int j = 0; j < N; ++j) {
            float d = f[i][j] - mean;
            sq += d * d;
          }
        }
      }
      float var = block_sum(sq, scratch) / H;
      rstd = rsqrtf(var + eps);
    }
    if (threadIdx.x == 0) {
      if (mean_out) mean_out[row] = mean;
      if (rstd_out) rstd_out[row] = rstd;
    }
    T* yr = y + (size_t)row * H;
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
      int v = threadIdx.x + i * blockDim.x;
      if (v < nvec) {
        float gf[N], bf[N], o[N];
        g[i].get(gf);
        if (!RMS && beta) b[i].get(bf);
#pragma unroll
        for (int j = 0; j < N; ++j) {
          float xh = (f[i][j] - mean) * rstd;
          o[j] = xh * gf[j] + ((!RMS && beta) ? bf[j] : 0.f);
        }
        Vec16<T> t;
        t.set(o);
        t.store(yr + v * N);
      }
    }
  }
}

// dx = rstd * (dy*g - mean(dy*g) - xhat * mean(dy*g*xhat))      (LayerNorm)
// dx = rstd * (dy*g - xhat * mean(dy*g*xhat))                   (RMSNorm, xhat = x*rstd)
// Optionally dx += dres (gradient arriving through the residual branch).
template <typename T, int VPT, bool RMS>
__global__ void norm_bwd_kernel(const T* __restrict__ dy, const T* __restrict__ x,
                                const T* __restrict__ gamma, const float* __restrict__ mean_in,
                                const float* __restrict__ rstd_in, const T* __restrict__ dres,
                                T* __restrict__ dx, float* __restrict__ dgamma,
                                float* __restrict__ dbeta, float* __restrict__ partial, int rows, int H) {
  constexpr int N = Vec16<T>::N;
  __shared__ float scratch[32];
  const int nvec = H / N;
  float gf[VPT][N], dg[VPT][N], db[VPT][N];
#pragma unroll
  for (int i = 0; i < VPT; ++i) {
    int v = threadIdx.x + i * blockDim.x;
#pragma unroll
    for (int j = 0; j < N; ++j) dg[i][j] = db[i][j] = gf[i][j] = 0.f;
    if (v < nvec) {
      Vec16<T> t;
      t.load_nc(gamma + v * N);
      t.get(gf[i]);
    }
  }
  // the next row's vectors are requested before this row's reductions, so their latency hides behind the block sums
  Vec16<T> nx[VPT], nd[VPT], nr[VPT];
  auto request = [&](int row) {
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
      int v = threadIdx.x + i * blockDim.x;
      if (v < nvec) {
        nx[i].load(x + (size_t)row * H + v * N);
        nd[i].load(dy + (size_t)row * H + v * N);
        if (dres) nr[i].load(dres + (size_t)row * H + v * N);
      }
    }
  };
  if ((int)blockIdx.x < rows) request(blockIdx.x);
  for (int row = blockIdx.x; row < rows; row += gridDim.x) {
    const float mean = RMS ? 0.f : mean_in[row];
    const float rstd = rstd_in[row];
    float xh[VPT][N], dyg[VPT][N], res[VPT][N];
    float s1 = 0.f, s2 = 0.f;
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
      int v = threadIdx.x + i * blockDim.x;
      if (v < nvec) {
        float xf[N], df[N];
        nx[i].get(xf);
        nd[i].get(df);
        if (dres) nr[i].get(res[i]);
#pragma unroll
        for (int j = 0; j < N; ++j) {
          xh[i][j] = (xf[j] - mean) * rstd;
          dyg[i][j] = df[j] * gf[i][j];
          dg[i][j] += df[j] * xh[i][j];
          db[i][j] += df[j];
          s1 += dyg[i][j];
          s2 += dyg[i][j] * xh[i][j];
        }
      }
    }
    if (row + (int)gridDim.x < rows) request(row + gridDim.x);
    if (!RMS) s1 = block_sum(s1, scratch) / H; else s1 = 0.f;
    s2 = block_sum(s2, scratch) / H;
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
      int v = threadIdx.x + i * blockDim.x;
      if (v < nvec) {
        float o[N];
#pragma unroll
        for (int j = 0; j < N; ++j) o[j] = dres ? res[i][j] : 0.f;
#pragma unroll
        for (int j = 0; j < N; ++j) o[j] += rstd * (dyg[i][j] - s1 - xh[i][j] * s2);
        Vec16<T> t;
        t.set(o);
        t.store(dx + (size_t)row * H + v * N);
      }
    }
  }
  // Per-CTA partial sums: written to the workspace (reduced by norm_bwd_reduce_kernel, no atomic
  // contention) or, without a workspace, added straight into the gradient with atomics.
#pragma unroll
  for (int i = 0; i < VPT; ++i) {
    int v = threadIdx.x + i * blockDim.x;
    if (v < nvec) {
      if (partial) {
        float* pg = partial + (size_t)blockIdx.x * 2 * H + v * N;
#pragma unroll
        for (int j = 0; j < N; j += 4) {
          *reinterpret_cast<float4*>(pg + j) = make_float4(dg[i][j], dg[i][j + 1], dg[i][j + 2], dg[i][j + 3]);
          if (!RMS) *reinterpret_cast<float4*>(pg + H + j) = make_float4(db[i][j], db[i][j + 1], db[i][j + 2], db[i][j + 3]);
        }
      } else {
#pragma unroll
        for (int j = 0; j < N; ++j) {
          if (dgamma) atomicAdd(dgamma + v * N + j, dg[i][j]);
          if (!RMS && dbeta) atomicAdd(dbeta + v * N + j, db[i][j]);
        }
      }
    }
  }
}

// ---------------------------------------------------------------------------------------------------------------
// Warp-per-row form of the forward for rows of at most 32 * VPL 16-byte vectors (H <= 2048 bf16, 1024 fp32). A warp owns a row: its
// statistics are two shuffle reductions with no block barrier, eight rows are in flight per CTA and the next row of
// every warp is requested before the current one is reduced. With one CTA per row a 2 KB row left too few bytes in
// flight per SM and two block barriers per row on the critical path (0.43 of the copy bandwidth at 32768 x 1024).
constexpr int NORM_WARPS = 8;

template <typename T, int VPL, bool RMS>
__global__ void __launch_bounds__(NORM_WARPS * 32, VPL <= 4 ? 2 : 1) norm_fwd_warp_kernel(
    const T* __restrict__ x, const T* __restrict__ gamma, const T* __restrict__ beta, T* __restrict__ y,
    float* __restrict__ mean_out, float* __restrict__ rstd_out, int rows, int H, float eps) {
  constexpr int N = Vec16<T>::N;
  const int lane = threadIdx.x & 31;
  const int nvec = H / N;
  const int nwarps = gridDim.x * NORM_WARPS;
  Vec16<T> g[VPL], b[VPL], nxt[VPL];
#pragma unroll
  for (int i = 0; i < VPL; ++i) {
    const int v = lane + 32 * i;
    if (v < nvec) {
      g[i].load_nc(gamma + v * N);
      if (!RMS && beta) b[i].load_nc(beta + v * N);
    }
  }
  int row = blockIdx.x * NORM_WARPS + (threadIdx.x >> 5);
  if (row < rows) {
#pragma unroll
    for (int i = 0; i < VPL; ++i)
      if (lane + 32 * i < nvec) nxt[i].load(x + (size_t)row * H + (lane + 32 * i) * N);
  }
  const float inv_h = 1.f / (float)H;
  for (; row < rows; row += nwarps) {
    float f[VPL][N];
    float s = 0.f;
#pragma unroll
    for (int i = 0; i < VPL; ++i) {
      if (lane + 32 * i < nvec) {
        nxt[i].get(f[i]);
#pragma unroll
        for (int j = 0; j < N; ++j) s += RMS ? f[i][j] * f[i][j] : f[i][j];
      }
    }
    if (row + nwarps < rows) {
#pragma unroll
      for (int i = 0; i < VPL; ++i)
        if (lane + 32 * i < nvec) nxt[i].load(x + (size_t)(row + nwarps) * H + (lane + 32 * i) * N);
    }
    float mean = 0.f, rstd;
    if (RMS) {
      rstd = rsqrtf(warp_sum(s) * inv_h + eps);
    } else {
      mean = warp_sum(s) * inv_h;
      float sq = 0.f;
#pragma unroll
      for (int i = 0; i < VPL; ++i) {
        if (lane + 32 * i < nvec) {
#pragma unroll
          for (int j = 0; j < N; ++j) {
            const float d = f[i][j] - mean;
            sq += d * d;
          }
        }
      }
      rstd = rsqrtf(warp_sum(sq) * inv_h + eps);
    }
    if (lane == 0) {
      if (mean_out) mean_out[row] = mean;
      if (rstd_out) rstd_out[row] = rstd;
    }
    T* yr = y + (size_t)row * H;
#pragma unroll
    for (int i = 0; i < VPL; ++i) {
      const int v = lane + 32 * i;
      if (v < nvec) {
        float gf[N], bf[N], o[N];
        g[i].get(gf);
        if (!RMS && beta) b[i].get(bf);
#pragma unroll
        for (int j = 0; j < N; ++j) {
          o[j] = (f[i][j] - mean) * rstd * gf[j];
          if (!RMS && beta) o[j] += bf[j];
        }
        Vec16<T> t;
        t.set(o);
        t.store(yr + v * N);
      }
    }
  }
}

// Backward for rows of up to 8192 elements: same arithmetic as norm_bwd_kernel. A team of G warps owns a row (16 elements a
// lane, 8 where that leaves fewer lanes idle) and walks rows with the next two or three already on their way: every lane
// copies its own vectors of x, dy and dres into a ring in shared memory (cp.async without a barrier: a lane reads only what it
// copied), and the statistics travel one row ahead. With the next row in registers there was room for 8 warps at 255
// registers, and every row began with a load of its mean: 82 us at 32768 x 1024 bf16, where this form takes 48 (31 at the copy
// rate); 8192 x 1024 with a residual gradient 32.5 -> 18.2, 1999 x 4096 fp32 29.3 -> 18.2, 20000 x 1600 89.6 -> 59.6. d(gamma) / d(beta) partial
// sums stay in registers for all rows of a team, meet in shared memory once and leave as one partial row per CTA.
__device__ __forceinline__ void cp_async16(void* smem, const void* g) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(smem)), "l"(g) : "memory");
}

// ONE: a CTA of a single team, one row per CTA.
template <typename T, int VPL, int NW, bool RMS, bool ONE>
__global__ void __launch_bounds__(NW * 32, 1) norm_bwd_ring_kernel(
    const T* __restrict__ dy, const T* __restrict__ x, const T* __restrict__ gamma, const float* __restrict__ mean_in,
    const float* __restrict__ rstd_in, const T* __restrict__ dres, T* __restrict__ dx, float* __restrict__ dgamma,
    float* __restrict__ dbeta, float* __restrict__ partial, int rows, int H, int G) {
  constexpr int N = Vec16<T>::N;
  extern __shared__ __align__(16) uint8_t nb_smem[];
  __shared__ float2 exch[2][NW];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int teams = ONE ? 1 : NW / G, team = ONE ? 0 : warp / G, member = warp - team * G;
  const int nvec = H / N, narr = dres ? 3 : 2, stages = dres ? 2 : 3;
  const bool active = team < teams;
  const int step = gridDim.x * teams;
  float2 dg[VPL][N / 2], db[VPL][N / 2];
  Vec16<T> gv[VPL];
#pragma unroll
  for (int i = 0; i < VPL; ++i) {
    const int v = member * 32 + lane + i * 32 * G;
#pragma unroll
    for (int j = 0; j < N / 2; ++j) dg[i][j] = db[i][j] = make_float2(0.f, 0.f);
    if (active && v < nvec) gv[i].load_nc(gamma + v * N);
    else gv[i].raw = make_uint4(0, 0, 0, 0);
  }
  auto slot = [&](int stage, int arr, int i) {
    return nb_smem + ((((size_t)stage * NW + warp) * narr + arr) * VPL + i) * 512 + lane * 16;
  };
  auto request = [&](int row, int stage) {
    if (row < rows) {
#pragma unroll
      for (int i = 0; i < VPL; ++i) {
        const int v = member * 32 + lane + i * 32 * G;
        if (v < nvec) {
          const size_t at = (size_t)row * H + v * N;
          cp_async16(slot(stage, 0, i), x + at);
          cp_async16(slot(stage, 1, i), dy + at);
          if (dres) cp_async16(slot(stage, 2, i), dres + at);
        }
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  const float inv_h = 1.f / (float)H;
  if (active) {
    int row = blockIdx.x * teams + team;
    for (int k = 0; k < stages; ++k) request(row + k * step, k);
    int stage = 0, par = 0;
    // the next row's statistics travel one row ahead, too: read when needed they put a memory latency into every row
    float mean_next = 0.f, rstd_next = 0.f;
    if (row < rows) {
      if (!RMS) mean_next = mean_in[row];
      rstd_next = rstd_in[row];
    }
    for (; row < rows; row += step) {
      const float mean = mean_next, rstd = rstd_next;
      if (row + step < rows) {
        if (!RMS) mean_next = mean_in[row + step];
        rstd_next = rstd_in[row + step];
      }
      if (dres) asm volatile("cp.async.wait_group 1;" ::: "memory");
      else asm volatile("cp.async.wait_group 2;" ::: "memory");
      // packed two-wide fp32 arithmetic: the row's instructions, not its bytes, were the larger share
      const float2 nm2 = make_float2(-mean, -mean), r2 = make_float2(rstd, rstd);
      float2 s1v = make_float2(0.f, 0.f), s2v = make_float2(0.f, 0.f);
      Vec16<T> xv[VPL], dv[VPL];
#pragma unroll
      for (int i = 0; i < VPL; ++i) {
        if (member * 32 + lane + i * 32 * G < nvec) {
          xv[i].raw = *reinterpret_cast<const uint4*>(slot(stage, 0, i));
          dv[i].raw = *reinterpret_cast<const uint4*>(slot(stage, 1, i));
          float xf[N], df[N], gf[N];
          xv[i].get(xf);
          dv[i].get(df);
          gv[i].get(gf);
#pragma unroll
          for (int j = 0; j < N; j += 2) {
            const float2 d2 = make_float2(df[j], df[j + 1]);
            const float2 xh = __fmul2_rn(__fadd2_rn(make_float2(xf[j], xf[j + 1]), nm2), r2);
            const float2 dyg = __fmul2_rn(d2, make_float2(gf[j], gf[j + 1]));
            dg[i][j / 2] = __ffma2_rn(d2, xh, dg[i][j / 2]);
            if (!RMS) {
              db[i][j / 2] = __fadd2_rn(db[i][j / 2], d2);
              s1v = __fadd2_rn(s1v, dyg);
            }
            s2v = __ffma2_rn(dyg, xh, s2v);
          }
        }
      }
      float s1 = s1v.x + s1v.y, s2 = s2v.x + s2v.y;
      s1 = RMS ? 0.f : warp_sum(s1);
      s2 = warp_sum(s2);
      if (G > 1) {  // the team's warps add their sums in the same order (two buffers: the next row may be ahead)
        if (lane == 0) exch[par][warp] = make_float2(s1, s2);
        asm volatile("bar.sync %0, %1;" ::"r"(1 + team), "r"(G * 32) : "memory");
        s1 = s2 = 0.f;
        for (int m = 0; m < G; ++m) {
          const float2 e = exch[par][team * G + m];
          s1 += e.x;
          s2 += e.y;
        }
        par ^= 1;
      }
      const float2 ns1 = make_float2(-s1 * inv_h, -s1 * inv_h), ns2 = make_float2(-s2 * inv_h, -s2 * inv_h);
#pragma unroll
      for (int i = 0; i < VPL; ++i) {
        const int v = member * 32 + lane + i * 32 * G;
        if (v < nvec) {
          float xf[N], df[N], gf[N], o[N];
          xv[i].get(xf);
          dv[i].get(df);
          gv[i].get(gf);
          if (dres) {
            Vec16<T> r;
            r.raw = *reinterpret_cast<const uint4*>(slot(stage, 2, i));
            r.get(o);
          } else {
#pragma unroll
            for (int j = 0; j < N; ++j) o[j] = 0.f;
          }
#pragma unroll
          for (int j = 0; j < N; j += 2) {
            const float2 xh = __fmul2_rn(__fadd2_rn(make_float2(xf[j], xf[j + 1]), nm2), r2);
            float2 t2 = __ffma2_rn(make_float2(df[j], df[j + 1]), make_float2(gf[j], gf[j + 1]), ns1);
            t2 = __ffma2_rn(xh, ns2, t2);
            t2 = __ffma2_rn(t2, r2, make_float2(o[j], o[j + 1]));
            o[j] = t2.x;
            o[j + 1] = t2.y;
          }
          Vec16<T> t;
          t.set(o);
          t.store(dx + (size_t)row * H + v * N);
        }
      }
      request(row + stages * step, stage);
      if (++stage == stages) stage = 0;
    }
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();
  // every team with a row leaves its column sums in its own [2][H] floats (RMS: [H]) over the ring's memory, which they never
  // exceed, and the CTA adds them in the order of the teams. Taking turns at one [2][H], 8 to 24 barriers, was most of a call
  // with few rows.
  float* sums = reinterpret_cast<float*>(nb_smem);
  const int width = RMS ? H : 2 * H, filled = min(teams, rows - (int)blockIdx.x * teams);
  if (active && team < filled) {
#pragma unroll
    for (int i = 0; i < VPL; ++i) {
      const int v = member * 32 + lane + i * 32 * G;
      if (v < nvec) {
#pragma unroll
        for (int j = 0; j < N; j += 4) {
          float* at = sums + (size_t)team * width + v * N + j;
          *reinterpret_cast<float4*>(at) = make_float4(dg[i][j / 2].x, dg[i][j / 2].y, dg[i][j / 2 + 1].x, dg[i][j / 2 + 1].y);
          if (!RMS)
            *reinterpret_cast<float4*>(at + H) = make_float4(db[i][j / 2].x, db[i][j / 2].y, db[i][j / 2 + 1].x, db[i][j / 2 + 1].y);
        }
      }
    }
  }
  __syncthreads();
  const bool vec = partial && !((uintptr_t)partial & 15);
  for (int c = threadIdx.x * 4; c < width; c += blockDim.x * 4) {
    float4 a = *reinterpret_cast<const float4*>(sums + c);
#pragma unroll 4
    for (int t = 1; t < filled; ++t) {
      const float4 b = *reinterpret_cast<const float4*>(sums + (size_t)t * width + c);
      a.x += b.x; a.y += b.y; a.z += b.z; a.w += b.w;
    }
    if (vec) {
      *reinterpret_cast<float4*>(partial + (size_t)blockIdx.x * 2 * H + c) = a;
      continue;
    }
    const float s[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {   // H is a multiple of 4: the four are all of d(gamma) or all of d(beta)
      if (partial) partial[(size_t)blockIdx.x * 2 * H + c + j] = s[j];
      else if (c < H && dgamma) atomicAdd(dgamma + c + j, s[j]);
      else if (c >= H && dbeta) atomicAdd(dbeta + c - H + j, s[j]);
    }
  }
}

// dgamma[c] (+)= sum_b partial[b][0][c]; dbeta[c] (+)= sum_b partial[b][1][c]. `store`: 0 adds to fp32 buffers, 1 writes fp32,
// 2 writes bf16 (a gradient that starts here needs neither a zeroed buffer nor a cast).
// A CTA owns 32 columns; its 32 x 32 threads split the nblk partial rows 32 ways (coalesced 128-byte reads), then
// the 32 row-groups meet in shared memory. With hundreds of partial rows a one-thread-per-column loop is a chain of
// dependent cache misses (47 us measured for H = 1024); this form takes a few microseconds.
__global__ void __launch_bounds__(1024) norm_bwd_reduce_kernel(const float* __restrict__ partial,
                                                               void* __restrict__ dgamma, void* __restrict__ dbeta,
                                                               int nblk, int H, int store) {
  __shared__ float red[32][33];
  const int c = blockIdx.x * 32 + threadIdx.x;
  const int which = blockIdx.y;  // 0 = gamma, 1 = beta
  void* out = which == 0 ? dgamma : dbeta;
  if (!out) return;
  float s = 0.f;
  if (c < H) {
    const float* p = partial + (size_t)which * H + c;
    for (int b = threadIdx.y; b < nblk; b += 32) s += p[(size_t)b * 2 * H];
  }
  red[threadIdx.y][threadIdx.x] = s;
  __syncthreads();
  if (threadIdx.y == 0 && c < H) {
    float t = 0.f;
#pragma unroll
    for (int y = 0; y < 32; ++y) t += red[y][threadIdx.x];
    if (store == 2) reinterpret_cast<bf16*>(out)[c] = __float2bfloat16(t);
    else if (store == 1) reinterpret_cast<float*>(out)[c] = t;
    else reinterpret_cast<float*>(out)[c] += t;
  }
}

static inline int norm_bwd_grid(int rows) { return rows < sm_count() * 4 ? rows : sm_count() * 4; }

template <typename T, bool RMS>
static int norm_fwd_launch(const void* x, const void* gamma, const void* beta, void* y, float* mean,
                           float* rstd, int rows, int H, float eps, cudaStream_t st) {
  constexpr int N = Vec16<T>::N;
  if (H % N) TB_FAIL(TB_E_ARG, "norm: H=%d must be a multiple of %d", H, N);
  int nvec = H / N;
  if (nvec <= 32 * 8) {
    // resident CTAs only (two per SM up to four vectors per lane, one above): every warp then streams several rows
    // with the next one already requested
    const int want = (rows + NORM_WARPS - 1) / NORM_WARPS;
    const int cap = sm_count() * (nvec <= 128 ? 2 : 1);
    const int wgrid = want < cap ? want : cap;
#define TB_NFW(VPL_)                                                                                                  \
  norm_fwd_warp_kernel<T, VPL_, RMS><<<wgrid, NORM_WARPS * 32, 0, st>>>((const T*)x, (const T*)gamma, (const T*)beta, \
                                                                        (T*)y, mean, rstd, rows, H, eps);
    if (nvec <= 32) TB_NFW(1) else if (nvec <= 64) TB_NFW(2) else if (nvec <= 128) TB_NFW(4) else TB_NFW(8)
#undef TB_NFW
    TB_CUDA_CHECK(cudaGetLastError());
    return 0;
  }
  int grid = rows < sm_count() * 8 ? rows : sm_count() * 8;
#define TB_NF(VPT_)                                                                                 \
  {                                                                                                 \
    int threads = ((nvec + VPT_ - 1) / VPT_ + 31) / 32 * 32;                                        \
    norm_fwd_kernel<T, VPT_, RMS><<<grid, threads, 0, st>>>((const T*)x, (const T*)gamma,           \
                                                             (const T*)beta, (T*)y, mean, rstd,     \
                                                             rows, H, eps);                         \
  }
  if (nvec <= 256) TB_NF(1) else if (nvec <= 1024) TB_NF(2) else if (nvec <= 4096) TB_NF(4) else
    TB_FAIL(TB_E_ARG, "norm: H=%d too large", H);
#undef TB_NF
  TB_CUDA_CHECK(cudaGetLastError());
  return 0;
}

template <typename T, int VPL, int NW, bool RMS>
static int norm_bwd_ring_launch(const void* dy, const void* x, const void* gamma, const float* mean, const float* rstd,
                                const void* dres, void* dx, float* dgamma, float* dbeta, float* partial, int rows, int H, int G,
                                int* used, cudaStream_t st) {
  // No more rows than SMs: a CTA of one team each starts and ends sooner than a few of 16 or 24 warps (LayerNorm 16 x 1024 fp32
  // with gradients that accumulate 8.8 -> 7.8 us, 100 x 1600 fp32 8.4 -> 7.6, 16 x 1600 bf16 9.6 -> 8.7).
  const bool one = rows <= sm_count();
  auto kern = one ? norm_bwd_ring_kernel<T, VPL, NW, RMS, true> : norm_bwd_ring_kernel<T, VPL, NW, RMS, false>;
  const size_t smem = (size_t)(dres ? 2 * 3 : 3 * 2) * NW * VPL * 512;
  // the column sums of the teams take the ring's place: NW / G teams of 2 * H floats, H <= G * VPL * 512 / sizeof(T)
  static_assert(2 * sizeof(float) / sizeof(T) <= 6, "column sums must fit into the ring");
  static std::atomic<uint64_t> in_one{0}, in_many{0};
  if (int r = smem_opt_in(one ? in_one : in_many, kern, 200 * 1024)) return r;
  const int teams = one ? 1 : NW / G, want = (rows + teams - 1) / teams, cap = sm_count();  // never above norm_bwd_grid(rows)
  *used = want < cap ? want : cap;
  kern<<<*used, (one ? G : NW) * 32, smem, st>>>((const T*)dy, (const T*)x, (const T*)gamma, mean, rstd, (const T*)dres, (T*)dx, dgamma,
                                                 dbeta, partial, rows, H, G);
  TB_CUDA_CHECK(cudaGetLastError());
  return 0;
}

template <typename T, bool RMS>
static int norm_bwd_launch(const void* dy, const void* x, const void* gamma, const float* mean,
                           const float* rstd, const void* dres, void* dx, void* dgamma_, void* dbeta_, float* partial, int rows,
                           int H, int store, cudaStream_t st) {
  constexpr int N = Vec16<T>::N;
  if (H % N) TB_FAIL(TB_E_ARG, "norm: H=%d must be a multiple of %d", H, N);
  float *dgamma = (float*)dgamma_, *dbeta = (float*)dbeta_;  // only touched by the kernels when there is no workspace
  int nvec = H / N;
  int grid = norm_bwd_grid(rows);
  if (H <= 8192) {
    // 16 elements a lane and 16 warps, or 8 elements and 24 warps: whichever leaves fewer lanes without a vector
    constexpr int V2 = 16 / N, V1 = 8 / N;
    const int g2 = (nvec + 32 * V2 - 1) / (32 * V2), g1 = (nvec + 32 * V1 - 1) / (32 * V1);
    const bool narrow = g1 <= 3 && g1 * V1 < g2 * V2;
    int used = 0, r;
    if (narrow) r = norm_bwd_ring_launch<T, V1, 24, RMS>(dy, x, gamma, mean, rstd, dres, dx, dgamma, dbeta, partial, rows, H, g1, &used, st);
    else r = norm_bwd_ring_launch<T, V2, 16, RMS>(dy, x, gamma, mean, rstd, dres, dx, dgamma, dbeta, partial, rows, H, g2, &used, st);
    if (r) return r;
    if (partial) {
      dim3 rgrid((H + 31) / 32, RMS ? 1 : 2);
      norm_bwd_reduce_kernel<<<rgrid, dim3(32, 32), 0, st>>>(partial, dgamma_, dbeta_, used, H, store);
    }
    TB_CUDA_CHECK(cudaGetLastError());
    return 0;
  }
#define TB_NB(VPT_)                                                                               \
  {                                                                                               \
    int threads = ((nvec + VPT_ - 1) / VPT_ + 31) / 32 * 32;                                      \
    norm_bwd_kernel<T, VPT_, RMS><<<grid, threads, 0, st>>>((const T*)dy, (const T*)x,            \
                                                             (const T*)gamma, mean, rstd,         \
                                                             (const T*)dres, (T*)dx, dgamma,      \
                                                             dbeta, partial, rows, H);            \
  }
  if (nvec <= 4096) TB_NB(4) else TB_FAIL(TB_E_ARG, "norm: H=%d too large", H);
#undef TB_NB
  if (partial) {
    dim3 rgrid((H + 31) / 32, RMS ? 1 : 2);
    norm_bwd_reduce_kernel<<<rgrid, dim3(32, 32), 0, st>>>(partial, dgamma_, dbeta_, grid, H, store);
  }
  TB_CUDA_CHECK(cudaGetLastError());
  return 0;
}

}  // namespace tb
using namespace tb;

// dtype: 0 = bf16, 1 = fp32. rms: 0 = LayerNorm, 1 = RMSNorm. beta / mean may be null.
TB_EXPORT int tb_norm_fwd(const void* x, const void* gamma, const void* beta, void* y, float* mean,
                          float* rstd, int rows, int H, float eps, int rms, int dtype,
                          cudaStream_t st) {
  TB_ENSURE_DEVICE();
  if (rows <= 0) return 0;
  if (dtype == 0)
    return rms ? norm_fwd_launch<bf16, true>(x, gamma, beta, y, mean, rstd, rows, H, eps, st)
               : norm_fwd_launch<bf16, false>(x, gamma, beta, y, mean, rstd, rows, H, eps, st);
  return rms ? norm_fwd_launch<float, true>(x, gamma, beta, y, mean, rstd, rows, H, eps, st)
             : norm_fwd_launch<float, false>(x, gamma, beta, y, mean, rstd, rows, H, eps, st);
}

// Number of fp32 elements of scratch memory tb_norm_bwd wants for (rows, H).
TB_EXPORT long tb_norm_bwd_workspace(int rows, int H) {
  if (rows <= 0) return 0;
  if (tb::ensure_device()) return 0;
  return (long)norm_bwd_grid(rows) * 2 * H;
}

namespace tb {
static int norm_bwd_dispatch(const void* dy, const void* x, const void* gamma, const float* mean, const float* rstd,
                             const void* dres, void* dx, void* dgamma, void* dbeta, float* partial, int rows, int H, int rms,
                             int dtype, int store, cudaStream_t st) {
  if (dtype == 0)
    return rms ? norm_bwd_launch<bf16, true>(dy, x, gamma, mean, rstd, dres, dx, dgamma, dbeta, partial, rows, H, store, st)
               : norm_bwd_launch<bf16, false>(dy, x, gamma, mean, rstd, dres, dx, dgamma, dbeta, partial, rows, H, store, st);
  return rms ? norm_bwd_launch<float, true>(dy, x, gamma, mean, rstd, dres, dx, dgamma, dbeta, partial, rows, H, store, st)
             : norm_bwd_launch<float, false>(dy, x, gamma, mean, rstd, dres, dx, dgamma, dbeta, partial, rows, H, store, st);
}
}  // namespace tb

// dgamma / dbeta are fp32 buffers that the kernel ACCUMULATES into (zero them for a fresh
// gradient). dres (optional) is added to dx. `partial` is scratch memory of
// tb_norm_bwd_workspace(rows, H) floats holding per-CTA partial sums that a second kernel
// reduces; with partial == null the partial sums are added with atomics instead (slower).
TB_EXPORT int tb_norm_bwd(const void* dy, const void* x, const void* gamma, const float* mean,
                          const float* rstd, const void* dres, void* dx, float* dgamma,
                          float* dbeta, float* partial, int rows, int H, int rms, int dtype,
                          cudaStream_t st) {
  TB_ENSURE_DEVICE();
  if (rows <= 0) return 0;
  return norm_bwd_dispatch(dy, x, gamma, mean, rstd, dres, dx, dgamma, dbeta, partial, rows, H, rms, dtype, 0, st);
}

// The same with dgamma / dbeta WRITTEN in grad_dtype (0 bf16, 1 fp32), rows > 0; the workspace is required.
TB_EXPORT int tb_norm_bwd_store(const void* dy, const void* x, const void* gamma, const float* mean, const float* rstd,
                                const void* dres, void* dx, void* dgamma, void* dbeta, float* partial, int rows, int H, int rms,
                                int dtype, int grad_dtype, cudaStream_t st) {
  TB_ENSURE_DEVICE();
  if (rows <= 0 || !partial) TB_FAIL(TB_E_ARG, "norm_bwd_store: needs rows and a workspace");
  return norm_bwd_dispatch(dy, x, gamma, mean, rstd, dres, dx, dgamma, dbeta, partial, rows, H, rms, dtype, grad_dtype == 0 ? 2 : 1, st);
}

// ---------------------------------------------------------------------------------------------
// Allocation-free variant of tb_norm_bwd (declared in csrc/include/torsh_b200_noalloc.h).
//
// tb_norm_bwd needs scratch memory for its per-CTA partial sums and expects the caller to provide
// it. Some callers cannot: code running inside a CUDA-graph capture or a real-time serving loop must
// not touch an allocator, and a plain C / FFI host has no caching allocator to ask. For them the
// scratch lives in the library image itself, in a file-scope device array of fixed size. Every GPU
// that loads the library holds these 8 MiB until the process exits.
//
// Rules that follow from sharing one array:
//  * the request is refused (TB_E_TOO_LARGE) when it needs more than the array holds;
//  * the array keeps whatever the previous call left in it. Nothing has to start at zero here: every
//    partial-sum row that the reduce kernel reads is fully overwritten by the CTA that owns it;
//  * two calls whose kernels overlap on the GPU (different streams, or graphs replayed concurrently)
//    race on the array. Issue them on one stream, or serialise them with events.
// The first call on a device looks up the array's device address (cudaGetSymbolAddress, with that
// device current) and caches it; make that first call before any stream capture begins.
namespace tb {
constexpr long NOALLOC_SCRATCH_FLOATS = 2L * 1024 * 1024;  // 8 MiB
static __device__ __align__(256) float g_norm_bwd_scratch[NOALLOC_SCRATCH_FLOATS];
// In host code the name above is only a handle for the symbol, never a device address.
static float* g_norm_bwd_scratch_dev[64] = {nullptr};

static int noalloc_scratch_ptr(float** out) {
  int dev = 0;
  TB_CUDA_CHECK(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64) TB_FAIL(TB_E_ARG, "tb_norm_bwd_static: device index %d out of range", dev);
  if (!g_norm_bwd_scratch_dev[dev]) {
    float* p = nullptr;
    TB_CUDA_CHECK(cudaGetSymbolAddress((void**)&p, g_norm_bwd_scratch));
    if (!p) TB_FAIL(TB_E_CUDA, "tb_norm_bwd_static: cudaGetSymbolAddress returned a null address");
    g_norm_bwd_scratch_dev[dev] = p;
  }
  *out = g_norm_bwd_scratch_dev[dev];
  return 0;
}
}  // namespace tb

TB_EXPORT long tb_norm_bwd_static_capacity() { return tb::NOALLOC_SCRATCH_FLOATS; }

TB_EXPORT int tb_norm_bwd_static(const void* dy, const void* x, const void* gamma, const float* mean,
                                 const float* rstd, const void* dres, void* dx, float* dgamma, float* dbeta,
                                 int rows, int H, int rms, int dtype, cudaStream_t st) {
  TB_ENSURE_DEVICE();
  if (rows <= 0) return 0;
  const long need = (long)tb::norm_bwd_grid(rows) * 2 * H;
  if (need > tb::NOALLOC_SCRATCH_FLOATS)
    TB_FAIL(tb::TB_E_TOO_LARGE,
            "tb_norm_bwd_static: rows=%d, H=%d needs %ld floats of scratch, the built-in array holds %ld; "
            "use tb_norm_bwd with caller-provided scratch",
            rows, H, need, tb::NOALLOC_SCRATCH_FLOATS);
  float* scratch = nullptr;
  if (int r = tb::noalloc_scratch_ptr(&scratch)) return r;
  return tb_norm_bwd(dy, x, gamma, mean, rstd, dres, dx, dgamma, dbeta, scratch, rows, H, rms, dtype, st);
}
