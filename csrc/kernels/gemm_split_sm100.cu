// bf16 GEMM for grids that leave the chip idle: D[M,N] = A[M,K] * B[N,K]^T with the contraction split over the CTAs of a
// cluster, which add their partial tiles through distributed shared memory.
//
// What bounds a product of few tiles is how fast one SM can take operands in (about 64 bytes a clock, 0.28 us for the
// 32 KB of a K block), not the tensor core: 512 x 1024 x 4096 has 32 tiles of 128 x 128 and each walked 64 K blocks, 24 us
// on 32 of 148 SMs. A cluster of S CTAs takes one tile, each CTA every K block of its S-th of K, so S times as many
// SMs stream operands. The partial sums stay fp32 all the way: TMEM -> shared memory of the CTA that owns BN / S of the
// tile's columns -> one sum in rank order, so the result does not depend on timing and needs no zeroed fp32 buffer,
// no atomics and no cast pass.
//
// 192 threads, one tile per cluster: warp 0 TMA producer, warp 1 MMA issuer, warps 2..5 epilogue (one TMEM lane quarter
// each). Bias, residual and pre-activation of the owned columns are requested before the accumulator is waited for.
#include <string.h>

#include "gemm_pair.cuh"
#include "host_util.h"
#include "sm100.cuh"

namespace tb {

namespace ksplit {

constexpr int BK = 64;
constexpr int THREADS = 192;
constexpr int STAGES = 5;
constexpr int A_BYTES = 128 * BK * 2;
constexpr int STAGE_BYTES = A_BYTES + 128 * BK * 2;   // B uses BN * 128 bytes of its half
constexpr int RED_OFF = STAGES * STAGE_BYTES;         // partial sums from the cluster: [source][BN / S / 4][128 rows][4] fp32
constexpr int RED_BYTES = 128 * 128 * 4;
constexpr int BAR_OFF = RED_OFF + RED_BYTES;
constexpr int ALLOC = BAR_OFF + (2 * STAGES + 1) * 8 + 16;
static_assert(ALLOC <= 232448, "shared memory budget of one CTA exceeded");

struct Params {
  int M, N, bn, flags, S, tiles_m, tiles_n, kb_total;
  int ldd, ldr;
  __nv_bfloat16* D;
  const __nv_bfloat16 *bias, *residual, *aux;
  __nv_bfloat16* preact;
  int* status;
};

__device__ __forceinline__ void unpack8(uint4 a, float* f) {
  const uint32_t w[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    f[2 * e] = bf16_lo(w[e]);
    f[2 * e + 1] = bf16_hi(w[e]);
  }
}
__device__ __forceinline__ uint4 pack8(const float* f) {
  return make_uint4(pack_bf16x2(f[0], f[1]), pack_bf16x2(f[2], f[3]), pack_bf16x2(f[4], f[5]), pack_bf16x2(f[6], f[7]));
}

template <int A_MAJOR, int B_MAJOR>
__global__ void __launch_bounds__(THREADS, 1)
gemm_split_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b, const Params p) {
  extern __shared__ __align__(1024) uint8_t smem[];
  uint64_t* full = (uint64_t*)(smem + BAR_OFF);
  uint64_t* empty = full + STAGES;
  uint64_t* acc_full = empty + STAGES;
  uint32_t* tmem_ptr = (uint32_t*)(acc_full + 1);
  volatile int* abort_flag = (volatile int*)(tmem_ptr + 1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  uint32_t rank;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
  const int S = p.S, tile = blockIdx.x / S;
  const int n_t = tile / p.tiles_m, m_t = tile - n_t * p.tiles_m;
  const int kb0 = (int)((long)p.kb_total * rank / S), kb1 = (int)((long)p.kb_total * (rank + 1) / S);
  const int cw = p.bn / S;   // columns of the tile that this CTA finishes (a multiple of 8)

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    mbar_init(acc_full, 1);
    *abort_flag = (smem_u32(smem) & 1023u) ? 1 : 0;  // the 128-byte swizzle needs this alignment
    if (*abort_flag && p.status) atomicCAS(p.status, 0, TB_ERR_BAD_ARG);
    fence_barrier_init();
  }
  if (warp == 1) {
    tmem_alloc(tmem_ptr, 128);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_ptr;
  // the partial sums below go to CTAs that have started by then: every CTA arrives here, and waits just before it sends
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");

  if (warp == 0) {
    if (elect_one()) {
      int s = 0;
      uint32_t phase = 0;
      const int row = m_t * 128, col = n_t * p.bn;
      for (int kb = kb0; kb < kb1; ++kb) {
        if (*abort_flag || !mbar_wait(&empty[s], phase ^ 1, abort_flag, p.status, TB_ERR_WAIT_EMPTY)) break;
        uint8_t *sa = smem + s * STAGE_BYTES, *sb = sa + A_BYTES;
        mbar_expect_tx(&full[s], A_BYTES + p.bn * BK * 2);
        if (A_MAJOR == 0) {
          tma_load_2d(sa, &map_a, &full[s], kb * BK, row);
        } else {
          tma_load_2d(sa, &map_a, &full[s], row, kb * BK);
          tma_load_2d(sa + 64 * BK * 2, &map_a, &full[s], row + 64, kb * BK);
        }
        if (B_MAJOR == 0) {
          tma_load_2d(sb, &map_b, &full[s], kb * BK, col);
        } else {
          for (int c = 0; c < p.bn; c += 64) tma_load_2d(sb + c * BK * 2, &map_b, &full[s], col + c, kb * BK);
        }
        if (++s == STAGES) {
          s = 0;
          phase ^= 1;
        }
      }
      if (*abort_flag) {  // copies still in flight land before the shared memory is released
        const uint64_t t0 = globaltimer_ns();
        while (globaltimer_ns() - t0 < 2000000ull) {
        }
      }
    }
  } else if (warp == 1) {
    if (elect_one()) {
      const uint32_t idesc = make_idesc_bf16(128, p.bn, A_MAJOR, B_MAJOR);
      const uint64_t adesc0 = make_smem_desc_sw128(smem_u32(smem), A_MAJOR == 0 ? 16 : 64 * BK * 2, 1024);
      const uint64_t bdesc0 = make_smem_desc_sw128(smem_u32(smem) + A_BYTES, B_MAJOR == 0 ? 16 : 64 * BK * 2, 1024);
      int s = 0;
      uint32_t phase = 0;
      for (int kb = kb0; kb < kb1; ++kb) {
        mbar_wait(&full[s], phase, abort_flag, p.status, TB_ERR_WAIT_FULL);
        tc_fence_after();
        const uint64_t adesc = desc_at(adesc0, s * STAGE_BYTES), bdesc = desc_at(bdesc0, s * STAGE_BYTES);
#pragma unroll
        for (int k = 0; k < BK / 16; ++k)
          umma_ss(tmem_base, desc_at(adesc, k * (A_MAJOR == 0 ? 32 : 2048)), desc_at(bdesc, k * (B_MAJOR == 0 ? 32 : 2048)), idesc,
                 (kb > kb0 || k > 0) ? 1u : 0u);
        umma_commit(&empty[s]);
        if (++s == STAGES) {
          s = 0;
          phase ^= 1;
        }
      }
      umma_commit(acc_full);
    }
  }
  __syncwarp();
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");

  const int q = warp & 3, row_in = q * 32 + lane, row = m_t * 128 + row_in;
  const int col0 = n_t * p.bn + (int)rank * cw;
  const bool row_ok = warp >= 2 && row < p.M;
  const uint32_t lane_off = (uint32_t)(q * 32) << 16;
  // first 8 owned columns of the auxiliary matrix, requested ahead of the accumulator
  const __nv_bfloat16* aux_row = (p.flags & EPI_RESIDUAL) ? p.residual + (size_t)row * p.ldr
                                 : (p.flags & EPI_MUL_DGELU) ? p.aux + (size_t)row * p.ldd : nullptr;
  uint4 aux_next = make_uint4(0, 0, 0, 0), bias_next = make_uint4(0, 0, 0, 0);
  auto request = [&](int c) {
    const int n = col0 + c;
    if (c < cw && n < p.N) {
      if (aux_row && row_ok) aux_next = *reinterpret_cast<const uint4*>(aux_row + n);
      if (p.flags & EPI_BIAS) bias_next = __ldg(reinterpret_cast<const uint4*>(p.bias + n));
    }
  };
  float* red = reinterpret_cast<float*>(smem + RED_OFF);
  if (warp >= 2) {
    request(0);
    mbar_wait(acc_full, 0, abort_flag, p.status, TB_ERR_WAIT_TMEM_FULL);
    tc_fence_after();
    if (S > 1 && m_t * 128 + q * 32 < p.M) {   // rows beyond M are zero and nobody reads them
      const uint32_t red_addr = smem_u32(red);
      for (int c = 0; c < p.bn; c += 16) {
        uint32_t v[16];
        tmem_ld16(tmem_base + c + lane_off, v);
        tmem_wait_ld();
#pragma unroll
        for (int g = 0; g < 4; ++g) {
          const int cc = c + 4 * g, owner = cc / cw, cl = cc - owner * cw;
          uint32_t dst;
          asm volatile("mapa.shared::cluster.u32 %0, %1, %2;"
                       : "=r"(dst)
                       : "r"(red_addr + (uint32_t)((((int)rank * cw + cl) >> 2) * 2048 + row_in * 16)), "r"(owner));
          asm volatile("st.shared::cluster.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(dst), "r"(v[4 * g]), "r"(v[4 * g + 1]),
                       "r"(v[4 * g + 2]), "r"(v[4 * g + 3])
                       : "memory");
        }
      }
    }
  }
  __syncwarp();
  if (S > 1) {
    asm volatile("barrier.cluster.arrive.release.aligned;\n barrier.cluster.wait.acquire.aligned;" ::: "memory");
  }
  if (warp >= 2) {
    const bool warp_rows = m_t * 128 + q * 32 < p.M;
    for (int c = 0; c < cw && col0 + c < p.N && warp_rows; c += 8) {
      float f[8];
      if (S > 1) {
#pragma unroll
        for (int j = 0; j < 8; ++j) f[j] = 0.f;
        for (int src = 0; src < S; ++src) {
#pragma unroll
          for (int g = 0; g < 2; ++g) {
            const float4 x = *reinterpret_cast<const float4*>(red + ((src * cw + c + 4 * g) >> 2) * 512 + row_in * 4);
            f[4 * g] += x.x; f[4 * g + 1] += x.y; f[4 * g + 2] += x.z; f[4 * g + 3] += x.w;
          }
        }
      } else {
        uint32_t v[8];
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                     : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
                     : "r"(tmem_base + c + lane_off)
                     : "memory");
        tmem_wait_ld();
#pragma unroll
        for (int j = 0; j < 8; ++j) f[j] = __uint_as_float(v[j]);
      }
      const uint4 aux = aux_next, bias = bias_next;
      request(c + 8);
      if (!row_ok) continue;
      float t[8];
      if (p.flags & EPI_BIAS) {
        unpack8(bias, t);
#pragma unroll
        for (int j = 0; j < 8; ++j) f[j] += t[j];
      }
      const size_t off = (size_t)row * p.ldd + col0 + c;
      if (p.flags & EPI_STORE_PREACT) *reinterpret_cast<uint4*>(p.preact + off) = pack8(f);
      if (p.flags & EPI_GELU) {
#pragma unroll
        for (int j = 0; j < 8; ++j) f[j] = gelu_tanh(f[j]);
      }
      if (aux_row) {
        unpack8(aux, t);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          if (p.flags & EPI_RESIDUAL) f[j] += t[j];
          else f[j] *= gelu_tanh_grad(t[j]);
        }
      }
      *reinterpret_cast<uint4*>(p.D + off) = pack8(f);
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 128);
  }
}

template <int A_MAJOR, int B_MAJOR>
static int launch(const CUtensorMap& ma, const CUtensorMap& mb, const Params& p, cudaStream_t stream) {
  auto kern = gemm_split_kernel<A_MAJOR, B_MAJOR>;
  static std::atomic<uint64_t> opted_in{0};
  if (int r = smem_opt_in(opted_in, kern, ALLOC)) return r;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)(p.tiles_m * p.tiles_n * p.S));
  cfg.blockDim = dim3(THREADS);
  cfg.dynamicSmemBytes = ALLOC;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)p.S;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  TB_CUDA_CHECK(cudaLaunchKernelEx(&cfg, kern, ma, mb, p));
  return TB_LAUNCH_OK;
}

}  // namespace ksplit

bool gemm_split_ok(const GemmArgs& a) {
  auto al16 = [](const void* q) { return ((uintptr_t)q & 15) == 0; };
  if (a.flags & (EPI_OUT_F32 | EPI_ATOMIC | EPI_ACCUM)) return false;
  if (a.N % 8 || a.ldd % 8 || !al16(a.A) || !al16(a.B) || !al16(a.D)) return false;
  if ((a.flags & EPI_RESIDUAL) && (a.flags & EPI_MUL_DGELU)) return false;
  if ((a.flags & EPI_BIAS) && !al16(a.bias)) return false;
  if ((a.flags & EPI_RESIDUAL) && (!al16(a.residual) || a.ldr % 8)) return false;
  if ((a.flags & EPI_MUL_DGELU) && !al16(a.aux)) return false;
  if ((a.flags & EPI_STORE_PREACT) && !al16(a.preact)) return false;
  return true;
}

int gemm_split_launch(const GemmArgs& a, int bn, int S, cudaStream_t stream) {
  using namespace ksplit;
  if (!gemm_split_ok(a) || (bn != 64 && bn != 128) || (S != 1 && S != 2 && S != 4 && S != 8))
    TB_FAIL(TB_E_ARG, "gemm_split: shape, alignment or epilogue not supported");
  Params p{};
  p.M = a.M; p.N = a.N; p.bn = bn; p.flags = a.flags; p.S = S;
  p.tiles_m = (a.M + 127) / 128;
  p.tiles_n = (a.N + bn - 1) / bn;
  p.kb_total = (a.K + BK - 1) / BK;
  if (S > p.kb_total) TB_FAIL(TB_E_ARG, "gemm_split: more K splits than K blocks");
  p.ldd = a.ldd; p.ldr = a.ldr;
  p.D = (__nv_bfloat16*)a.D;
  p.bias = (const __nv_bfloat16*)a.bias;
  p.residual = (const __nv_bfloat16*)a.residual;
  p.aux = (const __nv_bfloat16*)a.aux;
  p.preact = (__nv_bfloat16*)a.preact;
  p.status = a.status;
  CUtensorMap ma, mb;
  uint64_t dims[2], str[1];
  uint32_t box[2];
  int r;
  if (a.a_major == 0) { dims[0] = a.K; dims[1] = a.M; box[0] = BK; box[1] = 128; }
  else                { dims[0] = a.M; dims[1] = a.K; box[0] = 64; box[1] = BK; }
  str[0] = (uint64_t)a.lda * 2;
  if ((r = make_tmap(&ma, a.A, 2, 2, dims, str, box))) return r;
  if (a.b_major == 0) { dims[0] = a.K; dims[1] = a.N; box[0] = BK; box[1] = bn; }
  else                { dims[0] = a.N; dims[1] = a.K; box[0] = 64; box[1] = BK; }
  str[0] = (uint64_t)a.ldb * 2;
  if ((r = make_tmap(&mb, a.B, 2, 2, dims, str, box))) return r;
  if (a.a_major == 0) return a.b_major == 0 ? launch<0, 0>(ma, mb, p, stream) : launch<0, 1>(ma, mb, p, stream);
  return a.b_major == 0 ? launch<1, 0>(ma, mb, p, stream) : launch<1, 1>(ma, mb, p, stream);
}

}  // namespace tb
