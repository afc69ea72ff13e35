// bf16 GEMM on CTA pairs (tcgen05 cta_group::2) for sm_100a: D[M,N] = A[M,K] * B[N,K]^T, fp32 accumulation in TMEM.
//
// Two CTAs of one cluster (the two SMs of a TPC) work on one 256 x 256 tile. Each loads its own 128 rows of A and its own
// 128 rows of B, and the tensor cores of both SMs read both halves of B, so a K block costs each SM 32 KB of shared
// memory traffic where the one-CTA 128 x 256 tile costs 48 KB: 1.5x the arithmetic per byte staged. That is what bounds
// the one-CTA kernel at large sizes (measured on both sides at route() in gemm_sm100.cu).
//
// 320 threads per CTA, persistent over a static deal of the tiles:
//   warp 0      TMA producer of this CTA's A and B halves; every copy reports to the full barrier of the pair's leader
//   warp 1      MMA issuer (leader CTA only, one thread): 256 x 256 x 16 MMAs; its commits release the stage in both CTAs
//   warps 2..9  epilogue, two warps per TMEM lane quarter taking turns at 64-column groups. Everything that the epilogue
//               moves goes through 128B-swizzled shared-memory tiles and TMA: the output, the pre-activation, the fp32
//               accumulation (TMA reduce-add) and, loaded while the tile's MMAs still run, the residual or the
//               pre-activation of the GELU backward. No thread touches global memory row by row.
// TMEM: two accumulators of 256 columns, so the epilogue of one tile runs under the MMAs of the next.
// Weight gradients (A = dy, stored [tokens, outputs]) can carry the bias gradient: four more warps per CTA add up the A tiles
// of the first column of output tiles over K, reading them from the stage between the MMAs that used it and its release.
// As a kernel of its own the sum read dy once more from memory: 16 us of the 8192 x 1024 x 4096 MLP's backward and 0.78 ms
// of a GPT-2-medium step; with it here, 8192 x 4096 x 1024 50.1 + 9.1 -> 52.5 us, 8192 x 3072 x 1024 39.3 + 7.2 -> 40.5.
//
// Every wait is bounded (sm100.cuh); a CTA that gives up drains its loops, and its peer runs into its own limits.
#include <stdlib.h>
#include <string.h>

#include "gemm_pair.cuh"
#include "host_util.h"
#include "sm100.cuh"

namespace tb {

namespace pair {

constexpr int BN = 256;                 // a pair's tile is 256 x BN; 128- and 192-wide tiles measured slower at every size
constexpr int BK = 64;
constexpr int THREADS = 320;
constexpr int EPI_WARPS = 8;
constexpr int A_BYTES = 128 * BK * 2;   // this CTA's half of A per stage
constexpr int B_BYTES = BN / 2 * BK * 2;   // this CTA's half of B per stage
constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
constexpr int STAGES = 5;
constexpr int SLOT_BYTES = 32 * 128;    // one staged group: 32 rows x 64 bf16 or 32 fp32 columns
constexpr int EPI_OFF = STAGES * STAGE_BYTES;
constexpr int BAR_OFF = EPI_OFF + EPI_WARPS * 2 * SLOT_BYTES;
// full[STAGES], empty[STAGES], tmem_full[2], tmem_empty[2], aux_full[EPI_WARPS][2], tmem pointer, abort flag
constexpr int NBARS = 3 * STAGES + 4 + 2 * EPI_WARPS;  // used[STAGES] last
constexpr int ALLOC = BAR_OFF + NBARS * 8 + 16;
static_assert(ALLOC <= 232448, "shared memory budget of one CTA exceeded");

struct Params {
  int M, N, flags, split_k, tiles_m, tiles_n, kb_total, kb_per_split;
  const __nv_bfloat16* bias;
  int* status;
  void* colsum;
  int colsum_store;
};

struct Maps {
  CUtensorMap a, b, d, pre, aux;
};

__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// address of the same shared-memory location in CTA `rank` of the cluster
__device__ __forceinline__ uint32_t mapa(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t addr) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(addr) : "memory");
}
__device__ __forceinline__ void tma_load_2d_pair(uint32_t dst, const CUtensorMap* map, uint32_t bar, int x, int y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%3, %4}], [%2];" ::"r"(dst),
      "l"(map), "r"(bar), "r"(x), "r"(y)
      : "memory");
}
__device__ __forceinline__ void umma_pair(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n}" ::"r"(d_tmem),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// arrives on the barrier at this offset in both CTAs of the pair
__device__ __forceinline__ void umma_commit_pair(uint64_t* bar) {
  asm volatile(
      "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(smem_u32(bar)),
      "h"((uint16_t)3)
      : "memory");
}
__device__ __forceinline__ void tma_store(const CUtensorMap* map, const void* src, int x, int y) {
  asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%1, %2}], [%3];" ::"l"(map), "r"(x), "r"(y),
               "r"(smem_u32(src))
               : "memory");
}
__device__ __forceinline__ void tma_reduce_add(const CUtensorMap* map, const void* src, int x, int y) {
  asm volatile("cp.reduce.async.bulk.tensor.2d.global.shared::cta.add.bulk_group [%0, {%1, %2}], [%3];" ::"l"(map), "r"(x),
               "r"(y), "r"(smem_u32(src))
               : "memory");
}
__device__ __forceinline__ void bulk_wait_read_1() { asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory"); }

__device__ __forceinline__ bool decode(const Params& p, int work, int& m_t, int& n_t, int& kb0, int& kb1) {
  if (work >= p.tiles_m * p.tiles_n * p.split_k) return false;
  const int tile = work / p.split_k, ks = work - tile * p.split_k;
  if (p.flags & EPI_RASTER_M) {
    n_t = tile / p.tiles_m;
    m_t = tile - n_t * p.tiles_m;
  } else {
    m_t = tile / p.tiles_n;
    n_t = tile - m_t * p.tiles_n;
  }
  kb0 = ks * p.kb_per_split;
  kb1 = min(p.kb_total, kb0 + p.kb_per_split);
  return true;
}

__device__ __forceinline__ void add_bf16x8(float* f, uint4 a) {
  const uint32_t w[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    f[2 * e] += bf16_lo(w[e]);
    f[2 * e + 1] += bf16_hi(w[e]);
  }
}
__device__ __forceinline__ uint4 pack8(const float* f) {
  return make_uint4(pack_bf16x2(f[0], f[1]), pack_bf16x2(f[2], f[3]), pack_bf16x2(f[4], f[5]), pack_bf16x2(f[6], f[7]));
}

template <int A_MAJOR, int B_MAJOR, bool COLSUM>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(THREADS + (COLSUM ? 128 : 0), 1)
gemm_pair_kernel(const __grid_constant__ Maps maps, const Params p) {
  extern __shared__ __align__(1024) uint8_t smem[];
  if (smem_u32(smem) & 1023u) {  // the 128-byte swizzle needs this alignment; the same in both CTAs
    if (threadIdx.x == 0 && p.status) atomicCAS(p.status, 0, TB_ERR_BAD_ARG);
    return;
  }
  uint64_t* full = (uint64_t*)(smem + BAR_OFF);   // used in the leader only
  uint64_t* empty = full + STAGES;
  uint64_t* tmem_full = empty + STAGES;
  uint64_t* tmem_empty = tmem_full + 2;           // used in the leader only
  uint64_t* aux_full = tmem_empty + 2;
  uint64_t* used = aux_full + 2 * EPI_WARPS;      // COLSUM: the MMAs of a stage are done, its A tile may be summed
  uint32_t* tmem_ptr = (uint32_t*)(used + STAGES);
  volatile int* abort_flag = (volatile int*)(tmem_ptr + 1);
  __shared__ float colsum_ex[COLSUM ? 128 : 1];

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_rank();
  const int worker = blockIdx.x >> 1, nworkers = gridDim.x >> 1;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], COLSUM ? 4 : 1);
      mbar_init(&used[s], 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(&tmem_full[a], 1);
      mbar_init(&tmem_empty[a], 2 * EPI_WARPS);
    }
    for (int i = 0; i < 2 * EPI_WARPS; ++i) mbar_init(&aux_full[i], 1);
    *abort_flag = 0;
    fence_barrier_init();
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_ptr)), "r"(512u) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync();  // the peer's barriers exist before anything reports to them
  tc_fence_after();
  const uint32_t tmem_base = *tmem_ptr;

  if (warp == 0) {
    // ---------------------------------------------------------------- TMA producer
    if (elect_one()) {
      tma_prefetch_desc(&maps.a);
      tma_prefetch_desc(&maps.b);
      int s = 0;
      uint32_t phase = 0;
      int m_t, n_t, kb0, kb1;
      for (int w = worker; !*abort_flag && decode(p, w, m_t, n_t, kb0, kb1); w += nworkers) {
        const int row = m_t * 256 + (int)rank * 128, col = n_t * BN + (int)rank * (BN / 2);
        for (int kb = kb0; kb < kb1; ++kb) {
          // once a wait has given up nothing more is loaded, and the MMA role drains on its own limits
          if (!mbar_wait(&empty[s], phase ^ 1, abort_flag, p.status, TB_ERR_WAIT_EMPTY)) break;
          const uint32_t sa = smem_u32(smem + s * STAGE_BYTES), sb = sa + A_BYTES;
          const uint32_t bar = mapa(smem_u32(&full[s]), 0);
          if (rank == 0) mbar_expect_tx(&full[s], 2 * STAGE_BYTES);  // both CTAs' copies
          if (A_MAJOR == 0) {
            tma_load_2d_pair(sa, &maps.a, bar, kb * BK, row);
          } else {
            tma_load_2d_pair(sa, &maps.a, bar, row, kb * BK);
            tma_load_2d_pair(sa + 64 * BK * 2, &maps.a, bar, row + 64, kb * BK);
          }
          if (B_MAJOR == 0) {
            tma_load_2d_pair(sb, &maps.b, bar, kb * BK, col);
          } else {
            tma_load_2d_pair(sb, &maps.b, bar, col, kb * BK);
            tma_load_2d_pair(sb + 64 * BK * 2, &maps.b, bar, col + 64, kb * BK);
          }
          if (++s == STAGES) {
            s = 0;
            phase ^= 1;
          }
        }
      }
      if (*abort_flag) {  // copies still in flight land before the shared memory is released
        const uint64_t t0 = globaltimer_ns();
        while (globaltimer_ns() - t0 < 2000000ull) {
        }
      }
    }
  } else if (warp == 1) {
    // ---------------------------------------------------------------- MMA issuer
    if (rank == 0 && elect_one()) {
      const uint32_t idesc = make_idesc_bf16(256, BN, A_MAJOR, B_MAJOR);
      const uint64_t adesc0 = make_smem_desc_sw128(smem_u32(smem), A_MAJOR == 0 ? 16 : 64 * BK * 2, 1024);
      const uint64_t bdesc0 = make_smem_desc_sw128(smem_u32(smem) + A_BYTES, B_MAJOR == 0 ? 16 : 64 * BK * 2, 1024);
      int s = 0, acc = 0;
      uint32_t phase = 0, acc_phase = 0;
      int m_t, n_t, kb0, kb1;
      for (int w = worker; decode(p, w, m_t, n_t, kb0, kb1); w += nworkers) {
        mbar_wait(&tmem_empty[acc], acc_phase ^ 1, abort_flag, p.status, TB_ERR_WAIT_TMEM_EMPTY);
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + acc * 256;
        for (int kb = kb0; kb < kb1; ++kb) {
          mbar_wait(&full[s], phase, abort_flag, p.status, TB_ERR_WAIT_FULL);
          tc_fence_after();
          const uint64_t adesc = desc_at(adesc0, s * STAGE_BYTES), bdesc = desc_at(bdesc0, s * STAGE_BYTES);
#pragma unroll
          for (int k = 0; k < BK / 16; ++k)
            umma_pair(d_tmem, desc_at(adesc, k * (A_MAJOR == 0 ? 32 : 2048)), desc_at(bdesc, k * (B_MAJOR == 0 ? 32 : 2048)), idesc,
                   (kb > kb0 || k > 0) ? 1u : 0u);
          umma_commit_pair(COLSUM ? &used[s] : &empty[s]);
          if (++s == STAGES) {
            s = 0;
            phase ^= 1;
          }
        }
        umma_commit_pair(&tmem_full[acc]);
        if (++acc == 2) {
          acc = 0;
          acc_phase ^= 1;
        }
      }
    }
  } else if (COLSUM && warp >= 2 + EPI_WARPS) {
    // ---------------------------------------------------------------- column sums of A
    // Two warps per 64-column chunk, 32 rows of a stage each: lane l reads the 16-byte vector l % 8 of rows l / 8, l / 8 + 4, ...
    // (vectors are xored with row % 8), all eight before the first is added. The stage waits for this, so it has to be quick:
    // with one warp per chunk and 4-byte reads the kernel took 75 us instead of 50.
    const int id = warp - 2 - EPI_WARPS, chunk = id >> 1, r0 = (id & 1) * 32 + (lane >> 3);
    int s = 0;
    uint32_t phase = 0;
    int m_t, n_t, kb0, kb1;
    for (int w = worker; decode(p, w, m_t, n_t, kb0, kb1); w += nworkers) {
      float2 total[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) total[j] = make_float2(0.f, 0.f);
      for (int kb = kb0; kb < kb1; ++kb) {
        const bool ok = mbar_wait(&used[s], phase, abort_flag, p.status, TB_ERR_WAIT_FULL);
        if (n_t == 0 && ok) {
          const uint8_t* base = smem + s * STAGE_BYTES + chunk * (64 * BK * 2);
          uint4 x[8];
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const int k = r0 + 4 * i;
            x[i] = *reinterpret_cast<const uint4*>(base + k * 128 + (((lane & 7) ^ (k & 7)) << 4));
          }
          __syncwarp();
          if (lane == 0) mbar_arrive(&empty[s]);   // everything this warp needs of the stage is in registers
          float2 part[4];
#pragma unroll
          for (int j = 0; j < 4; ++j) part[j] = make_float2(0.f, 0.f);
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const uint32_t u[4] = {x[i].x, x[i].y, x[i].z, x[i].w};
#pragma unroll
            for (int j = 0; j < 4; ++j) part[j] = __fadd2_rn(part[j], make_float2(bf16_lo(u[j]), bf16_hi(u[j])));
          }
#pragma unroll
          for (int j = 0; j < 4; ++j) total[j] = __fadd2_rn(total[j], part[j]);
        } else if (lane == 0) {
          mbar_arrive(&empty[s]);
        }
        if (++s == STAGES) {
          s = 0;
          phase ^= 1;
        }
      }
      if (n_t != 0) continue;
#pragma unroll
      for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int o = 8; o < 32; o <<= 1) {
          total[j].x += __shfl_xor_sync(0xffffffffu, total[j].x, o);
          total[j].y += __shfl_xor_sync(0xffffffffu, total[j].y, o);
        }
      const int m = m_t * 256 + (int)rank * 128 + chunk * 64 + (lane & 7) * 8;   // M is a multiple of 8
      if (p.colsum_store) {
        float4* ex = reinterpret_cast<float4*>(colsum_ex + chunk * 64 + (lane & 7) * 8);
        if ((id & 1) && lane < 8) {
          ex[0] = make_float4(total[0].x, total[0].y, total[1].x, total[1].y);
          ex[1] = make_float4(total[2].x, total[2].y, total[3].x, total[3].y);
        }
        asm volatile("bar.sync %0, 64;" ::"r"(1 + chunk) : "memory");
        if (!(id & 1) && lane < 8 && m < p.M) {
          const float4 a = ex[0], c = ex[1];
          *reinterpret_cast<uint4*>(reinterpret_cast<__nv_bfloat16*>(p.colsum) + m) =
              make_uint4(pack_bf16x2(total[0].x + a.x, total[0].y + a.y), pack_bf16x2(total[1].x + a.z, total[1].y + a.w),
                         pack_bf16x2(total[2].x + c.x, total[2].y + c.y), pack_bf16x2(total[3].x + c.z, total[3].y + c.w));
        }
        asm volatile("bar.sync %0, 64;" ::"r"(1 + chunk) : "memory");
      } else if (lane < 8 && m < p.M) {
        float* out = reinterpret_cast<float*>(p.colsum) + m;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          atomicAdd(out + 2 * j, total[j].x);
          atomicAdd(out + 2 * j + 1, total[j].y);
        }
      }
    }
  } else {
    // ---------------------------------------------------------------- epilogue
    const int e = warp - 2, q = warp & 3, set = e >> 2;   // TMEM lane quarter; which of the quarter's two warps
    uint8_t* slots = smem + EPI_OFF + e * 2 * SLOT_BYTES;
    uint64_t* aux_bar = aux_full + 2 * e;
    const uint32_t lane_off = (uint32_t)(q * 32) << 16;
    const int flags = p.flags;
    const bool f32_out = flags & EPI_OUT_F32;
    const bool has_aux = flags & (EPI_RESIDUAL | EPI_MUL_DGELU);
    const uint32_t empty_bar[2] = {mapa(smem_u32(&tmem_empty[0]), 0), mapa(smem_u32(&tmem_empty[1]), 0)};
    int acc = 0;
    uint32_t acc_phase = 0, aux_phase[2] = {0, 0}, cnt = 0;
    int m_t, n_t, kb0, kb1;
    for (int w = worker; decode(p, w, m_t, n_t, kb0, kb1); w += nworkers) {
      const int row0 = m_t * 256 + (int)rank * 128 + q * 32;
      const int col0 = n_t * BN;
      const int groups = (min(BN, p.N - col0) + 63) >> 6;   // 64-column groups of this tile; this warp takes set, set + 2
      if (has_aux && lane == 0) {
        // residual / pre-activation tiles of this warp's (at most two) groups: requested before the accumulator is done
        bulk_wait_read_all();
        for (int g = set, k = 0; g < groups; g += 2, ++k) {
          mbar_expect_tx(&aux_bar[k], SLOT_BYTES);
          tma_load_2d(slots + k * SLOT_BYTES, &maps.aux, &aux_bar[k], col0 + g * 64, row0);
        }
      }
      mbar_wait(&tmem_full[acc], acc_phase, abort_flag, p.status, TB_ERR_WAIT_TMEM_FULL);
      tc_fence_after();
      const bool add_bias = (flags & EPI_BIAS) && kb0 == 0;
      for (int g = set, k = 0; g < groups; g += 2, ++k) {
        if (has_aux) {
          mbar_wait(&aux_bar[k], aux_phase[k], abort_flag, p.status, TB_ERR_WAIT_FULL);
          aux_phase[k] ^= 1;
        }
        uint8_t* slot = slots + (has_aux ? k : (cnt & 1)) * SLOT_BYTES;
#pragma unroll 1
        for (int half = 0; half < 2; ++half) {
          const int c = g * 64 + half * 32, n0 = col0 + c;
          uint32_t v[32];
          tmem_ld32(tmem_base + acc * 256 + c + lane_off, v);
          tmem_wait_ld();
          float f[32];
#pragma unroll
          for (int j = 0; j < 32; ++j) f[j] = __uint_as_float(v[j]);
          if (add_bias) {
            const uint4* bp = reinterpret_cast<const uint4*>(p.bias + n0);
#pragma unroll
            for (int i = 0; i < 4; ++i)
              if (n0 + 8 * i < p.N) add_bf16x8(f + 8 * i, __ldg(bp + i));
          }
          if (f32_out) {
            // 32 fp32 columns are one staged group of their own
            uint8_t* fs = slots + (cnt & 1) * SLOT_BYTES;
            if (lane == 0) bulk_wait_read_1();
            __syncwarp();
#pragma unroll
            for (int i = 0; i < 8; ++i)
              *reinterpret_cast<float4*>(fs + lane * 128 + ((i ^ (lane & 7)) << 4)) =
                  make_float4(f[4 * i], f[4 * i + 1], f[4 * i + 2], f[4 * i + 3]);
            fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) {
              if (n0 < p.N && row0 < p.M) {
                if (flags & (EPI_ATOMIC | EPI_ACCUM)) tma_reduce_add(&maps.d, fs, n0, row0);
                else tma_store(&maps.d, fs, n0, row0);
              }
              bulk_commit();
            }
            ++cnt;
            continue;
          }
          const int ch = half * 4;
          if (flags & EPI_STORE_PREACT) {
            // the pre-activation takes the slot in turn, the output the other one
            if (half == 0) {
              if (lane == 0) bulk_wait_read_1();
              __syncwarp();
            }
#pragma unroll
            for (int i = 0; i < 4; ++i)
              *reinterpret_cast<uint4*>(slots + lane * 128 + (((ch + i) ^ (lane & 7)) << 4)) = pack8(f + 8 * i);
            if (half == 1) {
              fence_proxy_async_smem();
              __syncwarp();
              if (lane == 0) {
                if (row0 < p.M) tma_store(&maps.pre, slots, col0 + g * 64, row0);
                bulk_commit();
              }
            }
            slot = slots + SLOT_BYTES;
          }
          if (flags & EPI_GELU) {
#pragma unroll
            for (int j = 0; j < 32; ++j) f[j] = gelu_tanh(f[j]);
          }
          if (has_aux) {
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              const uint4 a = *reinterpret_cast<const uint4*>(slot + lane * 128 + (((ch + i) ^ (lane & 7)) << 4));
              if (flags & EPI_RESIDUAL) {
                add_bf16x8(f + 8 * i, a);
              } else {
                const uint32_t u[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                  f[8 * i + 2 * j] *= gelu_tanh_grad(bf16_lo(u[j]));
                  f[8 * i + 2 * j + 1] *= gelu_tanh_grad(bf16_hi(u[j]));
                }
              }
            }
          } else if (half == 0) {
            // the slot's last store has been read: with the pre-activation its own store is the newer one
            if (lane == 0) {
              if (flags & EPI_STORE_PREACT) bulk_wait_read_all(); else bulk_wait_read_1();
            }
            __syncwarp();
          }
#pragma unroll
          for (int i = 0; i < 4; ++i)
            *reinterpret_cast<uint4*>(slot + lane * 128 + (((ch + i) ^ (lane & 7)) << 4)) = pack8(f + 8 * i);
          if (half == 1) {
            fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) {
              if (row0 < p.M) tma_store(&maps.d, slot, col0 + g * 64, row0);
              bulk_commit();
            }
            ++cnt;
          }
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(empty_bar[acc]);
      if (++acc == 2) {
        acc = 0;
        acc_phase ^= 1;
      }
    }
    if (lane == 0) bulk_wait_all();  // everything sent has left shared memory and landed
  }

  tc_fence_before();
  __syncthreads();
  cluster_sync();  // neither CTA leaves while the other may still report to its barriers
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512u) : "memory");
  }
}

template <int A_MAJOR, int B_MAJOR, bool COLSUM = false>
static int launch(const Maps& maps, const Params& p, cudaStream_t stream) {
  auto kern = gemm_pair_kernel<A_MAJOR, B_MAJOR, COLSUM>;
  static std::atomic<uint64_t> opted_in{0};
  if (int r = smem_opt_in(opted_in, kern, ALLOC)) return r;
  const long total = (long)p.tiles_m * p.tiles_n * p.split_k;
  const int pairs = sm_count() / 2;
  kern<<<2 * (int)(total < pairs ? total : pairs), THREADS + (COLSUM ? 128 : 0), ALLOC, stream>>>(maps, p);
  TB_CUDA_CHECK(cudaGetLastError());
  return TB_LAUNCH_OK;
}

}  // namespace pair

bool gemm_pair_ok(const GemmArgs& a) {
  auto al16 = [](const void* q) { return ((uintptr_t)q & 15) == 0; };
  const int ebytes = (a.flags & EPI_OUT_F32) ? 4 : 2;
  if (a.N % 8 || !al16(a.A) || !al16(a.B) || !al16(a.D) || ((long)a.ldd * ebytes) % 16) return false;
  if (a.flags & EPI_OUT_F32) {
    // fp32 outputs: bias and accumulation only
    if (a.flags & (EPI_GELU | EPI_RESIDUAL | EPI_STORE_PREACT | EPI_MUL_DGELU)) return false;
  } else if (a.flags & (EPI_ATOMIC | EPI_ACCUM)) {
    return false;
  }
  // rows that overlap (a residual expanded over the rows: stride 0) are for the kernels that read with plain loads
  if (a.ldd < a.N || ((a.flags & EPI_RESIDUAL) && a.ldr < a.N)) return false;
  if (a.bias && !al16(a.bias)) return false;
  const bool res = a.flags & EPI_RESIDUAL, dgelu = a.flags & EPI_MUL_DGELU, pre = a.flags & EPI_STORE_PREACT;
  if (res + dgelu + pre > 1) return false;   // one auxiliary matrix through the two staging slots of a warp
  if (res && (!al16(a.residual) || a.ldr % 8)) return false;
  if ((dgelu && !al16(a.aux)) || (pre && !al16(a.preact))) return false;
  return true;
}

int gemm_pair_launch(const GemmArgs& a, cudaStream_t stream) {
  using namespace pair;
  if (!gemm_pair_ok(a)) TB_FAIL(TB_E_ARG, "gemm_pair: shape, alignment or epilogue not supported");
  Params p{};
  p.M = a.M; p.N = a.N; p.flags = a.flags;
  p.tiles_m = (a.M + 255) / 256;
  p.tiles_n = (a.N + BN - 1) / BN;
  p.kb_total = (a.K + BK - 1) / BK;
  int split = a.split_k < 1 ? 1 : a.split_k > p.kb_total ? p.kb_total : a.split_k;
  p.kb_per_split = (p.kb_total + split - 1) / split;
  p.split_k = (p.kb_total + p.kb_per_split - 1) / p.kb_per_split;
  if (p.split_k > 1 && !(a.flags & EPI_ATOMIC)) TB_FAIL(TB_E_ARG, "gemm_pair: split_k > 1 needs EPI_ATOMIC");
  p.bias = (const __nv_bfloat16*)a.bias;
  p.status = a.status;
  Maps m;
  memset(&m, 0, sizeof(m));
  uint64_t dims[2], str[1];
  uint32_t box[2];
  int r;
  if (a.a_major == 0) { dims[0] = a.K; dims[1] = a.M; box[0] = BK; box[1] = 128; }
  else                { dims[0] = a.M; dims[1] = a.K; box[0] = 64; box[1] = BK; }
  str[0] = (uint64_t)a.lda * 2;
  if ((r = make_tmap(&m.a, a.A, 2, 2, dims, str, box))) return r;
  if (a.b_major == 0) { dims[0] = a.K; dims[1] = a.N; box[0] = BK; box[1] = BN / 2; }
  else                { dims[0] = a.N; dims[1] = a.K; box[0] = 64; box[1] = BK; }
  str[0] = (uint64_t)a.ldb * 2;
  if ((r = make_tmap(&m.b, a.B, 2, 2, dims, str, box))) return r;
  const bool f32 = a.flags & EPI_OUT_F32;
  dims[0] = a.N; dims[1] = a.M;
  box[0] = f32 ? 32 : 64; box[1] = 32;
  str[0] = (uint64_t)a.ldd * (f32 ? 4 : 2);
  if ((r = make_tmap(&m.d, a.D, f32 ? 4 : 2, 2, dims, str, box))) return r;
  if (a.flags & EPI_STORE_PREACT)
    if ((r = make_tmap(&m.pre, a.preact, 2, 2, dims, str, box))) return r;
  if (a.flags & EPI_MUL_DGELU)
    if ((r = make_tmap(&m.aux, a.aux, 2, 2, dims, str, box))) return r;
  if (a.flags & EPI_RESIDUAL) {
    str[0] = (uint64_t)a.ldr * 2;
    if ((r = make_tmap(&m.aux, a.residual, 2, 2, dims, str, box))) return r;
  }
  if (a.colsum) {
    if (a.a_major != 1 || a.b_major != 1 || (a.colsum_store && p.split_k > 1) || ((uintptr_t)a.colsum & 15) || a.M % 8)
      TB_FAIL(TB_E_ARG, "gemm_pair: column sums need MN-major operands, M a multiple of 8, 16-byte alignment and, to be written, no split");
    p.colsum = a.colsum;
    p.colsum_store = a.colsum_store;
    return launch<1, 1, true>(m, p, stream);
  }
  if (a.a_major == 0) return a.b_major == 0 ? launch<0, 0>(m, p, stream) : launch<0, 1>(m, p, stream);
  return a.b_major == 0 ? launch<1, 0>(m, p, stream) : launch<1, 1>(m, p, stream);
}

}  // namespace tb
