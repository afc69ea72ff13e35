// Flash attention backward for sm_100a (tcgen05 / TMEM / TMA), causal or full, head dim 64 / 128.
//
// One CTA per (batch, head, 128-key block); it walks the query blocks that see those keys. Scores are kept transposed
// (TMEM lane = key), so that P^T is a tensor-memory operand and never goes through shared memory:
//   S^T  = K_j Q_i^T         dP^T = V_j dO_i^T                   (tensor core, into TMEM)
//   P^T  = exp(S^T*scale - L_i)  dS^T = P^T * (dP^T - delta_i) * scale   (compute warps, fp32)
//   dV_j += P^T dO_i         dK_j += dS^T Q_i                    (accumulate in TMEM over i)
//   dQ_i += dS K_j                                               (TMEM -> shared memory -> bulk fp32 reduce-add in global)
// dS^T goes to shared memory once, in the 128-byte-swizzled layout of the MMA
// descriptors, and serves as the K-major A operand of dK and as the MN-major A operand of dQ.
//
// What bounds it is the chain of a query block (scores, exponentials, dP, dS, three products, dQ out), so the chain is cut
// into roles that work on different blocks at the same time. 16 warps:
//   warps 0-7    compute, two threads per key row, each owning 64 queries of the block
//   warps 8-11   dQ out: drain block t while the compute warps evaluate the exponentials of block t + 1
//   warp 12      MMA issuer: the scores of block t + 1 go out as soon as block t has left their columns
//   warp 13      TMA producer (Q two blocks deep, dO one);  warp 14  L and delta rows into a two-deep ring
// TMEM: S^T | dP^T (128 columns each) | dV | dK (D each), and with D = 64 dQ | P^T (64 each).
// Registers are moved between the warpgroups with setmaxnreg: 512 threads x 128 at launch, 160 for the two compute groups,
// 88 and 104 for the others.
// One role after the other per block (P and dS both through shared memory) took 633 us where this takes 400 with everything
// around it (B2 S4096 H16 D128 causal), 214 where this takes 136 (B1 S2048 H32 D128), and 129 where this takes 117
// (B8 S1024 H16 D64). What bounds it now with D = 64 is shared memory: about 3400 clocks of 128 bytes per block for the MMA
// operands, the L and delta broadcasts, dS and dQ, against 1300 clocks of MMA and 1024 of exponentials. Four compute threads
// per row instead of two and conversions on the FMA pipe changed nothing.
//
// The reference has no attention backward at all (its autograd tape covers only
// add/sub/mul/matmul/pow/mean/sum: crates/torsh-tensor/src/core_ops/types.rs:1497-1658).
#include "host_util.h"
#include "sm100.cuh"

namespace tb {

constexpr int FB_THREADS = 512;

struct FaBwdParams {
  const float* LSE;    // [B, H, S]
  const float* delta;  // [B, H, S]  rowsum(dO * O)
  float* dQ_acc;       // fp32, accumulated: [B*H][groups of 32 queries][D / 32][the group's rows][32 columns, 16-byte chunks
                       // xor row % 8]; the last group of a sequence has S % 32 rows, so this is B*H*S*D floats
  __nv_bfloat16* dK;   // [B*S, dkv_stride], head h at column h*D
  __nv_bfloat16* dV;
  int B, S, H;
  long dkv_stride;
  float scale;
  int causal;
  int* status;
};

template <int D>
struct FaBwdSmem {
  static constexpr int TILE = 128 * D * 2;
  static constexpr int DOST = (D == 64) ? 2 : 1;  // dO ring depth
  static constexpr int K_OFF = 0;
  static constexpr int V_OFF = TILE;
  static constexpr int Q_OFF = 2 * TILE;
  static constexpr int DO_OFF = Q_OFF + 2 * TILE;
  static constexpr int DS_OFF = DO_OFF + DOST * TILE;
  static constexpr int DQ_OFF = DS_OFF + 32768;        // per dQ warp: 2 x (32 rows x 32 fp32 columns) on their way out
  static constexpr int LD_OFF = DQ_OFF + 4 * 8192;     // -L * log2(e) and -delta * scale of a query block, 2 stages
  static constexpr int BAR_OFF = LD_OFF + 2 * 2 * 512;
  // kv_full, q_full[2], q_empty[2], do_full[2], do_empty[2], ld_full[2], ld_empty[2], s_full, p_full, dp_full, ds_full,
  // ds_empty, dv_done, dq_full, dq_empty, dkv_full
  static constexpr int NBARS = 22;
  static constexpr int ALLOC = BAR_OFF + NBARS * 8 + 16;
  static_assert(ALLOC <= 232448, "shared memory budget of one CTA exceeded");
};

// e = exp2(S^T * sl2 - L) for 32 queries of one key row, and the same packed to bf16 pairs. `first` is the first query (as
// an index of this call's 32) that sees the key; MASK is a template parameter so that blocks away from the diagonal and the
// ragged edge carry no compare / select instructions. --L comes from shared memory (the same for every lane: broadcast).
template <bool MASK>
__device__ __forceinline__ void fa_bwd_p(const uint32_t (&sv)[32], const float* L, float sl2, int first, float (&e)[32],
                                         uint32_t (&pk)[16]) {
  const float2 s2 = make_float2(sl2, sl2);
#pragma unroll
  for (int i = 0; i < 32; i += 4) {
    const float4 l4 = *reinterpret_cast<const float4*>(L + i);
    const float2 t0 = __ffma2_rn(make_float2(__uint_as_float(sv[i]), __uint_as_float(sv[i + 1])), s2, make_float2(l4.x, l4.y));
    const float2 t1 = __ffma2_rn(make_float2(__uint_as_float(sv[i + 2]), __uint_as_float(sv[i + 3])), s2, make_float2(l4.z, l4.w));
    e[i] = exp2f(t0.x);
    e[i + 1] = exp2f(t0.y);
    e[i + 2] = exp2f(t1.x);
    e[i + 3] = exp2f(t1.y);
    if (MASK) {
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (i + j < first) e[i + j] = 0.f;
    }
    pk[i >> 1] = pack_bf16x2(e[i], e[i + 1]);
    pk[(i >> 1) + 1] = pack_bf16x2(e[i + 2], e[i + 3]);
  }
}

// dS^T = e * (dP^T * scale - delta * scale) for 32 queries, packed to bf16 pairs (the ring holds -delta * scale)
__device__ __forceinline__ void fa_bwd_ds(const uint32_t (&dv)[32], const float* ds_row, float scale, const float (&e)[32],
                                          uint32_t (&dd)[16]) {
  const float2 c2 = make_float2(scale, scale);
#pragma unroll
  for (int i = 0; i < 32; i += 4) {
    const float4 d4 = *reinterpret_cast<const float4*>(ds_row + i);
    const float2 g0 = __ffma2_rn(make_float2(__uint_as_float(dv[i]), __uint_as_float(dv[i + 1])), c2, make_float2(d4.x, d4.y));
    const float2 g1 = __ffma2_rn(make_float2(__uint_as_float(dv[i + 2]), __uint_as_float(dv[i + 3])), c2, make_float2(d4.z, d4.w));
    const float2 a = __fmul2_rn(make_float2(e[i], e[i + 1]), g0), b = __fmul2_rn(make_float2(e[i + 2], e[i + 3]), g1);
    dd[i >> 1] = pack_bf16x2(a.x, a.y);
    dd[(i >> 1) + 1] = pack_bf16x2(b.x, b.y);
  }
}

template <int D>
__global__ void __launch_bounds__(FB_THREADS, 1)
fa_bwd_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
              const __grid_constant__ CUtensorMap map_v, const __grid_constant__ CUtensorMap map_do,
              const FaBwdParams p) {
  using L = FaBwdSmem<D>;
  constexpr int KCH = D / 64;
  constexpr int DOST = L::DOST;
  constexpr uint32_t TM_S = 0, TM_DP = 128, TM_DV = 256, TM_DK = 256 + D;
  // With D = 64 there is room for P^T and dQ beside the rest, and the scores of the next block can be issued early. With
  // D = 128 P^T takes the first half of the S^T columns it came from (a compute half's 64 queries: 32 of its 64 columns)
  // and dQ the columns of dP^T once they have been read.
  constexpr bool ROOMY = D == 64;
  constexpr uint32_t TM_DQ = ROOMY ? 384 : TM_DP;
  constexpr uint32_t TM_P = ROOMY ? 448 : TM_S, P_HALF = ROOMY ? 32 : 64;
  extern __shared__ __align__(1024) uint8_t smem[];
  uint64_t* bars = (uint64_t*)(smem + L::BAR_OFF);
  uint64_t* kv_full = bars;
  uint64_t* q_full = bars + 1;
  uint64_t* q_empty = bars + 3;
  uint64_t* do_full = bars + 5;
  uint64_t* do_empty = bars + 7;
  uint64_t* ld_full = bars + 9;
  uint64_t* ld_empty = bars + 11;
  uint64_t* s_full = bars + 13;    // S^T[t] is in TMEM
  uint64_t* p_full = bars + 14;    // P^T[t] has replaced it
  uint64_t* dp_full = bars + 15;   // dP^T[t] is in TMEM
  uint64_t* ds_full = bars + 16;   // dP^T[t] has been read, dS^T[t] is in shared memory
  uint64_t* ds_empty = bars + 17;  // dK and dQ of block t have read dS^T[t]
  uint64_t* dv_done = bars + 18;   // dV of block t has read P^T[t]
  uint64_t* dq_full = bars + 19;   // dQ partial of block t is in TMEM
  uint64_t* dq_empty = bars + 20;  // ... and has been read
  uint64_t* dkv_full = bars + 21;
  uint32_t* tmem_ptr = (uint32_t*)(bars + L::NBARS);
  volatile int* abort_flag = (volatile int*)(tmem_ptr + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int n_blk = (p.S + 127) / 128;
  const int BH = p.B * p.H;
  const int jb = blockIdx.x / BH;     // key block; the early key blocks of all heads first: with a causal mask they are the long ones
  const int bh = blockIdx.x - jb * BH;
  const int h = bh % p.H, b = bh / p.H;
  const int kv0 = jb * 128;
  const int i0 = p.causal ? jb : 0;
  const int n_it = n_blk - i0;

  if (threadIdx.x == 0) {
    mbar_init(kv_full, 1);
    for (int i = 0; i < 2; ++i) {
      mbar_init(&q_full[i], 1);
      mbar_init(&q_empty[i], 1);
      mbar_init(&do_full[i], 1);
      mbar_init(&do_empty[i], 1);
      mbar_init(&ld_full[i], 32);
      mbar_init(&ld_empty[i], 256);
    }
    mbar_init(s_full, 1);
    mbar_init(p_full, 256);
    mbar_init(dp_full, 1);
    mbar_init(ds_full, 256);
    mbar_init(ds_empty, 1);
    mbar_init(dv_done, 1);
    mbar_init(dq_full, 1);
    mbar_init(dq_empty, 128);
    mbar_init(dkv_full, 1);
    // the 128-byte swizzle needs a 1024-byte aligned window; with the flag up no role loads or waits
    *abort_flag = (smem_u32(smem) & 1023u) ? 1 : 0;
    if (*abort_flag && p.status) atomicCAS(p.status, 0, TB_ERR_BAD_ARG);
    fence_barrier_init();
  }
  if (warp == 12) {
    tmem_alloc(tmem_ptr, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_ptr;
  const uint32_t lane_off = (uint32_t)((warp & 3) * 32) << 16;

  if (warp >= 12) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 104;");
    if (warp == 13) {
      // -------------------------------------------------------------- TMA producer
      if (elect_one() && !*abort_flag) {
        tma_prefetch_desc(&map_q);
        tma_prefetch_desc(&map_k);
        tma_prefetch_desc(&map_v);
        tma_prefetch_desc(&map_do);
        mbar_expect_tx(kv_full, 2 * L::TILE);
#pragma unroll
        for (int c = 0; c < KCH; ++c) {
          tma_load_4d(smem + L::K_OFF + c * 16384, &map_k, kv_full, c * 64, h, kv0, b);
          tma_load_4d(smem + L::V_OFF + c * 16384, &map_v, kv_full, c * 64, h, kv0, b);
        }
        for (int t = 0; t < n_it; ++t) {
          const int s = t & 1, sd = t % DOST;
          const int qrow0 = (i0 + t) * 128;
          // once a wait has given up, nothing more is loaded: loads without a free slot would pile transaction counts
          // on one barrier beyond its range
          if (!mbar_wait(&q_empty[s], ((t >> 1) & 1) ^ 1, abort_flag, p.status, TB_ERR_WAIT_EMPTY)) break;
          mbar_expect_tx(&q_full[s], L::TILE);
#pragma unroll
          for (int c = 0; c < KCH; ++c)
            tma_load_4d(smem + L::Q_OFF + s * L::TILE + c * 16384, &map_q, &q_full[s], c * 64, h, qrow0, b);
          if (!mbar_wait(&do_empty[sd], ((t / DOST) & 1) ^ 1, abort_flag, p.status, TB_ERR_WAIT_EMPTY)) break;
          mbar_expect_tx(&do_full[sd], L::TILE);
#pragma unroll
          for (int c = 0; c < KCH; ++c)
            tma_load_4d(smem + L::DO_OFF + sd * L::TILE + c * 16384, &map_do, &do_full[sd], c * 64, h, qrow0, b);
        }
        if (*abort_flag) {
          uint64_t t0 = globaltimer_ns();
          while (globaltimer_ns() - t0 < 2000000ull) {
          }
        }
      }
    } else if (warp == 14) {
      // -------------------------------------------------------------- L and delta rows
      for (int t = 0; t < n_it; ++t) {
        const int s = t & 1, q = (i0 + t) * 128 + lane * 4;
        float* ld = reinterpret_cast<float*>(smem + L::LD_OFF) + s * 256;
        const size_t at = ((size_t)b * p.H + h) * p.S + q;
        float lv[4], dv[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {   // queries beyond S: exp2(s - inf) = 0
          lv[j] = q + j < p.S ? p.LSE[at + j] * -1.4426950408889634f : -INFINITY;
          dv[j] = q + j < p.S ? p.delta[at + j] * -p.scale : 0.f;
        }
        mbar_wait(&ld_empty[s], ((t >> 1) & 1) ^ 1, abort_flag, p.status, TB_ERR_WAIT_EMPTY);
        *reinterpret_cast<float4*>(ld + lane * 4) = make_float4(lv[0], lv[1], lv[2], lv[3]);
        *reinterpret_cast<float4*>(ld + 128 + lane * 4) = make_float4(dv[0], dv[1], dv[2], dv[3]);
        mbar_arrive(&ld_full[s]);
      }
    } else if (warp == 12) {
      // -------------------------------------------------------------- MMA issuer
      if (elect_one()) {
        constexpr uint32_t idesc_s = make_idesc_bf16(128, 128, 0, 0);
        constexpr uint32_t idesc_kv = make_idesc_bf16(128, D, 0, 1);   // dV, dK: A K-major (TMEM / smem), B MN-major
        constexpr uint32_t idesc_dq = make_idesc_bf16(128, D, 1, 1);
        const uint32_t k_base = smem_u32(smem + L::K_OFF), v_base = smem_u32(smem + L::V_OFF);
        const uint32_t q_base = smem_u32(smem + L::Q_OFF), do_base = smem_u32(smem + L::DO_OFF);
        const uint32_t ds_base = smem_u32(smem + L::DS_OFF);
        const uint64_t k_kd = make_smem_desc_sw128(k_base, 16, 1024), k_mn = make_smem_desc_sw128(k_base, 16384, 1024);
        const uint64_t v_kd = make_smem_desc_sw128(v_base, 16, 1024);
        const uint64_t q_kd = make_smem_desc_sw128(q_base, 16, 1024), q_mn = make_smem_desc_sw128(q_base, 16384, 1024);
        const uint64_t do_kd = make_smem_desc_sw128(do_base, 16, 1024), do_mn = make_smem_desc_sw128(do_base, 16384, 1024);
        const uint64_t ds_kd = make_smem_desc_sw128(ds_base, 16, 1024), ds_mn = make_smem_desc_sw128(ds_base, 16384, 1024);
        auto issue_s = [&](int t) {   // S^T = K Q_t^T
          const uint32_t so = (t & 1) * L::TILE;
          mbar_wait(&q_full[t & 1], (t >> 1) & 1, abort_flag, p.status, TB_ERR_WAIT_FULL);
          tc_fence_after();
#pragma unroll
          for (int c = 0; c < KCH; ++c)
#pragma unroll
            for (int k = 0; k < 4; ++k)
              umma_ss(tmem_base + TM_S, desc_at(k_kd, c * 16384 + k * 32), desc_at(q_kd, so + c * 16384 + k * 32), idesc_s,
                      (c | k) ? 1u : 0u);
          umma_commit(s_full);
        };
        auto issue_dp = [&](int t) {  // dP^T = V dO_t^T; its columns were read before ds_full[t - 1]
          const uint32_t sdo = (t % DOST) * L::TILE;
          mbar_wait(&do_full[t % DOST], (t / DOST) & 1, abort_flag, p.status, TB_ERR_WAIT_FULL);
          tc_fence_after();
#pragma unroll
          for (int c = 0; c < KCH; ++c)
#pragma unroll
            for (int k = 0; k < 4; ++k)
              umma_ss(tmem_base + TM_DP, desc_at(v_kd, c * 16384 + k * 32), desc_at(do_kd, sdo + c * 16384 + k * 32), idesc_s,
                      (c | k) ? 1u : 0u);
          umma_commit(dp_full);
        };
        mbar_wait(kv_full, 0, abort_flag, p.status, TB_ERR_WAIT_FULL);
        issue_s(0);
        issue_dp(0);
        for (int t = 0; t < n_it; ++t) {
          const uint32_t so = (t & 1) * L::TILE, sdo = (t % DOST) * L::TILE;
          mbar_wait(p_full, t & 1, abort_flag, p.status, TB_ERR_WAIT_MISC);
          if (ROOMY && t + 1 < n_it) issue_s(t + 1);   // S^T[t] has been read
          tc_fence_after();
#pragma unroll
          for (int kk = 0; kk < 8; ++kk)   // dV += P^T dO_t
            umma_ts(tmem_base + TM_DV, tmem_base + TM_P + (kk >> 2) * P_HALF + (kk & 3) * 8, desc_at(do_mn, sdo + kk * 2048), idesc_kv,
                    (t | kk) ? 1u : 0u);
          umma_commit(dv_done);
          umma_commit(&do_empty[t % DOST]);
          if (!ROOMY && t + 1 < n_it) {
            mbar_wait(dv_done, t & 1, abort_flag, p.status, TB_ERR_WAIT_MISC);  // P^T[t] is no longer read
            issue_s(t + 1);
          }
          mbar_wait(ds_full, t & 1, abort_flag, p.status, TB_ERR_WAIT_MISC);
          if (ROOMY && t + 1 < n_it) issue_dp(t + 1);
          if (ROOMY && t > 0) mbar_wait(dq_empty, (t - 1) & 1, abort_flag, p.status, TB_ERR_WAIT_TMEM_EMPTY);
          tc_fence_after();
#pragma unroll
          for (int kk = 0; kk < 8; ++kk)   // dQ before dK: its way out is the longer one
            umma_ss(tmem_base + TM_DQ, desc_at(ds_mn, kk * 2048), desc_at(k_mn, kk * 2048), idesc_dq, kk ? 1u : 0u);
          umma_commit(dq_full);
#pragma unroll
          for (int kk = 0; kk < 8; ++kk)
            umma_ss(tmem_base + TM_DK, desc_at(ds_kd, (kk >> 2) * 16384 + (kk & 3) * 32), desc_at(q_mn, so + kk * 2048), idesc_kv,
                    (t | kk) ? 1u : 0u);
          umma_commit(ds_empty);
          umma_commit(&q_empty[t & 1]);
          if (!ROOMY && t + 1 < n_it) {
            mbar_wait(dq_empty, t & 1, abort_flag, p.status, TB_ERR_WAIT_TMEM_EMPTY);
            issue_dp(t + 1);
          }
        }
        umma_commit(dkv_full);
      }
    }
  } else if (warp >= 8) {
    // ---------------------------------------------------------------- dQ out (4 warps, one TMEM lane quarter each)
    asm volatile("setmaxnreg.dec.sync.aligned.u32 88;");
    // A warp's rows leave as one 4 KB bulk reduce-add per 32 columns; the accumulator keeps the staged order (the cast
    // pass undoes it). As 16-byte reductions of every lane into its own row they reached 1.1 to 1.5 TB/s of L2.
    uint8_t* stage = smem + L::DQ_OFF + (warp & 3) * 8192;
    const int sw = lane & 7;
    for (int t = 0; t < n_it; ++t) {
      mbar_wait(dq_full, t & 1, abort_flag, p.status, TB_ERR_WAIT_TMEM_FULL);
      tc_fence_after();
#pragma unroll
      for (int c = 0; c < D / 32; c += 2) {
        // both columns groups to registers first: with the last pair the columns are free before anything is staged
        uint32_t v[2][32];
        tmem_ld32(tmem_base + TM_DQ + c * 32 + lane_off, v[0]);
        tmem_ld32(tmem_base + TM_DQ + c * 32 + 32 + lane_off, v[1]);
        tmem_wait_ld();
        if (c == D / 32 - 2) {
          tc_fence_before();
          mbar_arrive(dq_empty);
        }
        if (lane == 0) bulk_wait_read_all();  // the previous pair has left the staging rows
        __syncwarp();
#pragma unroll
        for (int k = 0; k < 2; ++k)
#pragma unroll
          for (int g = 0; g < 8; ++g)
            *reinterpret_cast<uint4*>(stage + k * 4096 + lane * 128 + ((g ^ sw) << 4)) =
                make_uint4(v[k][g * 4], v[k][g * 4 + 1], v[k][g * 4 + 2], v[k][g * 4 + 3]);
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) {
          // worked out here and not once per block: held across the block, the row count and the pointer cost the compute warps
          // registers (D = 128: spills, 0.5 to 1.5 us of a launch)
          const int row0 = (i0 + t) * 128 + (warp & 3) * 32, rows = min(32, p.S - row0);
          float* dq_grp = p.dQ_acc + ((size_t)bh * p.S + row0) * D;
          if (rows > 0) {   // else nothing of this warp's quarter is in the sequence
#pragma unroll
            for (int k = 0; k < 2; ++k)
              asm volatile("cp.reduce.async.bulk.global.shared::cta.bulk_group.add.f32 [%0], [%1], %2;" ::"l"(dq_grp + (c + k) * rows * 32),
                           "r"(smem_u32(stage + k * 4096)), "r"(rows * 128)
                           : "memory");
          }
          bulk_commit();
        }
      }
    }
    if (lane == 0) bulk_wait_all();
  } else {
    // ---------------------------------------------------------------- compute (8 warps)
    // Two warps per group of 32 key rows: warps 0-3 take queries 0-63 of every block (and the first half of the dK / dV
    // columns at the end), warps 4-7 the rest; no exchange is needed, L and delta are per query.
    asm volatile("setmaxnreg.inc.sync.aligned.u32 160;");
    const int half = warp >> 2;
    const int row = (warp & 3) * 32 + lane;
    const int key = kv0 + row;
    const float sl2 = p.scale * 1.4426950408889634f;
    uint8_t* ds_row = smem + L::DS_OFF + half * 16384 + row * 128;
    const int sw = row & 7;
    const uint32_t tp = tmem_base + TM_P + half * P_HALF + lane_off;
    const uint32_t ts = tmem_base + TM_S + half * 64 + lane_off, tdp = tmem_base + TM_DP + half * 64 + lane_off;
    for (int t = 0; t < n_it; ++t) {
      const float* ld = reinterpret_cast<const float*>(smem + L::LD_OFF) + (t & 1) * 256 + half * 64;
      const bool need_mask = (p.causal && t == 0) || kv0 + 128 > p.S;   // with a causal mask block 0 is the diagonal one
      // first query (relative to this half) that sees the key: none for a key beyond S
      const int first = key >= p.S ? 1 << 30 : p.causal ? key - ((i0 + t) * 128 + half * 64) : 0;
      float e0[32], e1[32];
      uint32_t v0[32], v1[32], pk[16];
      mbar_wait(&ld_full[t & 1], (t >> 1) & 1, abort_flag, p.status, TB_ERR_WAIT_FULL);
      mbar_wait(s_full, t & 1, abort_flag, p.status, TB_ERR_WAIT_TMEM_FULL);
      tc_fence_after();
      // all 64 scores at once: the load's latency is paid once, and P^T may land on the same half's columns
      tmem_ld32(ts, v0);
      tmem_ld32(ts + 32, v1);
      tmem_wait_ld();
      if (need_mask) fa_bwd_p<true>(v0, ld, sl2, first, e0, pk);
      else fa_bwd_p<false>(v0, ld, sl2, first, e0, pk);
      if (ROOMY && t > 0) mbar_wait(dv_done, (t - 1) & 1, abort_flag, p.status, TB_ERR_WAIT_TMEM_EMPTY);  // P^T[t - 1] is read
      tmem_st16(tp, pk);
      if (need_mask) fa_bwd_p<true>(v1, ld + 32, sl2, first - 32, e1, pk);
      else fa_bwd_p<false>(v1, ld + 32, sl2, first - 32, e1, pk);
      tmem_st16(tp + 16, pk);
      tmem_wait_st();
      tc_fence_before();
      mbar_arrive(p_full);
      mbar_wait(dp_full, t & 1, abort_flag, p.status, TB_ERR_WAIT_TMEM_FULL);
      tc_fence_after();
      tmem_ld32(tdp, v0);
      tmem_ld32(tdp + 32, v1);
      tmem_wait_ld();
      mbar_wait(ds_empty, (t & 1) ^ 1, abort_flag, p.status, TB_ERR_WAIT_EMPTY);  // dK / dQ of block t - 1 have read dS^T
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        fa_bwd_ds(c == 0 ? v0 : v1, ld + 128 + c * 32, p.scale, c == 0 ? e0 : e1, pk);
#pragma unroll
        for (int g = 0; g < 4; ++g)
          *reinterpret_cast<uint4*>(ds_row + (((c * 4 + g) ^ sw) << 4)) = make_uint4(pk[g * 4], pk[g * 4 + 1], pk[g * 4 + 2], pk[g * 4 + 3]);
      }
      fence_proxy_async_smem();
      tc_fence_before();
      mbar_arrive(ds_full);
      mbar_arrive(&ld_empty[t & 1]);
    }
    // dK, dV of this key block: thread = key row
    mbar_wait(dkv_full, 0, abort_flag, p.status, TB_ERR_WAIT_TMEM_FULL);
    tc_fence_after();
    const bool kv_ok = key < p.S;
    __nv_bfloat16* dk_row = p.dK + ((size_t)b * p.S + (kv_ok ? key : 0)) * p.dkv_stride + (size_t)h * D;
    __nv_bfloat16* dv_row = p.dV + ((size_t)b * p.S + (kv_ok ? key : 0)) * p.dkv_stride + (size_t)h * D;
#pragma unroll 1
    for (int c = half * (D / 64); c < (half + 1) * (D / 64); ++c) {
      uint32_t kvv[32], vvv[32];
      tmem_ld32(tmem_base + TM_DK + c * 32 + lane_off, kvv);
      tmem_ld32(tmem_base + TM_DV + c * 32 + lane_off, vvv);
      tmem_wait_ld();
      if (kv_ok) {
#pragma unroll
        for (int g = 0; g < 4; ++g) {
          uint4 a, d2;
          a.x = pack_bf16x2(__uint_as_float(kvv[g * 8 + 0]), __uint_as_float(kvv[g * 8 + 1]));
          a.y = pack_bf16x2(__uint_as_float(kvv[g * 8 + 2]), __uint_as_float(kvv[g * 8 + 3]));
          a.z = pack_bf16x2(__uint_as_float(kvv[g * 8 + 4]), __uint_as_float(kvv[g * 8 + 5]));
          a.w = pack_bf16x2(__uint_as_float(kvv[g * 8 + 6]), __uint_as_float(kvv[g * 8 + 7]));
          d2.x = pack_bf16x2(__uint_as_float(vvv[g * 8 + 0]), __uint_as_float(vvv[g * 8 + 1]));
          d2.y = pack_bf16x2(__uint_as_float(vvv[g * 8 + 2]), __uint_as_float(vvv[g * 8 + 3]));
          d2.z = pack_bf16x2(__uint_as_float(vvv[g * 8 + 4]), __uint_as_float(vvv[g * 8 + 5]));
          d2.w = pack_bf16x2(__uint_as_float(vvv[g * 8 + 6]), __uint_as_float(vvv[g * 8 + 7]));
          reinterpret_cast<uint4*>(dk_row + c * 32)[g] = a;
          reinterpret_cast<uint4*>(dv_row + c * 32)[g] = d2;
        }
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 12) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

// delta[b, h, s] = sum_d O[b, s, h, d] * dO[b, s, h, d]. Each thread reads one 16-byte vector of O
// and dO (8 elements); the D/8 lanes of a (token, head) pair combine with shuffles.
template <int D>
__global__ void fa_delta_kernel(const __nv_bfloat16* __restrict__ O, const __nv_bfloat16* __restrict__ dO,
                                float* __restrict__ delta, int B, int S, int H, long o_stride, long do_stride) {
  constexpr int LPG = D / 8;  // lanes per (token, head)
  const long gid = (long)blockIdx.x * blockDim.x + threadIdx.x;
  const long pair = gid / LPG;
  const int sub = (int)(gid % LPG);
  const long total = (long)B * S * H;
  float s = 0.f;
  int hh = 0;
  long tok = 0;
  if (pair < total) {
    hh = (int)(pair % H);
    tok = pair / H;
    const uint4 a = *reinterpret_cast<const uint4*>(O + tok * o_stride + (long)hh * D + sub * 8);
    const uint4 c = *reinterpret_cast<const uint4*>(dO + tok * do_stride + (long)hh * D + sub * 8);
    const uint32_t aw[4] = {a.x, a.y, a.z, a.w}, cw[4] = {c.x, c.y, c.z, c.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) s += bf16_lo(aw[i]) * bf16_lo(cw[i]) + bf16_hi(aw[i]) * bf16_hi(cw[i]);
  }
#pragma unroll
  for (int off = LPG / 2; off > 0; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
  if (pair < total && sub == 0) {
    const long bb = tok / S, ss = tok % S;
    delta[(bb * H + hh) * S + ss] = s;
  }
}

// dQ: the fp32 accumulator's groups (layout at FaBwdParams::dQ_acc) -> bf16 rows. One thread per 8 columns of a row.
__global__ void fa_cvt_dq_kernel(const float* __restrict__ src, __nv_bfloat16* __restrict__ dst, int B, int S, int H, int D,
                                 long dst_stride) {
  const int vpr = D / 8;  // vectors per (token, head)
  const long total = (long)B * S * H * vpr;
  const long stride = (long)gridDim.x * blockDim.x;
  for (long idx = (long)blockIdx.x * blockDim.x + threadIdx.x; idx < total; idx += stride) {
    const int v = (int)(idx % vpr);
    const long th = idx / vpr;
    const int h = (int)(th % H);
    const long tok = th / H;
    const int b = (int)(tok / S), s = (int)(tok - (long)b * S);
    const int row = s & 31, c = v >> 2, g = (v & 3) * 2, rows = min(32, S - (s - row));
    const float* blk = src + (((size_t)b * H + h) * S + (s - row)) * D + (c * rows + row) * 32;
    const float4 x = *reinterpret_cast<const float4*>(blk + ((g ^ (row & 7)) << 2));
    const float4 y = *reinterpret_cast<const float4*>(blk + (((g + 1) ^ (row & 7)) << 2));
    *reinterpret_cast<uint4*>(dst + tok * dst_stride + (long)h * D + v * 8) =
        make_uint4(pack_bf16x2(x.x, x.y), pack_bf16x2(x.z, x.w), pack_bf16x2(y.x, y.y), pack_bf16x2(y.z, y.w));
  }
}

inline int make_bshd_map_bwd(CUtensorMap* m, const void* base, int B, int S, int H, int D, long row_stride) {
  uint64_t dims[4] = {(uint64_t)D, (uint64_t)H, (uint64_t)S, (uint64_t)B};
  uint64_t str[3] = {(uint64_t)D * 2, (uint64_t)row_stride * 2, (uint64_t)S * row_stride * 2};
  uint32_t box[4] = {64, 1, 128, 1};
  return make_tmap(m, base, 2, 4, dims, str, box);
}

}  // namespace tb
using namespace tb;

// Workspace (caller-provided, 16-byte aligned): delta fp32 [B*H*S], dq_acc fp32 [B*S*H*D] (zeroed here).
// dq, dk, dv: bf16 [B*S, dqkv_stride] with head h at column h*D (may be the three column bands of
// one fused dQKV buffer).
TB_EXPORT int tb_flash_attn_bwd(const void* q, const void* k, const void* v, const void* o, const void* dout,
                                const float* lse, void* dq, void* dk, void* dv, float* delta, float* dq_acc,
                                int B, int S, int H, int D, long q_stride, long kv_stride, long o_stride,
                                long do_stride, long dqkv_stride, float scale, int causal, int* status,
                                cudaStream_t st) {
  TB_ENSURE_DEVICE();
  if (!q || !k || !v || !o || !dout || !lse || !dq || !dk || !dv || !delta || !dq_acc)
    TB_FAIL(TB_E_ARG, "flash_attn_bwd: null pointer");
  if (D != 64 && D != 128) TB_FAIL(TB_E_ARG, "flash_attn_bwd: head dim %d not supported (64 or 128)", D);
  if ((dqkv_stride & 7) || ((uintptr_t)dq & 15) || ((uintptr_t)dk & 15) || ((uintptr_t)dv & 15))
    TB_FAIL(TB_E_ARG, "flash_attn_bwd: gradients must be 16-byte aligned");
  CUtensorMap mq, mk, mv, mdo;
  int r;
  if ((r = make_bshd_map_bwd(&mq, q, B, S, H, D, q_stride))) return r;
  if ((r = make_bshd_map_bwd(&mk, k, B, S, H, D, kv_stride))) return r;
  if ((r = make_bshd_map_bwd(&mv, v, B, S, H, D, kv_stride))) return r;
  if ((r = make_bshd_map_bwd(&mdo, dout, B, S, H, D, do_stride))) return r;
  if ((o_stride & 7) || (do_stride & 7) || ((uintptr_t)o & 15) || ((uintptr_t)dout & 15))
    TB_FAIL(TB_E_ARG, "flash_attn_bwd: o / dout must be 16-byte aligned with strides that are multiples of 8");
  const long nthreads = (long)B * S * H * (D / 8);
  if (D == 64)
    fa_delta_kernel<64><<<(unsigned)((nthreads + 255) / 256), 256, 0, st>>>((const __nv_bfloat16*)o, (const __nv_bfloat16*)dout, delta, B, S, H, o_stride, do_stride);
  else
    fa_delta_kernel<128><<<(unsigned)((nthreads + 255) / 256), 256, 0, st>>>((const __nv_bfloat16*)o, (const __nv_bfloat16*)dout, delta, B, S, H, o_stride, do_stride);
  TB_CUDA_CHECK(cudaMemsetAsync(dq_acc, 0, sizeof(float) * (size_t)B * S * H * D, st));
  FaBwdParams p{lse, delta, dq_acc, (__nv_bfloat16*)dk, (__nv_bfloat16*)dv, B, S, H, dqkv_stride, scale, causal, status};
  const int n_blk = (S + 127) / 128;
  const long grid = (long)n_blk * B * H;
  if (D == 64) {
    static std::atomic<uint64_t> opted_in{0};
    if (int e = smem_opt_in(opted_in, fa_bwd_kernel<64>, FaBwdSmem<64>::ALLOC)) return e;
    fa_bwd_kernel<64><<<(unsigned)grid, FB_THREADS, FaBwdSmem<64>::ALLOC, st>>>(mq, mk, mv, mdo, p);
  } else {
    static std::atomic<uint64_t> opted_in{0};
    if (int e = smem_opt_in(opted_in, fa_bwd_kernel<128>, FaBwdSmem<128>::ALLOC)) return e;
    fa_bwd_kernel<128><<<(unsigned)grid, FB_THREADS, FaBwdSmem<128>::ALLOC, st>>>(mq, mk, mv, mdo, p);
  }
  const long items = (long)B * S * H * (D / 8);
  int g = (int)((items + 255) / 256 < (long)sm_count() * 16 ? (items + 255) / 256 : (long)sm_count() * 16);
  fa_cvt_dq_kernel<<<g, 256, 0, st>>>(dq_acc, (__nv_bfloat16*)dq, B, S, H, D, dqkv_stride);
  TB_CUDA_CHECK(cudaGetLastError());
  return 0;
}
