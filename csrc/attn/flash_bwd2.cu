// Flash attention backward, transposed-score formulation (sm_100a, tcgen05 + TMEM).
// Same interface, scratch buffers and memory layouts as flash_bwd.cu.
//
// One CTA per (batch, kv head, 128-key tile); K and V stay in shared memory, Q / dO tiles of the
// query heads of the GQA group stream through two (d = 128) or four (d = 64) shared-memory stages, Q and
// dO with barriers of their own.  Scores are computed transposed, keys on the TMEM lanes, so that P^T and dS^T feed the dV / dK products straight
// from tensor memory:
//     A  S^T  = K Q^T             SS   -> R_S  [0,128)      (columns = queries)
//     B  dP^T = V dO^T            SS   -> R_dP [128,256)
//     C  P^T = exp2(S^T c - lse_q), dS^T = P^T (dP^T - delta_q) scale
//        bf16 P^T over R_S, bf16 dS^T over R_dP, dS^T also to shared memory
//     D  dV += P^T dO             TS (A = P^T from TMEM)     -> [256, 256+D)
//     E  dK += dS^T Q             TS (A = dS^T from TMEM)    -> [256+D, 256+2D)
//     F  dQ  = dS K               SS (A = dS^T tile in shared memory, M-major) -> R_dP again
//     G  dQ -> fp32 accumulator in global memory (red.global.add.v4.f32, one query row per thread)
// The issuer queues D E F of step i and A of step i+1 back to back (the tensor pipe runs in
// issue order, so A(i+1) may overwrite R_S right behind D(i)); only B(i+1) waits until G(i) has
// drained dQ out of R_dP.  The compute warps start the exponentials of step i+1 (needs S^T only)
// while B(i+1) is still running.
//
// Warps 0-7: compute (0-3: query columns 0-63, 4-7: columns 64-127; each warp covers 32 key
// lanes), warp 8: TMA producer, warp 9: MMA issuer + TMEM owner.
// With TRACE the first `trace_ctas` CTAs record (clock64, code) per warp at phase boundaries.
#include "../common/host.h"
#include "../common/ptx.cuh"
#include "attn_bwd_common.h"
#include <type_traits>

namespace zb {

constexpr int BWD2_WARPS = 10;
constexpr int BWD2_TRACE_EV = 256;

template <int D>
struct AttnBwd2Cfg {
  static constexpr int TILE_BYTES = 128 * D * 2;
  static constexpr int QS = D == 128 ? 2 : 4;       // Q / dO stages
  static constexpr int DS_BYTES = 128 * 128 * 2;
  static constexpr int SMEM_BYTES = 2 * TILE_BYTES + QS * 2 * TILE_BYTES + DS_BYTES + 1024 + 256;
  static constexpr int TMEM_COLS = 512;
  static constexpr int DP_COL = 128, DV_COL = 256, DK_COL = 256 + D;
  static constexpr int S1_COL = 384;                // D = 64: second S^T buffer
};

enum : int {
  TB_S_READY = 1, TB_P_DONE = 2, TB_DP_READY = 3, TB_DS_DONE = 4, TB_DQ_READY = 5, TB_DQ_DRAINED = 6,
  TB_MMA_QDO_READY = 16, TB_MMA_PDS_READY = 17, TB_MMA_DEF_ISSUED = 18, TB_MMA_A_ISSUED = 19, TB_MMA_DQ_EMPTY = 20,
  TB_MMA_B_ISSUED = 21,
  TB_TMA_STAGE_FREE = 32, TB_TMA_ISSUED = 33,
};

__device__ __forceinline__ void red_add_v4_f32(float* p, float a, float b, float c, float d) {
  asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(p), "f"(a), "f"(b), "f"(c), "f"(d)
               : "memory");
}

__device__ __forceinline__ void red_add_f32(float* p, float a) {
  asm volatile("red.global.add.f32 [%0], %1;" ::"l"(p), "f"(a) : "memory");
}

__device__ __forceinline__ void cluster_barrier() {   // every thread of every CTA of the cluster
  asm volatile("barrier.cluster.arrive.release;\nbarrier.cluster.wait.acquire;" ::: "memory");
}
// the word at the same shared-memory offset in CTA `cta` of the cluster
__device__ __forceinline__ uint32_t ld_cluster_u32(uint32_t addr, uint32_t cta) {
  uint32_t ra, v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(ra) : "r"(addr), "r"(cta));
  asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(v) : "r"(ra) : "memory");
  return v;
}
__device__ __forceinline__ float ld_cluster_f32(uint32_t addr, uint32_t cta) {
  return __uint_as_float(ld_cluster_u32(addr, cta));
}

// DQ = false: the key-tile half of the two-kernel backward (dK and dV only): no dS^T copy in shared memory,
// no dQ product and no atomics; dQ then comes from flash_bwd_dq.cu.
// CL > 1 (DQ = false): a cluster of CL CTAs shares a key tile, each taking its part of the query heads of the GQA group;
// the fp32 sums are added up through distributed shared memory, in rank order, at the end.  One CTA per key tile leaves
// 2048 tokens with 8 kv heads at 128 CTAs of 4 to 64 steps: the time is that of the longest.
template <int D, bool TRACE, bool DQ, int CL>
__global__ void __launch_bounds__(32 * BWD2_WARPS, 1)
flash_bwd2_kernel(const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ CUtensorMap tmap_k,
                  const __grid_constant__ CUtensorMap tmap_v, const __grid_constant__ CUtensorMap tmap_do,
                  const __grid_constant__ CUtensorMap tmap_dk, const __grid_constant__ CUtensorMap tmap_dv,
                  const AttnBwdParams p, const float* stats, int s_pad,
                  unsigned long long* trace, int trace_ctas) {
  using Cfg = AttnBwd2Cfg<D>;
  constexpr int BM = 128, BN = 128, QS = Cfg::QS, DB = D / 64;
  // With d = 64 tensor memory has room for a second S^T (without the dQ part): the scores of the next step are then formed
  // ahead of this step's P^T, and the compute warps go from one step's dS^T to the next step's exponentials without
  // waiting for dV and S^T.  32 / 8 heads of 8192 tokens 718 -> 660 us, 2 x 4096 tokens 398 -> 365 (statistics included).
  constexpr int NSB = (D == 64 && !DQ) ? 2 : 1;
  constexpr int BLK = 128 * 128;  // bytes of one [128 rows x 64 cols] bf16 block
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sK = smem;
  uint8_t* sV = sK + Cfg::TILE_BYTES;
  uint8_t* sQ = sV + Cfg::TILE_BYTES;                 // QS tiles
  uint8_t* sDO = sQ + QS * Cfg::TILE_BYTES;           // QS tiles
  uint8_t* sDS = sDO + QS * Cfg::TILE_BYTES;          // dS^T: [128 keys][128 queries], two 64-query blocks
  uint64_t* bars = reinterpret_cast<uint64_t*>(sDS + Cfg::DS_BYTES);
  uint64_t* k_full = bars;              // 1
  uint64_t* v_full = bars + 1;          // 1
  uint64_t* q_full = bars + 2;          // QS
  uint64_t* q_empty = q_full + QS;      // QS
  uint64_t* do_full = q_empty + QS;     // QS
  uint64_t* do_empty = do_full + QS;    // QS
  uint64_t* s_full = do_empty + QS;     // NSB
  uint64_t* dp_full = s_full + NSB;     // 1
  uint64_t* pds_full = dp_full + 1;     // 1 (8 arrivals)
  uint64_t* dq_full = pds_full + 1;     // 1
  uint64_t* dq_empty = dq_full + 1;     // 1 (8 arrivals)
  uint64_t* p_full = dq_empty;          // without the dQ part: P^T is in tensor memory, one barrier per score buffer
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(dq_empty + NSB);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // grid = (kv heads, key tiles, batch): x-fastest dispatch starts every head's heaviest key tile
  // (tile 0 sees all query tiles under a causal mask) before any light one
  const int jt = blockIdx.y, kv_head = blockIdx.x / CL, batch = blockIdx.z;
  const int cl_rank = blockIdx.x % CL;      // rank in the cluster
  const int kv0 = jt * BN;
  const int rep = p.Hq / p.Hkv / CL;        // query heads this CTA walks over
  const int head0 = kv_head * (p.Hq / p.Hkv) + cl_rank * rep;
  const int n_qt = (p.S + BM - 1) / BM;
  const int i_lo = p.causal ? (kv0 / BM) : 0;
  int i_hi = n_qt;
  if (p.window > 0) i_hi = min(n_qt, (kv0 + BN - 1 + p.window - 1) / BM + 1);
  const int per_head = max(i_hi - i_lo, 0);
  const int n_iters = per_head * rep;
  WaitCtx wctx{abort_flag, p.status};

  const int cta_lin = int(blockIdx.x) + int(gridDim.x) * (int(blockIdx.y) + int(gridDim.y) * int(blockIdx.z));
  unsigned long long* tr_buf = nullptr;
  int tr_n = 0;
  if (TRACE && trace != nullptr && cta_lin < trace_ctas && lane == 0)
    tr_buf = trace + (size_t(cta_lin) * BWD2_WARPS + warp) * BWD2_TRACE_EV;
  auto tr = [&](int code) {
    if (TRACE) {
      if (tr_buf != nullptr && tr_n < BWD2_TRACE_EV)
        tr_buf[tr_n++] = (static_cast<unsigned long long>(clock64()) << 8) | static_cast<unsigned long long>(code);
    }
  };

  if (threadIdx.x == 0) {
    *abort_flag = 0;
    mbar_init(k_full, 1);
    mbar_init(v_full, 1);
    for (int i = 0; i < QS; ++i) {
      mbar_init(&q_full[i], 1);
      mbar_init(&q_empty[i], 1);
      mbar_init(&do_full[i], 1);
      mbar_init(&do_empty[i], 1);
    }
    for (int i = 0; i < NSB; ++i) mbar_init(&s_full[i], 1);
    mbar_init(dp_full, 1);
    mbar_init(pds_full, 8);
    mbar_init(dq_full, 1);
    for (int i = 0; i < NSB; ++i) mbar_init(&dq_empty[i], 8);
    mbar_fence_init();
  }
  if (warp == 9) {
    tmem_alloc(tmem_slot, Cfg::TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  if constexpr (!DQ) {
    chain_wait();
    chain_trigger();   // behind the wait: the dQ kernel starts on this, under the last CTAs here (chain_late in ptx.cuh)
  }

  if (warp == 8) {
    // ------------------------------ TMA producer ------------------------------
    if (lane == 0) {
      tma_prefetch_desc(&tmap_q);
      tma_prefetch_desc(&tmap_k);
      tma_prefetch_desc(&tmap_v);
      tma_prefetch_desc(&tmap_do);
      // K and the first Q are all that the first scores need: they go ahead of V and dO (nobody waits for them without a
      // step, and a copy must not outlive the CTA)
      auto load_kv = [&](uint8_t* dst, const CUtensorMap* tm, uint64_t* bar) {
        mbar_expect_tx(bar, Cfg::TILE_BYTES);
#pragma unroll
        for (int b = 0; b < DB; ++b) tma_load_4d(dst + b * BLK, tm, bar, b * 64, kv_head, kv0, batch);
      };
      if (n_iters > 0) load_kv(sK, &tmap_k, k_full);
      int head = head0, qt = i_lo;
      for (int it = 0; it < n_iters; ++it) {
        const int st = it % QS;
        const uint32_t ph = uint32_t(it / QS) & 1;
        const int q0 = qt * BM;
        if (!zb_in_bounds(q0 >= 0 && q0 < p.S && head < p.Hq && kv0 < p.S, p.status, 8)) break;
        // Q and dO have their own barriers: dO_i is free once dV_i is done, Q_i only after dK_i, more than half a step
        // later, and the first S^T needs Q alone
        auto load_q = [&]() -> bool {
          if (!mbar_wait(&q_empty[st], ph ^ 1, wctx, ST_TIMEOUT_EMPTY)) return false;
          tr(TB_TMA_STAGE_FREE);
          mbar_expect_tx(&q_full[st], Cfg::TILE_BYTES + (DQ ? 0 : 1024));
#pragma unroll
          for (int b = 0; b < DB; ++b)
            tma_load_4d(sQ + st * Cfg::TILE_BYTES + b * BLK, &tmap_q, &q_full[st], b * 64, head, q0, batch);
          if constexpr (!DQ) {
            // -lse (log2 units) and -delta of the tile's 128 queries: 512 bytes each, freed with Q_i, that is after
            // every compute warp has formed dS_i (rows of the statistics buffer are padded to a multiple of 128
            // entries, q0 is a multiple of 128)
            const float* row = stats + (size_t(batch) * p.Hq + head) * 2 * size_t(s_pad) + q0;
            bulk_load_1d(sDS + st * 1024, row, 512, &q_full[st]);
            bulk_load_1d(sDS + st * 1024 + 512, row + s_pad, 512, &q_full[st]);
          }
          return true;
        };
        auto load_do = [&]() -> bool {
          if (!mbar_wait(&do_empty[st], ph ^ 1, wctx, ST_TIMEOUT_EMPTY)) return false;
          mbar_expect_tx(&do_full[st], Cfg::TILE_BYTES);
#pragma unroll
          for (int b = 0; b < DB; ++b)
            tma_load_4d(sDO + st * Cfg::TILE_BYTES + b * BLK, &tmap_do, &do_full[st], b * 64, head, q0, batch);
          return true;
        };
        if (it == 0) {
          if (!load_q()) break;
          load_kv(sV, &tmap_v, v_full);
          if (!load_do()) break;
        } else if (it < QS ? !(load_q() && load_do()) : !(load_do() && load_q())) {
          break;
        }
        tr(TB_TMA_ISSUED);
        if (++qt == i_hi) { qt = i_lo; ++head; }
      }
    }
  } else if (warp == 9) {
    // ------------------------------ MMA issuer ------------------------------
    // The whole warp walks the loop, one elected lane issues (operands stay in uniform registers).  With that, P^T
    // announced ahead of dS^T and fp32 P in registers the dK / dV kernel and the statistics take, for 4096 tokens, 32
    // heads, d = 128, 272 instead of 390 us, and for 2048 tokens, 32 / 8 heads, d = 64, 108 instead of 181 us with one CTA
    // per key tile (clocks per step of the first: 1460 exponentials, 630 dS^T, 1020 waiting for S^T and dP^T; the tensor
    // pipe is busy for about 2260 of 3110).
    if (n_iters > 0) {
      const bool elected = elect_one();
      constexpr uint32_t idesc_s = umma_idesc_bf16(128, 128, false, false);  // K-major A and B
      constexpr uint32_t idesc_dkv = umma_idesc_bf16(128, D, false, true);   // A from TMEM, B = [q rows][d] (N-major)
      // D = 128: A = K (M = head dim, M-major), B = dS^T tile (N = queries, N-major); D = 64: A = dS^T tile, B = K
      constexpr uint32_t idesc_dq = umma_idesc_bf16(128, D == 128 ? 128 : D, true, true);
      const uint32_t k_addr = smem_u32(sK), v_addr = smem_u32(sV), ds_addr = smem_u32(sDS);
      const uint32_t r_dp = tmem_base + Cfg::DP_COL;
      auto r_s = [&](int it) { return tmem_base + (NSB == 2 && (it & 1) ? uint32_t(Cfg::S1_COL) : 0u); };
      bool ok = mbar_wait_warp(k_full, 0, wctx, ST_TIMEOUT_FULL);
      auto issue_a = [&](int it) {  // S^T = K Q^T
        if (elected) {
          const uint32_t q_addr = smem_u32(sQ + (it % QS) * Cfg::TILE_BYTES), d = r_s(it);
#pragma unroll
          for (int kk = 0; kk < D / 16; ++kk) {
            const uint32_t off = uint32_t(kk / 4) * BLK + uint32_t(kk % 4) * 32;
            umma_f16_ss(d, umma_desc_kmajor(k_addr + off), umma_desc_kmajor(q_addr + off), idesc_s, kk != 0 ? 1u : 0u);
          }
          umma_commit(&s_full[it % NSB]);
        }
        __syncwarp();
      };
      auto issue_b = [&](uint32_t do_addr) {  // dP^T = V dO^T
        if (elected) {
#pragma unroll
          for (int kk = 0; kk < D / 16; ++kk) {
            const uint32_t off = uint32_t(kk / 4) * BLK + uint32_t(kk % 4) * 32;
            umma_f16_ss(r_dp, umma_desc_kmajor(v_addr + off), umma_desc_kmajor(do_addr + off), idesc_s, kk != 0 ? 1u : 0u);
          }
          umma_commit(dp_full);
        }
        __syncwarp();
      };
      if (ok) ok = mbar_wait_warp(&q_full[0], 0, wctx, ST_TIMEOUT_FULL);
      if (ok) {
        tc_fence_after();
        issue_a(0);
        ok = mbar_wait_warp(v_full, 0, wctx, ST_TIMEOUT_FULL);
      }
      if (ok) ok = mbar_wait_warp(&do_full[0], 0, wctx, ST_TIMEOUT_FULL);
      if (ok) {
        tc_fence_after();
        issue_b(smem_u32(sDO));
        tr(TB_MMA_B_ISSUED);
      }
      for (int it = 0; it < n_iters && ok; ++it) {
        const int st = it % QS;
        const uint32_t q_addr = smem_u32(sQ + st * Cfg::TILE_BYTES), do_addr = smem_u32(sDO + st * Cfg::TILE_BYTES);
        if (NSB == 2 && it + 1 < n_iters) {   // its buffer last held P^T of step it - 1, read by the D queued before this
          const int sn = (it + 1) % QS;
          if (!mbar_wait_warp(&q_full[sn], uint32_t((it + 1) / QS) & 1, wctx, ST_TIMEOUT_FULL)) break;
          tr(TB_MMA_QDO_READY);
          tc_fence_after();
          issue_a(it + 1);
          tr(TB_MMA_A_ISSUED);
        }
        // With two score buffers the compute warps may announce P^T of step it + 1 before this wait has seen that of step
        // it (their next scores are there already), so each buffer has a barrier of its own: the next phase of this one
        // needs S^T of step it + 2, which is only issued behind this wait.
        if (!mbar_wait_warp(DQ ? pds_full : &p_full[it % NSB], uint32_t(DQ ? it : it / NSB) & 1, wctx, ST_TIMEOUT_MISC)) break;
        if (DQ) tr(TB_MMA_PDS_READY);
        tc_fence_after();
        // D: dV += P^T dO, E: dK += dS^T Q  (reduction over the 128 queries; bf16 A operands sit in the
        // first 32 columns of each 64-column half of R_S / R_dP)
        if (elected) {
#pragma unroll
          for (int kk = 0; kk < BM / 16; ++kk) {
            const uint32_t acol = uint32_t(kk / 4) * 64 + uint32_t(kk % 4) * 8;
            umma_f16_ts(tmem_base + Cfg::DV_COL, r_s(it) + acol, umma_desc_mnmajor(do_addr + kk * 2048, BLK), idesc_dkv,
                        (it | kk) != 0 ? 1u : 0u);
          }
          umma_commit(&do_empty[st]);     // B_i and D_i are dO_i's readers
        }
        __syncwarp();
        if constexpr (!DQ) {
          // D needs P^T only, and S^T of the next step goes right behind it (D was P^T's last reader): both run while
          // the compute warps form dS^T, and the next step's exponentials run under E and B
          if (NSB == 1 && it + 1 < n_iters) {
            const int sn = (it + 1) % QS;
            if (!mbar_wait_warp(&q_full[sn], uint32_t((it + 1) / QS) & 1, wctx, ST_TIMEOUT_FULL)) break;
            tr(TB_MMA_QDO_READY);
            tc_fence_after();
            issue_a(it + 1);
            tr(TB_MMA_A_ISSUED);
          }
          if (!mbar_wait_warp(pds_full, uint32_t(it) & 1, wctx, ST_TIMEOUT_MISC)) break;
          tr(TB_MMA_PDS_READY);
          tc_fence_after();
        }
        if (elected) {
#pragma unroll
          for (int kk = 0; kk < BM / 16; ++kk) {
            const uint32_t acol = uint32_t(kk / 4) * 64 + uint32_t(kk % 4) * 8;
            umma_f16_ts(tmem_base + Cfg::DK_COL, r_dp + acol, umma_desc_mnmajor(q_addr + kk * 2048, BLK), idesc_dkv,
                        (it | kk) != 0 ? 1u : 0u);
          }
          umma_commit(&q_empty[st]);
        }
        __syncwarp();
        if constexpr (!DQ) {
          if (it + 1 == n_iters && elected) umma_commit(dq_full);   // every dK / dV product is done: the write-out may start
          __syncwarp();
          tr(TB_MMA_DEF_ISSUED);
          if (it + 1 < n_iters) {
            const int sn = (it + 1) % QS;
            if (!mbar_wait_warp(&do_full[sn], uint32_t((it + 1) / QS) & 1, wctx, ST_TIMEOUT_FULL)) break;
            tc_fence_after();
            issue_b(smem_u32(sDO + sn * Cfg::TILE_BYTES));   // overwrites R_dP behind E, its last reader
            tr(TB_MMA_B_ISSUED);
          }
          continue;
        }
        if constexpr (DQ) {
        // F: dQ = dS K  (reduction over the 128 keys) into R_dP, right behind E which read dS^T from it.
        // For D = 128 the product is formed transposed, dQ^T = K^T dS^T (same two shared-memory tiles with
        // the operand roles swapped): head-dim index on the TMEM lanes, so that the 32 lanes of a warp add
        // to 32 consecutive floats of one query row (one full 128-byte line per instruction) in G.
        if (elected) {
#pragma unroll
          for (int kk = 0; kk < BN / 16; ++kk) {
            if constexpr (D == 128)
              umma_f16_ss(r_dp, umma_desc_mnmajor(k_addr + kk * 2048, BLK), umma_desc_mnmajor(ds_addr + kk * 2048, BLK),
                          idesc_dq, kk != 0 ? 1u : 0u);
            else
              umma_f16_ss(r_dp, umma_desc_mnmajor(ds_addr + kk * 2048, BLK), umma_desc_mnmajor(k_addr + kk * 2048, BLK),
                          idesc_dq, kk != 0 ? 1u : 0u);
          }
          umma_commit(dq_full);
        }
        __syncwarp();
        }
        tr(TB_MMA_DEF_ISSUED);
        if (it + 1 < n_iters) {
          const int sn = (it + 1) % QS;
          if (!mbar_wait_warp(&q_full[sn], uint32_t((it + 1) / QS) & 1, wctx, ST_TIMEOUT_FULL)) break;
          if (!mbar_wait_warp(&do_full[sn], uint32_t((it + 1) / QS) & 1, wctx, ST_TIMEOUT_FULL)) break;
          tr(TB_MMA_QDO_READY);
          tc_fence_after();
          issue_a(it + 1);
          tr(TB_MMA_A_ISSUED);
          if constexpr (DQ) {
            // dQ_it sits in R_dP until the compute warps have drained it
            if (!mbar_wait_warp(dq_empty, uint32_t(it) & 1, wctx, ST_TIMEOUT_TMEM_EMPTY)) break;
            tr(TB_MMA_DQ_EMPTY);
            tc_fence_after();
          }
          issue_b(smem_u32(sDO + sn * Cfg::TILE_BYTES));
          tr(TB_MMA_B_ISSUED);
        }
      }
    }
  } else {
    // ------------------------------ compute warps ------------------------------
    const int half = warp >> 2;                  // which 64 query columns of S^T / dP^T (C), which d half (G, final)
    const int t = (warp & 3) * 32 + lane;        // TMEM lane: key row (C, final write), query row (G)
    const uint32_t lane_addr = tmem_base + (uint32_t((warp & 3) * 32) << 16);
    const int key = kv0 + t;
    const bool key_ok = key < p.S;
    uint8_t* ds_row = sDS + half * BLK + t * 128;  // this thread's 128-byte row of its 64-query block
    bool ok = true;
    int head = head0, qt = i_lo - 1;   // (counted along: two divisions per step otherwise)
    for (int it = 0; it < n_iters; ++it) {
      if (++qt == i_hi) { qt = i_lo; ++head; }
      const int q0 = qt * BM;
      const int qc0 = q0 + half * 64;            // first query column of this thread
      // statistics of the tile's queries: global rows indexed by the absolute query (one-kernel form), or the
      // copy the producer placed in shared memory with the stage
      const float* lse_q = stats + (size_t(batch) * p.Hq + head) * 2 * size_t(s_pad);
      const float* delta_q = lse_q + s_pad;
      const uint32_t nlse_s = smem_u32(sDS + (it % QS) * 1024 + half * 256), ndelta_s = nlse_s + 512;
      if constexpr (!DQ) {
        if (!__all_sync(0xffffffffu, mbar_wait(&q_full[it % QS], uint32_t(it / QS) & 1, wctx, ST_TIMEOUT_FULL))) { ok = false; break; }
      }
      const bool need_mask = (p.causal && kv0 + BN - 1 > q0) || (p.window > 0 && kv0 < q0 + BM - p.window) ||
                             (kv0 + BN > p.S) || (q0 + BM > p.S);
      // ---- C1: P^T = exp2(S^T c - lse_q), kept as packed bf16 pairs (queries 2i, 2i+1) ----
      if (!__all_sync(0xffffffffu, mbar_wait(&s_full[it % NSB], uint32_t(it / NSB) & 1, wctx, ST_TIMEOUT_TMEM_FULL))) { ok = false; break; }
      tr(TB_S_READY);
      tc_fence_after();
      // queries of this half that this thread's key is seen by: columns [vis_lo, vis_lo + vis_n)
      const int vis_lo = p.causal ? max(key - qc0, 0) : 0;
      const int vis_hi = min((p.window > 0 ? min(key + p.window, p.S) : p.S) - qc0, 64);
      const uint32_t vis_n = key_ok ? uint32_t(max(vis_hi - vis_lo, 0)) : 0u;
      if constexpr (!DQ) {
        // P stays in fp32 registers between its two uses; two-wide fp32 math; the softmax scale of dS is applied to
        // dK once, when it is written out
        float pr[64];
        const uint32_t s_col = lane_addr + uint32_t(half * 64) + (NSB == 2 && (it & 1) ? uint32_t(Cfg::S1_COL) : 0u);
        {
          uint32_t rs0[32], rs1[32];
          tmem_ld32(s_col, rs0);
          tmem_ld32(s_col + 32u, rs1);
          tmem_wait_ld();
#pragma unroll
          for (int k = 0; k < 64; k += 4) {
            const float4 l = ld_shared_f4(nlse_s + k * 4);
            const uint32_t* rs = k < 32 ? &rs0[k] : &rs1[k - 32];
            float x0, x1, x2, x3;
            ffma2(x0, x1, __uint_as_float(rs[0]), __uint_as_float(rs[1]), p.scale_log2, p.scale_log2, l.x, l.y);
            ffma2(x2, x3, __uint_as_float(rs[2]), __uint_as_float(rs[3]), p.scale_log2, p.scale_log2, l.z, l.w);
            pr[k] = exp2f(x0); pr[k + 1] = exp2f(x1); pr[k + 2] = exp2f(x2); pr[k + 3] = exp2f(x3);
          }
        }
        if (need_mask) {
#pragma unroll
          for (int k = 0; k < 64; ++k) pr[k] = uint32_t(k - vis_lo) < vis_n ? pr[k] : 0.f;
        }
        {
          uint32_t lo16[16], hi16[16];
#pragma unroll
          for (int k = 0; k < 16; ++k) {
            lo16[k] = pack_bf16x2(pr[2 * k], pr[2 * k + 1]);
            hi16[k] = pack_bf16x2(pr[32 + 2 * k], pr[33 + 2 * k]);
          }
          tmem_st16(s_col, lo16);
          tmem_st16(s_col + 16u, hi16);
        }
        tmem_wait_st();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&p_full[it % NSB]);
        tr(TB_P_DONE);
        if (!__all_sync(0xffffffffu, mbar_wait(dp_full, uint32_t(it) & 1, wctx, ST_TIMEOUT_TMEM_FULL))) { ok = false; break; }
        tr(TB_DP_READY);
        tc_fence_after();
        {
          uint32_t rd0[32], rd1[32];
          tmem_ld32(lane_addr + uint32_t(Cfg::DP_COL + half * 64), rd0);
          tmem_ld32(lane_addr + uint32_t(Cfg::DP_COL + half * 64 + 32), rd1);
          tmem_wait_ld();
          uint32_t ds0[16], ds1[16];
#pragma unroll
          for (int k = 0; k < 64; k += 4) {
            const float4 d = ld_shared_f4(ndelta_s + k * 4);
            const uint32_t* rd = k < 32 ? &rd0[k] : &rd1[k - 32];
            uint32_t* ds = k < 32 ? &ds0[k >> 1] : &ds1[(k - 32) >> 1];
            float x0, x1, x2, x3;
            fadd2(x0, x1, __uint_as_float(rd[0]), __uint_as_float(rd[1]), d.x, d.y);
            fadd2(x2, x3, __uint_as_float(rd[2]), __uint_as_float(rd[3]), d.z, d.w);
            fmul2(x0, x1, x0, x1, pr[k], pr[k + 1]);
            fmul2(x2, x3, x2, x3, pr[k + 2], pr[k + 3]);
            ds[0] = pack_bf16x2(x0, x1);
            ds[1] = pack_bf16x2(x2, x3);
          }
          // the other half's threads read their own 64 columns only, so the packed values may cover this half's first 32
          tmem_st16(lane_addr + uint32_t(Cfg::DP_COL + half * 64), ds0);
          tmem_st16(lane_addr + uint32_t(Cfg::DP_COL + half * 64 + 16), ds1);
        }
        tmem_wait_st();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(pds_full);
        tr(TB_DS_DONE);
      } else {
      // -lse_q (in log2 units) and -delta_q are the same for every lane: 16-byte loads from the
      // padded statistics rows
      auto load4 = [&](const float* base, int q, float (&v)[4]) {
        const float4 a = __ldg(reinterpret_cast<const float4*>(base + q));
        v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
      };
      uint32_t pp[32];
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        uint32_t rs[32];
        tmem_ld32(lane_addr + uint32_t(half * 64 + c * 32), rs);
        tmem_wait_ld();
        // the mask test is hoisted out of the element loop: one branch per chunk, not one per element
        if (need_mask) {
#pragma unroll
          for (int k = 0; k < 32; k += 4) {
            float l4[4], e[4];
            load4(lse_q, qc0 + c * 32 + k, l4);
#pragma unroll
            for (int u = 0; u < 4; ++u) {
              const float pe = exp2f(fmaf(__uint_as_float(rs[k + u]), p.scale_log2, l4[u]));
              e[u] = uint32_t(c * 32 + k + u - vis_lo) < vis_n ? pe : 0.f;
            }
            pp[c * 16 + (k >> 1)] = pack_bf16x2(e[0], e[1]);
            pp[c * 16 + (k >> 1) + 1] = pack_bf16x2(e[2], e[3]);
          }
        } else {
#pragma unroll
          for (int k = 0; k < 32; k += 4) {
            float l4[4], e[4];
            load4(lse_q, qc0 + c * 32 + k, l4);
#pragma unroll
            for (int u = 0; u < 4; ++u) e[u] = exp2f(fmaf(__uint_as_float(rs[k + u]), p.scale_log2, l4[u]));
            pp[c * 16 + (k >> 1)] = pack_bf16x2(e[0], e[1]);
            pp[c * 16 + (k >> 1) + 1] = pack_bf16x2(e[2], e[3]);
          }
        }
      }
      {
        uint32_t lo16[16], hi16[16];
#pragma unroll
        for (int k = 0; k < 16; ++k) { lo16[k] = pp[k]; hi16[k] = pp[16 + k]; }
        tmem_st16(lane_addr + uint32_t(half * 64), lo16);
        tmem_st16(lane_addr + uint32_t(half * 64 + 16), hi16);
      }
      tr(TB_P_DONE);
      // ---- C2: dS^T = P^T (dP^T - delta_q) scale -> TMEM (bf16 over R_dP) and shared memory ----
      if (!__all_sync(0xffffffffu, mbar_wait(dp_full, uint32_t(it) & 1, wctx, ST_TIMEOUT_TMEM_FULL))) { ok = false; break; }
      tr(TB_DP_READY);
      tc_fence_after();
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        uint32_t rd[32];
        tmem_ld32(lane_addr + uint32_t(Cfg::DP_COL + half * 64 + c * 32), rd);
        tmem_wait_ld();
        uint32_t ds[16];
#pragma unroll
        for (int k = 0; k < 32; k += 4) {
          float d4[4];
          load4(delta_q, qc0 + c * 32 + k, d4);
          const float2 pa = unpack_bf16x2(pp[c * 16 + (k >> 1)]), pb = unpack_bf16x2(pp[c * 16 + (k >> 1) + 1]);
          const float s0 = pa.x * (__uint_as_float(rd[k]) + d4[0]) * p.scale;
          const float s1 = pa.y * (__uint_as_float(rd[k + 1]) + d4[1]) * p.scale;
          const float s2 = pb.x * (__uint_as_float(rd[k + 2]) + d4[2]) * p.scale;
          const float s3 = pb.y * (__uint_as_float(rd[k + 3]) + d4[3]) * p.scale;
          ds[k >> 1] = pack_bf16x2(s0, s1);
          ds[(k >> 1) + 1] = pack_bf16x2(s2, s3);
        }
        // the other half's threads read columns [64 h', 64 h' + 64) only, so writing the packed
        // values over this half's own first 32 columns cannot disturb them
        tmem_st16(lane_addr + uint32_t(Cfg::DP_COL + half * 64 + c * 16), ds);
#pragma unroll
        for (int v4 = 0; v4 < 4; ++v4) {
          const int ch = c * 4 + v4;  // 16-byte chunk (8 queries) within the 128-byte row
          uint4 u = make_uint4(ds[v4 * 4 + 0], ds[v4 * 4 + 1], ds[v4 * 4 + 2], ds[v4 * 4 + 3]);
          *reinterpret_cast<uint4*>(ds_row + ((ch ^ (t & 7)) << 4)) = u;
        }
      }
      tmem_wait_st();
      fence_proxy_async_smem();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(pds_full);
      tr(TB_DS_DONE);
      // ---- G: dQ tile (lanes = query rows now) -> global fp32 accumulator ----
      if (!__all_sync(0xffffffffu, mbar_wait(dq_full, uint32_t(it) & 1, wctx, ST_TIMEOUT_TMEM_FULL))) { ok = false; break; }
      tr(TB_DQ_READY);
      tc_fence_after();
      if constexpr (D == 128) {
        // lanes = head-dim index t, columns = queries: this thread adds element t of 64 query rows
        const size_t row_stride = size_t(p.Hq) * D;
        float* dq_col = p.dq_acc + (size_t(batch) * p.S + q0) * row_stride + size_t(head) * D + t;
#pragma unroll 1
        for (int c = half * 2; c < half * 2 + 2; ++c) {
          uint32_t r[32];
          tmem_ld32(lane_addr + uint32_t(Cfg::DP_COL + c * 32), r);
          tmem_wait_ld();
          const int nq = min(32, p.S - (q0 + c * 32));   // query rows of this chunk that exist (warp-uniform)
#pragma unroll
          for (int k = 0; k < 32; ++k)
            if (k < nq) red_add_f32(dq_col + size_t(c * 32 + k) * row_stride, __uint_as_float(r[k]));
        }
      } else {
      const int qrow = q0 + t;
      float* dq_row = p.dq_acc + (size_t(batch) * p.S + qrow) * (size_t(p.Hq) * D) + size_t(head) * D;
#pragma unroll 1
      for (int c = half * (D / 64); c < (half + 1) * (D / 64); ++c) {
        uint32_t r[32];
        tmem_ld32(lane_addr + uint32_t(Cfg::DP_COL + c * 32), r);
        tmem_wait_ld();
        if (qrow < p.S) {
#pragma unroll
          for (int v4 = 0; v4 < 8; ++v4)
            red_add_v4_f32(dq_row + c * 32 + v4 * 4, __uint_as_float(r[v4 * 4 + 0]), __uint_as_float(r[v4 * 4 + 1]),
                           __uint_as_float(r[v4 * 4 + 2]), __uint_as_float(r[v4 * 4 + 3]));
        }
      }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(dq_empty);
      tr(TB_DQ_DRAINED);
      }
    }
    if constexpr (!DQ) {
      // the single dq_full arrival follows the last dK / dV product
      if (ok && n_iters > 0) ok = mbar_wait(dq_full, 0, wctx, ST_TIMEOUT_TMEM_FULL);
      tc_fence_after();
    }
    // ------------------------------ dK / dV write-out ------------------------------
    // the last dq_full arrival also covers every dK / dV MMA issued before it
    ok = __all_sync(0xffffffffu, ok);
    const uint32_t sums = smem_u32(sQ) + uint32_t(t) * 4;   // CL > 1: [which][column][key] fp32 over the Q / dO stages
    if constexpr (CL > 1) {
      // every copy into the stages has landed and every product that reads them is done (dq_full)
#pragma unroll 1
      for (int u = 0; u < 2 * (D / 64); ++u) {
        const int which = u / (D / 64), c = half * (D / 64) + u % (D / 64);
        uint32_t r[32];
        if (n_iters > 0) {
          tmem_ld32(lane_addr + (which == 0 ? Cfg::DK_COL : Cfg::DV_COL) + uint32_t(c * 32), r);
          tmem_wait_ld();
        } else {
#pragma unroll
          for (int k = 0; k < 32; ++k) r[k] = 0u;
        }
#pragma unroll
        for (int k = 0; k < 32; ++k)
          asm volatile("st.shared.b32 [%0], %1;" ::"r"(sums + uint32_t((which * D + c * 32 + k) * 512)), "r"(r[k]) : "memory");
      }
      cluster_barrier();
      // A rank that gave up holds incomplete sums.  Every warp of it has been through this barrier (a wait that runs out
      // raises the CTA's abort word first), so all ranks see the same words here and none of them stores.
      const uint32_t abort_addr = smem_u32(const_cast<int*>(abort_flag));
#pragma unroll
      for (int q = 0; q < CL; ++q) ok = ok && ld_cluster_u32(abort_addr, q) == 0;
    }
    // The tiles leave through the places of K and V, whose last readers are done, and TMA, which drops the rows behind the
    // sequence.  Stores straight from the registers went to 32 rows per instruction, half a sector each: 1.9 us per CTA of
    // 12.7 (d = 64, 577 tokens), 4.1 of 36 (d = 128, 4096 tokens).
#pragma unroll 1
    for (int which = 0; which < 2; ++which) {
      if (CL == 2 && which != cl_rank) continue;           // rank 0 writes dK, rank 1 dV
      if (CL == 4 && which != (cl_rank >> 1)) continue;    // ranks 0 and 1: alternate row halves of dK, 2 and 3: of dV
      if (CL == 4 && ((warp & 3) >> 1) != (cl_rank & 1)) continue;
      const uint32_t col0 = which == 0 ? Cfg::DK_COL : Cfg::DV_COL;
      const float mul = !DQ && which == 0 ? p.scale : 1.f;   // the two-kernel form leaves dS unscaled
      const uint32_t row = smem_u32(which == 0 ? sK : sV) + uint32_t(t) * 128;
#pragma unroll 1
      for (int c = half * (D / 64); c < (half + 1) * (D / 64); ++c) {
        uint32_t r[32];
        if constexpr (CL > 1) {
#pragma unroll
          for (int k = 0; k < 32; ++k) {
            const uint32_t a = sums + uint32_t((which * D + c * 32 + k) * 512);
            float s = ld_cluster_f32(a, 0);
#pragma unroll
            for (int q = 1; q < CL; ++q) s += ld_cluster_f32(a, q);
            r[k] = __float_as_uint(s);
          }
        } else if (n_iters > 0) {
          tmem_ld32(lane_addr + col0 + uint32_t(c * 32), r);
          tmem_wait_ld();
        } else {
#pragma unroll
          for (int k = 0; k < 32; ++k) r[k] = 0u;
        }
#pragma unroll
        for (int k = 0; k < 32; ++k) r[k] = __float_as_uint(__uint_as_float(r[k]) * mul);
        // columns [32 c, 32 c + 32) of the tile: 16-byte pieces 4 (c & 1) ... of block c / 2
        const uint32_t at = row + uint32_t(c >> 1) * BLK;
#pragma unroll
        for (int v4 = 0; v4 < 4; ++v4)
          st_shared_v4(at + ((uint32_t((c & 1) * 4 + v4) ^ uint32_t(t & 7)) << 4),
                       pack_bf16x2(__uint_as_float(r[v4 * 8 + 0]), __uint_as_float(r[v4 * 8 + 1])),
                       pack_bf16x2(__uint_as_float(r[v4 * 8 + 2]), __uint_as_float(r[v4 * 8 + 3])),
                       pack_bf16x2(__uint_as_float(r[v4 * 8 + 4]), __uint_as_float(r[v4 * 8 + 5])),
                       pack_bf16x2(__uint_as_float(r[v4 * 8 + 6]), __uint_as_float(r[v4 * 8 + 7])));
      }
    }
    fence_proxy_async_smem();
    asm volatile("bar.sync 1, 256;" ::: "memory");   // the compute warps
    // (a warp that gave up has raised the abort word; with CL > 1 all ranks have seen each other's)
    if (warp == 0 && ok && *abort_flag == 0) {
      if (lane == 0) {
#pragma unroll
        for (int which = 0; which < 2; ++which) {
          if ((CL == 2 && which != cl_rank) || (CL == 4 && which != (cl_rank >> 1))) continue;
          const uint8_t* tile = which == 0 ? sK : sV;
          // boxes of 64 rows: CL = 4 stores one of the two
#pragma unroll
          for (int hr = 0; hr < 2; ++hr) {
            if (CL == 4 && hr != (cl_rank & 1)) continue;
            if (kv0 + hr * 64 >= p.S) continue;
#pragma unroll
            for (int b = 0; b < DB; ++b)
              tma_store_4d(which == 0 ? &tmap_dk : &tmap_dv, tile + b * BLK + hr * 64 * 128, b * 64, kv_head, kv0 + hr * 64, batch);
          }
        }
        bulk_commit();
        bulk_wait_read<0>();
      }
      __syncwarp();
    }
  }

  __syncwarp();
  if constexpr (CL > 1) {
    if (warp >= 8) cluster_barrier();   // the compute warps' barrier in front of their write-out
    cluster_barrier();                  // nobody leaves while its sums are read
  }
  if (*abort_flag) {
    for (int i = 0; i < 64; ++i) __nanosleep(1000);
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 9) {
    tc_fence_after();
    tmem_dealloc(tmem_base, Cfg::TMEM_COLS);
  }
}

// stats[(b, h)][0][s] = -lse * log2(e), stats[(b, h)][1][s] = -sum_d dO * O; rows padded to s_pad
// entries, zeros behind the last query.  A CTA takes 64 tokens of one head: D / 8 lanes
// read a token's row in 16-byte pieces, all rows of a thread in flight at once, and the 64 results leave as two row
// segments. 32 heads of
// 4096 tokens, d = 128 32 -> 12 us, 32 heads of 2048, d = 64 15 -> 4 us (one warp per token and head, four-byte loads).
template <int D>
__global__ void __launch_bounds__(256)
attn_bwd2_stats_kernel(const __nv_bfloat16* o, const __nv_bfloat16* d_o,
                       const float* lse, float* stats, int S, int Hq, int s_pad, int o_vec) {
  chain_trigger();
  chain_wait();
  constexpr int LANES = D / 8, GROUPS = 256 / LANES, N = 64 / GROUPS;   // lanes per token, tokens at a time, tokens per group
  __shared__ float sm[64];
  const int s0 = blockIdx.x * 64, h = blockIdx.y, b = blockIdx.z;
  const int g = threadIdx.x / LANES, l = threadIdx.x % LANES;
  uint4 x[N], y[N];
#pragma unroll
  for (int i = 0; i < N; ++i) {
    const int s = s0 + i * GROUPS + g;
    x[i] = y[i] = make_uint4(0u, 0u, 0u, 0u);
    if (s < S) {
      const size_t at = ((size_t(b) * S + s) * Hq + h) * D + l * 8;
      y[i] = ld_v4(d_o + at);
      if (o_vec) {
        x[i] = ld_v4(o + at);
      } else {
        const uint32_t* p = reinterpret_cast<const uint32_t*>(o + at);
        x[i] = make_uint4(p[0], p[1], p[2], p[3]);
      }
    }
  }
#pragma unroll
  for (int i = 0; i < N; ++i) {
    const uint32_t xs[4] = {x[i].x, x[i].y, x[i].z, x[i].w}, ys[4] = {y[i].x, y[i].y, y[i].z, y[i].w};
    float acc = 0.f;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const float2 u = unpack_bf16x2(xs[k]), v = unpack_bf16x2(ys[k]);
      acc += u.x * v.x + u.y * v.y;
    }
#pragma unroll
    for (int off = LANES / 2; off > 0; off >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, off);
    if (l == 0) sm[i * GROUPS + g] = acc;
  }
  __syncthreads();
  const int s = s0 + int(threadIdx.x);
  if (threadIdx.x < 64) {   // (the padding too: its P is masked, but 0 times what lies there has to be 0)
    const size_t bh = size_t(b) * Hq + h;
    float* row = stats + bh * 2 * size_t(s_pad);
    row[s] = s < S ? lse[bh * S + s] * -1.4426950408889634f : 0.f;
    row[s_pad + s] = -sm[threadIdx.x];
  }
}

static int launch_stats(const __nv_bfloat16* o, const __nv_bfloat16* d_o, const float* lse, float* stats, int B, int S, int Hq,
                        int D, int s_pad, cudaStream_t stream) {
  const dim3 grid(s_pad / 64, Hq, B);
  const int o_vec = (reinterpret_cast<uintptr_t>(o) & 15) == 0;   // (dO is fetched by TMA and aligned anyway)
  if (reinterpret_cast<uintptr_t>(d_o) & 15) ZB_FAIL(-4, "attention: dO not 16-byte aligned");
  if (D == 128) ZB_CUDA_OK(launch_pass(attn_bwd2_stats_kernel<128>, grid, 256, 0, stream, o, d_o, lse, stats, S, Hq, s_pad,
                                       o_vec));
  else ZB_CUDA_OK(launch_pass(attn_bwd2_stats_kernel<64>, grid, 256, 0, stream, o, d_o, lse, stats, S, Hq, s_pad, o_vec));
  ZB_CUDA_OK(cudaGetLastError());
  return 0;
}

static int make_head_tmap_bwd2(CUtensorMap* out, const __nv_bfloat16* base, int B, int S, int heads, int D, int width,
                               uint32_t rows = 128) {
  uint64_t dims[4] = {uint64_t(D), uint64_t(heads), uint64_t(S), uint64_t(B)};
  uint64_t strides[3] = {uint64_t(D) * 2, uint64_t(width) * 2, uint64_t(width) * 2 * uint64_t(S)};
  uint32_t box[4] = {64, 1, rows, 1};
  return make_tmap_nd_bf16(out, base, 4, dims, strides, box);
}

template <int D, bool TRACE, bool DQ = true, int CL = 1>
static int launch_bwd2(const __nv_bfloat16* qkv, const __nv_bfloat16* d_o, const AttnBwdParams& p, const float* stats,
                       int s_pad, unsigned long long* trace, int trace_ctas, cudaStream_t stream) {
  using Cfg = AttnBwd2Cfg<D>;
  const int width = (p.Hq + 2 * p.Hkv) * D;
  CUtensorMap tq, tk, tv, tdo, tdk, tdv;
  int rc;
  if ((rc = make_head_tmap_bwd2(&tdk, p.dqkv + size_t(p.Hq) * D, p.B, p.S, p.Hkv, D, width, 64))) return rc;
  if ((rc = make_head_tmap_bwd2(&tdv, p.dqkv + size_t(p.Hq + p.Hkv) * D, p.B, p.S, p.Hkv, D, width, 64))) return rc;
  if ((rc = make_head_tmap_bwd2(&tq, qkv, p.B, p.S, p.Hq, D, width))) return rc;
  if ((rc = make_head_tmap_bwd2(&tk, qkv + size_t(p.Hq) * D, p.B, p.S, p.Hkv, D, width))) return rc;
  if ((rc = make_head_tmap_bwd2(&tv, qkv + size_t(p.Hq + p.Hkv) * D, p.B, p.S, p.Hkv, D, width))) return rc;
  if ((rc = make_head_tmap_bwd2(&tdo, d_o, p.B, p.S, p.Hq, D, p.Hq * D))) return rc;
  auto kern = flash_bwd2_kernel<D, TRACE, DQ, CL>;
  static bool attr_set = false;
  if (!attr_set) {
    ZB_CUDA_OK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::SMEM_BYTES));
    attr_set = true;
  }
  dim3 grid(p.Hkv * CL, (p.S + 127) / 128, p.B);
  if constexpr (!DQ) {
    ZB_CUDA_OK(launch_chained(kern, grid, 32 * BWD2_WARPS, Cfg::SMEM_BYTES, stream, CL > 1 ? CL : 0, tq, tk, tv, tdo, tdk, tdv, p, stats,
                              s_pad, trace, trace_ctas));
  } else {
    kern<<<grid, 32 * BWD2_WARPS, Cfg::SMEM_BYTES, stream>>>(tq, tk, tv, tdo, tdk, tdv, p, stats, s_pad, trace, trace_ctas);
    ZB_CUDA_OK(cudaGetLastError());
  }
  return 0;
}

// CTAs per key tile of the dK / dV kernel.  Splitting pays where one CTA per tile leaves SMs idle or waiting for the
// longest.  One / two / four CTAs, us from cold caches with the statistics: 2048 tokens, 32 / 8 heads (128 tiles), d = 64
// 108 / 70 / 91, d = 128 152 / 95 / 124; 512 tokens, d = 128 (32 tiles) 46 / 36 / 30.  From two waves on the second prologue
// and the sum at the end cost as much or more: 4608 tokens, d = 128 (288 tiles) 294 / 314 / 386, 8 x 512, d = 64 (256 tiles)
// 69 / 73 / 106, 8192 tokens, d = 64 (512 tiles) 662 / 650 / 816.
static int bwd_cluster(int B, int S, int Hq, int Hkv) {
  const int rep = Hq / Hkv;
  const long ctas = long(Hkv) * ((S + 127) / 128) * B;
  if (rep % 4 == 0 && 4 * ctas <= num_sms()) return 4;
  return rep % 2 == 0 && ctas <= num_sms() ? 2 : 1;
}

int attn_bwd_dq(const __nv_bfloat16* qkv, const __nv_bfloat16* d_o, const AttnBwdParams& p, const float* stats, int s_pad,
                int D, int late, cudaStream_t stream);   // flash_bwd_dq.cu

}  // namespace zb

extern "C" {

int zb_flash_bwd2_trace_events() { return zb::BWD2_TRACE_EV; }
int zb_flash_bwd2_trace_warps() { return zb::BWD2_WARPS; }

int zb_flash_bwd2_stats_floats(int B, int S, int Hq) { return B * Hq * 2 * ((S + 127) / 128 * 128); }

// Scratch: stats fp32 [zb_flash_bwd2_stats_floats(B, S, Hq)]; dq_acc fp32 [B*S*Hq*D], zero on entry (left zero).
// trace: nullptr, or a zeroed device buffer of trace_ctas * warps * events 64-bit words.
int zb_flash_bwd2(const void* d_o, const void* qkv, const void* o, const float* lse, void* dqkv, float* stats,
                  float* dq_acc, int B, int S, int Hq, int Hkv, int D, int causal, int window, float softmax_scale,
                  int* status, unsigned long long* trace, int trace_ctas, cudaStream_t stream) {
  using namespace zb;
  if (B <= 0 || S <= 0) return 0;
  if (Hkv <= 0 || Hq % Hkv != 0) ZB_FAIL(-1, "attention: Hq=%d not a multiple of Hkv=%d", Hq, Hkv);
  if (D != 64 && D != 128) ZB_FAIL(-1, "attention: head dim %d unsupported (64 or 128)", D);
  auto DO = static_cast<const __nv_bfloat16*>(d_o);
  auto O = static_cast<const __nv_bfloat16*>(o);
  auto QKV = static_cast<const __nv_bfloat16*>(qkv);
  const int s_pad = (S + 127) / 128 * 128;
  if (int rc_st = launch_stats(O, DO, lse, stats, B, S, Hq, D, s_pad, stream)) return rc_st;
  AttnBwdParams p;
  p.lse = lse; p.delta = nullptr; p.dq_acc = dq_acc;
  p.dqkv = static_cast<__nv_bfloat16*>(dqkv);
  p.B = B; p.S = S; p.Hq = Hq; p.Hkv = Hkv;
  p.window = window; p.causal = causal;
  p.scale = softmax_scale;
  p.scale_log2 = softmax_scale * 1.4426950408889634f;
  p.status = status;
  const bool trc = trace != nullptr && trace_ctas > 0;
  int rc;
  if (D == 128) rc = trc ? launch_bwd2<128, true>(QKV, DO, p, stats, s_pad, trace, trace_ctas, stream)
                         : launch_bwd2<128, false>(QKV, DO, p, stats, s_pad, nullptr, 0, stream);
  else rc = trc ? launch_bwd2<64, true>(QKV, DO, p, stats, s_pad, trace, trace_ctas, stream)
                : launch_bwd2<64, false>(QKV, DO, p, stats, s_pad, nullptr, 0, stream);
  if (rc) return rc;
  return attn_bwd_finish_dq(dq_acc, p.dqkv, B, S, Hq, Hkv, D, stream);
}

// Two-kernel backward without atomics: statistics pass, then dK / dV per key tile (this file's kernel without
// its dQ part) and dQ per query tile (flash_bwd_dq.cu); the two main kernels are independent of each other.
// Scratch: stats fp32 [zb_flash_bwd2_stats_floats(B, S, Hq)].
int zb_flash_bwd3(const void* d_o, const void* qkv, const void* o, const float* lse, void* dqkv, float* stats,
                  int B, int S, int Hq, int Hkv, int D, int causal, int window, float softmax_scale, int* status,
                  int parts, unsigned long long* trace, int trace_ctas, cudaStream_t stream) {
  // parts: 3 = the whole backward; 1 = statistics + dK / dV kernel only, 2 = dQ kernel only (needs the
  // statistics of an earlier call) - for timing the two halves separately
  using namespace zb;
  if (B <= 0 || S <= 0) return 0;
  if (Hkv <= 0 || Hq % Hkv != 0) ZB_FAIL(-1, "attention: Hq=%d not a multiple of Hkv=%d", Hq, Hkv);
  if (D != 64 && D != 128) ZB_FAIL(-1, "attention: head dim %d unsupported (64 or 128)", D);
  auto DO = static_cast<const __nv_bfloat16*>(d_o);
  auto O = static_cast<const __nv_bfloat16*>(o);
  auto QKV = static_cast<const __nv_bfloat16*>(qkv);
  const int s_pad = (S + 127) / 128 * 128;
  if (parts & 1) {
    if (int rc_st = launch_stats(O, DO, lse, stats, B, S, Hq, D, s_pad, stream)) return rc_st;
  }
  AttnBwdParams p;
  p.lse = lse; p.delta = nullptr; p.dq_acc = nullptr;
  p.dqkv = static_cast<__nv_bfloat16*>(dqkv);
  p.B = B; p.S = S; p.Hq = Hq; p.Hkv = Hkv;
  p.window = window; p.causal = causal;
  p.scale = softmax_scale;
  p.scale_log2 = softmax_scale * 1.4426950408889634f;
  p.status = status;
  int rc = 0;
  const bool trc = trace != nullptr && trace_ctas > 0;     // phase trace of the dK / dV kernel (as in zb_flash_bwd2)
  if (parts & 1) {
    auto run = [&](auto d) {
      constexpr int DD = decltype(d)::value;
      if (trc) return launch_bwd2<DD, true, false>(QKV, DO, p, stats, s_pad, trace, trace_ctas, stream);
      switch (bwd_cluster(B, S, Hq, Hkv)) {
        case 4: return launch_bwd2<DD, false, false, 4>(QKV, DO, p, stats, s_pad, nullptr, 0, stream);
        case 2: return launch_bwd2<DD, false, false, 2>(QKV, DO, p, stats, s_pad, nullptr, 0, stream);
        default: return launch_bwd2<DD, false, false>(QKV, DO, p, stats, s_pad, nullptr, 0, stream);
      }
    };
    rc = D == 128 ? run(std::integral_constant<int, 128>()) : run(std::integral_constant<int, 64>());
  }
  if (rc) return rc;
  return (parts & 2) ? attn_bwd_dq(QKV, DO, p, stats, s_pad, D, parts == 3, stream) : 0;
}

}  // extern "C"
