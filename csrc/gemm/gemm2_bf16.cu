// bf16 GEMM on CTA pairs: tcgen05.mma.cta_group::2 with a 256 x 256 (or 256 x 128) output tile per pair.
//
// Two CTAs of a cluster (2,1,1) share one tile: each holds 128 rows of A and of the fp32
// accumulators (its own tensor memory) and loads HALF of the B tile (128 of the 256 rows);
// the MMA issued by the leader CTA reads A and B from both CTAs' shared memory.  Per k-block a
// pair moves 64 KB for 256x256x64 MACs, 1.5x the arithmetic intensity of the single-CTA
// 128x256 kernel, which is what the L2 -> SM path needs at tensor-core rate.
//   * every TMA load is issued by the CTA that receives the data, WITHOUT cluster multicast;
//     its mbarrier completion is routed to the leader's barrier (cta_group::2 form),
//   * tcgen05.commit with cluster multicast hands stages / accumulators back to both CTAs,
//   * warp roles per CTA: 0 = TMA producer, 1 = MMA issuer (leader only) + TMEM owner,
//     2..5 = epilogue for the CTA's own 128 rows.
// Operand layouts and epilogue options are those of gemm_bf16.cu.
#include "../common/host.h"
#include "../common/ptx.cuh"
#include "../elementwise/act_math.cuh"
#include "gemm_common.cuh"
#include <algorithm>
#include <type_traits>

namespace zb {

constexpr uint32_t PEER_BIT_MASK = 0xFEFFFFFFu;  // clears the CTA-rank bit of a shared::cluster address

__device__ __forceinline__ uint32_t cluster_ctarank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.aligned;\nbarrier.cluster.wait.aligned;" ::: "memory");
}
// arrive on the barrier at the same shared-memory offset in CTA `cta` of the cluster
__device__ __forceinline__ void mbar_arrive_cluster(uint64_t* bar, uint32_t cta) {
  asm volatile(
      "{\n\t.reg .b32 ra;\n\t"
      "mapa.shared::cluster.u32 ra, %0, %1;\n\t"
      "mbarrier.arrive.shared::cluster.b64 _, [ra];\n\t}" ::"r"(smem_u32(bar)),
      "r"(cta)
      : "memory");
}
__device__ __forceinline__ void tma_load_2d_pair(void* smem_dst, const void* tmap, uint64_t* leader_bar, int x, int y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, "
      "{%3, %4}], [%2];"
      :
      : "r"(smem_u32(smem_dst)), "l"(tmap), "r"(smem_u32(leader_bar) & PEER_BIT_MASK), "r"(x), "r"(y)
      : "memory");
}
__device__ __forceinline__ void tma_load_3d_pair(void* smem_dst, const void* tmap, uint64_t* leader_bar, int x, int y,
                                                 int z) {
  asm volatile(
      "cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, "
      "{%3, %4, %5}], [%2];"
      :
      : "r"(smem_u32(smem_dst)), "l"(tmap), "r"(smem_u32(leader_bar) & PEER_BIT_MASK), "r"(x), "r"(y), "r"(z)
      : "memory");
}
__device__ __forceinline__ void tmem_alloc_pair(uint32_t* smem_result, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(smem_result)),
               "r"(ncols)
               : "memory");
}
__device__ __forceinline__ void tmem_relinquish_pair() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc_pair(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void umma_f16_ss_pair(uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t idesc,
                                                 uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, {%5, %6, %7, %8, %9, %10, %11, %12}, p;\n\t}"
      :
      : "r"(tmem_d), "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate), "r"(0), "r"(0), "r"(0), "r"(0), "r"(0),
        "r"(0), "r"(0), "r"(0)
      : "memory");
}
// arrives (once all MMAs issued so far are complete) on the barrier at this offset in BOTH CTAs
__device__ __forceinline__ void umma_commit_pair(uint64_t* bar) {
  asm volatile(
      "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(
          smem_u32(bar)),
      "h"(uint16_t(3))
      : "memory");
}

// BN_: columns of a pair's tile, 256 or 128; each CTA loads half of them as rows of B.
template <int BN_>
struct Gemm2Cfg {
  static constexpr int BM = 256;   // per pair; 128 per CTA
  static constexpr int BN = BN_;
  static constexpr int BK = 64;
  static constexpr int A_BYTES = 128 * BK * 2;
  static constexpr int B_BYTES = BN / 2 * BK * 2;
  static constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
  static constexpr int TMEM_COLS = 2 * BN;
  static constexpr int EP_BYTES = 32 * 128;    // epilogue box: 32 rows x 128 bytes
  // Shared memory is split at launch: 32 KB of epilogue boxes (EP_SMALL) and 6 operand stages, or 64 KB and 5.  The sixth
  // stage is worth 3 - 5 % of the main loop (4096 x 22016 x 4096: 486 -> 472 us), two boxes per epilogue warp instead of one
  // shorten the epilogue of a tile (load, add, store in flight at once).  The epilogue of a tile runs under the main loop of
  // the next one, so the boxes only count where that loop is short: K < 2048.
  // Tiles of 128 columns have stages of 24 KB instead of 32: 8, or 6.
  static constexpr int MAX_STAGES = 8, EP_SMALL = 8, EP_LARGE = 16;   // boxes
  static constexpr int STAGES_S = BN == 256 ? 6 : 8, STAGES_L = BN == 256 ? 5 : 6;
  static constexpr int RING_BYTES = STAGES_S * STAGE_BYTES + EP_SMALL * EP_BYTES;
  static_assert(STAGES_L * STAGE_BYTES + EP_LARGE * EP_BYTES <= RING_BYTES, "both splits fit the same space");
  static constexpr int SMEM_BYTES = RING_BYTES + 1024 + 512;
};

// How the accumulators leave the SM.  DIRECT: one output row per thread, loads and stores straight to global memory
// (any alignment, any combination of options).  BF16 / F32: 32 x 128-byte boxes through shared memory and TMA; the old
// C tile or the addend of a bf16 output arrives by TMA as well, two boxes ahead; an accumulating fp32 output is added
// in L2 (cp.reduce), so it is never read into the SM.  The direct form issues 16-byte accesses of 32 different rows per
// instruction and waits for the old C values chunk by chunk: about 20 us per 256 x 256 tile that accumulates, longer
// than the tile's main loop below K = 4096.  Weight gradients with the boxes: 3072 x 768 x 2048 fp32 34.7 -> 17.9 us,
// 20480 x 5120 x 2048 bf16 432 -> 335 us; plain bf16 outputs 1018 x 49152 x 512 61 -> 48 us.
enum : int { EP_DIRECT = 0, EP_BF16 = 1, EP_F32 = 2 };

struct Gemm2Extra {
  TileOrder order;
  int ep;          // EP_*
  int ep_load;     // EP_BF16: add the tensor behind tmap_x (old C or addend)
  // Split last wave: items [0, full) are whole tiles; the rest are tiles full, full + 1, ... in `splits` parts of their
  // k-blocks each, whose fp32 sums go to the workspace behind tmap_w, one slot of 256 rows per part (gemm2_fixup_kernel
  // adds them up).  Every pair gets at most one such part, as its last item.
  int items, full, splits;
  int a_3d, b_3d;  // MN-major operand fetched with one 3-D TMA box {64, BK, 64-column blocks} instead of 2-D boxes
};

// SCATTER: the epilogue sends every output row to the staging slot of the rank that owns it in a
// row-wise reduce-scatter (plain stores over NVLink, tile by tile while the main loop goes on) and
// the last CTA raises the arrival flags; the owners add the slots up (csrc/comm/tp_rs.cu).
// FUSED_AG (Params = GemmAgParams): four more warps per CTA pull the peers' parameter shards into the local
// unsharded buffer while the tiles whose B rows are already present run; each CTA's producer waits for the
// chunks that cover its own 128 rows of B.
// EP_WARPS: 4, or 8 in two groups that take the tile's boxes in turns.  A box takes a warp about 0.5 us (accumulators out of
// tensor memory, conversion, shared memory, fence, store), so with four the end of a product's last tiles lasted 2 us, and
// at K < 1000 the epilogue of a tile (with an activation above all) was longer than the main loop it has to hide under.
template <bool A_MN, bool B_MN, typename Params, int BN, int EP_WARPS, int EP_BUFS>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(64 + 32 * EP_WARPS + (std::is_same<Params, GemmAgParams>::value ? 128 : 0), 1)
gemm2_bf16_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b,
                  const __grid_constant__ CUtensorMap tmap_c, const __grid_constant__ CUtensorMap tmap_x,
                  const __grid_constant__ CUtensorMap tmap_w, const Params p, const Gemm2Extra ex) {
  using Cfg = Gemm2Cfg<BN>;
  constexpr bool SCATTER = std::is_same<Params, GemmScatterParams>::value;
  constexpr bool FUSED_AG = std::is_same<Params, GemmAgParams>::value;
  constexpr int FE = FusedEp<Params>::value;
  constexpr int BK = Cfg::BK, MAXS = Cfg::MAX_STAGES, HALF_N = BN / 2;
  constexpr int STAGES = EP_WARPS * EP_BUFS == Cfg::EP_SMALL ? Cfg::STAGES_S : Cfg::STAGES_L;
  static_assert(EP_WARPS * EP_BUFS == Cfg::EP_SMALL || EP_WARPS * EP_BUFS == Cfg::EP_LARGE, "a split of shared memory");
  constexpr int EP_GROUPS = EP_WARPS / 4;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sE = smem + STAGES * Cfg::STAGE_BYTES;   // epilogue boxes, EP_BUFS per epilogue warp
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + Cfg::RING_BYTES);
  uint64_t* full = bars;                          // leader's copy is the one in use
  uint64_t* empty = bars + MAXS;                  // each CTA waits on its own
  uint64_t* tmem_full = bars + 2 * MAXS;          // [2], each CTA waits on its own
  uint64_t* tmem_empty = bars + 2 * MAXS + 2;     // [2], leader's copy, one arrival per epilogue warp of both CTAs
  uint64_t* x_full = bars + 2 * MAXS + 4;         // [EP_WARPS][EP_BUFS]: a box of tmap_x has landed
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(x_full + Cfg::EP_LARGE);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t cta = cluster_ctarank();
  const bool leader = cta == 0;
  const int pair = blockIdx.x >> 1, num_pairs = gridDim.x >> 1;
  const int num_items = ex.items;
  const int num_kb = (p.K + BK - 1) / BK;
  auto tile_of = [&](int item) { return item < ex.full ? item : ex.full + (item - ex.full) / ex.splits; };
  auto kb_range = [&](int item, int& kb0, int& kb1) {
    kb0 = 0;
    kb1 = num_kb;
    if (item >= ex.full) {
      const int part = (item - ex.full) % ex.splits;
      kb0 = num_kb * part / ex.splits;
      kb1 = num_kb * (part + 1) / ex.splits;
    }
  };
  WaitCtx wctx{abort_flag, p.status};

  if (threadIdx.x == 0) {
    *abort_flag = 0;
    for (int i = 0; i < STAGES; ++i) {
      mbar_init(&full[i], 1);
      mbar_init(&empty[i], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&tmem_full[i], 1);
      mbar_init(&tmem_empty[i], 2 * EP_WARPS);
    }
    for (int i = 0; i < EP_WARPS * EP_BUFS; ++i) mbar_init(&x_full[i], 1);
    mbar_fence_init();
    tma_prefetch_desc(&tmap_a);   // (parameters of the kernel: nothing the kernel before this one writes)
    tma_prefetch_desc(&tmap_b);
  }
  if (warp == 1) {
    tmem_alloc_pair(tmem_slot, Cfg::TMEM_COLS);
    tmem_relinquish_pair();
  }
  tc_fence_before();
  cluster_sync_all();  // barriers of both CTAs are initialised before anyone signals them
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  const bool late = (p.flags & GEMM_LATE) != 0;
  if constexpr (!SCATTER && !FUSED_AG) {
    if (!late) chain_wait();
    chain_trigger();
  }

  if (warp == 0) {
    // ------------------------------ TMA producer (both CTAs) ------------------------------
    {
      const bool elected = elect_one();
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int item = pair; item < num_items && ok; item += num_pairs) {
        int tm, tn, kb0, kb1;
        const int tile = tile_of(item);
        kb_range(item, kb0, kb1);
        tile_at(ex.order, tile, tm, tn);
        const int m0 = tm * Cfg::BM + int(cta) * 128;
        // (a gated unit's tile: rows of the gate's weights in the first CTA, the same rows of the other half in the second)
        const int n0 = FE == FE_GLU_FWD ? tn * HALF_N + int(cta) * p.N : tn * BN + int(cta) * HALF_N;
        // (the second CTA's half may start past the edge of a ragged tile: its loads then read the fill value)
        if (!zb_in_bounds(m0 - int(cta) * 128 < p.M && tn * (FE == FE_GLU_FWD ? HALF_N : BN) < p.N && tile >= 0, p.status, 1)) break;
        if constexpr (FUSED_AG) {
          if (p.gate_flags != nullptr && n0 < p.N) {
            // rows [n0, n0 + HALF_N) of B inside the flat buffer: wait for every chunk of a peer's shard they touch
            const long b0 = p.gate_base + long(n0) * p.gate_row_bytes;
            const long b1 = p.gate_base + long(min(n0 + HALF_N, p.N)) * p.gate_row_bytes - 1;
            const long i0 = (b0 / p.gate_shard_bytes) * p.gate_cps + (b0 % p.gate_shard_bytes) / p.gate_chunk_bytes;
            const long i1 = (b1 / p.gate_shard_bytes) * p.gate_cps + (b1 % p.gate_shard_bytes) / p.gate_chunk_bytes;
            for (long c = i0; c <= i1 && ok; ++c) {
              if (int(c / p.gate_cps) == p.gate_self) continue;
              ok = flag_wait_ge(p.gate_flags + c, p.gate_epoch, ZB_WAIT_NS, p.status, ST_TIMEOUT_FLAG);
            }
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) { *abort_flag = 1; break; }
            asm volatile("fence.proxy.async.global;" ::: "memory");   // the gathered rows were written with plain stores
          }
        }
        for (int kb = kb0; kb < kb1; ++kb) {
          if (!mbar_wait_warp(&empty[stage], phase ^ 1, wctx, ST_TIMEOUT_EMPTY)) { ok = false; break; }
          uint8_t* sa = smem + stage * Cfg::STAGE_BYTES;
          uint8_t* sb = sa + Cfg::A_BYTES;
          if (elected) {
            if (leader) mbar_expect_tx(&full[stage], 2 * Cfg::STAGE_BYTES);
            if (!A_MN) {
              tma_load_2d_pair(sa, &tmap_a, &full[stage], kb * BK, m0);
            } else if (ex.a_3d) {
              tma_load_3d_pair(sa, &tmap_a, &full[stage], 0, kb * BK, m0 >> 6);
            } else {
              tma_load_2d_pair(sa, &tmap_a, &full[stage], m0, kb * BK);
              tma_load_2d_pair(sa + BK * 128, &tmap_a, &full[stage], m0 + 64, kb * BK);
            }
            if (!B_MN) {
              tma_load_2d_pair(sb, &tmap_b, &full[stage], kb * BK, n0);
            } else if (ex.b_3d) {
              tma_load_3d_pair(sb, &tmap_b, &full[stage], 0, kb * BK, n0 >> 6);
            } else {
#pragma unroll
              for (int j = 0; j < HALF_N / 64; ++j)
                tma_load_2d_pair(sb + j * BK * 128, &tmap_b, &full[stage], n0 + j * 64, kb * BK);
            }
          }
          __syncwarp();
          if (++stage == STAGES) { stage = 0; phase ^= 1; }
        }
      }
      // The leader's commits arrive on the stage barriers of both CTAs: those of the last stages are waited for too, so that
      // none is on its way to a CTA that has left.  The waits are those of one more round of loads.
      for (int i = 0; i < STAGES && ok; ++i) {
        ok = mbar_wait_warp(&empty[stage], phase ^ 1, wctx, ST_TIMEOUT_EMPTY);
        if (++stage == STAGES) { stage = 0; phase ^= 1; }
      }
    }
  } else if (warp == 1) {
    // ------------------------------ MMA issuer (leader CTA only) ------------------------------
    // The whole warp walks the loop and one elected lane issues: addresses and descriptors stay warp-uniform.  With the
    // loop inside `if (lane == 0)` issuing the four products of a k-block took longer than the tensor core needs for
    // them (4096 x 22016 x 4096: 519 -> 494 us).
    if (leader) {
      constexpr uint32_t idesc = umma_idesc_bf16(256, BN, A_MN, B_MN);
      const bool elected = elect_one();
      int stage = 0;
      uint32_t phase = 0;
      int local = 0;
      bool ok = true;
      for (int item = pair; item < num_items && ok; item += num_pairs, ++local) {
        int kb0, kb1;
        kb_range(item, kb0, kb1);
        const int buf = local & 1;
        const uint32_t use = uint32_t(local >> 1);
        ok = mbar_wait_warp(&tmem_empty[buf], (use & 1) ^ 1, wctx, ST_TIMEOUT_TMEM_EMPTY);
        if (!ok) break;
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + uint32_t(buf * BN);
        for (int kb = kb0; kb < kb1; ++kb) {
          if (!mbar_wait_warp(&full[stage], phase, wctx, ST_TIMEOUT_FULL)) { ok = false; break; }
          tc_fence_after();
          const uint32_t sa = smem_u32(smem + stage * Cfg::STAGE_BYTES);
          const uint32_t sb = sa + Cfg::A_BYTES;
          if (elected) {
#pragma unroll
            for (int kk = 0; kk < BK / 16; ++kk) {
              uint64_t da = A_MN ? umma_desc_mnmajor(sa + kk * 16 * 128, BK * 128) : umma_desc_kmajor(sa + kk * 32);
              uint64_t db = B_MN ? umma_desc_mnmajor(sb + kk * 16 * 128, BK * 128) : umma_desc_kmajor(sb + kk * 32);
              umma_f16_ss_pair(d_tmem, da, db, idesc, kb > kb0 || kk != 0 ? 1u : 0u);
            }
            umma_commit_pair(&empty[stage]);
          }
          __syncwarp();
          if (++stage == STAGES) { stage = 0; phase ^= 1; }
        }
        if (ok && elected) umma_commit_pair(&tmem_full[buf]);
        __syncwarp();
      }
      // The second CTA's epilogue warps arrive on these barriers from another SM, and the last arrivals release accumulators
      // that no tile wants any more: without a wait this CTA could be gone, and its shared memory another's, when one lands
      // (the barrier at the end orders no memory).  The waits are those of two more tiles, one per buffer.
      for (int i = 0; i < 2 && ok; ++i, ++local)
        ok = mbar_wait_warp(&tmem_empty[local & 1], (uint32_t(local >> 1) & 1) ^ 1, wctx, ST_TIMEOUT_TMEM_EMPTY);
    }
  } else if (warp < 2 + EP_WARPS) {
    // ------------------------------ epilogue (own 128 rows) ------------------------------
    const int q = warp & 3;                        // which 32 rows (the lanes of tensor memory this warp may read)
    const int h = EP_GROUPS > 1 ? (warp - 2) >> 2 : 0;   // boxes h, h + EP_GROUPS, ... of a tile
    const EpilogueCfg ecfg = epilogue_cfg(p);
    uint8_t* my_boxes = sE + (warp - 2) * EP_BUFS * Cfg::EP_BYTES;
    uint64_t* my_full = x_full + (warp - 2) * EP_BUFS;
    static_assert(EP_BUFS == 2 || EP_BUFS == 4, "a power of two");
    constexpr uint32_t slot_mask = uint32_t(EP_BUFS) - 1, phase_shift = EP_BUFS == 4 ? 2 : 1;
    auto mine = [&](int n) { return n > h ? (n - h + EP_GROUPS - 1) / EP_GROUPS : 0; };   // of a tile's n boxes
    uint32_t ep_count = 0;   // boxes this warp has stored: slot and barrier phase of the next one
    int local = 0;
    for (int item = pair; item < num_items; item += num_pairs, ++local) {
      int tm, tn;
      tile_at(ex.order, tile_of(item), tm, tn);
      const bool split = item >= ex.full;   // a part of a tile: plain fp32 sums to the workspace
      const int m0 = tm * Cfg::BM + int(cta) * 128;
      const int n0 = tn * BN;
      const int buf = local & 1;
      const uint32_t use = uint32_t(local >> 1);
      if constexpr (FE != FE_NONE) {
        // ---- activation or rotation in the epilogue: groups of 64 columns, each one to three boxes ----
        constexpr int COLS = FE == FE_GLU_FWD ? HALF_N : BN;
        // FE_ROPE: a group is 32 pairs of columns, half a head's width apart: a head of 64, or half of one of 128 (two boxes of
        // 32 columns).  The cosines and sines of a thread's row for them stay in its registers: those of a head of 64 for all
        // heads of the tile; the halves of wider heads go to the two warps of the rows, or come one after the other where
        // there is one.
        const int head = FE == FE_ROPE ? p.act : 64, halves = FE == FE_ROPE ? head / 64 : 1;
        const bool half_each = FE == FE_ROPE && EP_GROUPS == 2 && halves == 2;
        constexpr int LOADS = FE == FE_ACT_BWD ? 1 : FE == FE_GLU_BWD ? 2 : 0;
        const int row0 = m0 + q * 32, c0 = tn * COLS;
        const int heads = row0 < p.M ? min(COLS / head, (p.N - c0 + head - 1) / head) : 0;
        const int groups = mine(heads * halves);
        auto half_of = [&](int g) { return halves == 1 ? 0 : half_each ? h : int(g >= heads); };
        auto col_of = [&](int g) {
          return halves == 1 ? c0 + (h + g * EP_GROUPS) * 64 : c0 + (half_each || g < heads ? g : g - heads) * 128 + half_of(g) * 32;
        };
        const int per_group = LOADS > 0 ? LOADS : p.keep ? (FE == FE_GLU_FWD ? 3 : 2) : 1;
        auto box_of = [&](uint32_t k) { return my_boxes + (k & slot_mask) * Cfg::EP_BYTES; };
        auto load_group = [&](int g) {   // the pre-activations of group g (lane 0)
#pragma unroll
          for (int u = 0; u < LOADS; ++u) {
            const uint32_t k = ep_count + uint32_t(g * LOADS + u);
            mbar_expect_tx(&my_full[k & slot_mask], Cfg::EP_BYTES);
            if (FE == FE_GLU_BWD) tma_load_3d(box_of(k), &tmap_x, &my_full[k & slot_mask], col_of(g), u, row0);
            else tma_load_2d(box_of(k), &tmap_x, &my_full[k & slot_mask], col_of(g), row0);
          }
        };
        static_assert(EP_BUFS == 2, "a group has two boxes at a time");
        const TileBias bias(p, c0, COLS, lane);
        constexpr int DEPTH = LOADS > 0 ? EP_BUFS / LOADS : 1;   // groups whose loads the boxes hold
        if (LOADS > 0 && lane == 0) {
          bulk_wait_read<0>();
          for (int g = 0; g < DEPTH && g < groups; ++g) load_group(g);
        }
        [[maybe_unused]] float co[FE == FE_ROPE ? 32 : 1], si[FE == FE_ROPE ? 32 : 1];
        [[maybe_unused]] auto load_angles = [&](int c) {
          if constexpr (FE == FE_ROPE) {
            const float4* at = reinterpret_cast<const float4*>(p.cs + size_t((row0 + lane) % p.S) * head + 32 * c);
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              const uint4 a = ld_v4(at + j), b = ld_v4(at + (head >> 3) + j);
              co[4 * j] = __uint_as_float(a.x); co[4 * j + 1] = __uint_as_float(a.y);
              co[4 * j + 2] = __uint_as_float(a.z); co[4 * j + 3] = __uint_as_float(a.w);
              si[4 * j] = __uint_as_float(b.x); si[4 * j + 1] = __uint_as_float(b.y);
              si[4 * j + 2] = __uint_as_float(b.z); si[4 * j + 3] = __uint_as_float(b.w);
            }
          }
        };
        if (FE == FE_ROPE && groups > 0 && c0 < p.rope_cols) load_angles(half_of(0));   // under the main loop
        if (!__all_sync(0xffffffffu, mbar_wait(&tmem_full[buf], use & 1, wctx, ST_TIMEOUT_TMEM_FULL))) break;
        tc_fence_after();
        auto release_tmem = [&] {
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive_cluster(&tmem_empty[buf], 0);
        };
        bool ok = true;
        if (groups == 0) release_tmem();
#pragma unroll 1
        for (int g = 0; g < groups; ++g) {
          const uint32_t k = ep_count + uint32_t(g * per_group);
          const uint32_t row_off = uint32_t(lane) * 128, sw = uint32_t(lane & 7);
          const uint32_t box0 = smem_u32(box_of(k)) + row_off, box1 = smem_u32(box_of(k + 1)) + row_off;
          const int col = col_of(g);
          const uint32_t t_addr = tmem_base + (uint32_t(q * 32) << 16) + uint32_t(buf * BN + col - c0);
          uint32_t r[32], s[32];
          tmem_ld32(t_addr, r);
          tmem_ld32(t_addr + (FE == FE_GLU_FWD ? uint32_t(HALF_N) : FE == FE_ROPE ? uint32_t(head >> 1) : 32u), s);
          if (lane == 0) {
            if (LOADS > 0) {
              if (g > 0 && g - 1 + DEPTH < groups) {   // the boxes of group g - 1 take the loads of group g - 1 + DEPTH
                bulk_wait_read<0>();
                load_group(g - 1 + DEPTH);
              }
            } else if (per_group == 1) {
              bulk_wait_read<EP_BUFS - 1>();
            } else {
              bulk_wait_read<0>();   // two or three boxes: all
            }
          }
          tmem_wait_ld();
          if constexpr (FE == FE_ROPE) {
            const int far = head >> 1;   // from a column to the other of its pair
            if (halves == 2 && !half_each && g == heads && c0 < p.rope_cols) load_angles(1);
            if (g == groups - 1) release_tmem();
            else __syncwarp();
            bias.add(p, col - c0, r);
            bias.add(p, col - c0 + far, s);
            // the values as they would be stored, like a pass over them sees them
            uint4 x[4], y[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              x[j] = pack_f32x8(r, 8 * j);
              y[j] = pack_f32x8(s, 8 * j);
              if (col < p.rope_cols) {
                uint32_t xs[4] = {x[j].x, x[j].y, x[j].z, x[j].w}, ys[4] = {y[j].x, y[j].y, y[j].z, y[j].w};
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                  const float2 a = unpack_bf16x2(xs[u]), b = unpack_bf16x2(ys[u]);
                  const int i = 8 * j + 2 * u;
                  xs[u] = pack_bf16x2(a.x * co[i] - b.x * si[i], a.y * co[i + 1] - b.y * si[i + 1]);
                  ys[u] = pack_bf16x2(b.x * co[i] + a.x * si[i], b.y * co[i + 1] + a.y * si[i + 1]);
                }
                x[j] = make_uint4(xs[0], xs[1], xs[2], xs[3]);
                y[j] = make_uint4(ys[0], ys[1], ys[2], ys[3]);
              }
            }
            if (halves == 1) {
#pragma unroll
              for (int j = 0; j < 4; ++j) {
                st_shared_v4(box0 + ((uint32_t(j) ^ sw) << 4), x[j].x, x[j].y, x[j].z, x[j].w);
                st_shared_v4(box0 + ((uint32_t(4 + j) ^ sw) << 4), y[j].x, y[j].y, y[j].z, y[j].w);
              }
            } else {   // two boxes of 32 rows of 64 bytes, their 16-byte pieces swizzled by two bits of the row
              const uint32_t at = smem_u32(box_of(k)) + uint32_t(lane) * 64, sw2 = uint32_t(lane >> 1) & 3;
#pragma unroll
              for (int j = 0; j < 4; ++j) {
                st_shared_v4(at + ((uint32_t(j) ^ sw2) << 4), x[j].x, x[j].y, x[j].z, x[j].w);
                st_shared_v4(at + uint32_t(Cfg::EP_BYTES / 2) + ((uint32_t(j) ^ sw2) << 4), y[j].x, y[j].y, y[j].z, y[j].w);
              }
            }
            fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) {
              if (zb_in_bounds(row0 >= 0 && row0 < p.M && col >= 0 && col + far < p.N, p.status, 2)) {
                tma_store_2d(&tmap_w, box_of(k), col, row0);
                if (halves == 2) tma_store_2d(&tmap_w, box_of(k) + Cfg::EP_BYTES / 2, col + far, row0);
              }
              bulk_commit();
            }
          } else if constexpr (FE == FE_GLU_FWD) {
            uint4 a[8];
#pragma unroll
            for (int c = 0; c < 2; ++c) {
              if (c == 1) {
                tmem_ld32(t_addr + 32u, r);
                tmem_ld32(t_addr + uint32_t(HALF_N) + 32u, s);
                tmem_wait_ld();
                if (g == groups - 1) release_tmem();
              } else {
                __syncwarp();
              }
#pragma unroll
              for (int j = 0; j < 4; ++j) {
                const uint4 x = pack_f32x8(r, 8 * j), y = pack_f32x8(s, 8 * j);
                const uint32_t off = (uint32_t(c * 4 + j) ^ sw) << 4;
                if (p.keep) {
                  st_shared_v4(box0 + off, x.x, x.y, x.z, x.w);
                  st_shared_v4(box1 + off, y.x, y.y, y.z, y.w);
                }
                // of the values as they are stored, like a pass over them would see them
                const uint32_t xs[4] = {x.x, x.y, x.z, x.w}, ys[4] = {y.x, y.y, y.z, y.w};
                uint32_t o[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                  const float2 gate = unpack_bf16x2(xs[u]), up = unpack_bf16x2(ys[u]);
                  o[u] = pack_bf16x2(swiglu_fwd(gate.x, up.x), swiglu_fwd(gate.y, up.y));
                }
                a[c * 4 + j] = make_uint4(o[0], o[1], o[2], o[3]);
              }
            }
            uint8_t* last = box_of(k + uint32_t(per_group - 1));
            if (p.keep) {
              fence_proxy_async_smem();
              __syncwarp();
              if (lane == 0) {
                if (zb_in_bounds(row0 >= 0 && row0 < p.M && col >= 0 && col < p.N, p.status, 2)) {
                  tma_store_3d(&tmap_c, box_of(k), col, 0, row0);
                  tma_store_3d(&tmap_c, box_of(k + 1), col, 1, row0);
                }
                bulk_commit();
                bulk_wait_read<0>();   // the third box takes the place of the first
              }
              __syncwarp();
            }
            const uint32_t at = smem_u32(last) + row_off;
#pragma unroll
            for (int j = 0; j < 8; ++j) st_shared_v4(at + ((uint32_t(j) ^ sw) << 4), a[j].x, a[j].y, a[j].z, a[j].w);
            fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) {
              if (zb_in_bounds(row0 >= 0 && row0 < p.M && col >= 0 && col < p.N, p.status, 2)) tma_store_2d(&tmap_w, last, col, row0);
              bulk_commit();
            }
          } else {
            if (g == groups - 1) release_tmem();
            if constexpr (FE == FE_ACT_FWD) {
              bias.add(p, col - c0, r);
              bias.add(p, col - c0 + 32, s);
              __syncwarp();
            } else {
              __syncwarp();
#pragma unroll
              for (int u = 0; u < LOADS; ++u)
                ok = ok && __all_sync(0xffffffffu, mbar_wait(&my_full[(k + u) & slot_mask], ((k + u) >> phase_shift) & 1, wctx, ST_TIMEOUT_FULL));
              if (!ok) break;
            }
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              const uint4 x = j < 4 ? pack_f32x8(r, 8 * j) : pack_f32x8(s, 8 * (j - 4));   // h, or the gradient of the activation
              const uint32_t off = (uint32_t(j) ^ sw) << 4;
              const uint32_t xs[4] = {x.x, x.y, x.z, x.w};
              uint32_t o[4], o2[4];
              if constexpr (FE == FE_ACT_FWD) {
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                  const float2 a = act_fwd2(unpack_bf16x2(xs[u]), p.act);
                  o[u] = pack_bf16x2(a.x, a.y);
                }
                if (p.keep) st_shared_v4(box0 + off, x.x, x.y, x.z, x.w);
                st_shared_v4((p.keep ? box1 : box0) + off, o[0], o[1], o[2], o[3]);
              } else if constexpr (FE == FE_ACT_BWD) {
                const uint4 h = ld_shared_v4(box0 + off);
                const uint32_t hs[4] = {h.x, h.y, h.z, h.w};
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                  const float2 d = unpack_bf16x2(xs[u]), slope = act_bwd2(unpack_bf16x2(hs[u]), p.act);
                  o[u] = pack_bf16x2(d.x * slope.x, d.y * slope.y);
                }
                st_shared_v4(box0 + off, o[0], o[1], o[2], o[3]);
              } else {
                const uint4 gv = ld_shared_v4(box0 + off), uv = ld_shared_v4(box1 + off);
                const uint32_t gs[4] = {gv.x, gv.y, gv.z, gv.w}, us[4] = {uv.x, uv.y, uv.z, uv.w};
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                  const float2 d = unpack_bf16x2(xs[u]), gate = unpack_bf16x2(gs[u]), up = unpack_bf16x2(us[u]);
                  float dg0, dg1, du0, du1;
                  swiglu_bwd(gate.x, up.x, d.x, dg0, du0);
                  swiglu_bwd(gate.y, up.y, d.y, dg1, du1);
                  o[u] = pack_bf16x2(dg0, dg1);
                  o2[u] = pack_bf16x2(du0, du1);
                }
                st_shared_v4(box0 + off, o[0], o[1], o[2], o[3]);
                st_shared_v4(box1 + off, o2[0], o2[1], o2[2], o2[3]);
              }
            }
            fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) {
              const bool in = zb_in_bounds(row0 >= 0 && row0 < p.M && col >= 0 && col < p.N, p.status, 2);
              if constexpr (FE == FE_ACT_FWD) {
                if (p.keep) {
                  if (in) tma_store_2d(&tmap_c, box_of(k), col, row0);
                  bulk_commit();
                }
                if (in) tma_store_2d(&tmap_w, box_of(k + uint32_t(per_group - 1)), col, row0);
              } else if constexpr (FE == FE_ACT_BWD) {
                if (in) tma_store_2d(&tmap_c, box_of(k), col, row0);
              } else {
                if (in) tma_store_3d(&tmap_c, box_of(k), col, 0, row0);
                if (in) tma_store_3d(&tmap_c, box_of(k + 1), col, 1, row0);
              }
              bulk_commit();
            }
          }
        }
        ep_count += uint32_t(groups * per_group);
        if (!ok) break;
      } else if (!SCATTER && ex.ep != EP_DIRECT) {
        const bool f32 = split || ex.ep == EP_F32;
        const int row0 = m0 + q * 32;
        const int wide = f32 ? 32 : 64;                    // columns of a box
        const int boxes = mine(split ? BN / 32 : row0 < p.M ? min(BN / wide, (p.N - n0 + wide - 1) / wide) : 0);
        auto col_of = [&](int i) { return n0 + (h + i * EP_GROUPS) * wide; };   // this warp's i-th box
        auto load_box = [&](int i) {   // old C or addend -> its ring slot (lane 0)
          const uint32_t k = ep_count + uint32_t(i);
          mbar_expect_tx(&my_full[k & slot_mask], Cfg::EP_BYTES);
          tma_load_2d(my_boxes + (k & slot_mask) * Cfg::EP_BYTES, &tmap_x, &my_full[k & slot_mask], col_of(i), row0);
        };
        const TileBias bias(p, n0, BN, lane);
        if (ex.ep_load && !split && lane == 0) {
          bulk_wait_read<0>();   // stores of earlier boxes (issued a main loop ago) still hold the slots
          for (int i = 0; i < EP_BUFS && i < boxes; ++i) load_box(i);
        }
        if (!__all_sync(0xffffffffu, mbar_wait(&tmem_full[buf], use & 1, wctx, ST_TIMEOUT_TMEM_FULL))) break;
        tc_fence_after();
        auto release_tmem = [&] {   // this warp has read its part of the accumulators
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive_cluster(&tmem_empty[buf], 0);
        };
        auto wait_slot = [&] { bulk_wait_read<EP_BUFS - 1>(); };   // the store of box k - EP_BUFS has left the slot of box k
        bool ok = true;
        if (boxes == 0) release_tmem();
        for (int c = 0; c < boxes; ++c) {
          const uint32_t k = ep_count + uint32_t(c);
          const uint32_t box = smem_u32(my_boxes + (k & slot_mask) * Cfg::EP_BYTES) + uint32_t(lane) * 128;
          const int col0 = col_of(c);
          const uint32_t t_addr = tmem_base + (uint32_t(q * 32) << 16) + uint32_t(buf * BN + col0 - n0);
          if (f32) {
            uint32_t r[32];
            tmem_ld32(t_addr, r);
            if (lane == 0) wait_slot();
            tmem_wait_ld();
            if (c == boxes - 1) release_tmem();
            if (!split) { bias.add(p, col0 - n0, r); epilogue_act(p, r); }
            __syncwarp();
#pragma unroll
            for (int j = 0; j < 8; ++j)
              st_shared_v4(box + uint32_t((j ^ (lane & 7)) << 4), r[4 * j], r[4 * j + 1], r[4 * j + 2], r[4 * j + 3]);
          } else {
            uint32_t r[32], s[32];
            tmem_ld32(t_addr, r);
            tmem_ld32(t_addr + 32u, s);
            if (lane == 0) {
              if (!ex.ep_load) {
                wait_slot();
              } else if (c > 0 && c - 1 + EP_BUFS < boxes) {
                bulk_wait_read<0>();   // box c - 1 has left: its slot takes the next one
                load_box(c - 1 + EP_BUFS);
              }
            }
            tmem_wait_ld();
            if (c == boxes - 1) release_tmem();
            bias.add(p, col0 - n0, r);
            bias.add(p, col0 - n0 + 32, s);
            epilogue_act(p, r);
            epilogue_act(p, s);
            __syncwarp();
            if (ex.ep_load) {
              ok = __all_sync(0xffffffffu, mbar_wait(&my_full[k & slot_mask], (k >> phase_shift) & 1, wctx, ST_TIMEOUT_FULL));
              if (!ok) break;
#pragma unroll
              for (int j = 0; j < 4; ++j) {
                add_bf16x8(r, 8 * j, ld_shared_v4(box + uint32_t((j ^ (lane & 7)) << 4)));
                add_bf16x8(s, 8 * j, ld_shared_v4(box + uint32_t(((j + 4) ^ (lane & 7)) << 4)));
              }
            }
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              const uint4 a = pack_f32x8(r, 8 * j), b = pack_f32x8(s, 8 * j);
              st_shared_v4(box + uint32_t((j ^ (lane & 7)) << 4), a.x, a.y, a.z, a.w);
              st_shared_v4(box + uint32_t(((j + 4) ^ (lane & 7)) << 4), b.x, b.y, b.z, b.w);
            }
          }
          fence_proxy_async_smem();
          __syncwarp();
          if (lane == 0) {
            const void* src = my_boxes + (k & slot_mask) * Cfg::EP_BYTES;
            if (split) {
              tma_store_2d(&tmap_w, src, col0 - n0, (item - ex.full) * Cfg::BM + int(cta) * 128 + q * 32);
            } else if (zb_in_bounds(row0 >= 0 && row0 < p.M && col0 >= 0 && col0 < p.N, p.status, 2)) {
              if (ex.ep == EP_F32 && ecfg.accum) tma_reduce_add_2d(&tmap_c, src, col0, row0);
              else tma_store_2d(&tmap_c, src, col0, row0);
            }
            bulk_commit();
          }
        }
        ep_count += uint32_t(boxes);
        if (!ok) break;
      } else {
      if (!__all_sync(0xffffffffu, mbar_wait(&tmem_full[buf], use & 1, wctx, ST_TIMEOUT_TMEM_FULL))) break;
      tc_fence_after();
      const int row = m0 + q * 32 + lane;
      const bool row_ok = row < p.M;
      __nv_bfloat16* crow = nullptr;   // SCATTER: this thread's destination row
      if constexpr (SCATTER) if (row_ok) {
        const int owner = row / p.sc_rows;
        crow = static_cast<__nv_bfloat16*>(p.sc_dst[owner]) + size_t(row - owner * p.sc_rows) * p.ldc;
      }
#pragma unroll 1
      for (int c = h; c < BN / 32; c += EP_GROUPS) {
        const int col0 = n0 + c * 32;
        if (col0 >= p.N) break;
        uint32_t r[32];
        tmem_ld32(tmem_base + (uint32_t(q * 32) << 16) + uint32_t(buf * BN + c * 32), r);
        tmem_wait_ld();
        if (!row_ok) continue;
        if constexpr (SCATTER) epilogue_scatter_chunk(crow, col0, p.N, ecfg.vec_ok, r);
        else epilogue_store_chunk(p, ecfg, row, col0, r);
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(&tmem_empty[buf], 0);
      }
    }
    if constexpr (SCATTER) __threadfence_system();   // this thread's rows are visible to their owners before the flags
  }

  if constexpr (FUSED_AG) if (warp >= 2 + EP_WARPS) {
    // ------------------------------ all-gather copy warps ------------------------------
    const AgParams& ag = p.ag;
    const int ct = threadIdx.x - (64 + 32 * EP_WARPS);  // 0..127
    __shared__ int s_peer_ok;
    const int total = (ag.R - 1) * ag.cps;
    const long chunk16 = ag.chunk_bytes / 16;
    const long shard16 = ag.shard_bytes / 16;
    int checked_peer = -1;
    bool ok = true;
    for (int w = blockIdx.x; w < total && ok; w += gridDim.x) {
      // ascending chunk order inside each peer, peers visited starting after this rank
      const int c = w / (ag.R - 1);
      const int pi = w % (ag.R - 1);
      const int peer = (ag.r + 1 + pi) % ag.R;
      if (peer != checked_peer) {
        if (ct == 0)
          s_peer_ok = flag_wait_ge(ag.version_flags + peer, ag.need_version, ZB_WAIT_NS, p.status, ST_TIMEOUT_FLAG) ? 1 : 0;
        asm volatile("bar.sync 1, 128;" ::: "memory");
        ok = s_peer_ok != 0;
        asm volatile("bar.sync 1, 128;" ::: "memory");
        checked_peer = peer;
        if (!ok) break;
      }
      const long beg = long(c) * chunk16;
      const long end = min(beg + chunk16, shard16);
      if (!zb_in_bounds(peer >= 0 && peer < ag.R && peer != ag.r && beg >= 0 && end <= shard16 && beg <= end, p.status, 3)) break;
      if (!zb_in_bounds(peer * ag.cps + c < ag.R * ag.cps && c >= 0, p.status, 4)) break;
      const uint4* src = ag.src[peer];
      uint4* dst = ag.dst + long(peer) * shard16;
      long i = beg + ct;
      // Software-pipelined copy: the 8 requests of the next batch are issued before the 8 values of the current one are
      // stored, so a thread always has 8 - 16 peer loads of 16 bytes in flight (up to 32 KiB per CTA, 4.7 MB per GPU)
      // instead of draining to zero between batches.
      constexpr int UB = 8;
      const long step = long(UB) * 128;
      if (i + (UB - 1) * 128 < end) {
        uint4 cur[UB], nxt[UB];
#pragma unroll
        for (int u = 0; u < UB; ++u) cur[u] = ld_v4_relaxed_sys(src + i + u * 128);
        for (; i + step + (UB - 1) * 128 < end; i += step) {
#pragma unroll
          for (int u = 0; u < UB; ++u) nxt[u] = ld_v4_relaxed_sys(src + i + step + u * 128);
#pragma unroll
          for (int u = 0; u < UB; ++u) dst[i + u * 128] = cur[u];
#pragma unroll
          for (int u = 0; u < UB; ++u) cur[u] = nxt[u];
        }
#pragma unroll
        for (int u = 0; u < UB; ++u) dst[i + u * 128] = cur[u];
        i += step;
      }
      for (; i < end; i += 128) dst[i] = ld_v4_relaxed_sys(src + i);
      // the rows go from these stores (generic proxy) to the TMA loads of some CTA's producer (async proxy)
      __threadfence();
      asm volatile("fence.proxy.async.global;" ::: "memory");
      asm volatile("bar.sync 1, 128;" ::: "memory");
      if (ct == 0) st_release_sys(ag.chunk_flags + peer * ag.cps + c, ag.epoch);
    }
    if (!ok) *abort_flag = 1;
  }

  // ------------------------------ teardown ------------------------------
  __syncwarp();
  if (*abort_flag) {
    for (int i = 0; i < 64; ++i) __nanosleep(1000);
  }
  tc_fence_before();
  // The leader's MMAs read the peer's shared memory: leave together.  Where nothing written before is read behind this
  // barrier it need not order memory: a releasing arrival waits for the epilogue's own writes, 0.5 us at the end of a short
  // product (1018 x 2048 x 512 6.25 -> 5.75 us, 3072 x 768 x 768 7.24 -> 6.64, 3072 x 3072 x 768 13.3 -> 12.9).  Arrivals on the other CTA's barriers are no such writes: the issuer of the leader has waited for them above.
  // The stores of the last boxes are still being read meanwhile (their writes are complete when the grid is).
  if constexpr (SCATTER || FUSED_AG) asm volatile("barrier.cluster.arrive.aligned;" ::: "memory");
  else asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");
  if (warp >= 2 && lane == 0) bulk_wait_read<0>();
  __syncwarp();
  asm volatile("barrier.cluster.wait.aligned;" ::: "memory");
  if constexpr (!SCATTER && !FUSED_AG) {
    if (late) chain_wait();
  }
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc_pair(tmem_base, Cfg::TMEM_COLS);
  }
  if constexpr (SCATTER) if (threadIdx.x == 0) {
    // last CTA of the grid: every row has been stored and fenced; tell the owners (not after a timeout:
    // the status word is then non-zero and the owners' bounded wait reports it)
    if (atomicAdd(p.sc_counter, 1u) == gridDim.x - 1) {
      __threadfence_system();
      if (*reinterpret_cast<volatile int*>(p.status) == 0)
        for (int q = 0; q < p.sc_R; ++q) st_release_sys(p.sc_flags[q] + p.sc_flag_index, p.sc_epoch);
      *p.sc_counter = 0u;
    }
  }
}

// 3-D view of an MN-major operand stored [K rows, MN cols]: {64 within a block, K, MN/64 blocks}
static int make_tmap_mn3d(CUtensorMap* out, const void* base, uint64_t krows, uint64_t mn, uint64_t ld, uint32_t blocks) {
  uint64_t dims[3] = {64, krows, mn / 64};
  uint64_t strides[2] = {ld * 2, 128};
  uint32_t box[3] = {64, 64, blocks};
  return make_tmap_nd_bf16(out, base, 3, dims, strides, box);
}

// Tile order.  The operand of the band (the one with fewer tiles) is read from DRAM once per band and stays in L2 while
// the other operand streams through once per band, so a band as wide as that dimension reads both operands once.  It
// has to fit: with a band of more than BAND_BYTES (about a third of L2, each die keeps its own copy of what its SMs
// read) every wave reads the band again, and then the narrower bands win whose waves are close to square (74 pairs:
// 8 - 10 tiles).  The all-gather kernel keeps rows of B ascending, the order in which its chunks arrive.
// Weight gradient 22016 x 4096 x 4096 (fp32 bucket): 826 us with rows fastest, which read dY^T once per 256 columns,
// 674 us so.
template <typename Params, int BN>
static TileOrder gemm2_tile_order(int M, int N, int K) {
  constexpr long BAND_BYTES = 40l << 20;
  TileOrder o;
  o.tiles_m = (M + Gemm2Cfg<BN>::BM - 1) / Gemm2Cfg<BN>::BM;
  o.tiles_n = (N + BN - 1) / BN;
  o.n_fast = !std::is_same<Params, GemmAgParams>::value && o.tiles_n < o.tiles_m;
  const int nf = o.n_fast ? o.tiles_n : o.tiles_m;
  o.band = nf;
  if (!std::is_same<Params, GemmAgParams>::value && (nf > 16 || long(nf) * (o.n_fast ? BN : 256) * K * 2 > BAND_BYTES)) {
    const int bands = (nf + 9) / 10;
    o.band = (nf + bands - 1) / bands;
  }
  return o;
}

// Adds up the parts of the split tiles, in their order, and finishes them like the epilogue: bias, activation, addend, old C.
// One thread per 8 columns of a row; rows of C and of the addend are 16-byte aligned.
template <int BN>
__global__ void __launch_bounds__(256)
gemm2_fixup_kernel(const float* ws, const GemmParams p, const TileOrder order, int first_tile, int splits) {
  chain_trigger();
  chain_wait();
  constexpr int CHUNKS = 256 * BN / 8;
  const int w = blockIdx.x * 256 + threadIdx.x;
  const int t = w / CHUNKS, e = w - t * CHUNKS;
  const int rr = e / (BN / 8), cc = e % (BN / 8) * 8;
  int tm, tn;
  tile_at(order, first_tile + t, tm, tn);
  const int row = tm * 256 + rr, col = tn * BN + cc;
  if (row >= p.M || col >= p.N) return;
  const float* src = ws + size_t(t) * splits * (256 * BN) + size_t(rr) * BN + cc;
  float v[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  for (int s = 0; s < splits; ++s, src += 256 * BN) {
    const float4 a = reinterpret_cast<const float4*>(src)[0], b = reinterpret_cast<const float4*>(src)[1];
    v[0] += a.x; v[1] += a.y; v[2] += a.z; v[3] += a.w;
    v[4] += b.x; v[5] += b.y; v[6] += b.z; v[7] += b.w;
  }
  const int n = min(8, p.N - col);
  const bool acc = (p.flags & GEMM_ACCUMULATE) != 0;
  for (int j = 0; j < 8; ++j) {
    if (p.bias != nullptr && j < n) v[j] += __bfloat162float(p.bias[col + j]);
    if (p.flags & GEMM_GELU) v[j] = gelu_tanh(v[j]);
    else if (p.flags & GEMM_RELU) v[j] = fmaxf(v[j], 0.f);
  }
  auto add8 = [&](const __nv_bfloat16* at) {
    if (n == 8) {
      const uint4 u = *reinterpret_cast<const uint4*>(at);
      const float2 a = unpack_bf16x2(u.x), b = unpack_bf16x2(u.y), c = unpack_bf16x2(u.z), d = unpack_bf16x2(u.w);
      v[0] += a.x; v[1] += a.y; v[2] += b.x; v[3] += b.y; v[4] += c.x; v[5] += c.y; v[6] += d.x; v[7] += d.y;
    } else {
      for (int j = 0; j < n; ++j) v[j] += __bfloat162float(at[j]);
    }
  };
  if (p.addend != nullptr) add8(p.addend + size_t(row) * p.ld_addend + col);
  if (p.flags & GEMM_OUT_F32) {
    float* c = static_cast<float*>(p.C) + size_t(row) * p.ldc + col;
    for (int j = 0; j < n; ++j) c[j] = acc ? c[j] + v[j] : v[j];
  } else {
    __nv_bfloat16* c = static_cast<__nv_bfloat16*>(p.C) + size_t(row) * p.ldc + col;
    if (acc) add8(c);
    if (n == 8) {
      uint4 o;
      o.x = pack_bf16x2(v[0], v[1]); o.y = pack_bf16x2(v[2], v[3]);
      o.z = pack_bf16x2(v[4], v[5]); o.w = pack_bf16x2(v[6], v[7]);
      *reinterpret_cast<uint4*>(c) = o;
    } else {
      for (int j = 0; j < n; ++j) c[j] = __float2bfloat16(v[j]);
    }
  }
}

// Width of a pair's tile.  A wave of 128-column tiles over the 74 pairs takes between 0.58 (K = 20480) and 0.67 (K = 2048)
// of the time of a wave of 256-column tiles (A is read again for half as many columns, and the tile's fixed cost stays), so
// the narrow tile wins where the wide one leaves many pairs without a tile or the last wave nearly empty.
// Wide -> narrow, us: 1018 x 512 x 49152 225 -> 145, 3072 x 768 x 3072 25.4 -> 21.3, weight gradients 768 x 768 x 3072
// 25.3 -> 20.5 and 3072 x 768 x 4616 34.8 -> 28.7 (fp32), 2048 x 2304 x 768 21.3 -> 17.3.  The line is drawn at 0.67:
// 2048 x 5120 x 20480 (three waves against five) lost 5 %, 3072 x 2048 x 3000 (two against three) 4 %.
//
// Parts of a last wave: with a workspace the R tiles that are left behind the last full wave can be cut into
// min(pairs / R, 16) parts of at least 8 k-blocks each.  That saves up to a wave and costs about 18 us (fp32 sums out and in
// again, one more launch), the time of a 256-column wave at
// K = 3000.  2048 x 5120 x 20480 (160 tiles, 12 left, six parts each) 331 -> 259 us, x 5120 87 -> 79; 4096 x 4096 x 22016 492 ->
// 458; 3000 x 2048 x 8192 91 -> 75; 1018 x 512 x 49152 (all eight tiles in nine parts) 149 -> 56; weight gradient
// 6144 x 4096 x 8192 280 -> 249.  Error against fp64 as before, in fp32 outputs a little smaller.
struct Gemm2Plan {
  int bn, splits;
};
static Gemm2Plan gemm2_plan(int M, int N, int K, int pairs, bool may_split) {
  constexpr long SPLIT_COST = 3000 * 100;
  Gemm2Plan best = {256, 1};
  long best_cost = -1;
  for (int bn = 256; bn >= 128; bn -= 128) {
    const long unit = bn == 256 ? 100 : 67;   // cost of a wave per column of K
    const long tiles = long((M + 255) / 256) * ((N + bn - 1) / bn), full = tiles / pairs, rest = tiles % pairs;
    auto consider = [&](long cost, int splits) {
      if (best_cost < 0 || cost < best_cost) {
        best_cost = cost;
        best = {bn, splits};
      }
    };
    consider((full + (rest > 0)) * unit * K, 1);
    if (may_split && rest > 0) {
      const int parts = int(std::min(std::min(pairs / rest, 16l), long((K + 63) / 64 / 8)));
      if (parts > 1) consider(full * unit * K + unit * K / parts + SPLIT_COST, parts);
    }
  }
  return best;
}

// Bytes of the fp32 sums of a plan's split tiles (at most one slot per pair).
static long gemm2_ws_bytes(const Gemm2Plan& plan, int M, int N, int pairs) {
  if (plan.splits <= 1) return 0;
  const long tiles = long((M + 255) / 256) * ((N + plan.bn - 1) / plan.bn);
  return tiles % pairs * plan.splits * 256 * plan.bn * 4;
}

template <bool A_MN, bool B_MN, typename Params = GemmParams, int BN = 256>
static int launch_gemm2(const void* A, const void* B, const Params& p, int lda, int ldb, int max_ctas,
                        cudaStream_t stream, float* ws = nullptr, long ws_bytes = 0) {
  using Cfg = Gemm2Cfg<BN>;
  int pairs = num_sms() / 2;
  if (max_ctas > 0 && max_ctas / 2 < pairs) pairs = max_ctas / 2 > 0 ? max_ctas / 2 : 1;
  CUtensorMap ta, tb;
  Gemm2Extra ex = {};
  // TMA epilogue: 16-byte aligned rows that do not overlap (a broadcast addend has a row stride of 0, which no tensor map
  // takes), rows of C that end on a 16-byte boundary (a store writes whole 16-byte pieces: it would clear what follows the
  // last column of a wider matrix), and at most one tensor to add to a bf16 output
  CUtensorMap tc = {}, tx = {}, tw = {};
  const bool f32 = (p.flags & GEMM_OUT_F32) != 0, acc = (p.flags & GEMM_ACCUMULATE) != 0, add = p.addend != nullptr;
  auto rows_ok = [&](const void* base, long ld, int size) {
    return (reinterpret_cast<uintptr_t>(base) & 15) == 0 && ld * size % 16 == 0 && ld >= p.N;
  };
  if (std::is_same<Params, GemmParams>::value && rows_ok(p.C, p.ldc, f32 ? 4 : 2) && p.N % (f32 ? 4 : 8) == 0 &&
      !(f32 ? add : (add && acc)) && (!add || rows_ok(p.addend, p.ld_addend, 2))) {
    ex.ep = f32 ? EP_F32 : EP_BF16;
    ex.ep_load = !f32 && (acc || add);
  }
  Gemm2Plan plan = {BN, 1};
  if constexpr (std::is_same<Params, GemmParams>::value) {
    // Parts need the boxes of the TMA epilogue and room for the sums of the plan this device gives; whole tiles otherwise.
    plan = gemm2_plan(p.M, p.N, p.K, pairs, ws != nullptr && ex.ep != EP_DIRECT);
    if (gemm2_ws_bytes(plan, p.M, p.N, pairs) > ws_bytes) plan = gemm2_plan(p.M, p.N, p.K, pairs, false);
    if (BN == 256 && plan.bn == 128)
      return launch_gemm2<A_MN, B_MN, Params, 128>(A, B, p, lda, ldb, max_ctas, stream, ws, ws_bytes);
  }
  if (ex.ep != EP_DIRECT) {
    int rc_ep = make_tmap_2d_out(&tc, p.C, p.M, p.N, p.ldc, f32, 32);
    if (rc_ep) return rc_ep;
    if (add) rc_ep = make_tmap_2d_out(&tx, p.addend, p.M, p.N, p.ld_addend, false, 32);
    else tx = tc;
    if (rc_ep) return rc_ep;
  }
  int rc;
  if (!A_MN) rc = make_tmap_2d_bf16(&ta, A, p.M, p.K, lda, 128, 64);
  else if (p.M % 64 == 0) { rc = make_tmap_mn3d(&ta, A, p.K, p.M, lda, 2); ex.a_3d = 1; }
  else rc = make_tmap_2d_bf16(&ta, A, p.K, p.M, lda, 64, 64);
  if (rc) return rc;
  if (!B_MN) rc = make_tmap_2d_bf16(&tb, B, p.N, p.K, ldb, BN / 2, 64);
  else if (p.N % 64 == 0) { rc = make_tmap_mn3d(&tb, B, p.K, p.N, ldb, BN / 128); ex.b_3d = 1; }
  else rc = make_tmap_2d_bf16(&tb, B, p.K, p.N, ldb, 64, 64);
  if (rc) return rc;
  // fewer stages and two boxes per warp where the tile's epilogue is not hidden by a long main loop (comment at Gemm2Cfg)
  constexpr bool PLAIN = std::is_same<Params, GemmParams>::value;
  constexpr int WARPS = 4;
  const bool short_k = PLAIN && ex.ep != EP_DIRECT && p.K < 2048;
  auto kern = gemm2_bf16_kernel<A_MN, B_MN, Params, BN, WARPS, Gemm2Cfg<BN>::EP_SMALL / WARPS>;
  if constexpr (PLAIN) {
    if (short_k) kern = gemm2_bf16_kernel<A_MN, B_MN, Params, BN, WARPS, Gemm2Cfg<BN>::EP_LARGE / WARPS>;
  }
  static bool attr_set[2] = {false, false};
  if (!attr_set[short_k]) {
    ZB_CUDA_OK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::SMEM_BYTES));
    attr_set[short_k] = true;
  }
  ex.order = gemm2_tile_order<Params, BN>(p.M, p.N, p.K);
  const int tiles = ex.order.tiles_m * ex.order.tiles_n;
  ex.items = ex.full = tiles;
  ex.splits = 1;
  if (plan.splits > 1) {
    ex.full = tiles / pairs * pairs;
    ex.splits = plan.splits;
    ex.items = ex.full + (tiles - ex.full) * ex.splits;
    if ((rc = make_tmap_2d_out(&tw, ws, uint64_t(ex.items - ex.full) * 256, BN, BN, true, 32))) return rc;
  }
  if (ex.items < pairs) pairs = ex.items;
  if constexpr (std::is_same<Params, GemmParams>::value) {
    ZB_CUDA_OK(launch_chained(kern, dim3(2 * pairs), 64 + 32 * WARPS, Cfg::SMEM_BYTES, stream, 0, ta, tb, tc, tx, tw, p, ex));
  } else {
    kern<<<2 * pairs, 64 + 32 * WARPS + (std::is_same<Params, GemmAgParams>::value ? 128 : 0), Cfg::SMEM_BYTES, stream>>>(ta, tb, tc, tx, tw, p, ex);
    ZB_CUDA_OK(cudaGetLastError());
  }
  if constexpr (std::is_same<Params, GemmParams>::value) {
    if (ex.splits > 1) {
      ZB_CUDA_OK(launch_pass(gemm2_fixup_kernel<BN>, (tiles - ex.full) * (BN / 8), 256, 0, stream, ws, p, ex.order, ex.full,
                             ex.splits));
      ZB_CUDA_OK(cudaGetLastError());
    }
  }
  return 0;
}

// [rows][2][F] view of a gated unit's pre-activations (gate | up): boxes of 32 rows x 64 columns of one half, clipped at F
static int make_tmap_halves(CUtensorMap* out, const void* base, uint64_t rows, uint64_t F) {
  uint64_t dims[3] = {F, 2, rows};
  uint64_t strides[2] = {F * 2, F * 4};
  uint32_t box[3] = {64, 1, 32};
  return make_tmap_nd_bf16(out, base, 3, dims, strides, box);
}

// Products with an activation in the epilogue.  FE_ACT_FWD: act(A B^T + bias) -> out, A B^T + bias -> pre.  FE_GLU_FWD: the
// same for a gated unit (B: gate and up weights, N = F).  FE_ACT_BWD / FE_GLU_BWD: (A B) times the activation's derivative
// at `pre` -> out.  FE_ROPE: A B^T + bias with its first heads rotated -> out.  All matrices but A and B are dense.
//
// As passes of their own the activations read and write everything once more (4096 x 11008, gated: 47 us forward, 79
// backward) and cost a launch each; here the forward one works on accumulators, and the backward one fetches only what it
// needs, under the main loop of the next tile.
// The rotation, one more pass over the projection, has both halves of its pairs in the accumulators.  As two calls, as one, and
// the product alone: 8192 x 2560 x 2048, heads of 64, 69.1, 59.9 and 59.1 us; 3000 x 3072 x 1024, heads of 128, 23.0, 19.0
// and 19.8; 1024 x 1536 x 512 8.3, 6.5 and 5.5.
template <int FE, int BN>
static int launch_gemm2_fused(const void* A, const void* B, void* pre, void* out, const GemmFusedParams<FE>& p, int lda, int ldb,
                              cudaStream_t stream) {
  using Cfg = Gemm2Cfg<BN>;
  using Params = GemmFusedParams<FE>;
  constexpr bool FWD = FE == FE_ACT_FWD || FE == FE_GLU_FWD || FE == FE_ROPE, GLU = FE == FE_GLU_FWD || FE == FE_GLU_BWD;
  const int cols = FE == FE_GLU_FWD ? 2 * p.N : p.N;   // of the accumulators
  int pairs = num_sms() / 2;
  if (BN == 256 && gemm2_plan(p.M, cols, p.K, pairs, false).bn == 128)
    return launch_gemm2_fused<FE, 128>(A, B, pre, out, p, lda, ldb, stream);
  CUtensorMap ta, tb, tc = {}, tx = {}, tw = {};
  Gemm2Extra ex = {};
  ex.ep = EP_BF16;
  int rc = make_tmap_2d_bf16(&ta, A, p.M, p.K, lda, 128, 64);
  if (rc) return rc;
  if (FWD) rc = make_tmap_2d_bf16(&tb, B, cols, p.K, ldb, BN / 2, 64);
  else if (p.N % 64 == 0) { rc = make_tmap_mn3d(&tb, B, p.K, p.N, ldb, BN / 128); ex.b_3d = 1; }
  else rc = make_tmap_2d_bf16(&tb, B, p.K, p.N, ldb, 64, 64);
  if (rc) return rc;
  if (FWD) {
    if ((rc = make_tmap_2d_out(&tw, out, p.M, p.N, p.N, false, 32, FE == FE_ROPE && p.act == 128 ? 64 : 128))) return rc;
    if (p.keep) {
      rc = GLU ? make_tmap_halves(&tc, pre, p.M, p.N) : make_tmap_2d_out(&tc, pre, p.M, p.N, p.N, false, 32);
      if (rc) return rc;
    }
  } else {
    rc = GLU ? make_tmap_halves(&tx, pre, p.M, p.N) : make_tmap_2d_out(&tx, pre, p.M, p.N, p.N, false, 32);
    if (rc) return rc;
    rc = GLU ? make_tmap_halves(&tc, out, p.M, p.N) : make_tmap_2d_out(&tc, out, p.M, p.N, p.N, false, 32);
    if (rc) return rc;
  }
  // two boxes per warp: eight warps and fewer stages where the main loop is short, four and the full ring elsewhere
  const bool short_k = p.K < 2048;
  auto kern = short_k ? gemm2_bf16_kernel<false, !FWD, Params, BN, 8, 2> : gemm2_bf16_kernel<false, !FWD, Params, BN, 4, 2>;
  static bool attr_set[2] = {false, false};
  if (!attr_set[short_k]) {
    ZB_CUDA_OK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::SMEM_BYTES));
    attr_set[short_k] = true;
  }
  ex.order = gemm2_tile_order<Params, BN>(p.M, cols, p.K);
  ex.items = ex.full = ex.order.tiles_m * ex.order.tiles_n;
  ex.splits = 1;
  if (ex.items < pairs) pairs = ex.items;
  ZB_CUDA_OK(launch_chained(kern, dim3(2 * pairs), short_k ? 320 : 192, Cfg::SMEM_BYTES, stream, 0, ta, tb, tc, tx, tw, p, ex));
  return 0;
}

template <int FE>
static int gemm2_fused_entry(const void* A, const void* B, const void* bias, void* pre, void* out, int M, int N, int K, int lda,
                             int ldb, int act, int keep, int* status, cudaStream_t stream, const float* cs = nullptr, int S = 0,
                             int rope_cols = 0) {
  GemmFusedParams<FE> p = {};
  p.C = out;
  p.bias = static_cast<const __nv_bfloat16*>(bias);
  p.M = M; p.N = N; p.K = K;
  p.ldc = N;
  p.status = status;
  p.act = act;
  p.keep = keep;
  p.cs = cs;
  p.S = S;
  p.rope_cols = rope_cols;
  return launch_gemm2_fused<FE, 256>(A, B, pre, out, p, lda, ldb, stream);
}

static int gemm2_entry(const void* A, const void* B, void* C, int M, int N, int K, int lda, int ldb, int ldc,
                       int a_mn_major, int b_mn_major, const void* bias, const void* addend, int ld_addend, int flags,
                       int max_ctas, float* ws, long ws_bytes, int* status, cudaStream_t stream) {
  if (M <= 0 || N <= 0 || K <= 0) ZB_FAIL(-1, "gemm2: empty problem %d x %d x %d", M, N, K);
  GemmParams p;
  p.C = C;
  p.bias = static_cast<const __nv_bfloat16*>(bias);
  p.addend = static_cast<const __nv_bfloat16*>(addend);
  p.M = M; p.N = N; p.K = K;
  p.ldc = ldc; p.ld_addend = ld_addend;
  p.flags = flags;
  p.status = status;
  p.gate_flags = nullptr;
  p.gate_epoch = 0;
  p.gate_base = 0; p.gate_row_bytes = 0; p.gate_shard_bytes = 1;
  p.gate_chunk_bytes = 1; p.gate_cps = 1; p.gate_self = -1;
  if (!a_mn_major && !b_mn_major) return launch_gemm2<false, false>(A, B, p, lda, ldb, max_ctas, stream, ws, ws_bytes);
  if (!a_mn_major && b_mn_major) return launch_gemm2<false, true>(A, B, p, lda, ldb, max_ctas, stream, ws, ws_bytes);
  if (a_mn_major && b_mn_major) return launch_gemm2<true, true>(A, B, p, lda, ldb, max_ctas, stream, ws, ws_bytes);
  return launch_gemm2<true, false>(A, B, p, lda, ldb, max_ctas, stream, ws, ws_bytes);
}

}  // namespace zb

// Bytes of fp32 workspace (16-byte aligned) with which zb_gemm2_split_bf16 would cut the last wave of this product into
// parts; 0: it would not.
extern "C" int zb_gemm2_workspace(int M, int N, int K) {
  using namespace zb;
  if (M <= 0 || N <= 0 || K <= 0) return 0;
  const int pairs = num_sms() / 2;
  return int(gemm2_ws_bytes(gemm2_plan(M, N, K, pairs, true), M, N, pairs));
}

extern "C" int zb_gemm2_bf16(const void* A, const void* B, void* C, int M, int N, int K, int lda, int ldb, int ldc,
                             int a_mn_major, int b_mn_major, const void* bias, const void* addend, int ld_addend,
                             int flags, int max_ctas, int* status, cudaStream_t stream) {
  return zb::gemm2_entry(A, B, C, M, N, K, lda, ldb, ldc, a_mn_major, b_mn_major, bias, addend, ld_addend, flags, max_ctas,
                         nullptr, 0, status, stream);
}
// zb_gemm2_bf16 on the whole GPU with a workspace of `workspace_bytes`; one of fewer than the bytes zb_gemm2_workspace(M, N, K)
// gives on this device is not used.
extern "C" int zb_gemm2_split_bf16(const void* A, const void* B, void* C, int M, int N, int K, int lda, int ldb, int ldc,
                                   int a_mn_major, int b_mn_major, const void* bias, const void* addend, int ld_addend,
                                   int flags, void* workspace, long workspace_bytes, int* status, cudaStream_t stream) {
  return zb::gemm2_entry(A, B, C, M, N, K, lda, ldb, ldc, a_mn_major, b_mn_major, bias, addend, ld_addend, flags, 0,
                         static_cast<float*>(workspace), workspace_bytes, status, stream);
}
// MLP up-projection and activation: out = act(x w^T + bias).  act 0, 1, 2: as zb_act_fwd, w [N, K]; act 3: gated unit, w
// [2N, K] = gate | up, no bias.  pre: the pre-activations ([M, N], act 3 [M, 2N]) are stored there, nullptr: not at all.
// Returns 1, with nothing done, where the pair kernel or TMA cannot take it (fewer than 256 rows or columns, N % 8).
extern "C" int zb_gemm2_act_fwd(const void* x, const void* w, const void* bias, void* pre, void* out, int M, int N, int K, int lda,
                                int ldb, int act, int* status, cudaStream_t stream) {
  using namespace zb;
  if (M < 256 || N < 256 || K <= 0 || N % 8 || act < 0 || act > 3 || (act == 3 && bias != nullptr) ||
      ((reinterpret_cast<uintptr_t>(pre) | reinterpret_cast<uintptr_t>(out)) & 15))
    return 1;
  if (act == 3) return gemm2_fused_entry<FE_GLU_FWD>(x, w, nullptr, pre, out, M, N, K, lda, ldb, 0, pre != nullptr, status, stream);
  return gemm2_fused_entry<FE_ACT_FWD>(x, w, bias, pre, out, M, N, K, lda, ldb, act, pre != nullptr, status, stream);
}
// Projection to query, key and value heads with the rotation of the first `heads` (rotate-half within each head of d columns;
// row m is position m % S of cs, [S, d] fp32 cosines | sines): out = rope(x w^T + bias), [M, N] dense.  Returns 1, with nothing
// done, where it is not for this kernel: as zb_gemm2_act_fwd, heads of other widths than 64 and 128, and columns that are no
// whole heads.  Products whose last wave the plain kernel cuts into parts are taken too: 2048 x 12288 x 4096 is 133 us cut and 14
// for the pass, 147 as here.
extern "C" int zb_gemm2_rope_fwd(const void* x, const void* w, const void* bias, const float* cs, void* out, int M, int N, int K,
                                 int lda, int ldb, int S, int heads, int d, int* status, cudaStream_t stream) {
  using namespace zb;
  if (M < 256 || N < 256 || K <= 0 || (d != 64 && d != 128) || N % d || S <= 0 || heads <= 0 || heads > N / d ||
      ((reinterpret_cast<uintptr_t>(out) | reinterpret_cast<uintptr_t>(cs)) & 15))
    return 1;
  return gemm2_fused_entry<FE_ROPE>(x, w, bias, nullptr, out, M, N, K, lda, ldb, d, 0, status, stream, cs, S, heads * d);
}
// Gradient of the pre-activations: dpre = (dy w) act'(pre), w [K, N] (K: columns of dy); act 3: pre and dpre [M, 2N].
// Returns 1 as zb_gemm2_act_fwd.
extern "C" int zb_gemm2_act_bwd(const void* dy, const void* w, const void* pre, void* dpre, int M, int N, int K, int lda, int ldb,
                                int act, int* status, cudaStream_t stream) {
  using namespace zb;
  if (M < 256 || N < 256 || K <= 0 || N % 8 || act < 0 || act > 3 ||
      ((reinterpret_cast<uintptr_t>(pre) | reinterpret_cast<uintptr_t>(dpre)) & 15))
    return 1;
  void* h = const_cast<void*>(pre);
  if (act == 3) return gemm2_fused_entry<FE_GLU_BWD>(dy, w, nullptr, h, dpre, M, N, K, lda, ldb, 0, 0, status, stream);
  return gemm2_fused_entry<FE_ACT_BWD>(dy, w, nullptr, h, dpre, M, N, K, lda, ldb, act, 0, status, stream);
}
// C = A @ B^T (b_mn_major: A @ B) with the output rows scattered for a row-wise reduce-scatter over
// R ranks: rows [q * M / R, (q + 1) * M / R) go to dst_ptrs[q] (this rank's bf16 staging slot in rank
// q's memory, [M / R, N] with row stride ldc); when the grid is done `epoch` is stored to
// flag_ptrs[q][flag_index] for every q.  A: [M, K] K-major.  counter: zeroed device int.
extern "C" int zb_gemm2_rs_bf16(const void* A, const void* B, int M, int N, int K, int lda, int ldb, int ldc,
                                int b_mn_major, void* const* dst_ptrs, int* const* flag_ptrs, int R, int flag_index,
                                int epoch, unsigned int* counter, int max_ctas, int* status, cudaStream_t stream) {
  using namespace zb;
  if (M <= 0 || N <= 0 || K <= 0) ZB_FAIL(-1, "gemm2_rs: empty problem %d x %d x %d", M, N, K);
  if (R < 1 || R > 8 || M % R != 0) ZB_FAIL(-1, "gemm2_rs: %d rows do not split over %d ranks (1..8)", M, R);
  GemmScatterParams p;
  p.C = nullptr;
  p.bias = nullptr; p.addend = nullptr;
  p.M = M; p.N = N; p.K = K;
  p.ldc = ldc; p.ld_addend = 0;
  p.flags = 0;
  p.status = status;
  p.gate_flags = nullptr;
  p.gate_epoch = 0;
  p.gate_base = 0; p.gate_row_bytes = 0; p.gate_shard_bytes = 1;
  p.gate_chunk_bytes = 1; p.gate_cps = 1; p.gate_self = -1;
  for (int q = 0; q < 8; ++q) { p.sc_dst[q] = nullptr; p.sc_flags[q] = nullptr; }
  for (int q = 0; q < R; ++q) {
    if (reinterpret_cast<uintptr_t>(dst_ptrs[q]) & 15) ZB_FAIL(-1, "gemm2_rs: destination %d not 16-byte aligned", q);
    p.sc_dst[q] = dst_ptrs[q];
    p.sc_flags[q] = flag_ptrs[q];
  }
  p.C = dst_ptrs[0];   // alignment of the vector path is judged on a destination
  p.sc_rows = M / R; p.sc_R = R; p.sc_flag_index = flag_index; p.sc_epoch = epoch; p.sc_counter = counter;
  if (b_mn_major) return launch_gemm2<false, true, GemmScatterParams>(A, B, p, lda, ldb, max_ctas, stream);
  return launch_gemm2<false, false, GemmScatterParams>(A, B, p, lda, ldb, max_ctas, stream);
}

// All-gather fused with the GEMM that first consumes the gathered weights, on the 2-CTA core
// (same contract as zb_ag_gemm_bf16 in gemm_bf16.cu): C[M,N] = A[M,K] * B[N,K]^T (+bias)(+addend),
// B = a [N,K] weight inside the unit's flat unsharded buffer `full` at byte offset b_offset_bytes.
extern "C" int zb_ag_gemm2_bf16(const void* A, void* full, long b_offset_bytes, void* C, int M, int N, int K, int lda,
                                int ldc, const void* bias, const void* addend, int ld_addend, int flags,
                                const void* const* shard_ptrs, int R, int r, long shard_bytes, int chunk_bytes,
                                int* chunk_flags, int epoch, const int* version_flags, int need_version, int* status,
                                cudaStream_t stream) {
  using namespace zb;
  if (M <= 0 || N <= 0 || K <= 0) ZB_FAIL(-1, "ag_gemm2: empty problem %d x %d x %d", M, N, K);
  if (R < 2 || R > AG_MAX_R) ZB_FAIL(-1, "ag_gemm2: group size %d unsupported (2..%d)", R, AG_MAX_R);
  if (shard_bytes % 16 || chunk_bytes % 2048 || chunk_bytes <= 0) ZB_FAIL(-1, "ag_gemm2: bad shard/chunk size");
  if (b_offset_bytes % 16 || (long(K) * 2) % 16) ZB_FAIL(-1, "ag_gemm2: weight offset / row size not 16-byte aligned");
  GemmAgParams p;
  p.C = C;
  p.bias = static_cast<const __nv_bfloat16*>(bias);
  p.addend = static_cast<const __nv_bfloat16*>(addend);
  p.M = M; p.N = N; p.K = K;
  p.ldc = ldc; p.ld_addend = ld_addend;
  p.flags = flags;
  p.status = status;
  AgParams& ag = p.ag;
  for (int i = 0; i < AG_MAX_R; ++i) ag.src[i] = i < R ? static_cast<const uint4*>(shard_ptrs[i]) : nullptr;
  ag.dst = static_cast<uint4*>(full);
  ag.shard_bytes = shard_bytes;
  ag.R = R; ag.r = r;
  ag.chunk_bytes = chunk_bytes;
  ag.cps = int((shard_bytes + chunk_bytes - 1) / chunk_bytes);
  ag.chunk_flags = chunk_flags;
  ag.epoch = epoch;
  ag.version_flags = version_flags;
  ag.need_version = need_version;
  p.gate_flags = chunk_flags;
  p.gate_epoch = epoch;
  p.gate_base = b_offset_bytes;
  p.gate_row_bytes = long(K) * 2;
  p.gate_shard_bytes = shard_bytes;
  p.gate_chunk_bytes = chunk_bytes;
  p.gate_cps = ag.cps;
  p.gate_self = r;
  const void* B = static_cast<const char*>(full) + b_offset_bytes;
  return launch_gemm2<false, false, GemmAgParams>(A, B, p, lda, K, 0, stream);
}
