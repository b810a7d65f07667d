// dK and dQ of head dimensions above 128 in one pass over the (key tile, query tile) pairs, for sm_100a.
//
// Tensor memory does not hold dK and dV of a key tile of 128 keys beside the scores (256 columns each), so the single-pass
// backward ends at head dimension 128. Of the eight products that the split backward takes for five (S, dP, dK; S, dV; S, dP,
// dQ), two go when dQ is made where dK is: one kernel makes dV (bwd_dkdv_kernel, its dV items only), this one dK and dQ from four
// products. Per step, a key tile of 128 and a query sub-tile of 64:
//   S^T  = K Q^T            keys on tensor-memory lanes, 64 query columns
//   dP^T = V dO^T           V is the A operand out of tensor memory (copied there once an item), which leaves its shared memory for a
//                           second dO tile
//   dS^T = P^T (dP^T - delta)   compute warps; to shared memory as 16-bit, [keys][queries]
//   dQ^T = K^T dS^T         two products of 128 head-dim rows, over the columns of S^T and dP^T
//   dK  += dS^T Q
// A step is one chain: S^T 768 cycles (products of N = 64 from shared memory are bound by it: 48 cycles for 32), dP^T 512, dS^T some
// 600, dQ^T 768, and dK's 512, under which the drain takes dQ^T out. With what it shares of shared memory's bandwidth (480 KB a step)
// it takes 4780 cycles; the two kernels together 7400 a pair of tiles, the split form 9200. Step of 2 x 16384 tokens, 8 heads of
// 256: 5900 -> 5040 us; 2 x 8192 1540 -> 1270; packed samples of 517 to 4095 tokens a half, 8/4 heads of 192, 2115 -> 1850. Where
// it does not pay: bwd_wide_pays.
// dQ^T goes from tensor memory through a staging area into the fp32 accumulator with bulk reductions, as in the single-pass
// backward, and bwd_dq_convert_kernel rounds it; the order of the adds hangs on scheduling, so this serves deterministic == 0 only.
//
// The reference has one kernel for all head dimensions there (csrc/fda/mainloop_bwd_sm90_tma_gmma_ws.hpp:815-984).
#include <type_traits>

#include "bwd_common.cuh"

namespace fda {
namespace {

struct WideCfg {
  static constexpr int kHeadDim = 256;
  using T = TileCfg<kHeadDim>;
  static constexpr int kSubTileBytes = kSub * kHeadDim * 2;    // Q or dO sub-tile
  static constexpr int kSubPanelBytes = kSub * 128;
  static constexpr int kSlots = 2;                             // of Q and of dO; V lands in the two of dO
  static_assert(kSlots * kSubTileBytes == T::kTileBytes, "V goes through the dO slots");
  static constexpr int kStatBytes = 2 * kSub * 4;              // lse2[64], delta[64]
  static constexpr int kOffQ = T::kTileBytes, kOffDo = kOffQ + kSlots * kSubTileBytes;
  static constexpr int kOffDs = kOffDo + kSlots * kSubTileBytes;
  static constexpr int kStageChunk = 32 * 32 * 4;              // one warp's 32 head-dim rows x 32 query columns of dQ^T
  static constexpr int kOffStage = kOffDs + kTile * 128;
  static constexpr int kOffStat = kOffStage + 4 * kStageChunk;
  static constexpr int kOffBar = kOffStat + kSlots * kStatBytes;
  static constexpr int kSmemBytes = kOffBar + 448;             // barriers and headers 384, mailbox 64
  static_assert(kSmemBytes <= 232448 && kOffStage % 1024 == 0, "shared memory budget");
  // tensor memory: V, dK, and 128 columns for S^T (64) and dP^T (64), then for the two halves of dQ^T
  static constexpr int kTmemV = 0, kTmemDK = 128, kTmemS = 384, kTmemDP = 448, kTmemDQ = 384;
  static constexpr int kCols = kSub / 2;                       // query columns of a compute thread
  static constexpr int kThreads = 512, kLoadWarp = 8, kMmaWarp = 9, kDrainWarp0 = 12;
  static constexpr uint32_t kComputeRegs = 144, kProducerRegs = 64, kDrainRegs = 160;
  static_assert(128 * (2 * kComputeRegs + kProducerRegs + kDrainRegs) <= kThreads * 128, "register pool");
};

template <bool kBf16, bool kSoftcap>
__global__ void __launch_bounds__(WideCfg::kThreads, 1) bwd_wide_kernel(const __grid_constant__ BwdParams p) {
  using Cfg = WideCfg;
  using T = Cfg::T;
  extern __shared__ __align__(1024) uint8_t smem_wide[];   // starts where the block's window does; checked, as in the other kernels
  uint8_t* smem = smem_wide;
  uint8_t* sK = smem;
  uint8_t* sQ = smem + Cfg::kOffQ;
  uint8_t* sDo = smem + Cfg::kOffDo;
  uint8_t* sDs = smem + Cfg::kOffDs;
  uint8_t* sStage = smem + Cfg::kOffStage;
  uint8_t* sStat = smem + Cfg::kOffStat;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + Cfg::kOffBar);
  uint64_t* k_full = bars;
  uint64_t* k_empty = bars + 1;     // S^T and dQ^T of the item have read K
  uint64_t* v_full = bars + 2;      // V is in the dO slots
  uint64_t* q_full = bars + 3;      // [2] Q sub-tile, its statistics and the step header
  uint64_t* q_empty = bars + 5;     // [2]
  uint64_t* do_full = bars + 7;     // [2]
  uint64_t* do_empty = bars + 9;    // [2] dP^T has read the tile, or V has left for tensor memory
  uint64_t* s_full = bars + 11;
  uint64_t* dp_full = bars + 12;
  uint64_t* ds_full = bars + 13;    // dS^T in shared memory, S^T and dP^T in registers
  uint64_t* ds_free = bars + 14;    // dQ^T and dK have read dS^T
  uint64_t* dq_full = bars + 15;
  uint64_t* dq_free = bars + 16;    // dQ^T is in the drain warps' registers
  uint64_t* acc_full = bars + 17;
  uint64_t* acc_free = bars + 18;
  uint64_t* desc_full = bars + 19;  // [2] the step's description for the drain warps (see bwd_fused_kernel)
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 21);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  volatile int* dq_desc = reinterpret_cast<volatile int*>(bars + 22);       // [2][2]: {flags, first accumulator row}
  volatile int* hdr = reinterpret_cast<volatile int*>(bars + 24);           // [2][4]
  SchedMailbox* mbox = reinterpret_cast<SchedMailbox*>(reinterpret_cast<uint8_t*>(bars) + 384);
  static_assert(24 * 8 + Cfg::kSlots * 16 <= 384 && sizeof(SchedMailbox) <= 64, "barrier area");

  const int warp = ptx::uniform(static_cast<int>(threadIdx.x >> 5)), lane = threadIdx.x & 31;
  if ((ptx::smem_u32(smem) & 1023u) != 0) {
    if (threadIdx.x == 0 && atomicCAS(&g_fda_status[0], 0, 120) == 0) {
      g_fda_status[1] = static_cast<int>(blockIdx.x);
      g_fda_status[2] = 0;
      g_fda_status[3] = static_cast<int>(ptx::smem_u32(smem) & 1023u);
    }
    return;
  }
  if (threadIdx.x == 0) {
    *abort_flag = 0;
    sched_init(mbox, 8 + 2 + 4);   // compute, MMA and drain warps
    for (int i = 0; i < 21; ++i) {
      const bool of_compute = bars + i == ds_full, of_drain = bars + i == dq_free || bars + i == acc_free;
      ptx::mbar_init(bars + i, of_compute ? 8 : of_drain ? 4 : 1);
    }
    ptx::fence_mbar_init();
  }
  if (warp == Cfg::kLoadWarp) {
    ptx::tmem_alloc(tmem_slot, 512);
    ptx::tmem_relinquish();
  }
  ptx::tc_fence_before();
  __syncthreads();
  ptx::tc_fence_after();
  ptx::wait_for_stream();
  ptx::let_next_start();
  const uint32_t tmem = ptx::uniform(*tmem_slot);
  const int bs = p.block_size;
  const int group = p.heads / p.heads_k;
  const int total_items = kv_item_count(p);
  constexpr int kFmt = kBf16 ? 1 : 0;
  constexpr uint32_t kHi = ptx::smem_desc_hi(1024);

  if (warp >= Cfg::kDrainWarp0) {
    // --------------------------------------------------------------------------------------- dQ drain + dK epilogue
    ptx::reg_acquire_to<Cfg::kDrainRegs>();
    const int quad = warp & 3;
    const uint32_t lane_addr = static_cast<uint32_t>(quad * 32) << 16;
    uint8_t* stage = sStage + quad * Cfg::kStageChunk;
    uint32_t n_item = 0, gd = 0;
    bool alive = true;
    for (uint32_t n_sched = 0; alive; ++n_sched) {
      const int idx = ptx::uniform(sched_consume<true>(mbox, n_sched, abort_flag));
      if (idx < 0 || idx >= total_items) break;
      const KvItem it = decode_kv_item(p, idx);
      if (!it.valid) continue;
      for (bool last = false; alive && !last; ++gd) {
        const uint32_t par = gd & 1u;
        if (!ptx::mbar_wait(&desc_full[par], (gd >> 1) & 1u, abort_flag, 63)) { alive = false; break; }
        const int flags = ptx::uniform(dq_desc[2 * par]);
        const int acc_row = ptx::uniform(dq_desc[2 * par + 1]);
        last = (flags & 1) != 0;
        const int rows_left = flags >> 8;   // query rows of this sub-tile that exist (1..64)
        if (!ptx::mbar_wait(dq_full, par, abort_flag, 64)) { alive = false; break; }
        ptx::tc_fence_after();
        // All of dQ^T to registers, so that the columns are free for the next S^T and dP^T; then, under their products, pieces of
        // 32 head-dim rows x 16 queries through shared memory and out as one 2 KB bulk reduction each, two pieces in turn (one piece
        // of 4 KB, which is all there is room for, has to be read before the next is written: 2390 against 2350 us)
        uint32_t a[128];
#pragma unroll
        for (int c = 0; c < 4; ++c) ptx::tmem_ld32(tmem + Cfg::kTmemDQ + lane_addr + c * 32, a + c * 32);
        ptx::tmem_wait_ld();
        ptx::tc_fence_before();
        ptx::mbar_arrive_warp(dq_free);
        float* dst = p.dq_acc + static_cast<size_t>(acc_row) * Cfg::kHeadDim + quad * 1024;
#pragma unroll
        for (int c = 0; c < 8; ++c) {
          const int half = c >> 2, q0 = (c & 3) * 16;   // head-dim rows 128 half + 32 quad .., queries q0 ..
          if ((q0 & ~31) < rows_left && half * 128 + quad * 32 < p.head_dim) {
            uint8_t* piece = stage + (c & 1) * (Cfg::kStageChunk / 2);
            if (lane == 0) ptx::bulk_wait_group_read<1>();   // the last reduction but one out of these pieces has read its own
            __syncwarp();
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              const uint32_t* x = a + c * 16 + i * 4;
              ptx::st_shared_v4(piece + i * 512 + lane * 16, x[0], x[1], x[2], x[3]);
            }
            ptx::fence_async_smem();
            __syncwarp();
            if (lane == 0) {
              float* target = dst + (q0 & ~31) * Cfg::kHeadDim + half * 4 * 1024 + (c & 1) * 512;
              if (target >= p.dq_acc && target + 512 <= p.dq_acc + p.acc_floats) {
                ptx::bulk_reduce_add_f32(target, piece, Cfg::kStageChunk / 2);
                ptx::bulk_commit_group();
              } else if (atomicCAS(&g_fda_status[0], 0, 121) == 0) {   // never expected: recorded, not performed
                g_fda_status[1] = static_cast<int>(blockIdx.x);
                g_fda_status[2] = acc_row;
                g_fda_status[3] = flags;
              }
            }
          }
        }
      }
      if (!alive) break;
      const int row = quad * 32 + lane;
      const int rows_valid = imax(0, imin(32, it.n - (it.k0 + quad * 32)));
      const int64_t srow = static_cast<int64_t>(it.row0) + it.kh * it.n + it.k0 + row;
      uint16_t* dk_row = static_cast<uint16_t*>(p.dk) + it.bcoord * p.dk_bs + srow * p.dk_rs + it.hk * p.dk_hs;
      if (!ptx::mbar_wait(acc_full, n_item & 1, abort_flag, 62)) break;
      ++n_item;
      ptx::tc_fence_after();
#pragma unroll 1
      for (int c = 0; c < Cfg::kHeadDim; c += 64) {
        uint32_t accv[64];
        ptx::tmem_ld32(tmem + Cfg::kTmemDK + lane_addr + c, accv);
        ptx::tmem_ld32(tmem + Cfg::kTmemDK + lane_addr + c + 32, accv + 32);
        ptx::tmem_wait_ld();
        if (c == Cfg::kHeadDim - 64) {
          ptx::tc_fence_before();
          ptx::mbar_arrive_warp(acc_free);
        }
        if (lane < rows_valid) {
          ptx::store_row32<kBf16>(dk_row, c, accv, p.softmax_scale, p.head_dim, p.wide_store != 0);
          ptx::store_row32<kBf16>(dk_row, c + 32, accv + 32, p.softmax_scale, p.head_dim, p.wide_store != 0);
        }
      }
    }
    if (lane == 0) ptx::bulk_wait_group0();   // every reduction this warp issued has been performed
  } else if (warp >= Cfg::kLoadWarp) {
  ptx::reg_release_to<Cfg::kProducerRegs>();
  if (warp == Cfg::kLoadWarp) {
    // ------------------------------------------------------------------------------------------------ producer
    if (lane == 0) {
      uint32_t n_item = 0, gc = 0;
      uint32_t do_par = 3;   // bit s: parity to wait for before dO slot s is filled
      bool alive = true;
      auto wait_do = [&](uint32_t s) -> bool {
        if (!ptx::mbar_wait(&do_empty[s], (do_par >> s) & 1u, abort_flag, 43)) return false;
        do_par ^= 1u << s;
        return true;
      };
      for (uint32_t n_sched = 0; alive; ++n_sched) {
        const int idx = sched_produce(mbox, n_sched, p.ticket_q, abort_flag);
        if (idx < 0 || idx >= total_items) break;
        const KvItem it = decode_kv_item(p, idx);
        if (!it.valid) continue;
        const QueryPlan plan = make_query_plan(it.kh, it.k0, it.k1, it.n, bs, kTile);
        const KvSpans spans = make_kv_spans(it, bs);
        const int grow0 = p.cu_seqlens != nullptr ? it.row0 : it.b * p.seqlen;
        const int k_row = it.row0 + it.kh * it.n + it.k0;
        if (!wait_do(0) || !wait_do(1)) break;
        ptx::mbar_expect_tx(v_full, T::kTileBytes);
        load_tile<Cfg::kHeadDim>(sDo, &p.tm_v, v_full, k_row, it.hk, it.bcoord);
        if (!ptx::mbar_wait(k_empty, (n_item & 1) ^ 1, abort_flag, 44)) break;
        ptx::mbar_expect_tx(k_full, T::kTileBytes);
        load_tile<Cfg::kHeadDim>(sK, &p.tm_k, k_full, k_row, it.hk, it.bcoord);
        // The loader alone walks the item's steps; each carries a header (see bwd_fused_kernel). A step is sent when its successor
        // is known, so that the last one can be marked.
        auto emit = [&](const SubStep& st, bool last) -> bool {
          const uint32_t slot = gc & 1u;
          if (!ptx::mbar_wait(&q_empty[slot], ((gc >> 1) & 1u) ^ 1u, abort_flag, 42)) return false;
          volatile int* h4 = hdr + 4 * slot;
          h4[0] = (last ? 1 : 0) | (st.cls == kTileMasked ? 2 : 0) | (st.qh == it.kh ? 4 : 0) | ((st.sb - st.sa) << 8);
          h4[1] = st.sa;
          h4[2] = st.h * p.acc_tiles * 64 + acc_row_of(grow0, it.n, it.b, st.qh, st.sa);
          ptx::mbar_expect_tx(&q_full[slot], Cfg::kSubTileBytes + Cfg::kStatBytes);
          const int q_row = it.row0 + st.qh * it.n + st.sa;
          const int64_t seg = stat_segment(p, it.b, st.h, st.qh) + st.sa;
#pragma unroll
          for (int c = 0; c < T::kPanels; ++c) {
            ptx::tma_load_4d(sQ + slot * Cfg::kSubTileBytes + c * Cfg::kSubPanelBytes, &p.tm_q64, &q_full[slot], c * 64, q_row,
                             st.h, it.bcoord);
          }
          ptx::bulk_load_1d(sStat + slot * Cfg::kStatBytes, p.lse2_pad + seg, kSub * 4, &q_full[slot]);
          ptx::bulk_load_1d(sStat + slot * Cfg::kStatBytes + kSub * 4, p.delta_pad + seg, kSub * 4, &q_full[slot]);
          if (!wait_do(slot)) return false;
          ptx::mbar_expect_tx(&do_full[slot], Cfg::kSubTileBytes);
#pragma unroll
          for (int c = 0; c < T::kPanels; ++c) {
            ptx::tma_load_4d(sDo + slot * Cfg::kSubTileBytes + c * Cfg::kSubPanelBytes, &p.tm_do64, &do_full[slot], c * 64, q_row,
                             st.h, it.bcoord);
          }
          ++gc;
          return true;
        };
        SubStep pend{};
        bool have = false;
        alive = for_each_substep(it, plan, spans, group, [&](const SubStep& st) -> bool {
          if (have && !emit(pend, false)) return false;
          pend = st;
          have = true;
          return true;
        });
        // every valid key tile is seen at least by the queries of its own rows, so there is a last step
        if (alive && have) alive = emit(pend, true);
        ++n_item;
      }
      if (*abort_flag) __nanosleep(100000);
    }
  } else if (warp == Cfg::kMmaWarp) {
    // ------------------------------------------------------------------- MMA issuer 1: S^T = K Q^T, dP^T = V dO^T
    constexpr uint32_t kIdescS = ptx::make_idesc(kTile, kSub, kFmt, false, false);
    const uint32_t k_lo = ptx::smem_desc_lo(ptx::smem_u32(sK), 16);
    const uint32_t q_lo = ptx::smem_desc_lo(ptx::smem_u32(sQ), 16);
    const uint32_t do_lo = ptx::smem_desc_lo(ptx::smem_u32(sDo), 16);   // also V on its way to tensor memory
    uint32_t n_item = 0, g = 0;
    bool alive = true;
    for (uint32_t n_sched = 0; alive; ++n_sched) {
      const int idx = ptx::uniform(sched_consume<true>(mbox, n_sched, abort_flag));
      if (idx < 0 || idx >= total_items) break;
      if (!decode_kv_item(p, idx).valid) continue;
      // every dP^T of the last item is complete: its dO slots were free for V
      if (!ptx::mbar_wait(v_full, n_item & 1, abort_flag, 69)) break;
      ptx::tc_fence_after();
      if (ptx::elect_one()) {
#pragma unroll
        for (int kk = 0; kk < Cfg::kHeadDim / 16; ++kk) {
          ptx::tmem_cp_128x32b_lh(tmem + Cfg::kTmemV + kk * 8, do_lo + (((kk / 4) * T::kPanelBytes + (kk % 4) * 32) >> 4), kHi);
        }
        ptx::umma_commit(&do_empty[0]);
        ptx::umma_commit(&do_empty[1]);
      }
      if (!ptx::mbar_wait(k_full, n_item & 1, abort_flag, 51)) break;
      ++n_item;
      for (bool last = false; alive && !last; ++g) {
        const uint32_t slot = g & 1u, spar = (g >> 1) & 1u;
        const uint32_t t_off = slot * (Cfg::kSubTileBytes >> 4);
        if (!ptx::mbar_wait(&q_full[slot], spar, abort_flag, 52)) { alive = false; break; }
        last = (ptx::uniform(hdr[4 * slot]) & 1) != 0;
        if (!ptx::mbar_wait(dq_free, (g & 1u) ^ 1u, abort_flag, 58)) { alive = false; break; }
        ptx::tc_fence_after();
        if (ptx::elect_one()) {
#pragma unroll
          for (int kk = 0; kk < Cfg::kHeadDim / 16; ++kk) {
            ptx::umma_ss_f16_lh(tmem + Cfg::kTmemS, k_lo + (((kk / 4) * T::kPanelBytes + (kk % 4) * 32) >> 4),
                                q_lo + t_off + (((kk / 4) * Cfg::kSubPanelBytes + (kk % 4) * 32) >> 4), kHi, kIdescS, kk > 0);
          }
          ptx::umma_commit(s_full);
        }
        if (!ptx::mbar_wait(&do_full[slot], spar, abort_flag, 56)) { alive = false; break; }
        ptx::tc_fence_after();
        if (ptx::elect_one()) {
#pragma unroll
          for (int kk = 0; kk < Cfg::kHeadDim / 16; ++kk) {
            ptx::umma_ts_f16_lh(tmem + Cfg::kTmemDP, tmem + Cfg::kTmemV + kk * 8,
                                do_lo + t_off + (((kk / 4) * Cfg::kSubPanelBytes + (kk % 4) * 32) >> 4), kHi, kIdescS, kk > 0);
          }
          ptx::umma_commit(dp_full);
          ptx::umma_commit(&do_empty[slot]);
        }
      }
    }
  } else if (warp == Cfg::kMmaWarp + 1) {
    // -------------------------------------------------------------------- MMA issuer 2: dQ^T = K^T dS^T, dK += dS^T Q
    constexpr uint32_t kIdescQ = ptx::make_idesc(kTile, kSub, kFmt, true, true);
    constexpr uint32_t kIdescK = ptx::make_idesc(kTile, Cfg::kHeadDim, kFmt, false, true);
    const uint32_t k_mn = ptx::smem_desc_lo(ptx::smem_u32(sK), T::kPanelBytes);
    const uint32_t q_mn = ptx::smem_desc_lo(ptx::smem_u32(sQ), Cfg::kSubPanelBytes);
    const uint32_t ds_mn = ptx::smem_desc_lo(ptx::smem_u32(sDs), 16), ds_k = ds_mn;   // one panel either way
    uint32_t g = 0, n_item = 0;
    bool alive = true;
    for (uint32_t n_sched = 0; alive; ++n_sched) {
      const int idx = ptx::uniform(sched_consume<true>(mbox, n_sched, abort_flag));
      if (idx < 0 || idx >= total_items) break;
      if (!decode_kv_item(p, idx).valid) continue;
      bool acc = false;
      // the first dK product of an item overwrites the accumulator: the epilogue must have read the last item's
      if (!ptx::mbar_wait(acc_free, (n_item & 1u) ^ 1u, abort_flag, 57)) break;
      ++n_item;
      for (bool last = false; alive && !last; ++g) {
        const uint32_t slot = g & 1u;
        if (!ptx::mbar_wait(&q_full[slot], (g >> 1) & 1u, abort_flag, 55)) { alive = false; break; }
        last = (ptx::uniform(hdr[4 * slot]) & 1) != 0;
        if (!ptx::mbar_wait(ds_full, g & 1u, abort_flag, 59)) { alive = false; break; }
        ptx::tc_fence_after();
        if (ptx::elect_one()) {
          // dQ before dK: its drain then runs under dK
#pragma unroll
          for (int kk = 0; kk < kTile / 16; ++kk) {
            ptx::umma_ss_f16_lh(tmem + Cfg::kTmemDQ, k_mn + kk * (2048 >> 4), ds_mn + kk * (2048 >> 4), kHi, kIdescQ, kk > 0);
            ptx::umma_ss_f16_lh(tmem + Cfg::kTmemDQ + 64, k_mn + ((2 * T::kPanelBytes + kk * 2048) >> 4), ds_mn + kk * (2048 >> 4),
                                kHi, kIdescQ, kk > 0);
          }
          ptx::umma_commit(dq_full);
          if (last) ptx::umma_commit(k_empty);   // every S^T of the item is complete by now
#pragma unroll
          for (int kk = 0; kk < kSub / 16; ++kk) {
            ptx::umma_ss_f16_lh(tmem + Cfg::kTmemDK, ds_k + ((kk * 32) >> 4),
                                q_mn + slot * (Cfg::kSubTileBytes >> 4) + kk * (2048 >> 4), kHi, kIdescK, (acc || kk > 0) ? 1u : 0u);
          }
          ptx::umma_commit(&q_empty[slot]);
          ptx::umma_commit(ds_free);
        }
        acc = true;
      }
      if (!alive) break;
      if (ptx::elect_one()) ptx::umma_commit(acc_full);
    }
  }
  } else {
    // ----------------------------------------------------------------------------------------- softmax backward
    ptx::reg_acquire_to<Cfg::kComputeRegs>();
    const int wg = warp >> 2;                  // which half of the step's queries
    const int quad = warp & 3;
    const int row = quad * 32 + lane;          // key row inside the tile
    const uint32_t lane_addr = static_cast<uint32_t>(quad * 32) << 16;
    uint8_t* ds_row = sDs + row * 128;         // 16-byte piece c of row r sits at c ^ (r & 7)
    uint32_t gc = 0;
    bool alive = true;
    for (uint32_t n_sched = 0; alive; ++n_sched) {
      const int idx = ptx::uniform(sched_consume<true>(mbox, n_sched, abort_flag));
      if (idx < 0 || idx >= total_items) break;
      const KvItem it = decode_kv_item(p, idx);
      if (!it.valid) continue;
      const int kj = it.k0 + row;
      // queries that see this thread's key: same-half tiles and (clean keys only) noisy tiles of later blocks
      int same_lo, same_hi, cross_lo, cross_hi;
      query_interval(it.kh, it.kh, kj, it.n, bs, same_lo, same_hi);
      query_interval(0, 1, kj, it.n, bs, cross_lo, cross_hi);
      for (bool last = false; alive && !last; ++gc) {
        const uint32_t slot = gc & 1u, par = gc & 1u;
        const float4* stats = reinterpret_cast<const float4*>(sStat + slot * Cfg::kStatBytes) + wg * (Cfg::kCols / 4);
        // the Q barrier orders the header and the bulk copies of lse2 / delta before our reads
        if (!ptx::mbar_wait(&q_full[slot], (gc >> 1) & 1u, abort_flag, 60)) { alive = false; break; }
        const int hdr0 = ptx::uniform(hdr[4 * slot]), hdr1 = ptx::uniform(hdr[4 * slot + 1]), hdr2 = hdr[4 * slot + 2];
        last = (hdr0 & 1) != 0;
        const int lo = ((hdr0 & 4) ? same_lo : cross_lo) - (hdr1 + wg * Cfg::kCols);
        const int hi = ((hdr0 & 4) ? same_hi : cross_hi) - (hdr1 + wg * Cfg::kCols);
        float pr[Cfg::kCols];
        if (!ptx::mbar_wait(s_full, par, abort_flag, 61)) { alive = false; break; }
        ptx::tc_fence_after();
        ptx::tmem_ld32(tmem + Cfg::kTmemS + lane_addr + wg * Cfg::kCols, reinterpret_cast<uint32_t*>(pr));
        ptx::tmem_wait_ld();
        auto first_half = [&](auto masked_tag) {   // P, or with the score cap P (1 - tanh^2)
          constexpr bool kMasked = decltype(masked_tag)::value;
          const uint32_t seen = kMasked ? ptx::bits_below(hi) & ~ptx::bits_below(lo) : 0u;
#pragma unroll
          for (int i = 0; i < Cfg::kCols / 4; ++i) {
            const float4 nl2 = stats[i];
            const float nl2a[4] = {nl2.x, nl2.y, nl2.z, nl2.w};
#pragma unroll
            for (int j = 0; j < 4; j += 2) {
              const int c = 4 * i + j;
              float x0 = pr[c], x1 = pr[c + 1];
              if (kSoftcap) {
                ptx::mul2(x0, x1, x0, x1, p.softcap_pre, p.softcap_pre);
                x0 = ptx::tanh_fast(x0);
                x1 = ptx::tanh_fast(x1);
              }
              float y0, y1;
              ptx::fma2(y0, y1, x0, x1, p.scale_log2, p.scale_log2, nl2a[j], nl2a[j + 1]);
              float v0 = ptx::ex2(y0), v1 = ptx::ex2(y1);
              if (kMasked && !(seen & (1u << c))) v0 = 0.f;
              if (kMasked && !(seen & (2u << c))) v1 = 0.f;
              if (kSoftcap) ptx::mul2(v0, v1, v0, v1, 1.f - x0 * x0, 1.f - x1 * x1);
              pr[c] = v0;
              pr[c + 1] = v1;
            }
          }
        };
        if (hdr0 & 2) first_half(std::true_type{});
        else first_half(std::false_type{});
        if (!ptx::mbar_wait(dp_full, par, abort_flag, 65)) { alive = false; break; }
        if (!ptx::mbar_wait(ds_free, par ^ 1u, abort_flag, 66)) { alive = false; break; }
        ptx::tc_fence_after();
        uint32_t dpv[Cfg::kCols];
        ptx::tmem_ld32(tmem + Cfg::kTmemDP + lane_addr + wg * Cfg::kCols, dpv);
        ptx::tmem_wait_ld();
        // masked positions have P = 0, so dS = 0 there without another select unless dP is infinite or NaN
        const uint32_t seen = (hdr0 & 2) ? ptx::bits_below(hi) & ~ptx::bits_below(lo) : 0xffffffffu;
#pragma unroll
        for (int i = 0; i < Cfg::kCols / 8; ++i) {
          const float4 d0 = stats[kSub / 4 + 2 * i], d1 = stats[kSub / 4 + 2 * i + 1];
          const float dl[8] = {d0.x, d0.y, d0.z, d0.w, d1.x, d1.y, d1.z, d1.w};
          uint32_t pk[4];
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const int c = 8 * i + 2 * j;
            float t0, t1;
            // dP - delta: there is no packed subtraction, the FMA with -1 rounds once like one
            ptx::fma2(t0, t1, dl[2 * j], dl[2 * j + 1], -1.f, -1.f, __uint_as_float(dpv[c]), __uint_as_float(dpv[c + 1]));
            ptx::mul2(t0, t1, t0, t1, pr[c], pr[c + 1]);
            if (!(seen & (1u << c))) t0 = 0.f;
            if (!(seen & (2u << c))) t1 = 0.f;
            pk[j] = ptx::pack2<kBf16>(t0, t1);
          }
          ptx::st_shared_v4(ds_row + (((4 * wg + i) ^ (row & 7)) << 4), pk[0], pk[1], pk[2], pk[3]);
        }
        if (threadIdx.x == 0) {
          dq_desc[2 * par] = hdr0 & ~6;
          dq_desc[2 * par + 1] = hdr2;
          ptx::mbar_arrive(&desc_full[par]);
        }
        ptx::fence_async_smem();
        ptx::tc_fence_before();
        ptx::mbar_arrive_warp(ds_full);
      }
    }
  }
  ptx::tc_fence_before();
  __syncthreads();
  if (warp == Cfg::kLoadWarp) ptx::tmem_dealloc(tmem, 512);
}

template <bool kBf16, bool kSoftcap>
int launch_wide_instance(const BwdParams& p, int sm_count, cudaStream_t stream) {
  auto kernel = bwd_wide_kernel<kBf16, kSoftcap>;
  static PerDeviceFlags smem_set;
  const int rc = set_dynamic_smem(kernel, WideCfg::kSmemBytes, smem_set);
  if (rc) return rc;
  const int items = bwd_item_bound(p, p.heads_k);
  if (const int launched = launch_kernel(p.overlap != 0, kernel, items < sm_count ? items : sm_count, WideCfg::kThreads, WideCfg::kSmemBytes, stream, p)) return launched;
  return FDA_OK;
}

}  // namespace

int launch_bwd_wide(const BwdParams& p, bool bf16, bool softcap, int sm_count, cudaStream_t stream) {
  if (bf16) return softcap ? launch_wide_instance<true, true>(p, sm_count, stream) : launch_wide_instance<true, false>(p, sm_count, stream);
  return softcap ? launch_wide_instance<false, true>(p, sm_count, stream) : launch_wide_instance<false, false>(p, sm_count, stream);
}

int read_status_bwd_wide(int32_t* out4) {
  int zero[4] = {0, 0, 0, 0};
  FDA_CUDA_TRY(cudaMemcpyFromSymbol(out4, g_fda_status, sizeof(int) * 4));
  FDA_CUDA_TRY(cudaMemcpyToSymbol(g_fda_status, zero, sizeof(int) * 4));
  return FDA_OK;
}

}  // namespace fda
