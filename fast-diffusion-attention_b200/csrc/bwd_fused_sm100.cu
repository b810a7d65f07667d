// Single-pass backward of block-diffusion attention for sm_100a: dK, dV and dQ from five GEMMs per tile pair.
//
// One CTA per (128-key tile, KV head, sample, half), persistent. K and V stay in shared memory; the visible
// 128-row query tiles of every query head of the group stream through (few tokens and few KV heads: of a part of the heads,
// see bwd_fused_kv_split). Per (key tile, query tile) step:
//   S^T  = K Q^T                        keys on tensor-memory lanes, 128 query columns
//   P^T  = exp2(S^T c - LSE2)           compute warps; written back over S^T as 16-bit (with a score cap: of
//                                       cap * tanh(S^T / cap), and the factor kept for dS^T is P^T (1 - tanh^2))
//   dP^T = V dO^T                       a second 128-column buffer
//   dS^T = P^T (dP^T - delta)           compute warps; to shared memory as 16-bit, [keys][queries]
//   dV  += P^T dO, dK += dS^T Q         accumulators in tensor memory for the whole key tile
//   dQ^T = K^T dS^T                     head dim on lanes, 128 query columns, written over the consumed dP^T buffer
//                                       (head dim 64 leaves room for columns of its own; without score cap it is
//                                       dQ = dS K there, queries on lanes, 64 columns)
// The two halves of the arithmetic hang on different products, so they overlap different MMAs: P^T is computed while
// dP^T (and the tail of the previous step) runs, dS^T while dV runs. The partial dQ^T of a step is added into an fp32
// accumulator in global memory: the drain warps move it from tensor memory through a small shared-memory staging
// area and out as 4 KB bulk reductions (cp.reduce.async.bulk add.f32); `bwd_dq_convert_kernel` then scales and
// rounds the accumulator into dQ (and, where there are parts, adds up those of dK and dV).
// Some 20 bytes per clock and SM go towards L2 this way when all SMs do it (5.8 TB/s in a microbenchmark, whatever the
// instruction), 3300 cycles for the 64 KB of a step, so the drain runs under the next step's products.
//
// The reference does the same five GEMMs per pair with an fp32 dQ accumulator reduced through global memory
// (csrc/fda/mainloop_bwd_sm90_tma_gmma_ws.hpp:815-984 `bwd_step`, :605-664 `store_dq`, there with
// cp.reduce.async.bulk from shared memory) and converts afterwards (flash_bwd_postprocess_kernel.h:160-264).
// The order of the adds depends on scheduling, so this path serves deterministic == 0 only; the deterministic
// backward keeps the two-kernel split (dK/dV kernel + dQ kernel), which has no cross-CTA reduction.
#include <type_traits>

#include "bwd_common.cuh"


namespace fda {
namespace {

template <int kHeadDim, int kSlots, int kDoSlots>
struct FusedCfg {
  using T = TileCfg<kHeadDim>;
  static constexpr int kDsPanelBytes = kTile * 128;          // [128 keys][64 queries] 16-bit
  static constexpr int kDsBytes = 2 * kDsPanelBytes;         // dS^T: two 64-query panels
  static constexpr int kStatBytes = 2 * kTile * 4;           // lse2[128], delta[128] of a query tile
  static constexpr int kOffQ = 2 * T::kTileBytes;            // K, V first (V directly behind K)
  static constexpr int kOffDo = kOffQ + kSlots * T::kTileBytes;
  static constexpr int kOffDs = kOffDo + kDoSlots * T::kTileBytes;
  static constexpr int kStageChunk = 32 * 32 * 4;            // one warp's 32 head-dim rows x 32 query columns of dQ^T
  static constexpr int kOffStage = kOffDs + kDsBytes;        // [4 warps][2 slots][kStageChunk]
  static constexpr int kOffStat = kOffStage + 4 * 2 * kStageChunk;
  static constexpr int kOffBar = kOffStat + kSlots * kStatBytes;
  static constexpr int kSmemBytes = kOffBar + 768;   // barriers 384, mailbox 64, item descriptions
  // tensor memory: S^T / P^T at 0, dP^T / dQ^T at 128, dK and dV behind
  static constexpr int kTmemS = 0, kTmemDP = 128, kTmemDK = 256, kTmemDV = 256 + kHeadDim;
  // Head dimension 64 leaves 128 columns behind the accumulators: dQ^T (or dQ) gets them, and the next dP^T no longer waits
  // for the drain of this step's dQ^T. At 128 all 512 columns are taken and dQ^T overwrites dP^T. (The other use of the 128, a
  // second S^T buffer, with dQ over dP^T: kernel time 2361 instead of 2211 us on 4 x 8192 tokens, 32 heads.)
  static constexpr bool kOwnDq = 256 + 2 * kHeadDim + 128 <= 512;
  static constexpr int kTmemDQ = kOwnDq ? 256 + 2 * kHeadDim : kTmemDP;
  static_assert(kHeadDim == 64 || kHeadDim == 128, "the single-pass backward covers head dimensions up to 128");
  static_assert(kOffStat % 1024 == 0, "tiles stay 1024-byte aligned for the swizzle");
  static_assert(kSmemBytes <= 232448, "shared memory budget");
  static_assert((17 + 2 * kSlots + 2 * kDoSlots) * 8 + 8 + 16 + 16 * kSlots <= 384, "barrier area");
};

// Warp roles: compute warpgroups (a thread = a key row and kCols query columns), a producer warpgroup (TMA warp, two
// MMA warps, one idle), the drain and epilogue warpgroup. The register counts of a form add up to what its block has at
// launch.
//   Head dim 128: two compute warpgroups of 64 columns. 512 threads start with 128 registers, and the drain warps hold a
//     whole dQ^T (128 columns): the buffer it shares with dP^T is free 250 cycles after the product instead of after 48
//     of its 64 KB have left for L2 (backward of 4 x 8192 tokens, 32/8 heads of 128, blocks of 1024: 4.25 -> 3.98 ms).
//     It is bound by shared memory and by power: a step takes 4260 cycles there (of a clock of 1.46 to 1.65 GHz), of which
//     shared memory at 128 bytes a clock has some 4300 (operands 2300, the staging of dQ^T 1024, the loads 512, dS^T 256,
//     statistics 250), the tensor pipe's arithmetic 2560; without the reductions themselves it takes 11 % less time
//     (3 % less on 8 x 4096 tokens, 16 heads, blocks of 256). Vector reductions straight from the registers
//     would save the staging, but stall the load/store unit for the compute warps (4.1 ms).
//   Head dim 64: dQ^T has columns of its own, and the exponentials (and tanh) weigh more: four compute warpgroups of 32
//     columns keep the special-function unit busier than two (4 x 8192 tokens, 32 heads, score cap: 2.8 against 3.2 ms).
template <int kHeadDim>
struct FusedRoles {
  static constexpr int kCmpWG = kHeadDim == 128 ? 2 : 4;
  static constexpr int kCols = kTile / kCmpWG;
  static constexpr int kThreads = 128 * (kCmpWG + 2);
  static constexpr int kLoadWarp = 4 * kCmpWG;
  static constexpr int kMmaWarp = kLoadWarp + 1;
  static constexpr int kEpiWarp0 = kLoadWarp + 4;
  static constexpr int kLaunchRegs = kCmpWG == 2 ? 128 : 80;
  static constexpr uint32_t kComputeRegs = kCmpWG == 2 ? 144 : 88;
  static constexpr uint32_t kProducerRegs = 64;
  static constexpr uint32_t kDrainRegs = kCmpWG == 2 ? 160 : 64;
  static constexpr int kHold = kCmpWG == 2 ? 4 : 1;   // 32-column chunks of dQ^T that a drain warp holds at once
  // A warp of its own works the items out ahead of the loader. Head dim 128: backward of 8 x 4096 tokens, 16 heads, blocks
  // of 256, 1036 us without and 1017 with it. Head dim 64: 4 x 8192, 32 heads, scores capped, 2750 without and 2824 with
  // it; 64 x 256 tokens, 16 heads, 155 and 148; no difference on 4 x 4096, 32/8 heads.
  static constexpr bool kGeometryWarp = kHeadDim == 128;
  // dQ = dS K instead of dQ^T = K^T dS^T: at head dim 64, where dQ^T has only 64 rows, so that half of an M = 128 product is
  // thrown away and two of the four drain warps do all the work (backward of 4 x 4096 tokens, 32/8 heads, blocks of 64: 706 ->
  // 684 us; 4 x 8192, 32 heads, blocks of 256: 2358 -> 2320). With capped scores, whose arithmetic leaves time for both, it was
  // not faster (2710 / 2616 us on the latter shape, with a tanh cheaper than the present one).
  static constexpr bool dq_rows(bool softcap) { return kHeadDim == 64 && !softcap; }
  static_assert(128 * (kCmpWG * kComputeRegs + kProducerRegs + kDrainRegs) <= kThreads * kLaunchRegs, "register pool");
};

// Rows of the dQ accumulator come in blocks of 64. Every half of every sample starts at its own block: the
// "+ 2 b + qh" gives each of the 2 * batch halves one block of slack, so rounding the start down never lets two
// halves share a block. Returns the first accumulator row of query row `qa` (a multiple of 64) of half `qh` of a
// sample whose first row in the packed row space is `grow0`.
__device__ __forceinline__ int acc_row_of(int grow0, int n, int b, int qh, int qa) {
  return ((grow0 + qh * n) / 64 + 2 * b + qh) * 64 + qa;
}

// One step of an item: a visible 128-row query tile of one query head. At most `left` steps follow it.
struct QStep {
  int h, qh, qa, cls, left;
};

// What the roles need to know about an item. At head dim 128 a warp of its own takes the items, works this out (some
// twenty integer divisions and a ticket from global memory) while the last steps of the item before are under way, and
// leaves it beside the mailbox; where items are short that counts. At head dim 64 the loader does it between its loads.
struct FusedItem {
  KvItem it;
  QueryPlan plan;
  KvSpans spans;
  int grow0;   // first row of the sample in the packed row space
  int part;    // which of the kv_split parts of the group's query heads
};
// The next item is taken when at most this many steps of the current one are to be sent: early enough for the ticket's
// round trip, late enough that CTAs do not reserve work. It hardly matters (same backward with 1, 4, 16: 1018, 1017, 1024).
constexpr int kTicketSteps = 4;

template <typename Fn>
__device__ __forceinline__ bool for_each_qstep(const KvItem& it, const QueryPlan& plan, const KvSpans& spans, int group,
                                               int head0, int head1, Fn&& fn) {
  for (int g = head0; g < head1; ++g) {
    for (int s = 0; s < plan.steps(); ++s) {
      QStep st;
      int qt;
      plan.step(s, it.kh, st.qh, qt);
      st.qa = qt * kTile;
      const int qb = imin(st.qa + kTile, it.n);
      st.cls = spans.classify(st.qh, it.kh, st.qa, qb);
      if (st.cls == kTileSkip) continue;
      st.h = it.hk * group + g;
      st.left = (head1 - 1 - g) * plan.steps() + plan.steps() - 1 - s;
      if (!fn(st)) return false;
    }
  }
  return true;
}

template <int kHeadDim, int kSlots, int kDoSlots, bool kBf16, bool kSoftcap, bool kParts>
__global__ void __launch_bounds__(FusedRoles<kHeadDim>::kThreads, 1) bwd_fused_kernel(const __grid_constant__ BwdParams p) {
  using Cfg = FusedCfg<kHeadDim, kSlots, kDoSlots>;
  using T = TileCfg<kHeadDim>;
  using R = FusedRoles<kHeadDim>;
  constexpr bool kDqRows = R::dq_rows(kSoftcap);
  // The tiles need 1024-byte alignment for the 128-byte swizzle. Dynamic shared memory starts at the beginning of the
  // block's window, which is aligned that far; the budget leaves no room to round the base up, so a base that is not
  // aligned is reported through the status word instead.
  extern __shared__ __align__(1024) uint8_t smem[];
  uint8_t* sK = smem;
  uint8_t* sV = smem + T::kTileBytes;   // directly behind K: for head dim 64 it may be the second panel of the M = 128
                                        // operand of dQ^T (rows 64..127 of that product are never read)
  uint8_t* sQ = smem + Cfg::kOffQ;
  uint8_t* sDo = smem + Cfg::kOffDo;
  uint8_t* sDs = smem + Cfg::kOffDs;
  uint8_t* sStage = smem + Cfg::kOffStage;
  uint8_t* sStat = smem + Cfg::kOffStat;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + Cfg::kOffBar);
  uint64_t* k_full = bars;
  uint64_t* k_empty = bars + 1;                // S^T and dQ^T of the item have read K
  uint64_t* v_full = bars + 2;
  uint64_t* v_empty = bars + 3;                // dP^T of the item has read V
  uint64_t* q_full = bars + 4;                 // [kSlots] Q tile, its statistics and the step header
  uint64_t* q_empty = q_full + kSlots;
  uint64_t* do_full = q_empty + kSlots;        // [kDoSlots] dO tile
  uint64_t* do_empty = do_full + kDoSlots;
  uint64_t* s_full = do_empty + kDoSlots;      // S^T complete
  uint64_t* dp_full = s_full + 1;              // dP^T complete
  uint64_t* p_full = dp_full + 1;              // P^T written over S^T
  uint64_t* ds_full = p_full + 1;              // dS^T in shared memory, dP^T in registers
  uint64_t* s_free = ds_full + 1;              // dV has read P^T: the next S^T may overwrite it
  uint64_t* dq_full = s_free + 1;              // dQ complete
  uint64_t* dp_free = dq_full + 1;             // dQ is in the drain warps' registers: its columns may be overwritten
                                               // (by the next dP^T, or by the next dQ where it has columns of its own)
  uint64_t* ds_free = dp_free + 1;             // dQ^T and dK have read dS^T: the next step may overwrite it
  uint64_t* acc_full = ds_free + 1;
  uint64_t* acc_free = acc_full + 1;
  // [2] The step's description for the drain warps is in dq_desc[g & 1]. They do not wait for ds_full: where dQ has its
  // own columns, dS^T of step g + 1 can be complete before they look for step g, and a wait by parity that is one whole
  // round late waits for ever. A barrier for even and one for odd steps cannot be lapped (step g + 2 needs dp_free of g).
  uint64_t* desc_full = acc_free + 1;
  uint64_t* go = desc_full + 2;                // the loader is about to send the last steps of its item
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(go + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  volatile int* dq_desc = reinterpret_cast<volatile int*>(tmem_slot + 2);   // [2][2]: {flags, first accumulator row}
  volatile int* hdr = reinterpret_cast<volatile int*>(tmem_slot + 6);       // [kSlots][4]
  SchedMailbox* mbox = reinterpret_cast<SchedMailbox*>(reinterpret_cast<uint8_t*>(bars) + 384);
  FusedItem* items = reinterpret_cast<FusedItem*>(reinterpret_cast<uint8_t*>(bars) + 448);   // [2], like the mailbox
  static_assert(sizeof(SchedMailbox) <= 64 && 2 * sizeof(FusedItem) <= 320, "mailbox and item descriptions");

  const int warp = ptx::uniform(static_cast<int>(threadIdx.x >> 5)), lane = threadIdx.x & 31;
  if ((ptx::smem_u32(smem) & 1023u) != 0) {
    if (threadIdx.x == 0 && atomicCAS(&g_fda_status[0], 0, 120) == 0) {
      g_fda_status[1] = static_cast<int>(blockIdx.x);
      g_fda_status[2] = 0;
      g_fda_status[3] = static_cast<int>(ptx::smem_u32(smem) & 1023u);
    }
    ptx::wait_for_stream();
    return;
  }
  if (threadIdx.x == 0) {
    *abort_flag = 0;
    sched_init(mbox, 4 * R::kCmpWG + (R::kGeometryWarp ? 3 : 2) + 4);   // compute, (loader,) two MMA, four drain warps
    ptx::mbar_init(k_full, 1);
    ptx::mbar_init(k_empty, 1);
    ptx::mbar_init(v_full, 1);
    ptx::mbar_init(v_empty, 1);
    for (int i = 0; i < kSlots; ++i) {
      ptx::mbar_init(&q_full[i], 1);
      ptx::mbar_init(&q_empty[i], 1);
    }
    for (int i = 0; i < kDoSlots; ++i) {
      ptx::mbar_init(&do_full[i], 1);
      ptx::mbar_init(&do_empty[i], 2);   // dP^T (issuer 1) and dV (issuer 2) have both read the tile
    }
    ptx::mbar_init(s_full, 1);
    ptx::mbar_init(dp_full, 1);
    ptx::mbar_init(p_full, 4 * R::kCmpWG);
    ptx::mbar_init(ds_full, 4 * R::kCmpWG);
    ptx::mbar_init(s_free, 1);
    ptx::mbar_init(dq_full, 1);
    ptx::mbar_init(dp_free, 4);
    ptx::mbar_init(ds_free, 1);
    ptx::mbar_init(acc_full, 1);
    ptx::mbar_init(acc_free, 4);
    ptx::mbar_init(&desc_full[0], 1);
    ptx::mbar_init(&desc_full[1], 1);
    ptx::mbar_init(go, 1);
    ptx::fence_mbar_init();
  }
  if (warp == R::kLoadWarp) {
    ptx::tmem_alloc(tmem_slot, 512);
    ptx::tmem_relinquish();
  }
  ptx::tc_fence_before();
  __syncthreads();
  ptx::tc_fence_after();
  ptx::wait_for_stream();
  if (p.next_early) ptx::let_next_start();
  const uint32_t tmem = ptx::uniform(*tmem_slot);
  const int bs = p.block_size;
  const int group = p.heads / p.heads_k;
  const int split = kParts ? p.kv_split : 1;   // CTAs that share a key tile
  const int total_items = kv_item_count(p) * split;

  auto make_item = [&](int idx, FusedItem& d) -> bool {   // false: a tile that does not exist
    const KvItem it = decode_kv_item(p, idx / split);
    if (!it.valid) return false;
    d.it = it;
    d.plan = make_query_plan(it.kh, it.k0, it.k1, it.n, bs, kTile);
    d.spans = make_kv_spans(it, bs);
    d.grow0 = p.cu_seqlens != nullptr ? it.row0 : it.b * p.seqlen;
    d.part = idx % split;
    return true;
  };

  if (warp >= R::kEpiWarp0) {
    // ------------------------------------------------------------------------------------- dQ drain + dK/dV epilogue
    // Four warps, one per quarter of the tensor-memory lanes. Per step they add the partial dQ^T (lane = head-dim
    // row, 128 query columns) into the global accumulator; after the last step of an item they write dK and dV.
    if (R::kHold > 1) ptx::reg_acquire_to<R::kDrainRegs>();
    else ptx::reg_release_to<R::kDrainRegs>();
    const int quad = warp & 3;
    const int row = quad * 32 + lane;
    const uint32_t lane_addr = static_cast<uint32_t>(quad * 32) << 16;
    // dQ^T: a lane is a value of the head dimension, the columns are the step's queries. dQ: a lane is a query, the columns are
    // the head dimension.
    constexpr int kDqCols = kDqRows ? kHeadDim : kTile;
    uint32_t n_item = 0, gd = 0, n_bulk = 0;
    bool alive = true;
    for (uint32_t n_sched = 0; alive; ++n_sched) {
      const int idx = R::kGeometryWarp ? sched_peek<true>(mbox, n_sched, abort_flag) : sched_consume<true>(mbox, n_sched, abort_flag);
      if (idx < 0 || idx >= total_items) break;
      const KvItem it = R::kGeometryWarp ? items[n_sched & 1u].it : decode_kv_item(p, idx / split);
      const int part = R::kGeometryWarp ? items[n_sched & 1u].part : idx % split;
      const int grow0 = p.cu_seqlens != nullptr ? it.row0 : it.b * p.seqlen;
      if (R::kGeometryWarp) sched_release<true>(mbox, n_sched);
      else if (!it.valid) continue;
      for (bool last = false; alive && !last; ++gd) {
        const uint32_t par = gd & 1u;
        if (!ptx::mbar_wait_warp(&desc_full[par], (gd >> 1) & 1u, abort_flag, 63)) { alive = false; break; }
        const int flags = dq_desc[2 * par];
        const int acc_row = dq_desc[2 * par + 1];
        last = (flags & 1) != 0;
        const int rows_left = flags >> 8;   // query rows of this tile that exist (1..128)
        if (!ptx::mbar_wait_warp(dq_full, par, abort_flag, 64)) { alive = false; break; }
        ptx::tc_fence_after();
        // kHold chunks of 32 columns go to registers at once; when the last is there the columns are free and the adds
        // follow behind the next step's products. Blocks of 32 query rows of the accumulator are stored as
        // [head dim / 32][8][32][4]: 8 groups of 4 queries x 32 head-dim values (dQ^T), or 8 groups of 4 head-dim values x 32
        // queries (dQ). Either way a warp's 32 x 32 piece goes through shared memory (16 bytes a thread, a quarter of the
        // store instructions of single values) and out as ONE 4 KB bulk reduction issued by lane 0. Two staging slots per warp
        // alternate.
        float* dst = p.dq_acc + static_cast<size_t>(acc_row) * kHeadDim + quad * (kDqRows ? 32 * kHeadDim : 1024);
#pragma unroll 1
        for (int c0 = 0; c0 < kDqCols / 32; c0 += R::kHold) {
          uint32_t a[32 * R::kHold];
#pragma unroll
          for (int c = 0; c < R::kHold; ++c) ptx::tmem_ld32(tmem + Cfg::kTmemDQ + lane_addr + (c0 + c) * 32, a + c * 32);
          if (R::kHold == 1) {   // the slot is waited for while the load is under way
            if (lane == 0) ptx::bulk_wait_group_read<1>();
            __syncwarp();
          }
          ptx::tmem_wait_ld();
          if (c0 + R::kHold == kDqCols / 32) {
            ptx::tc_fence_before();
            ptx::mbar_arrive_warp(dp_free);
          }
#pragma unroll
          for (int c = 0; c < R::kHold; ++c) {
            // pieces of queries that do not exist or behind the head dimension hold nothing
            const int col = (c0 + c) * 32;
            if (kDqRows ? quad * 32 < rows_left && col < p.head_dim : col < rows_left && quad * 32 < p.head_dim) {
              uint8_t* stage = sStage + (quad * 2 + (n_bulk & 1u)) * Cfg::kStageChunk;
              // the bulk reduction that last read this slot (two chunks ago) must have finished reading it
              if (R::kHold > 1) {
                if (lane == 0) ptx::bulk_wait_group_read<1>();
                __syncwarp();
              }
#pragma unroll
              for (int i = 0; i < 8; ++i) {
                const uint32_t* x = a + c * 32 + i * 4;
                ptx::st_shared_v4(stage + i * 512 + lane * 16, x[0], x[1], x[2], x[3]);
              }
              ptx::fence_async_smem();
              __syncwarp();
              if (lane == 0) {
                float* target = dst + (c0 + c) * (kDqRows ? 1024 : 32 * kHeadDim);
                if (target >= p.dq_acc && target + 1024 <= p.dq_acc + p.acc_floats) {
                  ptx::bulk_reduce_add_f32(target, stage, Cfg::kStageChunk);
                  ptx::bulk_commit_group();
                } else if (atomicCAS(&g_fda_status[0], 0, 121) == 0) {   // never expected: recorded, not performed
                  g_fda_status[1] = static_cast<int>(blockIdx.x);
                  g_fda_status[2] = acc_row;
                  g_fda_status[3] = flags;
                }
              }
              ++n_bulk;
            }
          }
        }
      }
      if (!alive) break;
      const int kj = it.k0 + row;
      const int rows_valid = imax(0, imin(32, it.n - (it.k0 + quad * 32)));  // of this warp's 32 key rows
      const int64_t srow = static_cast<int64_t>(it.row0) + it.kh * it.n + kj;
      uint16_t* dk_row = static_cast<uint16_t*>(p.dk) + it.bcoord * p.dk_bs + srow * p.dk_rs + it.hk * p.dk_hs;
      uint16_t* dv_row = static_cast<uint16_t*>(p.dv) + it.bcoord * p.dv_bs + srow * p.dv_rs + it.hk * p.dv_hs;
      if (!ptx::mbar_wait_warp(acc_full, n_item & 1, abort_flag, 62)) break;
      ++n_item;
      ptx::tc_fence_after();
      if (kParts) {
        // A part of the group's heads: 32 x 32 pieces of dK and dV go out as they are, in the order of the dQ accumulator's
        // blocks ([head dim / 32][8 groups of 4 values][32 rows][4 values]); the convert kernel adds the parts up.
        const int arow = acc_row_of(grow0, it.n, it.b, it.kh, it.k0) + quad * 32;
#pragma unroll 1
        for (int c = 0; c < 2 * kHeadDim / 32; ++c) {
          uint32_t accv[32];
          ptx::tmem_ld32(tmem + Cfg::kTmemDK + lane_addr + c * 32, accv);
          if (lane == 0) ptx::bulk_wait_group_read<1>();
          __syncwarp();
          ptx::tmem_wait_ld();
          if (c == 2 * kHeadDim / 32 - 1) {
            ptx::tc_fence_before();
            ptx::mbar_arrive_warp(acc_free);
          }
          const int is_dv = c * 32 >= kHeadDim ? 1 : 0, col = c * 32 - is_dv * kHeadDim;
          if (rows_valid > 0 && col < p.head_dim) {
            uint8_t* stage = sStage + (quad * 2 + (n_bulk & 1u)) * Cfg::kStageChunk;
#pragma unroll
            for (int i = 0; i < 8; ++i) {
              ptx::st_shared_v4(stage + i * 512 + lane * 16, accv[4 * i], accv[4 * i + 1], accv[4 * i + 2], accv[4 * i + 3]);
            }
            ptx::fence_async_smem();
            __syncwarp();
            if (lane == 0) {
              const int64_t block = (static_cast<int64_t>(is_dv) * p.kv_split + part) * p.heads_k + it.hk;
              const int64_t at = (block * p.acc_tiles * 64 + arow) * kHeadDim + col * 32;
              if (at >= 0 && at + 1024 <= p.part_floats) {
                ptx::bulk_store_1d(p.dkv_part + at, stage, Cfg::kStageChunk);
                ptx::bulk_commit_group();
              } else if (atomicCAS(&g_fda_status[0], 0, 122) == 0) {   // never expected: recorded, not performed
                g_fda_status[1] = static_cast<int>(blockIdx.x);
                g_fda_status[2] = arow;
                g_fda_status[3] = c;
              }
            }
            ++n_bulk;
          }
        }
        continue;
      }
      // dK and dV sit side by side in tensor memory. With the registers for it (kHold > 1) both are rounded first, in three
      // rounds of loads (a load is answered after 250 cycles and more while the products run, however wide it is), and
      // the next item's products may overwrite them while the rows are stored. (Tile copies through the staging slots
      // were slower: they queue behind the reductions.)
      if constexpr (R::kHold > 1) {
        uint32_t w[kHeadDim];
        auto round = [&](auto cols_tag, int col0) {
          constexpr int kN = decltype(cols_tag)::value;
          uint32_t accv[kN];
#pragma unroll
          for (int c = 0; c < kN; c += 32) ptx::tmem_ld32(tmem + Cfg::kTmemDK + lane_addr + col0 + c, accv + c);
          ptx::tmem_wait_ld();
          const float sc = col0 >= kHeadDim ? 1.f : p.softmax_scale;
#pragma unroll
          for (int i = 0; i < kN / 2; ++i) {
            w[col0 / 2 + i] = ptx::pack2<kBf16>(__uint_as_float(accv[2 * i]) * sc, __uint_as_float(accv[2 * i + 1]) * sc);
          }
        };
        round(std::integral_constant<int, kHeadDim>{}, 0);
        round(std::integral_constant<int, kHeadDim / 2>{}, kHeadDim);
        round(std::integral_constant<int, kHeadDim / 2>{}, kHeadDim + kHeadDim / 2);
        ptx::tc_fence_before();
        ptx::mbar_arrive_warp(acc_free);
        if (lane < rows_valid) {
#pragma unroll
          for (int c = 0; c < 2 * kHeadDim; c += 32) {
            ptx::store_row32_packed(c >= kHeadDim ? dv_row : dk_row, c % kHeadDim, w + c / 2, p.head_dim, p.wide_store != 0);
          }
        }
      } else {
        constexpr int kAccChunks = 2 * kHeadDim / 32;
#pragma unroll 1
        for (int c = 0; c < kAccChunks; ++c) {
          const bool is_dv = c * 32 >= kHeadDim;
          uint32_t accv[32];
          ptx::tmem_ld32(tmem + Cfg::kTmemDK + lane_addr + c * 32, accv);
          ptx::tmem_wait_ld();
          if (c == kAccChunks - 1) {
            ptx::tc_fence_before();
            ptx::mbar_arrive_warp(acc_free);
          }
          if (lane < rows_valid) {
            ptx::store_row32<kBf16>(is_dv ? dv_row : dk_row, c * 32 - (is_dv ? kHeadDim : 0), accv,
                                    is_dv ? 1.f : p.softmax_scale, p.head_dim, p.wide_store != 0);
          }
        }
      }
    }
    if (lane == 0) ptx::bulk_wait_group0();   // every reduction this warp issued has been performed
  } else if (warp >= R::kLoadWarp) {
  ptx::reg_release_to<R::kProducerRegs>();
  if (warp == R::kLoadWarp) {
    // ------------------------------------------------------------------------------------------------ producer
    if (lane == 0) {
      uint32_t n_item = 0, gc = 0;
      bool alive = true;
      for (uint32_t n_sched = 0; alive; ++n_sched) {
        const int idx = R::kGeometryWarp ? sched_peek<false>(mbox, n_sched, abort_flag)
                                         : sched_produce(mbox, n_sched, p.ticket_kv, abort_flag);
        if (idx < 0 || idx >= total_items) break;
        FusedItem d;
        if (R::kGeometryWarp) {
          d = items[n_sched & 1u];
          sched_release<false>(mbox, n_sched);
        } else if (!make_item(idx, d)) {
          continue;
        }
        const KvItem& it = d.it;
        // V is free after the last item's last dP^T; K only after its last dQ^T, behind everything that the first step
        // loads.
        const int k_row = it.row0 + it.kh * it.n + it.k0;
        if (!ptx::mbar_wait(v_empty, (n_item & 1) ^ 1, abort_flag, 41)) break;
        ptx::mbar_expect_tx(v_full, T::kTileBytes);
        load_tile<kHeadDim>(sV, &p.tm_v, v_full, k_row, it.hk, it.bcoord);
        bool k_loaded = false, told = false;
        // The loader alone walks the item's steps. Each carries a header for the other roles:
        // {bit 0 last step of the item, bit 1 partially masked, bit 2 queries of the keys' own half, bits 8.. the
        // number of query rows that exist; first query row; first accumulator row of the step's dQ}. A step is sent
        // when its successor is known, so that the last one can be marked.
        auto emit = [&](const QStep& st, bool last) -> bool {
          const uint32_t slot = gc % kSlots, par = ((gc / kSlots) & 1u) ^ 1u;
          if (R::kGeometryWarp && !told && (last || st.left <= kTicketSteps)) {
            told = true;
            ptx::mbar_arrive(go);
          }
          if (!ptx::mbar_wait(&q_empty[slot], par, abort_flag, 42)) return false;
          volatile int* h4 = hdr + 4 * slot;
          h4[0] = (last ? 1 : 0) | (st.cls == kTileMasked ? 2 : 0) | (st.qh == it.kh ? 4 : 0) |
                  (imin(kTile, it.n - st.qa) << 8);
          h4[1] = st.qa;
          h4[2] = st.h * p.acc_tiles * 64 + acc_row_of(d.grow0, it.n, it.b, st.qh, st.qa);
          ptx::mbar_expect_tx(&q_full[slot], T::kTileBytes + Cfg::kStatBytes);
          const int q_row = it.row0 + st.qh * it.n + st.qa;
          load_tile<kHeadDim>(sQ + slot * T::kTileBytes, &p.tm_q, &q_full[slot], q_row, st.h, it.bcoord);
          const int64_t seg = stat_segment(p, it.b, st.h, st.qh) + st.qa;
          ptx::bulk_load_1d(sStat + slot * Cfg::kStatBytes, p.lse2_pad + seg, kTile * 4, &q_full[slot]);
          ptx::bulk_load_1d(sStat + slot * Cfg::kStatBytes + kTile * 4, p.delta_pad + seg, kTile * 4, &q_full[slot]);
          const uint32_t dslot = gc % kDoSlots, dpar = ((gc / kDoSlots) & 1u) ^ 1u;
          if (!ptx::mbar_wait(&do_empty[dslot], dpar, abort_flag, 43)) return false;
          ptx::mbar_expect_tx(&do_full[dslot], T::kTileBytes);
          load_tile<kHeadDim>(sDo + dslot * T::kTileBytes, &p.tm_do, &do_full[dslot], q_row, st.h, it.bcoord);
          ++gc;
          if (!k_loaded) {
            k_loaded = true;
            if (!ptx::mbar_wait(k_empty, (n_item & 1) ^ 1, abort_flag, 44)) return false;
            ptx::mbar_expect_tx(k_full, T::kTileBytes);
            load_tile<kHeadDim>(sK, &p.tm_k, k_full, k_row, it.hk, it.bcoord);
          }
          return true;
        };
        QStep pend{};
        bool have = false;
        const int part_heads = group / split;
        const int head0 = d.part * part_heads;
        alive = for_each_qstep(it, d.plan, d.spans, group, head0, head0 + part_heads, [&](const QStep& st) -> bool {
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
  } else if (R::kGeometryWarp && warp == R::kMmaWarp + 2) {
    // ---------------------------------------------------------------------------------------------- item geometry
    if (lane == 0) {
      for (uint32_t n = 0;; ++n) {
        if (n > 0 && !ptx::mbar_wait(go, (n - 1) & 1u, abort_flag, 45)) break;
        int idx = sched_take(mbox, n, p.ticket_kv, abort_flag);
        if (idx < 0) break;
        while (idx < total_items && !make_item(idx, items[n & 1u])) idx = sched_next(p.ticket_kv);
        sched_publish(mbox, n, idx);
        if (idx >= total_items) break;
      }
    }
  } else if (warp == R::kMmaWarp) {
    // ------------------------------------------------------------------- MMA issuer 1: S^T = K Q^T, dP^T = V dO^T
    // Two warps issue the MMAs of this kernel, so that the barrier waits and commits of one overlap the MMAs of
    // the other. The whole warp takes part in waits and loop control and one elected lane issues, which keeps descriptors and
    // counters in uniform registers (with a single thread in the loop every MMA moved them there first: step of packed samples
    // with blocks of 4, 32/8 heads of 128, 3790 -> 3630 us; 1 x 8192 tokens, 32/8 heads, 1325 -> 1252; 2 x 8192, 32 heads of 64,
    // capped, 1957 -> 1820). S^T of step g + 1 may overwrite P^T of step g once dV has read it (s_free); dP^T of step g + 1
    // may overwrite dQ^T of step g once the drain warps hold it (dp_free) or, where dQ has its own columns, dP^T of
    // step g once the compute warps hold it (ds_full).
    {
      constexpr int kFmt = kBf16 ? 1 : 0;
      const uint32_t idesc_s = ptx::make_idesc(kTile, kTile, kFmt, false, false);
      constexpr uint32_t kHi = ptx::smem_desc_hi(1024);
      const uint32_t k_lo = ptx::smem_desc_lo(ptx::smem_u32(sK), 16);
      const uint32_t v_lo = ptx::smem_desc_lo(ptx::smem_u32(sV), 16);
      const uint32_t q_lo = ptx::smem_desc_lo(ptx::smem_u32(sQ), 16);
      const uint32_t do_lo = ptx::smem_desc_lo(ptx::smem_u32(sDo), 16);
      uint32_t n_item = 0, g = 0;
      bool alive = true;
      for (uint32_t n_sched = 0; alive; ++n_sched) {
        const int idx = ptx::uniform(sched_consume<true>(mbox, n_sched, abort_flag));
        if (idx < 0 || idx >= total_items) break;
        if (!R::kGeometryWarp && !decode_kv_item(p, idx / split).valid) continue;
        if (!ptx::mbar_wait_warp(k_full, n_item & 1, abort_flag, 51)) break;
        bool first = true;
        for (bool last = false; alive && !last; ++g) {
          const uint32_t slot = g % kSlots, spar = (g / kSlots) & 1u;
          const uint32_t t_off = slot * (T::kTileBytes >> 4);
          if (!ptx::mbar_wait_warp(&q_full[slot], spar, abort_flag, 52)) { alive = false; break; }
          last = (ptx::uniform(hdr[4 * slot]) & 1) != 0;
          if (!ptx::mbar_wait_warp(s_free, (g & 1u) ^ 1u, abort_flag, 54)) { alive = false; break; }
          ptx::tc_fence_after();
          if (ptx::elect_one()) {
#pragma unroll
            for (int kk = 0; kk < kHeadDim / 16; ++kk) {
              const uint32_t off = ((kk / 4) * T::kPanelBytes + (kk % 4) * 32) >> 4;
              ptx::umma_ss_f16_lh(tmem + Cfg::kTmemS, k_lo + off, q_lo + t_off + off, kHi, idesc_s, kk > 0);
            }
            ptx::umma_commit(s_full);
          }
          const uint32_t dslot = g % kDoSlots;
          if (!ptx::mbar_wait_warp(&do_full[dslot], (g / kDoSlots) & 1u, abort_flag, 56)) { alive = false; break; }
          if (first && !ptx::mbar_wait_warp(v_full, n_item & 1, abort_flag, 69)) { alive = false; break; }
          first = false;
          if (!ptx::mbar_wait_warp(Cfg::kOwnDq ? ds_full : dp_free, (g & 1u) ^ 1u, abort_flag, 58)) { alive = false; break; }
          ptx::tc_fence_after();
          if (ptx::elect_one()) {
#pragma unroll
            for (int kk = 0; kk < kHeadDim / 16; ++kk) {
              const uint32_t off = ((kk / 4) * T::kPanelBytes + (kk % 4) * 32) >> 4;
              ptx::umma_ss_f16_lh(tmem + Cfg::kTmemDP, v_lo + off, do_lo + dslot * (T::kTileBytes >> 4) + off, kHi, idesc_s,
                                  kk > 0);
            }
            ptx::umma_commit(dp_full);
            ptx::umma_commit(&do_empty[dslot]);
            if (last) ptx::umma_commit(v_empty);
          }
        }
        ++n_item;
      }
    }
  } else if (warp == R::kMmaWarp + 1) {
    // -------------------------------------------------- MMA issuer 2: dV += P^T dO, dQ^T = K^T dS^T, dK += dS^T Q
    {
      constexpr int kFmt = kBf16 ? 1 : 0;
      const uint32_t idesc_g = ptx::make_idesc(kTile, kHeadDim, kFmt, false, true);   // A K-major, B MN-major
      // dQ^T = K^T dS^T or dQ = dS K: A and B MN-major (the reduction runs over key rows)
      const uint32_t idesc_q = ptx::make_idesc(kTile, kDqRows ? kHeadDim : kTile, kFmt, true, true);
      constexpr uint32_t kHi = ptx::smem_desc_hi(1024);
      const uint32_t q_mn = ptx::smem_desc_lo(ptx::smem_u32(sQ), T::kPanelBytes);     // Q / dO as MN-major B: rows of
      const uint32_t do_mn = ptx::smem_desc_lo(ptx::smem_u32(sDo), T::kPanelBytes);   // queries are the reduction
      const uint32_t k_mn = ptx::smem_desc_lo(ptx::smem_u32(sK), T::kPanelBytes);
      const uint32_t ds_mn = ptx::smem_desc_lo(ptx::smem_u32(sDs), Cfg::kDsPanelBytes);
      const uint32_t dq_a = kDqRows ? ds_mn : k_mn, dq_b = kDqRows ? k_mn : ds_mn;
      const uint32_t ds_k = ptx::smem_desc_lo(ptx::smem_u32(sDs), 16);                // dS^T as K-major A of dK
      uint32_t g = 0, n_item_b = 0;
      bool alive = true;
      for (uint32_t n_sched = 0; alive; ++n_sched) {
        const int idx = ptx::uniform(sched_consume<true>(mbox, n_sched, abort_flag));
        if (idx < 0 || idx >= total_items) break;
        if (!R::kGeometryWarp && !decode_kv_item(p, idx / split).valid) continue;
        bool acc = false;
        // the first dV / dK products of an item overwrite the accumulators: the epilogue must have read the last item's
        if (!ptx::mbar_wait_warp(acc_free, (n_item_b & 1u) ^ 1u, abort_flag, 57)) break;
        ++n_item_b;
        for (bool last = false; alive && !last; ++g) {
          const uint32_t slot = g % kSlots, spar = (g / kSlots) & 1u;
          const uint32_t t_off = slot * (T::kTileBytes >> 4);
          if (!ptx::mbar_wait_warp(&q_full[slot], spar, abort_flag, 55)) { alive = false; break; }
          last = (ptx::uniform(hdr[4 * slot]) & 1) != 0;
          if (!ptx::mbar_wait_warp(p_full, g & 1u, abort_flag, 53)) { alive = false; break; }
          // dO usually landed long ago (dP^T of this step reads it too), but nothing this thread has waited for so far
          // says so
          if (!ptx::mbar_wait_warp(&do_full[g % kDoSlots], (g / kDoSlots) & 1u, abort_flag, 67)) { alive = false; break; }
          ptx::tc_fence_after();
          // dV += P^T dO: P^T of the 16 queries of reduction step kk sits at column 32 (kk / 2) + 8 (kk % 2)
          if (ptx::elect_one()) {
#pragma unroll
            for (int kk = 0; kk < kTile / 16; ++kk) {
              ptx::umma_ts_f16_lh(tmem + Cfg::kTmemDV, tmem + Cfg::kTmemS + 32 * (kk / 2) + 8 * (kk % 2),
                                  do_mn + (g % kDoSlots) * (T::kTileBytes >> 4) + kk * (2048 >> 4), kHi, idesc_g,
                                  (acc || kk > 0) ? 1u : 0u);
            }
            ptx::umma_commit(s_free);
            ptx::umma_commit(&do_empty[g % kDoSlots]);
          }
          if (!ptx::mbar_wait_warp(ds_full, g & 1u, abort_flag, 59)) { alive = false; break; }
          ptx::tc_fence_after();
          // dQ before dK: its drain (tensor memory -> registers -> global adds) then runs under dK
          if (Cfg::kOwnDq) {
            // the drain warps hold dQ of the previous step
            if (!ptx::mbar_wait_warp(dp_free, (g & 1u) ^ 1u, abort_flag, 68)) { alive = false; break; }
            ptx::tc_fence_after();
          }
          if (ptx::elect_one()) {
#pragma unroll
            for (int kk = 0; kk < kTile / 16; ++kk) {
              ptx::umma_ss_f16_lh(tmem + Cfg::kTmemDQ, dq_a + kk * (2048 >> 4), dq_b + kk * (2048 >> 4), kHi, idesc_q, kk > 0);
            }
            ptx::umma_commit(dq_full);
            // K is read by S^T (complete for every step of this item by now) and by dQ^T: after the last dQ^T the next
            // item's K may load. (The rows of dQ^T that come from V at head dim 64, where V may be changing by then, are
            // the ones nobody reads.)
            if (last) ptx::umma_commit(k_empty);
#pragma unroll
            for (int kk = 0; kk < kTile / 16; ++kk) {
              ptx::umma_ss_f16_lh(tmem + Cfg::kTmemDK, ds_k + (((kk / 4) * Cfg::kDsPanelBytes + (kk % 4) * 32) >> 4),
                                  q_mn + t_off + kk * (2048 >> 4), kHi, idesc_g, (acc || kk > 0) ? 1u : 0u);
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
  }
  } else {
    ptx::reg_acquire_to<R::kComputeRegs>();
    // -------------------------------------------------------------------------------------- softmax backward
    const int wg = warp >> 2;                  // which kCols query columns of the step
    constexpr int kChunks = R::kCols / 32;
    const int quad = warp & 3;
    const int row = quad * 32 + lane;          // key row inside the tile
    const uint32_t lane_addr = static_cast<uint32_t>(quad * 32) << 16;
    const uint32_t s_t = tmem + Cfg::kTmemS + lane_addr + wg * R::kCols;
    const uint32_t dp_t = tmem + Cfg::kTmemDP + lane_addr + wg * R::kCols;
    // this thread's row of the dS^T panel that holds its queries: 16-byte pieces from ds_piece0 on (128-byte swizzle:
    // piece c of row r sits at c ^ (r & 7))
    uint8_t* ds_row = sDs + (wg * R::kCols / 64) * Cfg::kDsPanelBytes + row * 128;
    const int ds_piece0 = R::kCols == 64 ? 0 : 4 * (wg & 1);
    uint32_t gc = 0;
    bool alive = true;
    for (uint32_t n_sched = 0; alive; ++n_sched) {
      const int idx = R::kGeometryWarp ? sched_peek<true>(mbox, n_sched, abort_flag) : sched_consume<true>(mbox, n_sched, abort_flag);
      if (idx < 0 || idx >= total_items) break;
      const KvItem it = R::kGeometryWarp ? items[n_sched & 1u].it : decode_kv_item(p, idx / split);
      if (R::kGeometryWarp) sched_release<true>(mbox, n_sched);
      else if (!it.valid) continue;
      const int kj = it.k0 + row;
      // queries that see this thread's key: same-half tiles and (clean keys only) noisy tiles of later blocks
      int same_lo, same_hi, cross_lo, cross_hi;
      query_interval(it.kh, it.kh, kj, it.n, bs, same_lo, same_hi);
      query_interval(0, 1, kj, it.n, bs, cross_lo, cross_hi);
      for (bool last = false; alive && !last; ++gc) {
        const uint32_t slot = gc % kSlots, par = gc & 1u;
        const float* stats = reinterpret_cast<const float*>(sStat + slot * Cfg::kStatBytes) + wg * R::kCols;
        // the Q barrier orders the header and the bulk copies of lse2 / delta before our reads
        if (!ptx::mbar_wait_warp(&q_full[slot], (gc / kSlots) & 1u, abort_flag, 60)) { alive = false; break; }
        const int hdr0 = hdr[4 * slot], hdr1 = hdr[4 * slot + 1], hdr2 = hdr[4 * slot + 2];
        last = (hdr0 & 1) != 0;
        const bool masked = (hdr0 & 2) != 0;
        // visible query columns of this thread's key, relative to its first column of the step
        const int lo = ((hdr0 & 4) ? same_lo : cross_lo) - (hdr1 + wg * R::kCols);
        const int hi = ((hdr0 & 4) ? same_hi : cross_hi) - (hdr1 + wg * R::kCols);
        {
          // First half, once S^T is complete: P^T (16-bit, back to tensor memory for dV) and, kept in registers, the
          // factor of the second half: P, or with the score cap P (1 - tanh^2).
          float pr[R::kCols];
          if (!ptx::mbar_wait_warp(s_full, par, abort_flag, 61)) { alive = false; break; }
          ptx::tc_fence_after();
#pragma unroll
          for (int half = 0; half < kChunks; ++half) ptx::tmem_ld32(s_t + 32 * half, reinterpret_cast<uint32_t*>(pr) + 32 * half);
          ptx::tmem_wait_ld();
          const float4* l2v = reinterpret_cast<const float4*>(stats);
          // the fully visible tile (the common one) carries no per-element compare
          auto first_half = [&](auto masked_tag) {
            constexpr bool kMasked = decltype(masked_tag)::value;
#pragma unroll
            for (int half = 0; half < kChunks; ++half) {
              uint32_t pk[16];
              const uint32_t seen = kMasked ? ptx::bits_below(hi - 32 * half) & ~ptx::bits_below(lo - 32 * half) : 0u;
#pragma unroll
              for (int i = 0; i < 8; ++i) {
                const float4 nl2 = l2v[8 * half + i];
                const float nl2a[4] = {nl2.x, nl2.y, nl2.z, nl2.w};
#pragma unroll
                for (int j = 0; j < 4; j += 2) {
                  const int c = 32 * half + 4 * i + j;
                  float x0 = pr[c], x1 = pr[c + 1];
                  float dt0 = 1.f, dt1 = 1.f;
                  if (kSoftcap) {
                    ptx::mul2(x0, x1, x0, x1, p.softcap_pre, p.softcap_pre);
                    x0 = ptx::tanh_fast(x0);
                    x1 = ptx::tanh_fast(x1);
                    dt0 = 1.f - x0 * x0;
                    dt1 = 1.f - x1 * x1;
                  }
                  float y0, y1;
                  ptx::fma2(y0, y1, x0, x1, p.scale_log2, p.scale_log2, nl2a[j], nl2a[j + 1]);
                  float v0 = ptx::ex2(y0), v1 = ptx::ex2(y1);
                  if (kMasked && !(seen & (1u << (4 * i + j)))) v0 = 0.f;
                  if (kMasked && !(seen & (2u << (4 * i + j)))) v1 = 0.f;
                  pk[2 * i + j / 2] = ptx::pack2<kBf16>(v0, v1);
                  if (kSoftcap) ptx::mul2(v0, v1, v0, v1, dt0, dt1);
                  pr[c] = v0;
                  pr[c + 1] = v1;
                }
              }
              // a warp overwrites only columns it has itself already loaded: the 16-bit P^T of 32 queries goes to the
              // first 16 of their 32 columns
              ptx::tmem_st16(s_t + 32 * half, pk);
            }
          };
          if (masked) first_half(std::true_type{});
          else first_half(std::false_type{});
          ptx::tmem_wait_st();
          ptx::tc_fence_before();
          ptx::mbar_arrive_warp(p_full);
          if (!ptx::mbar_wait_warp(dp_full, par, abort_flag, 65)) { alive = false; break; }
          // dQ^T and dK of the previous step have read the dS^T tile (long ago in the steady state)
          if (!ptx::mbar_wait_warp(ds_free, par ^ 1u, abort_flag, 66)) { alive = false; break; }
          ptx::tc_fence_after();
          const float4* dlv = reinterpret_cast<const float4*>(stats + kTile);
          uint32_t dpv[R::kCols];
#pragma unroll
          for (int half = 0; half < kChunks; ++half) ptx::tmem_ld32(dp_t + 32 * half, dpv + 32 * half);
          ptx::tmem_wait_ld();
          // masked positions have P = 0, so dS = 0 there without another compare
#pragma unroll
          for (int i = 0; i < R::kCols / 8; ++i) {
            const float4 d0 = dlv[2 * i], d1 = dlv[2 * i + 1];
            const float dl[8] = {d0.x, d0.y, d0.z, d0.w, d1.x, d1.y, d1.z, d1.w};
            uint32_t pk[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              const int c = 8 * i + 2 * j;
              float t0, t1;
              // dP - delta: there is no packed subtraction, the FMA with -1 rounds once like one
              ptx::fma2(t0, t1, dl[2 * j], dl[2 * j + 1], -1.f, -1.f, __uint_as_float(dpv[c]), __uint_as_float(dpv[c + 1]));
              ptx::mul2(t0, t1, t0, t1, pr[c], pr[c + 1]);
              pk[j] = ptx::pack2<kBf16>(t0, t1);
            }
            ptx::st_shared_v4(ds_row + (((ds_piece0 + i) ^ (row & 7)) << 4), pk[0], pk[1], pk[2], pk[3]);
          }
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
  if (warp == R::kLoadWarp) ptx::tmem_dealloc(tmem, 512);
}

// ------------------------------------------------------------------------------------------------------------
// dQ = round(accumulator * softmax_scale) and, where the heads of a group were dealt out, dK and dV = rounded sums of the parts
// (dK scaled too). One block per 64 rows of a (sample, query or KV head, half); stands where the reference converts its
// accumulator (csrc/fda/flash_bwd_postprocess_kernel.h:160-264 there).
// ------------------------------------------------------------------------------------------------------------
template <int kHeadDim, bool kBf16, bool kSoftcap, bool kParts>
__global__ void __launch_bounds__(256) bwd_dq_convert_kernel(const __grid_constant__ BwdParams p) {
  ptx::wait_for_stream();
  ptx::let_next_start();
  const int hh = blockIdx.y >> 1, half = blockIdx.y & 1;
  const int b = blockIdx.z;
  const Sample sm = sample_of(p, b);
  const int qa = blockIdx.x * 64;
  if (qa >= sm.n) return;
  const int grow0 = p.cu_seqlens != nullptr ? sm.row0 : b * p.seqlen;
  // a query head's dQ, or (behind all of them, where the heads of a group were dealt out) a KV head's dK or dV
  const int kv = kParts ? hh - p.heads : -1, is_dv = kv >= p.heads_k ? 1 : 0;
  const int h = kv < 0 ? hh : kv - is_dv * p.heads_k;
  const size_t rows = static_cast<size_t>(p.acc_tiles) * 64, row = acc_row_of(grow0, sm.n, b, half, qa);
  const float* src = kv < 0 ? p.dq_acc + (h * rows + row) * kHeadDim
                            : p.dkv_part + ((static_cast<size_t>(is_dv) * p.kv_split * p.heads_k + h) * rows + row) * kHeadDim;
  const int parts = kv < 0 ? 1 : p.kv_split;
  const bool row_lanes = FusedRoles<kHeadDim>::dq_rows(kSoftcap) || (kParts && kv >= 0);
  // The accumulator is read in its own order (see the drain; 16 bytes a lane), rounded, transposed through shared memory and
  // written in rows. The pad of 16 bytes keeps the row reads of 16
  // bytes aligned and the 2-byte writes of a warp (32 neighbouring values of a row) free of conflicts.
  constexpr int kRowElems = kHeadDim + 8;
  __shared__ __align__(16) uint16_t tile[64 * kRowElems];
  const float sc = kv >= 0 && is_dv ? 1.f : p.softmax_scale;
#pragma unroll
  for (int i = threadIdx.x; i < 16 * kHeadDim; i += 256) {
    const int e = i % 32, g = (i / 32) % 8, panel = (i / 256) % (kHeadDim / 32), q32 = i / (8 * kHeadDim);
    if (panel * 32 >= p.head_dim) continue;
    float4 x = reinterpret_cast<const float4*>(src)[i];
#pragma unroll 4
    for (int part = 1; kParts && part < parts; ++part) {   // always in this order: dK and dV are the same in every run
      const float4 y = reinterpret_cast<const float4*>(src + part * p.heads_k * rows * kHeadDim)[i];
      x = make_float4(x.x + y.x, x.y + y.y, x.z + y.z, x.w + y.w);
    }
    const uint32_t w0 = ptx::pack2<kBf16>(x.x * sc, x.y * sc), w1 = ptx::pack2<kBf16>(x.z * sc, x.w * sc);
    if (row_lanes) {   // 4 values of row e
      *reinterpret_cast<uint2*>(tile + (q32 * 32 + e) * kRowElems + panel * 32 + g * 4) = make_uint2(w0, w1);
    } else {           // value e of 4 rows
      uint16_t* t = tile + (q32 * 32 + g * 4) * kRowElems + panel * 32 + e;
      t[0] = static_cast<uint16_t>(w0);
      t[kRowElems] = static_cast<uint16_t>(w0 >> 16);
      t[2 * kRowElems] = static_cast<uint16_t>(w1);
      t[3 * kRowElems] = static_cast<uint16_t>(w1 >> 16);
    }
  }
  __syncthreads();
  constexpr int kPieces = kHeadDim / 8;
#pragma unroll
  for (int i = threadIdx.x; i < 64 * kPieces; i += 256) {
    const int qr = i / kPieces, piece = i % kPieces;
    if (qa + qr >= sm.n || piece * 8 >= p.head_dim) continue;
    const int64_t srow = static_cast<int64_t>(sm.row0) + half * sm.n + qa + qr;
    uint16_t* dst = static_cast<uint16_t*>(kv < 0 ? p.dq : is_dv ? p.dv : p.dk) +
                    sm.bcoord * (kv < 0 ? p.dq_bs : is_dv ? p.dv_bs : p.dk_bs) +
                    srow * (kv < 0 ? p.dq_rs : is_dv ? p.dv_rs : p.dk_rs) +
                    h * (kv < 0 ? p.dq_hs : is_dv ? p.dv_hs : p.dk_hs) + piece * 8;
    *reinterpret_cast<uint4*>(dst) = *reinterpret_cast<const uint4*>(tile + qr * kRowElems + piece * 8);
  }
}

// A row of the convert kernel's grid is one half of a query head's dQ or, with parts, of a KV head's dK or dV.
int convert_rows(int heads, int heads_k, bool parts) { return 2 * (heads + (parts ? 2 * heads_k : 0)); }
constexpr int kMaxGridY = 65535;

template <int kHeadDim, int kSlots, int kDoSlots, bool kBf16, bool kSoftcap, bool kParts>
int launch_fused_instance(const BwdParams& p, int sm_count, unsigned stages, cudaStream_t stream) {
  if (stages & 2u) {
    using Cfg = FusedCfg<kHeadDim, kSlots, kDoSlots>;
    auto kernel = bwd_fused_kernel<kHeadDim, kSlots, kDoSlots, kBf16, kSoftcap, kParts>;
    static PerDeviceFlags smem_set;
    const int rc = set_dynamic_smem(kernel, Cfg::kSmemBytes, smem_set);
    if (rc) return rc;
    if (p.zero_acc16 == 0) {
      FDA_CUDA_TRY(cudaMemsetAsync(p.dq_acc, 0, static_cast<size_t>(p.heads) * p.acc_tiles * 64 * kHeadDim * 4, stream));
    }
    const int64_t items = static_cast<int64_t>(bwd_item_bound(p, p.heads_k)) * p.kv_split;
    const int grid = items < sm_count ? static_cast<int>(items) : sm_count;
    const int launched = launch_kernel(p.overlap != 0, kernel, grid, FusedRoles<kHeadDim>::kThreads, Cfg::kSmemBytes, stream, p);
    if (launched) return launched;
  }
  if (stages & 4u) {
    dim3 grid(p.n_pad / 64, convert_rows(p.heads, p.heads_k, p.kv_split > 1), p.batch);
    return launch_kernel(p.overlap != 0, bwd_dq_convert_kernel<kHeadDim, kBf16, kSoftcap, kParts>, grid, 256, 0, stream, p);
  }
  return FDA_OK;
}

template <bool kParts>
int dispatch_fused(const BwdParams& p, int d_round, bool bf16, bool softcap, int sm_count, unsigned stages,
                   cudaStream_t stream) {
  auto go = [&](auto bf16_tag, auto softcap_tag) {
    constexpr bool kB = decltype(bf16_tag)::value, kC = decltype(softcap_tag)::value;
    return d_round == 64 ? launch_fused_instance<64, 3, 3, kB, kC, kParts>(p, sm_count, stages, stream)
                         : launch_fused_instance<128, 2, 1, kB, kC, kParts>(p, sm_count, stages, stream);
  };
  if (bf16) return softcap ? go(std::true_type{}, std::true_type{}) : go(std::true_type{}, std::false_type{});
  return softcap ? go(std::false_type{}, std::true_type{}) : go(std::false_type{}, std::false_type{});
}

}  // namespace

// Number of 64-row blocks of the dQ accumulator per query head (see acc_row_of): every half of every sample starts at
// its own block, and the last 128-row step of a half may reach one block past the half's rows.
int64_t bwd_fused_acc_tiles(const FdaProblem& pr) {
  return static_cast<int64_t>(pr.total) / 64 + 2 * static_cast<int64_t>(pr.batch) + 3;
}

size_t bwd_fused_acc_bytes(const FdaProblem& pr) {
  const int d_round = pr.head_dim <= 64 ? 64 : 128;
  return static_cast<size_t>(pr.heads) * bwd_fused_acc_tiles(pr) * 64 * d_round * 4;
}

namespace {

constexpr int64_t kMaxPartBytes = 512ll << 20, kMaxPartBytesMixed = 256ll << 20;

// fp32 dK and dV of `split` parts, in the accumulator's layout
int64_t part_bytes(const FdaProblem& pr, int split) {
  const int d_round = pr.head_dim <= 64 ? 64 : 128;
  return 2ll * split * pr.heads_k * bwd_fused_acc_tiles(pr) * 64 * d_round * 4;
}

}  // namespace

namespace {

// What the host knows of the samples, in tiles: the longest, their sum, the sum of their squares (bounded from below where packed
// samples are not all as long as max_seqlen says: one sample as long as that, the rest equal). Returns whether they are.
bool known_tiles(const FdaProblem& pr, double& longest, double& all, double& squares) {
  longest = (pr.seqlen / 2 + kTile - 1) / kTile;
  all = longest * pr.batch;
  squares = longest * all;
  const bool one_length = pr.cu_seqlens == nullptr || pr.total == static_cast<int64_t>(pr.batch) * pr.seqlen;
  if (!one_length) {
    all = pr.total / (2.0 * kTile);
    if (longest > all) longest = all;
    squares = longest * longest + (pr.batch > 1 ? (all - longest) * (all - longest) / (pr.batch - 1) : 0);
  }
  return one_length;
}

// The longest chain, 2 x longest steps of a query head, is at most 1.23 times a CTA's share of all steps where these are at least
// kLine x longest (kLine = 2 x 148 / 1.23).
constexpr double kLine = 240;

}  // namespace

// Samples of that many tokens a half, the longest and on average, and no chain of a key tile's steps over all heads of a group longer
// than 1.23 times a CTA's share.
bool bwd_chains_fit(const FdaProblem& pr, int tokens) {
  if (pr.heads_k <= 0 || pr.batch <= 0 || pr.seqlen / 2 < tokens) return false;
  if (pr.total / 2 < static_cast<int64_t>(pr.batch) * tokens) return false;
  double longest, all, squares;
  known_tiles(pr, longest, all, squares);
  return pr.heads_k * (squares + 2 * all) >= kLine * longest;
}

// Parts into which the query heads of a group are dealt. A key tile's steps are a chain, and those of the longest sample's first
// clean tile (2 x tiles x group, with tiles = n / 128) are more than a CTA's share of all steps (tiles (tiles + 2) x group for
// each KV head and sample, over 148 CTAs) where few tokens and few KV heads leave most of the chip idle. Then as many parts as
// make the chain at most 1.23 times that share, as far as the group goes.
// (Backward of 2 x 1000 tokens, 8 heads of 128 on one: 164 -> 62 us; 1 x 8192 tokens, 8/2 heads: 613 -> 233; 1 x 4096 tokens,
// 32/8 heads: 416 -> 281, with a chain of at most the share itself, which takes four parts instead of two, 307.)
// Lengths of packed samples are on the device. What is known of them here, the longest (or a bound of it) and their sum, bounds
// their steps from below: one sample as long as that, the rest equal. Samples of one length count like a batch of them.
// All samples are dealt alike, so one long sample among many short ones would need much memory: parts of samples of unlike lengths
// take kMaxPartBytesMixed at most, others kMaxPartBytes (4 x 6000 tokens, 14/2 heads of 128 need 337 MiB: 1260 -> 995 us).
// Where a block is half of the longest sample or more, that chain is shorter and the others are more like it, so that whole chains
// fill the chip better than the sums above say. Parts then have to save at least 12 of its steps (8 x 1280 tokens, 8/2 heads of 128,
// blocks of 512: 121 us whole, 143 in parts; 4 x 2000 tokens, 12/4 heads, one block each 202 and 229).
// Chains of up to 32 steps stay whole although they would gain too (3 x 666 tokens, 12/4 heads of 96, 18 steps: 66 -> 55 us): the
// sums of parts round differently, and on small problems the two forms of the backward give the same bits of dK and dV.
// They stay whole, too, where the convert kernel's grid has no rows left for dK and dV (more than 32700 heads or so).
// sm_margin does not count: it changes no result.
int bwd_fused_kv_split(const FdaProblem& pr) {
  constexpr double kCtas = 148;
  const int group = pr.heads_k > 0 ? pr.heads / pr.heads_k : 1;
  if (group <= 1 || pr.batch <= 0) return 1;
  double longest, all, squares;
  const bool one_length = known_tiles(pr, longest, all, squares);
  if (2 * longest * group <= 32 || convert_rows(pr.heads, pr.heads_k, true) > kMaxGridY) return 1;
  const double steps = pr.heads_k * (squares + 2 * all);   // of one query head of each group
  int split = 1;
  while (split * steps < kLine * longest) {
    int next = split + 1;
    while (next < group && group % next != 0) ++next;
    if (next > group || part_bytes(pr, next) > (one_length ? kMaxPartBytes : kMaxPartBytesMixed)) break;
    split = next;
  }
  const double block = pr.block_size >= pr.seqlen / 2 || pr.block_size / kTile > longest ? longest : pr.block_size / kTile;
  if (2 * block >= longest) {
    const double whole = (2 * longest - block) * group;
    const double share = (steps + pr.heads_k * (one_length ? all : longest) * (block > 2 ? block - 2 : 0)) * group / kCtas;
    if (whole - (share > whole / split ? share : whole / split) < 12) return 1;
  }
  return split;
}

size_t bwd_fused_part_bytes(const FdaProblem& pr) {
  const int split = bwd_fused_kv_split(pr);
  return split == 1 ? 0 : static_cast<size_t>(part_bytes(pr, split));
}

// stages: bit 1 = accumulator zero-fill + single-pass kernel, bit 2 = dQ convert.
int launch_bwd_fused(const BwdParams& p, int d_round, bool bf16, bool softcap, int sm_count, unsigned stages,
                     cudaStream_t stream) {
  return p.kv_split > 1 ? dispatch_fused<true>(p, d_round, bf16, softcap, sm_count, stages, stream)
                        : dispatch_fused<false>(p, d_round, bf16, softcap, sm_count, stages, stream);
}

int read_status_bwd_fused(int32_t* out4) {
  int zero[4] = {0, 0, 0, 0};
  FDA_CUDA_TRY(cudaMemcpyFromSymbol(out4, g_fda_status, sizeof(int) * 4));
  FDA_CUDA_TRY(cudaMemcpyToSymbol(g_fda_status, zero, sizeof(int) * 4));
  return FDA_OK;
}

}  // namespace fda
