// Forward pass of block-diffusion attention for sm_100a.
//
// Replaces the reference's forward stack (csrc/fda/flash_fwd_kernel_sm90.h:165-325,
// csrc/fda/mainloop_fwd_sm90_tma_gmma_ws.hpp:334-880, csrc/fda/epilogue_fwd.hpp:126-272,
// csrc/fda/softmax.h:92-168 and the forward scheduler csrc/fda/tile_scheduler.hpp:51-185) with a design
// built around tcgen05:
//
//   * a work item is kQTiles consecutive 128-row query tiles of one half of one (sample, head); both tiles
//     walk ONE list of key slots (clean prefix, then the noisy diagonal) in sub-steps of 64 keys, so K and V fetched
//     once by TMA feed both; a sub-step that one of the query tiles cannot see is skipped for that query tile only;
//   * warp roles: kQTiles softmax warpgroups (thread = one query row), one TMA producer warp, one MMA warp for each
//     query tile;
//   * S = Q K^T and O += P V are tcgen05.mma with fp32 accumulators in tensor memory; P is written back over
//     S in the type of the inputs and consumed from tensor memory as the A operand; V is used MN-major straight from its
//     TMA layout;
//   * online softmax with the scale folded into one FMA + exp2, a running row maximum that (after the first 128 keys, and
//     for 16-bit types) is only advanced when it grows by more than 2^8 (O is rescaled in tensor memory only then), LSE in
//     natural-log units;
//   * only visible sub-steps are enumerated, only those crossing a block boundary (or the end of a half) get the
//     element mask;
//   * persistent CTAs; items are ordered longest first (query tiles near the end of a half see most keys).
//
// Numerics contract kept from the reference: fp32 accumulation, softcap applied before the mask
// (mainloop_fwd...hpp:679-683), P rounded to the input dtype before P V (:782), row sums accumulated in fp32
// from the unrounded P, LSE = max * scale + ln(sum) (softmax.h:137-154).
#include <type_traits>

#include "geometry.h"
#include "host_util.h"
#include "ptx.cuh"
#include "sched.cuh"
#include "varlen_list.cuh"


#ifndef FDA_SHORT8_FWD
#define FDA_SHORT8_FWD 2   // eighths of a (sample, head)'s items that count as short
#endif

namespace fda {
namespace {


constexpr int kBlockM = 128;  // query rows per tile (= tensor-memory lanes)
constexpr int kSubKeys = 64;  // keys per sub-step (columns of one S buffer)
constexpr int kBufs = 2;      // S buffers per query tile
constexpr int kQPanelBytes = kBlockM * 128;
constexpr float kLog2e = 1.4426950408889634f;
constexpr float kLn2 = 0.6931471805599453f;
constexpr float kRescaleThreshold = 8.0f;  // in log2 units

struct FwdParams {
  CUtensorMap tm_q, tm_k, tm_v;
  CUtensorMap tm_o;    // out, boxes of 64 columns x 32 rows (used when o_tma != 0)
  int o_tma;           // out's strides allow tile stores
  void* out;
  float* lse;
  int64_t o_batch_stride, o_row_stride, o_head_stride;
  const int32_t* cu_seqlens;
  int batch, seqlen, total, heads, heads_k, head_dim, block_size;
  int items_per_half;  // ceil(max n / rows per item)
  int n_long;          // of the 2 * items_per_half items of a (sample, head): how many count as long
  int total_items;     // batched layout; packed batches read the count from the work list
  VarlenList vl;       // packed batches: samples longest first with running item counts (base == nullptr otherwise)
  int* ticket;         // global work counter, zeroed before the launch
  int wide_store;      // rows of out allow 32-byte stores
  int overlap;         // host: overlapped_launches
  int next_early;      // the next kernel may start early: no SMs are kept free
  const float* q_descale;  // FP8 only: (batch, heads_k) factors, element strides below; nullptr = 1
  const float* k_descale;
  const float* v_descale;
  int64_t descale_bs[3], descale_hs[3];
  float scale_log2;    // exponent scale: softmax_scale*log2(e), or softcap*log2(e) with softcapping
  float softcap_pre;   // softmax_scale / softcap (tanh argument scale)
  float lse_scale;     // natural-log scale of the row maximum: softmax_scale, or softcap
};

struct Item {
  int b, h, hk, qh, qa, qb, n;
  int row0;    // tensor row of the first token of the sample
  int bcoord;  // batch coordinate for TMA (0 when packed)
  bool valid;
};

template <int kQTiles>
__device__ __forceinline__ Item decode_item(const FwdParams& p, int idx) {
  // (sample, head)-major so that the CTAs running at the same time share the K/V of a few heads in L2; inside a
  // head the items with the most key tiles (late query rows) come first.
  Item it;
  int rem, items_per_half;
  if (p.vl.base != nullptr) {
    // packed batch: the work list holds exactly the items that exist, longest sample first; inside a sample the
    // heads follow each other, inside a head the items with the most key tiles come first
    const VarlenPos pos = varlen_locate(p.vl, idx, 2 * p.heads);
    items_per_half = pos.units;
    it.b = pos.b;
    it.h = pos.rem / (2 * pos.units);
    rem = pos.rem - it.h * (2 * pos.units);
  } else {
    const int per_bh = 2 * p.items_per_half;
    int bh;
    two_phase_order(idx, per_bh, p.n_long, p.batch * p.heads, bh, rem);
    items_per_half = p.items_per_half;
    it.b = bh / p.heads;
    it.h = bh - it.b * p.heads;
  }
  it.qh = rem & 1;
  const int p_rev = rem >> 1;
  it.hk = it.h / (p.heads / p.heads_k);
  const int pidx = items_per_half - 1 - p_rev;
  if (p.cu_seqlens != nullptr) {
    const int s = p.cu_seqlens[it.b];
    const int e = p.cu_seqlens[it.b + 1];
    it.n = (e - s) / 2;
    it.row0 = s;
    it.bcoord = 0;
  } else {
    it.n = p.seqlen / 2;
    it.row0 = 0;
    it.bcoord = it.b;
  }
  it.qa = pidx * kQTiles * kBlockM;
  it.valid = it.qa < it.n;
  it.qb = imin(it.qa + kQTiles * kBlockM, it.n);
  return it;
}

// Key spans of query tile t of the item, one per key half (index 0 noisy, 1 clean). Built once per item (the
// divisions by the block size happen here); classifying a key tile afterwards is a few compares. A query tile
// without rows gets empty spans, so every key tile is "skip" for it.
struct TileSpans {
  Span half[2];
  // selects instead of half[kh]: a run-time index would put the spans in local memory
  __device__ __forceinline__ int classify(int kh, int k0) const {
    Span s;
    s.lo_first = kh ? half[1].lo_first : half[0].lo_first;
    s.hi_first = kh ? half[1].hi_first : half[0].hi_first;
    s.lo_last = kh ? half[1].lo_last : half[0].lo_last;
    s.hi_last = kh ? half[1].hi_last : half[0].hi_last;
    return s.classify(k0, kSubKeys);
  }
};

__device__ __forceinline__ TileSpans make_tile_spans(const Item& it, int t, int bs) {
  TileSpans ts;
  const int ta = it.qa + t * kBlockM;
  if (ta >= it.qb) {
    ts.half[0] = Span{0, 0, 0, 0};
    ts.half[1] = Span{0, 0, 0, 0};
    return ts;
  }
  const int tb = imin(ta + kBlockM, it.qb);
  ts.half[0] = key_span(it.qh, 0, ta, tb, it.n, bs);
  ts.half[1] = key_span(it.qh, 1, ta, tb, it.n, bs);
  return ts;
}

// What the roles need to know about an item. The TMA warp works it out once (that is where the divisions by the
// block size and the head counts happen) and leaves it in shared memory next to the scheduler's mailbox; the softmax
// warps copy it from there. (The MMA warps need less: a word of flags beside every K slot.)
struct ItemDesc {
  Item it;
  KeyPlan plan;
  TileSpans spans[2];
};

// kType: 0 bf16, 1 fp16, 2 fp8 e4m3 (forward only; the output is bf16)
template <int kHeadDim, int kQTiles, int kType, bool kSoftcap, bool kQInTmem>
struct FwdConfig {
  static constexpr bool kFp8 = kType == 2;
  static constexpr int kElemBytes = kFp8 ? 1 : 2;
  static constexpr int kTileBytes = kBlockM * kHeadDim * kElemBytes;  // one query tile
  static constexpr int kPanelElems = 128 / kElemBytes;                // elements per 128-byte panel row
  static constexpr int kPanels = kHeadDim / kPanelElems;
  static constexpr int kStepElems = 32 / kElemBytes;                  // reduction elements per MMA (32 bytes)
  static_assert(kHeadDim % kPanelElems == 0, "head dimension must fill whole 128-byte panels");
  // K and V travel in slots of kSlotKeys keys. 16-bit rows of 256 leave room for four slots of 64 keys only.
  static constexpr int kSlotKeys = kTileBytes > 32768 ? 64 : 128;
  static constexpr int kSlotBytes = kSlotKeys * kHeadDim * kElemBytes;
  static constexpr int kSlotPanelBytes = kSlotKeys * 128;
  static constexpr int kHalves = kSlotKeys / kSubKeys;                // sub-steps per slot
  // Two query tiles: the two softmax warpgroups need more registers than an even split of the file gives them
  // (168 per thread with the block rounded up to whole warpgroups), so the block is padded to three whole
  // warpgroups and the third (TMA warp, two MMA warps, an idle warp) hands registers to the other two.
  static constexpr bool kRegRealloc = kQTiles == 2;
  static constexpr int kThreads = kRegRealloc ? 384 : 128 * kQTiles + 64;
  static constexpr uint32_t kSoftmaxRegs = 200, kProducerRegs = 104;
  // the pool is what the block got at launch, 384 threads x 168 registers: 2 * 128 * 200 + 128 * 104 = 384 * 168.
  // Asking for more than the pool holds would block the warpgroup for ever.
  static_assert(2 * 128 * kSoftmaxRegs + 128 * kProducerRegs <= 384 * 168, "register pool");
  static constexpr int kLoadWarp = 4 * kQTiles;
  static constexpr int kMmaWarp = 4 * kQTiles + 1;                    // one issuing warp per query tile
  // epilogue staging: per query tile one [128 rows][64 columns] 16-bit tile, stored to out as a whole
  static constexpr int kStageOBytes = kBlockM * 128;
  // 16-bit Q on its way to tensor memory comes through the ring: a pair of slots holds it, and the ring has a
  // pair more. With two pairs the loads' latency set the pace (nothing but loads took 894 of 1090 us on 2 x 16384 tokens, 8 heads: now
  // 890; packed samples of 517 to 4095 tokens a half, 8 heads of 192, 438 -> 342; 51 x 640 tokens, 16/8 heads 602 -> 546, 256 x 384
  // 529 -> 445, which read Q from shared memory before).
  static constexpr bool kQInRing = kQInTmem && !kFp8;
  static_assert(!kQInRing || kTileBytes == 2 * kSlotBytes, "a pair of slots holds a query tile");
  static constexpr int kFixedBytes = kQTiles * ((kQInRing ? 0 : kTileBytes) + kStageOBytes) + 1024 /*alignment slack*/ +
                                     1024 /*barriers, mailbox, item descriptions*/;
  static constexpr int kFit = (232448 - kFixedBytes) / (2 * kSlotBytes);
  static constexpr int kPairs = kFit < 4 ? kFit : 4;                  // the ring holds pairs of a K and a V slot
  static_assert(kPairs >= 2, "two V slots owed to P V and the K slots ahead of them");
  static constexpr int kSmemBytes = kFixedBytes + 2 * kPairs * kSlotBytes;
  // tensor memory: S of query tile t, buffer b at (t * kBufs + b) * 64 (P over its first columns), O behind
  static constexpr int kTmemO = kQTiles * kBufs * kSubKeys;
  static_assert(kTmemO + kQTiles * kHeadDim <= 512, "tensor memory budget");
  // ... and, for head dim 256, Q behind that. The S product then fetches only K from shared memory (16 instead
  // of 48 cycles a reduction step of 32 bytes): 1225 -> 1154 us on 2 x 16384 tokens, 8 heads, e4m3 916 -> 903. Head dim 64, where
  // columns are left too, gains nothing (256 / 254 us on 4 x 4096 tokens, 32/8 heads; 806 / 830 on 4 x 8192, 32 heads).
  static constexpr bool kTmemHasQ = kQInTmem;
  static constexpr int kTmemQ = kTmemO + kQTiles * kHeadDim;
  static_assert(!kTmemHasQ || (kQTiles == 1 && kTmemQ + kHeadDim * kElemBytes / 4 <= 512), "tensor memory budget");
  // The loop over fully visible sub-steps takes two of them, one a buffer, where that is not too much code: head dim 64 (4 x 8192
  // tokens, 32 heads: 768 / 753 us; capped 1284 / 1253) and e4m3 (2 x 16384 tokens, 8 heads of 256: 813 / 788; 4 x 8192, 16/4
  // heads of 128: 531 / 519).
  static constexpr bool kUnrollFull = kHeadDim == 64 || kFp8;
  static constexpr int kPCols = kSubKeys * kElemBytes / 4;            // tensor-memory columns of the packed P
};

// The keys advance in sub-steps of 64 and every query tile has two 64-column S buffers (kBufs), used in turn, P written
// over the S it came from. While the softmax warps turn one buffer into P, the tensor pipe runs P V of the other and
// then the S product that refills it, so neither waits for the other's latency. With ONE 128-column buffer per tile the
// chain S -> softmax -> P V -> next S was serial. The price is the shared-memory traffic of N = 64 products (6 KB per 32
// cycles of arithmetic, 48 cycles at 128 bytes per clock). On 4 x 8192 tokens, 32/8 heads of 128, blocks of 1024: 1.24 ->
// 1.14 ms, 4400 -> 4000 cycles of kernel time for two query tiles against 128 keys, of which the tensor pipe has 2300 (that mix
// of products measured alone) and the special-function unit 2048 to do. The rest is the softmax warps' own chain of a sub-step: wait,
// load (some 300 cycles), maximum, vote, pack, store, hand over. Without exponentials and products the kernel still takes half its
// time, and what shortens that chain by instructions helps. (Loads ahead, turns at the exponentials and more warps a tile do not:
// each adds hand-overs, 3-40 % slower.)
//
// Every query tile has its own issuing warp, and that warp does next to nothing but wait and issue: the TMA warp, which
// has time, walks the geometry and leaves one word of flags beside every K slot. (A single thread that decoded items and
// classified tiles between the products spent 1200 cycles a round on that while the pipe ran dry; the whole warp takes
// part in waits and loop control, one elected lane issues, which keeps descriptors and counters in uniform registers.)
// Bit 2 t + h: tile t sees half h.
constexpr uint32_t kInfoFirst = 16, kInfoLast = 32, kInfoHalf1 = 64, kInfoStop = 128, kInfoTile0 = 256, kInfoQ = 1024;

// kFullLoop: fully visible sub-steps have a loop of their own (see forward_full_loop).
template <int kHeadDim, int kQTiles, int kType, bool kSoftcap, bool kQInTmem, bool kFullLoop>
__global__ void __launch_bounds__(kQTiles == 2 ? 384 : 128 * kQTiles + 64, 1) fwd_kernel(const __grid_constant__ FwdParams p) {
  using Cfg = FwdConfig<kHeadDim, kQTiles, kType, kSoftcap, kQInTmem>;
  constexpr int kStages = 2 * Cfg::kPairs;         // slot 2 i: K of pair i, slot 2 i + 1: its V
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sQ = smem;
  uint8_t* sKV = smem + (Cfg::kQInRing ? 0 : kQTiles * Cfg::kTileBytes);
  uint8_t* sStageO = sKV + kStages * Cfg::kSlotBytes;
  uint64_t* bars = reinterpret_cast<uint64_t*>(sStageO + kQTiles * Cfg::kStageOBytes);
  uint64_t* q_full = bars;                         // 1
  uint64_t* q_empty = bars + 1;                    // 1
  uint64_t* kv_full = bars + 2;                    // kStages
  uint64_t* kv_empty = kv_full + kStages;          // kStages
  uint64_t* s_full = kv_empty + kStages;           // [kQTiles][kBufs] S complete
  uint64_t* p_full = s_full + kQTiles * kBufs;     // [kQTiles][kBufs] P written over it
  uint64_t* pv_done = p_full + kQTiles * kBufs;    // [kQTiles][kBufs] P V has updated O
  uint64_t* o_full = pv_done + kQTiles * kBufs;    // kQTiles
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(o_full + kQTiles);
  static_assert((2 + 2 * kStages + 3 * kQTiles * kBufs + kQTiles) * 8 + 8 + 16 <= 320, "barrier area");
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  volatile uint32_t* slot_info = tmem_slot + 2;    // one word per pair
  SchedMailbox* mbox = reinterpret_cast<SchedMailbox*>(reinterpret_cast<uint8_t*>(bars) + 320);
  ItemDesc* desc = reinterpret_cast<ItemDesc*>(reinterpret_cast<uint8_t*>(bars) + 512);  // two slots
  static_assert(Cfg::kMmaWarp + kQTiles <= Cfg::kThreads / 32, "roles");
  static_assert(sizeof(SchedMailbox) <= 192 && 2 * sizeof(ItemDesc) <= 512, "mailbox and item descriptions");

  const int warp = ptx::uniform(static_cast<int>(threadIdx.x >> 5));
  const int lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    *abort_flag = 0;
    sched_init(mbox, 4 * kQTiles);
    ptx::mbar_init(q_full, 1);
    ptx::mbar_init(q_empty, kQTiles);
    for (int i = 0; i < kStages; ++i) {
      ptx::mbar_init(&kv_full[i], 1);
      ptx::mbar_init(&kv_empty[i], kQTiles);   // every issuer lets go of every slot
    }
    for (int i = 0; i < kQTiles * kBufs; ++i) {
      ptx::mbar_init(&s_full[i], 1);
      ptx::mbar_init(&p_full[i], 4);  // one arrival per softmax warp
      ptx::mbar_init(&pv_done[i], 1);
    }
    for (int t = 0; t < kQTiles; ++t) ptx::mbar_init(&o_full[t], 1);
    ptx::fence_mbar_init();
  }
  if (warp == Cfg::kLoadWarp) {
    ptx::tmem_alloc(tmem_slot, 512);
    ptx::tmem_relinquish();
    if (lane == 0) {
      ptx::prefetch_tensormap(&p.tm_q);
      ptx::prefetch_tensormap(&p.tm_k);
      ptx::prefetch_tensormap(&p.tm_v);
    }
  }
  ptx::tc_fence_before();
  __syncthreads();
  ptx::tc_fence_after();
  ptx::wait_for_stream();
  if (p.next_early) ptx::let_next_start();
  const uint32_t tmem = ptx::uniform(*tmem_slot);
  const int bs = p.block_size;
  const int total_items = p.vl.base != nullptr ? p.vl.base[0] * 2 * p.heads : p.total_items;

  // The register counts are set inside the role branches: after a point where the branches meet again the
  // compiler would have to assume the smaller count for everything.
  if (warp >= 4 * kQTiles) {
  if (Cfg::kRegRealloc) ptx::reg_release_to<Cfg::kProducerRegs>();
  if (warp == Cfg::kLoadWarp) {
    // ------------------------------------------------------------------------------------------- TMA producer
    if (lane == 0) {
      uint32_t pair = 0, empty_par = 1, n_item = 0;
      bool alive = true;
      for (uint32_t n_sched = 0; alive; ++n_sched) {
        const int idx = sched_take(mbox, n_sched, p.ticket, abort_flag);
        if (idx < 0) break;
        if (idx >= total_items) {
          sched_publish(mbox, n_sched, idx);
          if (ptx::mbar_wait(&kv_empty[2 * pair], empty_par, abort_flag, 11)) {
            slot_info[pair] = kInfoStop;
            ptx::mbar_arrive(&kv_full[2 * pair]);
          }
          break;
        }
        const Item it = decode_item<kQTiles>(p, idx);
        KeyPlan plan{};
        TileSpans spans[kQTiles];
        {
          ItemDesc& d = desc[n_sched & 1u];
          d.it = it;
          if (it.valid) {
            plan = make_key_plan(it.qh, it.qa, it.qb, it.n, bs, Cfg::kSlotKeys);
            d.plan = plan;
#pragma unroll
            for (int t = 0; t < kQTiles; ++t) {
              spans[t] = make_tile_spans(it, t, bs);
              d.spans[t] = spans[t];
            }
          }
        }
        sched_publish(mbox, n_sched, idx);
        if (!it.valid) continue;
        const int tiles = plan.steps();
        const int q_row = it.row0 + it.qh * it.n + it.qa;
        const int ntiles = ceil_div(it.qb - it.qa, kBlockM);
        auto visible = [&](int s, int sub) -> uint32_t {   // bit 2 t + sub: tile t sees these 64 keys of slot s
          int kh, kt;
          plan.step(s, kh, kt);
          const int k0 = kt * Cfg::kSlotKeys + (Cfg::kHalves == 2 ? sub * kSubKeys : 0);
          uint32_t bits = 0;
#pragma unroll
          for (int t = 0; t < kQTiles; ++t) bits |= spans[t].classify(kh, k0) != kTileSkip ? 1u << (2 * t + sub) : 0u;
          return bits;
        };
        if (Cfg::kQInRing) {
          // the item's Q, half of it in each slot of a pair
          for (int which = 0; which < 2; ++which) {
            const uint32_t slot = 2 * pair + which;
            if (!ptx::mbar_wait(&kv_empty[slot], empty_par, abort_flag, 12)) { alive = false; break; }
            if (which == 0) slot_info[pair] = kInfoQ;
            ptx::mbar_expect_tx(&kv_full[slot], Cfg::kSlotBytes);
#pragma unroll
            for (int c = 0; c < Cfg::kPanels / 2; ++c) {
              ptx::tma_load_4d(sKV + slot * Cfg::kSlotBytes + c * kQPanelBytes, &p.tm_q, &kv_full[slot],
                               (which * (Cfg::kPanels / 2) + c) * Cfg::kPanelElems, q_row, it.h, it.bcoord);
            }
          }
          if (++pair == Cfg::kPairs) { pair = 0; empty_par ^= 1; }
        }
        for (int s = 0; s < tiles && alive; ++s) {
          int kh, kt;
          plan.step(s, kh, kt);
          const int k_row = it.row0 + kh * it.n + kt * Cfg::kSlotKeys;
          for (int which = 0; which < 2; ++which) {  // 0: K, 1: V
            const uint32_t slot = 2 * pair + which;
            if (!ptx::mbar_wait(&kv_empty[slot], empty_par, abort_flag, 11)) { alive = false; break; }
            if (which == 0 && (Cfg::kHalves == 2 || (s & 1) == 0)) {
              // flags of the two sub-steps that start here: both halves of this slot, or this slot and the next
              const bool two = Cfg::kHalves == 2 || s + 1 < tiles;
              uint32_t w = visible(s, 0);
              if (two) w |= visible(Cfg::kHalves == 2 ? s : s + 1, 1) | kInfoHalf1;
              if (s == 0) w |= kInfoFirst;
              if (s + (Cfg::kHalves == 2 ? 1 : 2) >= tiles) w |= kInfoLast;
              w |= ((1u << ntiles) - 1u) * kInfoTile0;
              slot_info[pair] = w;
            }
            ptx::mbar_expect_tx(&kv_full[slot], Cfg::kSlotBytes);
            uint8_t* dst = sKV + slot * Cfg::kSlotBytes;
            const CUtensorMap* tm = which == 0 ? &p.tm_k : &p.tm_v;
#pragma unroll
            for (int c = 0; c < Cfg::kPanels; ++c) {
              ptx::tma_load_4d(dst + c * Cfg::kSlotPanelBytes, tm, &kv_full[slot], c * Cfg::kPanelElems, k_row, it.hk,
                               it.bcoord);
            }
            if (!Cfg::kQInRing && s == 0 && which == 0) {
              // Q after the first K slot: the first MMA needs both, the previous item may still own Q.
              if (!ptx::mbar_wait(q_empty, (n_item & 1) ^ 1, abort_flag, 12)) { alive = false; break; }
              ptx::mbar_expect_tx(q_full, ntiles * Cfg::kTileBytes);
              for (int t = 0; t < ntiles; ++t) {
#pragma unroll
                for (int c = 0; c < Cfg::kPanels; ++c) {
                  ptx::tma_load_4d(sQ + t * Cfg::kTileBytes + c * kQPanelBytes, &p.tm_q, q_full, c * Cfg::kPanelElems,
                                   q_row + t * kBlockM, it.h, it.bcoord);
                }
              }
            }
          }
          if (++pair == Cfg::kPairs) { pair = 0; empty_par ^= 1; }
        }
        ++n_item;
      }
      if (*abort_flag) __nanosleep(100000);  // let copies in flight land before the CTA exits
    }
  } else if (warp < Cfg::kMmaWarp + kQTiles) {
    // ------------------------------------------------------------------------------- MMA issuer of one query tile
    // Two sub-steps of 64 keys a round: P V of the last round's half h, then S of this round's half h into the buffer
    // that this P V has read (the products of one thread run in order).
    constexpr int kFmt = kType == 0 ? 1 : 0;  // kind::f16: 1 = bf16, 0 = f16; kind::f8f6f4: 0 = e4m3
    constexpr uint32_t kIdescS = ptx::make_idesc(kBlockM, kSubKeys, kFmt, false, false);
    constexpr uint32_t kIdescO = ptx::make_idesc(kBlockM, kHeadDim, kFmt, false, true);
    constexpr uint32_t kDescHi = ptx::smem_desc_hi(1024);
    const int t = warp - Cfg::kMmaWarp;
    // descriptor low words of slot 0; a slot adds its bytes / 16, a k-step a constant
    const uint32_t q_lo = ptx::smem_desc_lo(ptx::smem_u32(sQ), 16) + t * (Cfg::kTileBytes >> 4);
    const uint32_t k_lo0 = ptx::smem_desc_lo(ptx::smem_u32(sKV), 16);
    const uint32_t v_lo0 = ptx::smem_desc_lo(ptx::smem_u32(sKV), Cfg::kSlotPanelBytes);
    const uint32_t tmem_st = tmem + t * kBufs * kSubKeys;
    const uint32_t tmem_ot = tmem + Cfg::kTmemO + t * kHeadDim;
    const uint32_t tmem_q = tmem + Cfg::kTmemQ;
    uint64_t* s_full_t = s_full + t * kBufs;
    uint64_t* p_full_t = p_full + t * kBufs;
    uint64_t* pv_done_t = pv_done + t * kBufs;

    uint32_t pair = 0, par = 0;            // ring position of the next K
    uint32_t v_pair[2] = {0, 0}, v_par[2] = {0, 0};
    uint32_t p_par[2] = {0, 0}, q_par = 0;
    bool owed[2] = {false, false};         // a V slot of the last round waits for its release ...
    bool pend[2] = {false, false};         // ... and a P V for being issued
    bool o_acc = false, alive = true;

    auto do_pv = [&](int h) {
      if (!owed[h]) return;
      const uint32_t slot = 2 * v_pair[h] + 1;
      if (Cfg::kHalves == 1 || h == 0) {
        if (!ptx::mbar_wait_warp(&kv_full[slot], v_par[h], abort_flag, 23)) { alive = false; return; }
      }
      if (pend[h]) {
        if (!ptx::mbar_wait_warp(&p_full_t[h], p_par[h], abort_flag, 24)) { alive = false; return; }
        p_par[h] ^= 1;
        ptx::tc_fence_after();
        const uint32_t b_lo = v_lo0 + slot * (Cfg::kSlotBytes >> 4) + (Cfg::kHalves == 2 ? h * ((kSubKeys * 128) >> 4) : 0);
        if (ptx::elect_one()) {
#pragma unroll
          for (int kk = 0; kk < kSubKeys / Cfg::kStepElems; ++kk) {
            // one MMA consumes 32 bytes of every P row (8 columns) and kStepElems rows of V (128 bytes each)
            const uint32_t b = b_lo + kk * ((Cfg::kStepElems * 128) >> 4);
            const uint32_t acc = (kk > 0 || o_acc) ? 1u : 0u;
            if (Cfg::kFp8) ptx::umma_ts_f8_lh(tmem_ot, tmem_st + h * kSubKeys + kk * 8, b, kDescHi, kIdescO, acc);
            else ptx::umma_ts_f16_lh(tmem_ot, tmem_st + h * kSubKeys + kk * 8, b, kDescHi, kIdescO, acc);
          }
          ptx::umma_commit(&pv_done_t[h]);
          if (Cfg::kHalves == 1 || h == 1) ptx::umma_commit(&kv_empty[slot]);
        }
        o_acc = true;
        pend[h] = false;
      } else if (Cfg::kHalves == 1 || h == 1) {
        if (ptx::elect_one()) ptx::umma_commit(&kv_empty[slot]);
      }
      owed[h] = false;
    };

    while (alive) {
      if (!ptx::mbar_wait_warp(&kv_full[2 * pair], par, abort_flag, 22)) break;
      const uint32_t info = ptx::uniform(slot_info[pair]);
      if (info & kInfoStop) break;
      if (Cfg::kQInRing && (info & kInfoQ)) {
        // Every S product of the last item is complete: this warp has waited for the P of each.
        if (!ptx::mbar_wait_warp(&kv_full[2 * pair + 1], par, abort_flag, 21)) break;
        ptx::tc_fence_after();
        if (ptx::elect_one()) {
          const uint32_t lo = k_lo0 + 2 * pair * (Cfg::kSlotBytes >> 4);
#pragma unroll
          for (int kk = 0; kk < kHeadDim / Cfg::kStepElems; ++kk) {
            ptx::tmem_cp_128x32b_lh(tmem_q + kk * 8, lo + (((kk / 4) * kQPanelBytes + (kk % 4) * 32) >> 4), kDescHi);
          }
          ptx::umma_commit(&kv_empty[2 * pair]);
          ptx::umma_commit(&kv_empty[2 * pair + 1]);
        }
        if (++pair == Cfg::kPairs) { pair = 0; par ^= 1; }
        o_acc = false;
        continue;
      }
      if (!Cfg::kQInRing && (info & kInfoFirst)) {
        if (!ptx::mbar_wait_warp(q_full, q_par, abort_flag, 21)) break;
        q_par ^= 1;
        o_acc = false;
        if (Cfg::kTmemHasQ) {
          // Every S product of the last item is complete: this warp has waited for the P of each.
          ptx::tc_fence_after();
          if (ptx::elect_one()) {
#pragma unroll
            for (int kk = 0; kk < kHeadDim / Cfg::kStepElems; ++kk) {
              ptx::tmem_cp_128x32b_lh(tmem_q + kk * 8, q_lo + (((kk / 4) * kQPanelBytes + (kk % 4) * 32) >> 4), kDescHi);
            }
            ptx::umma_commit(q_empty);   // the next item's Q may load
          }
        }
      }
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        do_pv(h);
        if (!alive) break;
        if (Cfg::kHalves == 1 && h == 1) {
          if (!(info & kInfoHalf1)) break;
          if (!ptx::mbar_wait_warp(&kv_full[2 * pair], par, abort_flag, 22)) { alive = false; break; }
        }
        const bool vis = (info >> (2 * t + h)) & 1u;
        const uint32_t slot = 2 * pair;
        const uint32_t b_lo = k_lo0 + slot * (Cfg::kSlotBytes >> 4) + (Cfg::kHalves == 2 ? h * ((kSubKeys * 128) >> 4) : 0);
        const bool ends = (info & kInfoLast) != 0 && (h == 1 || !(info & kInfoHalf1));
        ptx::tc_fence_after();
        if (ptx::elect_one()) {
          if (vis) {
#pragma unroll
            for (int kk = 0; kk < kHeadDim / Cfg::kStepElems; ++kk) {
              const uint32_t a = q_lo + (((kk / 4) * kQPanelBytes + (kk % 4) * 32) >> 4);
              const uint32_t b = b_lo + (((kk / 4) * Cfg::kSlotPanelBytes + (kk % 4) * 32) >> 4);
              if (Cfg::kTmemHasQ) {
                if (Cfg::kFp8) ptx::umma_ts_f8_lh(tmem_st + h * kSubKeys, tmem_q + kk * 8, b, kDescHi, kIdescS, kk > 0);
                else ptx::umma_ts_f16_lh(tmem_st + h * kSubKeys, tmem_q + kk * 8, b, kDescHi, kIdescS, kk > 0);
              } else {
                if (Cfg::kFp8) ptx::umma_ss_f8_lh(tmem_st + h * kSubKeys, a, b, kDescHi, kIdescS, kk > 0);
                else ptx::umma_ss_f16_lh(tmem_st + h * kSubKeys, a, b, kDescHi, kIdescS, kk > 0);
              }
            }
            ptx::umma_commit(&s_full_t[h]);
          }
          if (Cfg::kHalves == 1 || h == 1) ptx::umma_commit(&kv_empty[slot]);
          // Q is read by the S products only: after the last of them the next item's Q may load, while the last
          // P V products and the epilogue of this item still run
          if (!Cfg::kTmemHasQ && ends) ptx::umma_commit(q_empty);
        }
        pend[h] = vis;
        owed[h] = true;
        v_pair[h] = pair;
        v_par[h] = par;
        if (Cfg::kHalves == 1 || h == 1) {
          if (++pair == Cfg::kPairs) { pair = 0; par ^= 1; }
        }
      }
      if (!alive) break;
      if (info & kInfoLast) {
        do_pv(0);
        if (alive) do_pv(1);
        if (!alive) break;
        if ((info & (kInfoTile0 << t)) && ptx::elect_one()) ptx::umma_commit(&o_full[t]);
      }
    }
  }
  } else {
    // ------------------------------------------------------------------------------------ softmax + epilogue
    if (Cfg::kRegRealloc) ptx::reg_acquire_to<Cfg::kSoftmaxRegs>();
    // Loop bounds and addresses in uniform registers: one query tile and e4m3 (2 x 16384 tokens, 8 heads of 256, e4m3: 788 -> 765
    // us; 32 x 512, 16/8 heads of 256, 138 -> 133). With two tiles of 16 bits they are better where the compiler puts them from a
    // plain warp number (4 x 8192 tokens, 32 heads of 64: 771 / 744 us; 1 x 16384, 32/8 heads of 128 872 / 862).
    constexpr bool kUniform = Cfg::kFp8 || kQTiles == 1;
    auto uni = [](auto x) { return kUniform ? ptx::uniform(x) : x; };
    const int own_warp = uni(static_cast<int>(threadIdx.x >> 5));
    const uint32_t tmem_own = uni(*reinterpret_cast<volatile uint32_t*>(tmem_slot));
    const int t = own_warp >> 2;                   // query tile of this warpgroup
    const int quad = own_warp & 3;                     // tensor-memory lane quadrant of this warp
    const int row = quad * 32 + lane;              // row inside the tile
    const uint32_t lane_addr = static_cast<uint32_t>(quad * 32) << 16;
    const uint32_t tmem_s = tmem_own + t * kBufs * kSubKeys + lane_addr;
    const uint32_t tmem_o = tmem_own + Cfg::kTmemO + t * kHeadDim + lane_addr;
    uint32_t s_par = 0;   // bit b: parity of the next S in buffer b
    uint32_t cnt_o = 0;
    bool alive = true;
    uint8_t* stage_o = sStageO + t * Cfg::kStageOBytes;
    for (uint32_t n_sched = 0; alive; ++n_sched) {
      const int idx = sched_peek<true>(mbox, n_sched, abort_flag);
      if (idx < 0 || idx >= total_items) break;
      const Item it = desc[n_sched & 1u].it;
      const TileSpans spans = desc[n_sched & 1u].spans[t];
      const KeyPlan plan = desc[n_sched & 1u].plan;
      sched_release<true>(mbox, n_sched);
      if (!it.valid) continue;
      const int ta = it.qa + t * kBlockM;
      if (ta >= it.qb) continue;
      const int subs = uni(plan.steps() * Cfg::kHalves);
      const int r = ta + row;                      // position in the half
      const bool row_valid = r < it.n;
      const int r_eff = row_valid ? r : it.n - 1;
      const int blk0 = block_lo(r_eff, bs);
      const int blk1 = imin(blk0 + bs, it.n);
      // FP8: the per-(sample, KV head) descales of q and k fold into the score scale, the descale of v into the
      // final normalisation (the reference does the same, flash_fwd_kernel_sm90.h:299-305, mainloop_fwd...:818-822)
      float scale_log2 = p.scale_log2, softcap_pre = p.softcap_pre, lse_scale = p.lse_scale, out_scale = 1.f;
      if (Cfg::kFp8) {
        float qk = 1.f;
        if (p.q_descale != nullptr) qk *= p.q_descale[it.b * p.descale_bs[0] + it.hk * p.descale_hs[0]];
        if (p.k_descale != nullptr) qk *= p.k_descale[it.b * p.descale_bs[1] + it.hk * p.descale_hs[1]];
        if (p.v_descale != nullptr) out_scale = p.v_descale[it.b * p.descale_bs[2] + it.hk * p.descale_hs[2]];
        if (kSoftcap) {
          softcap_pre *= qk;
        } else {
          scale_log2 *= qk;
          lse_scale *= qk;
        }
      }
      // P is rounded to e4m3 for FP8: the exponent is shifted by 8 (the reference's Max_offset = 8, softmax.h:67-69
      // there) and the maximum advances at every increase, so P stays in (0, 2^8] and the largest P of a row is 2^8
      // itself, which e4m3 holds exactly. (P up to 2^8.8 would still fit below 448 and spare most of the rescales of O,
      // 557 instead of 610 us on 4 x 8192 tokens, 16/4 heads of 128, but would round the probability that matters most,
      // by up to 6 %, and the relative error of the output rises from 1.97e-2 to 2.06e-2.) 16-bit P may run up to 2^8
      // above 1 before the maximum is advanced.
      constexpr float kThreshold = Cfg::kFp8 ? 0.f : kRescaleThreshold;
      constexpr float kPShift = Cfg::kFp8 ? 8.f : 0.f;
      // fp8 rescales O often. That is done behind the exponentials, so that the last P V, which must be done first, runs under
      // them (2 x 16384 tokens, 8 heads of 256: 950 -> 897 us; 4 x 8192 tokens, 16/4 heads of 64, 128, 256: 607, 616, 1044 -> 596, 604,
      // 997). 16-bit P rescales O about once an item and gains nothing (1310 against 1326 us on 4 x 8192 tokens, 32/8 heads of 128).
      // Capped scores rescale less: there it is worth it with one query tile only (4 x 8192 tokens, 16/4 heads of 256
      // 1316 -> 1296; of 64 and 128, two tiles, 846 and 852 -> 864 and 871; 16-bit 1328 -> 1339 with 32 heads of 64).
      constexpr bool kLateRescale = Cfg::kFp8 && (!kSoftcap || kHeadDim == 256);
      float m_run = -INFINITY;  // reference maximum (unscaled scores, or tanh values with softcap)
      float l_run = 0.f;
      bool o_started = false, settled = false;   // one sub-step, two sub-steps of this tile are done
      // The clean keys come first, and the first n_full sub-steps of them this tile sees in full: with long samples they have a loop
      // of their own without classification and mask.
      const int n_full = kFullLoop ? uni(imin(spans.half[1].hi_first / kSubKeys, plan.n_clean * Cfg::kHalves)) : 0;
      auto sub_step = [&](auto full_tag, int u, const int buf) {
        constexpr bool kFull = decltype(full_tag)::value;
        int kh = 1, k0 = 0, cls = kTileFull;
        if (!kFull) {
          int kt;
          plan.step(u / Cfg::kHalves, kh, kt);
          k0 = kt * Cfg::kSlotKeys + (u % Cfg::kHalves) * kSubKeys;
          cls = spans.classify(kh, k0);
          if (cls == kTileSkip) return;
        }
        if (!ptx::mbar_wait_warp(&s_full[t * kBufs + buf], (s_par >> buf) & 1u, abort_flag, 31)) { alive = false; return; }
        s_par ^= 1u << buf;
        ptx::tc_fence_after();
        const uint32_t tmem_sb = tmem_s + buf * kSubKeys;
        float v[kSubKeys];
        {
          uint32_t* w = reinterpret_cast<uint32_t*>(v);
#pragma unroll
          for (int c = 0; c < kSubKeys / 32; ++c) ptx::tmem_ld32(tmem_sb + c * 32, w + c * 32);
          ptx::tmem_wait_ld();
        }
        if (kSoftcap) {
#pragma unroll
          for (int c = 0; c < kSubKeys; c += 2) {
            ptx::mul2(v[c], v[c + 1], v[c], v[c + 1], softcap_pre, softcap_pre);
            v[c] = ptx::tanh_fast(v[c]);
            v[c + 1] = ptx::tanh_fast(v[c + 1]);
          }
        }
        if (!kFull && cls == kTileMasked) {
          int lo, hi;
          if (it.qh == 1) { lo = 0; hi = blk1; }
          else if (kh == 1) { lo = 0; hi = blk0; }
          else { lo = blk0; hi = blk1; }
          lo -= k0;
          hi -= k0;
          // A word of visible columns and one select a column: a third of the instructions of two compares and a select each, for
          // every masked sub-step and in what the warps have to fetch (32 x 512 tokens, 16 heads of 128 / 64, blocks of 32: 83 -> 77
          // us, 58.0 -> 53.5; 64 x 200 tokens, blocks of 20: 103 -> 94).
#pragma unroll
          for (int c0 = 0; c0 < kSubKeys; c0 += 32) {
            const uint32_t seen = ptx::bits_below(hi - c0) & ~ptx::bits_below(lo - c0);
#pragma unroll
            for (int c = 0; c < 32; ++c) {
              if (!(seen & (1u << c))) v[c0 + c] = -INFINITY;
            }
          }
        }
        // eight independent running maxima (one chain of dependent max operations costs more than the exponentials
        // that follow)
        float mx[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) mx[i] = fmaxf(v[2 * i], v[2 * i + 1]);
#pragma unroll
        for (int c = 16; c < kSubKeys; c += 16) {
#pragma unroll
          for (int i = 0; i < 8; ++i) mx[i] = ptx::max3(mx[i], v[c + 2 * i], v[c + 2 * i + 1]);
        }
        const float m_tile = fmaxf(ptx::max3(mx[0], mx[1], mx[2]), ptx::max3(ptx::max3(mx[3], mx[4], mx[5]), mx[6], mx[7]));
        const float m_new = fmaxf(m_run, m_tile);
        // Advance the reference maximum only when it grew by more than the threshold. In the first two sub-steps at every
        // increase: the largest of the first 128 scores then has P = 1 exactly, and few rows have a larger one after that.
        // (Settling it on 64 keys saves a rescale of O an item, 289 instead of 298 us on 8 x 4096 tokens, 16 heads of 128,
        // but the relative error of the output, over 24 drawn shapes in bf16, is 2.21e-3 instead of 2.17e-3.)
        const bool need = (m_new - m_run) * scale_log2 > (settled ? kThreshold : 0.f);
        const bool any_need = __any_sync(0xffffffffu, need);
        float factor = 1.f;
        auto rescale = [&]() {
          // every P V of this tile so far must have updated O. In this buffer it has: S followed it through the
          // pipe. In the others the last one may still run (an unused buffer's barrier passes at once).
#pragma unroll
          for (int b = 0; b < kBufs; ++b) {
            if (b == buf) continue;
            if (!ptx::mbar_wait_warp(&pv_done[t * kBufs + b], ((s_par >> b) & 1u) ^ 1u, abort_flag, 33)) { alive = false; return; }
          }
          ptx::tc_fence_after();
          // A load is answered after some 250 cycles while products run, however wide it is. fp8 rescales often, and with
          // one query tile has the registers for 128 columns a round (2 x 16384 tokens, 8 heads of 256: 1017 -> 948 us;
          // with two tiles 64 are slower than 32, 646 against 610 us on 4 x 8192 tokens, 16/4 heads of 128).
          constexpr int kRound = Cfg::kFp8 && kQTiles == 1 ? 128 : 32;
#pragma unroll
          for (int c0 = 0; c0 < kHeadDim; c0 += kRound) {
            float o[kRound];
#pragma unroll
            for (int c = 0; c < kRound; c += 32) ptx::tmem_ld32(tmem_o + c0 + c, reinterpret_cast<uint32_t*>(o) + c);
            ptx::tmem_wait_ld();
#pragma unroll
            for (int i = 0; i < kRound; i += 2) ptx::mul2(o[i], o[i + 1], o[i], o[i + 1], factor, factor);
#pragma unroll
            for (int c = 0; c < kRound; c += 32) ptx::tmem_st32(tmem_o + c0 + c, reinterpret_cast<uint32_t*>(o) + c);
          }
        };
        if (any_need) {
          if (need) factor = ptx::ex2((m_run - m_new) * scale_log2);
          if (!kLateRescale && o_started) {
            rescale();
            if (!alive) return;
          }
          l_run *= factor;
          if (need) m_run = m_new;
        }
        const float m_ref = (m_run == -INFINITY) ? 0.f : m_run;
        const float neg_m = kPShift - m_ref * scale_log2;
        float sum4[4] = {0.f, 0.f, 0.f, 0.f};
        uint32_t pk[Cfg::kPCols];
        {
          // Two elements per FMA and per ADD: the sums run as four pairs of partial sums. What a warp issues counts here as much
          // as the special-function unit: packed arithmetic for e4m3 too, and packed products for the rescale and the argument of
          // tanh, took 4 x 8192 tokens, 16/4 heads of 128, e4m3 from 598 to 555 us, 8 x 4096 tokens, 16 heads of 128, capped, from 407
          // to 389.
          float sumb[4] = {0.f, 0.f, 0.f, 0.f};
          constexpr int kWord = 4 / Cfg::kElemBytes;   // elements a word of P
#pragma unroll
          for (int c = 0; c < kSubKeys; c += kWord) {
            float e[kWord];
#pragma unroll
            for (int i = 0; i < kWord; i += 2) {
              float y0, y1;
              ptx::fma2(y0, y1, v[c + i], v[c + i + 1], scale_log2, scale_log2, neg_m, neg_m);
              e[i] = ptx::ex2(y0);
              e[i + 1] = ptx::ex2(y1);
              const int s = ((c + i) / 2) & 3;
              ptx::add2(sum4[s], sumb[s], sum4[s], sumb[s], e[i], e[i + 1]);
            }
            pk[c / kWord] = Cfg::kFp8 ? ptx::pack_e4m3x4(e[0], e[1], e[kWord - 2], e[kWord - 1]) : ptx::pack2<kType == 0>(e[0], e[1]);
          }
#pragma unroll
          for (int i = 0; i < 4; ++i) sum4[i] += sumb[i];
        }
        l_run += (sum4[0] + sum4[1]) + (sum4[2] + sum4[3]);
        if (Cfg::kPCols == 32) ptx::tmem_st32(tmem_sb, pk);
        else ptx::tmem_st16(tmem_sb, pk);
        if (kLateRescale && any_need && o_started) {
          rescale();
          if (!alive) return;
        }
        ptx::tmem_wait_st();
        ptx::tc_fence_before();
        ptx::mbar_arrive_warp(&p_full[t * kBufs + buf]);
        settled = o_started;
        o_started = true;
      };
      int u = 0;
      if (Cfg::kUnrollFull) {
#pragma unroll 1
        for (; u + 2 <= n_full && alive; u += 2) {
          sub_step(std::true_type{}, u, 0);
          if (alive) sub_step(std::true_type{}, u + 1, 1);
        }
      } else {
#pragma unroll 1
        for (; u < n_full && alive; ++u) sub_step(std::true_type{}, u, u & 1);
      }
#pragma unroll 1
      for (; u < subs && alive; ++u) sub_step(std::false_type{}, u, u & 1);
      if (!alive) break;
      // ---- epilogue: O / l -> global, LSE
      if (!ptx::mbar_wait_warp(&o_full[t], cnt_o & 1, abort_flag, 32)) { alive = false; break; }
      ++cnt_o;
      ptx::tc_fence_after();
      const float inv_l = out_scale / l_run;
      const int64_t srow = static_cast<int64_t>(it.row0) + it.qh * it.n + r;
      bool lse_done = false;
      auto store_lse = [&]() {
        lse_done = true;
        if (row_valid) {
          const float m_ref = (m_run == -INFINITY) ? 0.f : m_run;
          const float lse = (l_run > 0.f) ? m_ref * lse_scale + (__log2f(l_run) - kPShift) * kLn2 : -INFINITY;
          const int64_t li = (p.cu_seqlens != nullptr)
                                 ? static_cast<int64_t>(it.h) * p.total + srow
                                 : (static_cast<int64_t>(it.b) * p.heads + it.h) * p.seqlen + (it.qh * it.n + r);
          p.lse[li] = lse;
        }
      };
      if (p.o_tma != 0 && ta + kBlockM <= it.n) {
        // Whole tile: through shared memory, 64 columns at a time, and out as tile copies, one per warp (32 rows),
        // so that no warp waits for another. (A row per thread written straight to global memory costs one
        // memory transaction per thread and instruction; for a 128 x 128 tile that is thousands of cycles in
        // which the load/store unit serves nobody else.)
        uint8_t* my_stage = stage_o + quad * (32 * 128);
#pragma unroll
        for (int pass = 0; pass < kHeadDim / 64; ++pass) {
          if (pass * 64 < p.head_dim) {
            uint32_t o[64];
            ptx::tmem_ld32(tmem_o + pass * 64, o);
            ptx::tmem_ld32(tmem_o + pass * 64 + 32, o + 32);
            ptx::tmem_wait_ld();
            uint32_t w[32];
#pragma unroll
            for (int i = 0; i < 32; ++i) {
              w[i] = ptx::pack2<kType != 1>(__uint_as_float(o[2 * i]) * inv_l, __uint_as_float(o[2 * i + 1]) * inv_l);
            }
            // the previous copy out of this warp's buffer (last pass or last item) must have read it completely
            if (lane == 0) ptx::bulk_wait_group_read0();
            __syncwarp();
            ptx::st_shared_row128_sw(my_stage, lane, w);
            ptx::fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) {
              ptx::tma_store_4d(&p.tm_o, my_stage, pass * 64, it.row0 + it.qh * it.n + ta + quad * 32, it.h, it.bcoord);
              ptx::bulk_commit_group();
            }
            // the log-sum-exp goes out while the tile copy reads the buffer
            if (!lse_done) store_lse();
          }
        }
      } else {
        uint16_t* orow = reinterpret_cast<uint16_t*>(p.out) + it.bcoord * p.o_batch_stride + srow * p.o_row_stride +
                         it.h * p.o_head_stride;
        // all loads first, one wait: the stores of a chunk then overlap the conversion of the next
        uint32_t o[kHeadDim <= 128 ? kHeadDim : 128];
        constexpr int kPass = kHeadDim <= 128 ? 1 : kHeadDim / 128;
#pragma unroll
        for (int pass = 0; pass < kPass; ++pass) {
          constexpr int kPassCols = kHeadDim <= 128 ? kHeadDim : 128;
#pragma unroll
          for (int c = 0; c < kPassCols / 32; ++c) ptx::tmem_ld32(tmem_o + pass * 128 + c * 32, o + c * 32);
          ptx::tmem_wait_ld();
          if (row_valid) {
#pragma unroll
            for (int c = 0; c < kPassCols / 32; ++c) {
              ptx::store_row32<kType != 1>(orow, pass * 128 + c * 32, o + c * 32, inv_l, p.head_dim, p.wide_store != 0);
            }
          }
        }
      }
      if (!lse_done) store_lse();
      ptx::tc_fence_before();
    }
    // shared memory must outlive the tile copies that read it
    if (lane == 0) ptx::bulk_wait_group0();
  }

  ptx::tc_fence_before();
  __syncthreads();
  if (warp == Cfg::kLoadWarp) ptx::tmem_dealloc(tmem, 512);
}

template <int kHeadDim, int kQTiles, int kType, bool kSoftcap, bool kQInTmem, bool kFullLoop>
int launch_fwd_instance(const FwdParams& p, int grid, cudaStream_t stream) {
  using Cfg = FwdConfig<kHeadDim, kQTiles, kType, kSoftcap, kQInTmem>;
  auto kernel = fwd_kernel<kHeadDim, kQTiles, kType, kSoftcap, kQInTmem, kFullLoop>;
  static PerDeviceFlags smem_set;
  const int rc = set_dynamic_smem(kernel, Cfg::kSmemBytes, smem_set);
  if (rc) return rc;
  return launch_kernel(p.overlap != 0, kernel, grid, Cfg::kThreads, Cfg::kSmemBytes, stream, p);
}

template <int kHeadDim, int kQTiles, int kType, bool kQInTmem>
int dispatch_fwd(const FwdParams& p, int grid, bool softcap, bool full_loop, cudaStream_t stream) {
  constexpr bool kHas = kHeadDim == 64 || kType == 2;   // the loop over fully visible sub-steps: see forward_full_loop
  if (kHas && full_loop) {
    return softcap ? launch_fwd_instance<kHeadDim, kQTiles, kType, true, kQInTmem, kHas>(p, grid, stream)
                   : launch_fwd_instance<kHeadDim, kQTiles, kType, false, kQInTmem, kHas>(p, grid, stream);
  }
  return softcap ? launch_fwd_instance<kHeadDim, kQTiles, kType, true, kQInTmem, false>(p, grid, stream)
                 : launch_fwd_instance<kHeadDim, kQTiles, kType, false, kQInTmem, false>(p, grid, stream);
}

template <int kHeadDim, int kQTiles, bool kQInTmem = false>
int dispatch_fwd16(const FwdParams& p, int grid, bool bf16, bool softcap, bool full_loop, cudaStream_t stream) {
  return bf16 ? dispatch_fwd<kHeadDim, kQTiles, 0, kQInTmem>(p, grid, softcap, full_loop, stream)
              : dispatch_fwd<kHeadDim, kQTiles, 1, kQInTmem>(p, grid, softcap, full_loop, stream);
}

}  // namespace

size_t fwd_workspace_bytes(const FdaProblem& pr) {
  // scheduler words, and for packed batches the work list
  return 256 + (pr.cu_seqlens != nullptr ? varlen_list_bytes(pr.batch) : 0);
}

// Whether fully visible sub-steps get a loop of their own. It saves their classification and mask, and makes a second
// and a third copy of a long body. Where CTAs take many items of few sub-steps each, or of few that the loop takes
// (noisy rows of large blocks see no clean key in full), the warps run from one copy into another and wait for
// instructions. One loop / two, us, d = 64, e4m3, e4m3 of 256 (16/8 heads, blocks of 64):
//   32 x 1024 tokens  111 / 142  135 / 188  238 / 277      4 x 6000   257 / 252  327 / 323  550 / 538
//   8 x 3000          157 / 164  197 / 219  332 / 355      3 x 8192   323 / 303  409 / 384  688 / 642
//   8 x 4096          248 / 252  314 / 331  535 / 550      1 x 16384  388 / 362  487 / 454  823 / 754
// 3 x 8192 in blocks of 1024: 355 / 345, 470 / 440, 798 / 746; in one block: 558 / 580, 744 / 723, 1216 / 1181. Capped,
// 3 x 8192: 501 / 486, 600 / 565, 892 / 828. With at most eight items a CTA the loop loses nothing from 600 tokens a
// half on (blocks of 16): 16 x 512, 16 heads 20.6 / 20.6, 21.0 / 22.7, 33.1 / 33.6; 1 x 1400, 16/4 heads 17.2 / 16.7,
// 20.3 / 19.5, 22.7 / 23.5; 4 x 1400 35.1 / 34.8, 39.4 / 39.1, 63.5 / 62.4; 1 x 3000, 16 heads 35.7 / 33.1, 43.3 /
// 40.8, 55.9 / 55.4; 1 x 6000, 3 heads 38.8 / 35.2, 46.8 / 43.3, 49.7 / 49.9; 1 x 4096, 16 heads in one block 69.1 /
// 69.9, 88.7 / 88.0, 141 / 137. 16-bit heads of 128 have one loop (1 x 16384, 32/8 heads, blocks of 64, 256 and 1024
// 941 / 963, 953 / 984, 1033 / 1063; 3 x 8192, 16/8, blocks of 1024 427 / 448), and those of 256, which wait for K and
// V (1 % the other way).
bool forward_full_loop(const FdaProblem& pr) {
  const bool fp8 = pr.dtype == FDA_E4M3;
  if (pr.batch <= 0 || (!fp8 && pr.head_dim > 64)) return false;
  const int64_t tokens = pr.total / (2 * static_cast<int64_t>(pr.batch));   // of a half, on average
  const int item_rows = pr.head_dim > 128 ? kBlockM : 2 * kBlockM;
  const int64_t items = (tokens + item_rows - 1) / item_rows * 2 * pr.heads * pr.batch;
  const bool few = items <= 8 * 148;
  if (tokens < (few ? 600 : fp8 ? 3000 : 4096)) return false;
  return fp8 || (few ? 2 : 4) * static_cast<int64_t>(pr.block_size) <= tokens;
}

int launch_fwd(const FdaFwdArgs& a, cudaStream_t stream) {
  const FdaProblem& pr = a.p;
  DeviceInfo info;
  int rc = current_device_info(&info);
  if (rc) return rc;
  if (info.cc_major != 10) return FDA_ERR_ARCH;

  const int d = pr.head_dim;
  const bool fp8 = pr.dtype == FDA_E4M3;
  // FP8 rows are padded to whole 128-byte panels, so the smallest FP8 kernel is the 128-wide one
  const int d_round = (d <= 64 && !fp8) ? 64 : (d <= 128 ? 128 : 256);
  const int slot_keys = (d_round == 256 && !fp8) ? 64 : 128;   // FwdConfig::kSlotKeys
  const int eb = fp8 ? 1 : 2;
  const int box_cols = 128 / eb;
  const bool varlen = pr.cu_seqlens != nullptr;
  const int64_t rows = varlen ? pr.total : pr.seqlen;
  const int tma_batch = varlen ? 1 : pr.batch;
  const bool fp16 = pr.dtype == FDA_FP16;

  int grid = info.sm_count - (pr.sm_margin > 0 ? pr.sm_margin : 0);
  if (grid < 1) grid = 1;
  // Items of two query tiles share the K and V they read. Where even items of one tile find an SM each, one tile per
  // item halves the time of the longest item instead. (Packed batches: by the upper bound that the host knows.)
  auto item_bound = [&](int tiles) -> int64_t {
    if (varlen) return (static_cast<int64_t>(pr.total) / (2 * tiles * kBlockM) + pr.batch) * 2 * pr.heads;
    return static_cast<int64_t>(ceil_div(pr.seqlen / 2, tiles * kBlockM)) * 2 * pr.heads * pr.batch;
  };
  const int q_tiles = d_round > 128 || item_bound(1) <= grid ? 1 : 2;

  FwdParams p;
  memset(&p, 0, sizeof(p));
  rc = encode_tile_map(&p.tm_q, a.q.ptr, eb, fp8, fp16, d, rows, pr.heads, tma_batch, a.q.row_stride,
                       a.q.head_stride, a.q.batch_stride, box_cols, kBlockM);
  if (rc) return rc;
  rc = encode_tile_map(&p.tm_k, a.k.ptr, eb, fp8, fp16, d, rows, pr.heads_k, tma_batch, a.k.row_stride,
                       a.k.head_stride, a.k.batch_stride, box_cols, slot_keys);
  if (rc) return rc;
  rc = encode_tile_map(&p.tm_v, a.v.ptr, eb, fp8, fp16, d, rows, pr.heads_k, tma_batch, a.v.row_stride,
                       a.v.head_stride, a.v.batch_stride, box_cols, slot_keys);
  if (rc) return rc;
  if (fp8) {
    p.q_descale = a.q_descale;
    p.k_descale = a.k_descale;
    p.v_descale = a.v_descale;
    for (int i = 0; i < 3; ++i) {
      p.descale_bs[i] = a.descale_batch_stride[i];
      p.descale_hs[i] = a.descale_head_stride[i];
    }
  }
  {
    // out: 16-bit whatever the inputs are. What the tile copy wants of out (16-byte aligned base and strides) is
    // also what the row stores of partial tiles need, so a refusal here is final.
    const int orc = encode_tile_map(&p.tm_o, a.out.ptr, 2, false, fp16, d, rows, pr.heads, tma_batch, a.out.row_stride,
                                    a.out.head_stride, a.out.batch_stride, 64, 32);
    if (orc != FDA_OK) return orc;
    p.o_tma = 1;
  }
  p.out = a.out.ptr;
  p.lse = a.lse;
  p.o_batch_stride = varlen ? 0 : a.out.batch_stride;
  p.o_row_stride = a.out.row_stride;
  p.o_head_stride = a.out.head_stride;
  p.wide_store = (d % 16 == 0 && (reinterpret_cast<uintptr_t>(a.out.ptr) & 31) == 0 && a.out.row_stride % 16 == 0 &&
                  a.out.head_stride % 16 == 0 && (varlen || a.out.batch_stride % 16 == 0))
                     ? 1
                     : 0;
  p.cu_seqlens = pr.cu_seqlens;
  p.batch = pr.batch;
  p.seqlen = pr.seqlen;
  p.total = pr.total;
  p.heads = pr.heads;
  p.heads_k = pr.heads_k;
  p.overlap = overlapped_launches(pr, 0) ? 1 : 0;
  p.next_early = pr.sm_margin <= 0 ? 1 : 0;
  p.head_dim = d;
  p.block_size = pr.block_size;
  const int max_n = pr.seqlen / 2;
  p.items_per_half = ceil_div(max_n, q_tiles * kBlockM);
  p.total_items = p.items_per_half * 2 * pr.heads * pr.batch;
  const bool softcap = pr.softcap > 0.f;
  if (softcap) {
    p.scale_log2 = pr.softcap * kLog2e;
    p.softcap_pre = pr.softmax_scale / pr.softcap;
    p.lse_scale = pr.softcap;
  } else {
    p.scale_log2 = pr.softmax_scale * kLog2e;
    p.softcap_pre = 0.f;
    p.lse_scale = pr.softmax_scale;
  }
  if (p.total_items <= 0) return FDA_OK;
  if (!a.workspace || a.workspace_bytes < fwd_workspace_bytes(pr)) return FDA_ERR_WORKSPACE;
  p.ticket = static_cast<int*>(a.workspace);
  // the shortest eighths of every (sample, head) run at the end; few items per CTA: rank for rank over all of them
  p.n_long = order_n_long(2 * p.items_per_half, FDA_SHORT8_FWD, p.total_items, grid);
  if (varlen) {
    // the work list is built on the device from cu_seqlens (no host synchronisation): the host only knows an upper
    // bound of the number of items, blocks beyond the real number find no work and leave
    int* list = reinterpret_cast<int*>(static_cast<uint8_t*>(a.workspace) + 256);
    const int rc = launch_varlen_prepare(pr.cu_seqlens, pr.batch, q_tiles * kBlockM, list, p.ticket, stream, p.overlap != 0);
    if (rc) return rc;
    p.vl.base = list;
    p.vl.batch = pr.batch;
    if (grid > item_bound(q_tiles)) grid = static_cast<int>(item_bound(q_tiles));
  } else if (grid >= p.total_items) {
    grid = p.total_items;   // a block for every item: no work counter, nothing to zero
    p.ticket = nullptr;
  } else {
    FDA_CUDA_TRY(cudaMemsetAsync(p.ticket, 0, kTicketInts * 4, stream));
  }
  const bool bf16 = pr.dtype == FDA_BF16;
  const bool full_loop = forward_full_loop(pr);
  if (fp8) {
    if (d_round == 256) return dispatch_fwd<256, 1, 2, true>(p, grid, softcap, full_loop, stream);
    return q_tiles == 2 ? dispatch_fwd<128, 2, 2, false>(p, grid, softcap, full_loop, stream)
                        : dispatch_fwd<128, 1, 2, false>(p, grid, softcap, full_loop, stream);
  }
  if (d_round == 256) return dispatch_fwd16<256, 1, true>(p, grid, bf16, softcap, full_loop, stream);
  if (d_round == 128) {
    return q_tiles == 2 ? dispatch_fwd16<128, 2>(p, grid, bf16, softcap, full_loop, stream)
                        : dispatch_fwd16<128, 1>(p, grid, bf16, softcap, full_loop, stream);
  }
  return q_tiles == 2 ? dispatch_fwd16<64, 2>(p, grid, bf16, softcap, full_loop, stream)
                      : dispatch_fwd16<64, 1>(p, grid, bf16, softcap, full_loop, stream);
}

int read_status_fwd(int32_t* out4) {
  int zero[4] = {0, 0, 0, 0};
  FDA_CUDA_TRY(cudaMemcpyFromSymbol(out4, g_fda_status, sizeof(int) * 4));
  FDA_CUDA_TRY(cudaMemcpyToSymbol(g_fda_status, zero, sizeof(int) * 4));
  return FDA_OK;
}

}  // namespace fda
