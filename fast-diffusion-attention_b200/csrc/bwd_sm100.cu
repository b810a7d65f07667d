// Backward pass of block-diffusion attention for sm_100a.
//
// The reference runs up to six launches (csrc/fda/flash_bwd_launch_template.h:26-284 there): a preprocess
// (flash_bwd_preprocess_kernel.h:106-208), an optional noisy-diagonal kernel, the dK/dV-stationary main kernel
// with an fp32 dQ accumulator reduced through global memory (mainloop_bwd_sm90_tma_gmma_ws.hpp:413-1014,
// epilogue_bwd.hpp:25-441), and convert passes (flash_bwd_postprocess_kernel.h:160-264). On B200 the tensor
// memory budget (512 columns) and the cost of a global fp32 reduction lead to a different split:
//
//   1. bwd_preprocess : delta = rowsum(dO * O) and -LSE * log2(e), written to a padded per-(sample, head, half)
//                       layout whose padding rows carry -inf for the latter (so padded query rows get P = 0). It also
//                       zeroes the work counters and small dQ accumulators of the kernels that follow.
//   2. bwd_dkdv       : one CTA per (128-key tile, KV head, sample, half); K, V stay in shared memory, the
//                       visible query tiles of every query head of the group stream through. S^T = K Q^T and
//                       dP^T = V dO^T land in tensor memory (keys on lanes); P^T and dS^T go back to tensor
//                       memory as 16-bit A operands of dV += P^T dO and dK += dS^T Q. GQA sums over the group
//                       inside the CTA: no fp32 dK/dV accumulators in global memory. Head dims above 128: an item makes
//                       either dK or dV.
//   3. bwd_dq         : forward-shaped, one CTA per 128-row query tile: S = Q K^T, dP = dO V^T, dS to tensor
//                       memory, dQ += dS K. No cross-CTA reduction at all, so dQ needs no atomics, no fp32
//                       accumulator, no zero-fill and no convert pass.
//
// Seven GEMMs per tile pair instead of five (eight for head dims above 128), in exchange for zero global reductions; every
// gradient has a fixed accumulation order, so the result is bitwise reproducible whether or not `deterministic` is set.
// Numerics kept from the reference: P = exp2(S*c - LSE * log2(e)) from the saved LSE, dS = P * (dP - delta)
// [* (1 - tanh^2) with softcap, before masking], P and dS rounded to the input dtype before the second GEMMs,
// dK and dQ scaled by softmax_scale once at the end (mainloop_bwd...hpp:836-893, :1009).
#include <type_traits>

#include "bwd_common.cuh"

namespace fda {
namespace {

// ------------------------------------------------------------------------------------------------------------
// 1. preprocess
// ------------------------------------------------------------------------------------------------------------
// rows per thread group; measured on the benchmark shape (268 MB read): 1 row 0.063 ms, 2 rows 0.053, 4 rows 0.066,
// 8 rows 0.072
constexpr int kPreUnroll = 2;

template <bool kBf16, int kLanes>
__global__ void __launch_bounds__(256) bwd_preprocess_kernel(const __grid_constant__ BwdParams p) {
  ptx::wait_for_stream();
  ptx::let_next_start();
  constexpr int kRowsPerWarp = 32 / kLanes;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int sub = lane / kLanes, l = lane % kLanes;
  const int hh = blockIdx.y;
  const int h = hh >> 1, half = hh & 1;
  const int b = blockIdx.z;
  // zero-fills for the kernels that follow, so that a small problem does not pay a launch for each of them
  if (p.zero_tickets != nullptr && (blockIdx.x | blockIdx.y | blockIdx.z) == 0 && threadIdx.x < kTicketInts) {
    p.zero_tickets[threadIdx.x] = 0;
  }
  if (p.zero_acc16 != 0) {
    const int64_t block = (static_cast<int64_t>(b) * gridDim.y + hh) * gridDim.x + blockIdx.x;
    const int64_t threads = static_cast<int64_t>(gridDim.x) * gridDim.y * gridDim.z * 256;
    for (int64_t i = block * 256 + threadIdx.x; i < p.zero_acc16; i += threads) {
      reinterpret_cast<uint4*>(p.dq_acc)[i] = make_uint4(0, 0, 0, 0);
    }
  }
  const Sample sm = sample_of(p, b);
  const int64_t seg = stat_segment(p, b, h, half);
  // row u of this thread group: position in the half (rows >= n, up to n_pad, only get their padding values)
  const int r0 = ((blockIdx.x * 8 + warp) * kPreUnroll) * kRowsPerWarp + sub;
  float acc[kPreUnroll];
  // head dimensions up to 8 * kLanes take one 16-byte piece of O and of dO per lane: all loads of the kPreUnroll rows
  // are issued before the first use
  uint4 ov[kPreUnroll], gv[kPreUnroll];
#pragma unroll
  for (int u = 0; u < kPreUnroll; ++u) {
    const int r = r0 + u * kRowsPerWarp;
    acc[u] = 0.f;
    ov[u] = make_uint4(0, 0, 0, 0);
    gv[u] = make_uint4(0, 0, 0, 0);
    if (r < sm.n && l * 8 < p.head_dim) {
      const int64_t srow = static_cast<int64_t>(sm.row0) + half * sm.n + r;
      const uint16_t* o = static_cast<const uint16_t*>(p.out) + sm.bcoord * p.o_bs + srow * p.o_rs + h * p.o_hs;
      const uint16_t* g = static_cast<const uint16_t*>(p.dout) + sm.bcoord * p.do_bs + srow * p.do_rs + h * p.do_hs;
      ov[u] = *reinterpret_cast<const uint4*>(o + l * 8);
      gv[u] = *reinterpret_cast<const uint4*>(g + l * 8);
    }
  }
#pragma unroll
  for (int u = 0; u < kPreUnroll; ++u) {
    const uint32_t aw[4] = {ov[u].x, ov[u].y, ov[u].z, ov[u].w};
    const uint32_t dw[4] = {gv[u].x, gv[u].y, gv[u].z, gv[u].w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      float2 fa, fd;
      if (kBf16) {
        fa = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&aw[i]));
        fd = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&dw[i]));
      } else {
        fa = __half22float2(*reinterpret_cast<const __half2*>(&aw[i]));
        fd = __half22float2(*reinterpret_cast<const __half2*>(&dw[i]));
      }
      acc[u] = fmaf(fa.x, fd.x, acc[u]);
      acc[u] = fmaf(fa.y, fd.y, acc[u]);
    }
#pragma unroll
    for (int off = kLanes / 2; off > 0; off >>= 1) acc[u] += __shfl_xor_sync(0xffffffffu, acc[u], off);
  }
  if (l == 0) {
#pragma unroll
    for (int u = 0; u < kPreUnroll; ++u) {
      const int r = r0 + u * kRowsPerWarp;
      if (r >= p.n_pad) continue;
      const bool valid = r < sm.n;
      float lse2 = -INFINITY;
      if (valid) {
        const int64_t srow = static_cast<int64_t>(sm.row0) + half * sm.n + r;
        const int64_t li = (p.cu_seqlens != nullptr)
                               ? static_cast<int64_t>(h) * p.total + srow
                               : (static_cast<int64_t>(b) * p.heads + h) * p.seqlen + (half * sm.n + r);
        const float lse = p.lse[li];
        lse2 = (lse == -INFINITY) ? 0.f : -lse * kLog2e;
      }
      p.delta_pad[seg + r] = valid ? acc[u] : 0.f;
      p.lse2_pad[seg + r] = lse2;
    }
  }
}

// ------------------------------------------------------------------------------------------------------------
// 2. dK / dV
// ------------------------------------------------------------------------------------------------------------

// kMakes: bit 0 dK, bit 1 dV (one without the other: head dims above 128).
template <int kHeadDim, int kStages, int kMakes>
struct DkdvCfg {
  using T = TileCfg<kHeadDim>;
  static constexpr int kSubTileBytes = kSub * kHeadDim * 2;     // Q or dO sub-tile
  static constexpr int kSubPanelBytes = kSub * 128;             // one 64-column panel of a sub-tile
  static constexpr int kThreads = kDkdvThreads;
  // buffer u: S^T at u*128, dP^T at u*128 + 64; accumulators behind
  // Head dimensions above 128 do not leave room for both accumulators next to the S^T / dP^T buffers: every key tile is
  // two items, one for dK (three products: S^T, dP^T, dS^T Q) and one for dV (two: S^T, P^T dO). Halving the columns of
  // both instead takes S^T and dP^T twice, six products for five. (Backward of 2 x 16384 tokens, 8 heads of 256, blocks of
  // 256: 7.34 -> 4.97 ms with the rings below.)
  static constexpr int kPasses = kHeadDim > 128 ? 2 : 1;
  static constexpr int kItems = kMakes == 3 ? kPasses : 1;   // a key tile
  static constexpr bool kDvOnly = kMakes == 2;
  static_assert(kMakes == 3 || kPasses == 2, "head dims above 128");
  static constexpr int kTmemDK = 256, kTmemDV = kPasses == 2 ? 256 : 256 + kHeadDim;
  static_assert(kTmemDV + kHeadDim <= 512, "tensor memory budget");
  // Rings of Q and dO sub-tiles of their own. With 128 KB of K and V there is room for three of 32 KB: two for Q, one for
  // dO, so that the next sub-step's tiles load while this one's are in use (one slot for both left the pipe waiting for
  // every load).
  // Without dK nobody reads V, and dO gets three slots: with one, a dV product waited for the load
  // behind the last (2 x 16384 tokens, 8 heads of 256: 1346 -> 934 us for dV).
  static constexpr int kQSlots = kPasses == 2 ? 2 : kStages, kDoSlots = kDvOnly ? 3 : kPasses == 2 ? 1 : kStages;
  // lse2[64], delta[64] and the header of a sub-step. The slot of step x is written when Q of step x - 2 is done with,
  // which for dV means S^T of x - 2 complete, so that step x - 4 is the last that every role has certainly left.
  static constexpr int kStatSlots = kPasses == 2 ? 4 : kStages;
  static constexpr int kHeaderOffset = 2 * kSub * 4, kStatBytes = kHeaderOffset + 32;
  static constexpr int kOffQ = (kDvOnly ? 1 : 2) * T::kTileBytes, kOffDo = kOffQ + kQSlots * kSubTileBytes;
  static constexpr int kOffStat = kOffDo + kDoSlots * kSubTileBytes;
  static constexpr int kOffBar = kOffStat + kStatSlots * kStatBytes;
  static constexpr int kSmemBytes = kOffBar + 512;
  static_assert(kSmemBytes <= 232448 && kOffBar % 16 == 0, "shared memory budget");
  static_assert((11 + 2 * kQSlots + 2 * kDoSlots + kStatSlots) * 8 + 8 <= 384, "barrier area");
};

// Calls fn(SubStep) for every non-skipped sub-step of the item, in order; stops early when fn returns false. A sub-step is one
// 64-row half of a visible 128-row query tile of one query head of the group; a half with no visible row is skipped.
template <typename Fn>
__device__ __forceinline__ bool for_each_substep(const KvItem& it, const QueryPlan& plan, const KvSpans& spans, int group, Fn&& fn) {
  for (int g = 0; g < group; ++g) {
    for (int s = 0; s < plan.steps(); ++s) {
      int qh, qt;
      plan.step(s, it.kh, qh, qt);
      const int qa = qt * kTile, qb = imin(qa + kTile, it.n);
      if (spans.classify(qh, it.kh, qa, qb) == kTileSkip) continue;
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        SubStep st;
        st.sa = qa + half * kSub;
        if (st.sa >= qb) continue;
        st.sb = imin(st.sa + kSub, qb);
        st.cls = spans.classify(qh, it.kh, st.sa, st.sb);
        if (st.cls == kTileSkip) continue;
        st.h = it.hk * group + g;
        st.qh = qh;
        if (!fn(st)) return false;
      }
    }
  }
  return true;
}

// One CTA per SM. A sub-step is one 64-row half of a visible 128-row query tile of one query head of the group; a half with
// no visible row is skipped.
template <int kHeadDim, int kStages, bool kBf16, bool kSoftcap, int kMakes>
__global__ void __launch_bounds__(kDkdvThreads, 1) bwd_dkdv_kernel(const __grid_constant__ BwdParams p) {
  using Cfg = DkdvCfg<kHeadDim, kStages, kMakes>;
  using T = TileCfg<kHeadDim>;
  // The tiles need 1024-byte alignment for the 128-byte swizzle. Dynamic shared memory starts at the beginning of the
  // block's window, which is aligned that far; head dimension 256 leaves no room to round the base up, so a base that is
  // not aligned is reported through the status word instead.
  extern __shared__ __align__(1024) uint8_t smem_dkdv[];
  uint8_t* smem = smem_dkdv;
  uint8_t* sK = smem;
  uint8_t* sV = smem + T::kTileBytes;
  uint8_t* sQ = smem + Cfg::kOffQ;
  uint8_t* sDo = smem + Cfg::kOffDo;
  uint8_t* sStat = smem + Cfg::kOffStat;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + Cfg::kOffBar);
  uint64_t* kv_full = bars;
  uint64_t* kv_empty = bars + 1;
  uint64_t* q_full = bars + 2;                    // [kQSlots]
  uint64_t* q_empty = q_full + Cfg::kQSlots;
  uint64_t* do_full = q_empty + Cfg::kQSlots;     // [kDoSlots]
  uint64_t* do_empty = do_full + Cfg::kDoSlots;
  uint64_t* stat_full = do_empty + Cfg::kDoSlots; // [kStatSlots] statistics and header
  uint64_t* sdp_full = stat_full + Cfg::kStatSlots;   // [2]
  uint64_t* pds_full = sdp_full + 2;         // [2]
  uint64_t* acc_full = pds_full + 2;
  uint64_t* buf_free = acc_full + 1;         // [2]
  uint64_t* acc_free = buf_free + 2;         // the epilogue warps have the accumulators in registers
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_free + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  SchedMailbox* mbox = reinterpret_cast<SchedMailbox*>(reinterpret_cast<uint8_t*>(bars) + 384);

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
    sched_init(mbox, 4 * kCmpWG + 2 + 4);   // compute warps, two MMA issuers, four epilogue warps
    ptx::mbar_init(kv_full, 1);
    ptx::mbar_init(kv_empty, 1);
    for (int i = 0; i < Cfg::kQSlots; ++i) {
      ptx::mbar_init(&q_full[i], 1);
      ptx::mbar_init(&q_empty[i], 1);
    }
    for (int i = 0; i < Cfg::kDoSlots; ++i) {
      ptx::mbar_init(&do_full[i], 1);
      ptx::mbar_init(&do_empty[i], 1);
    }
    for (int i = 0; i < Cfg::kStatSlots; ++i) ptx::mbar_init(&stat_full[i], 1);
    for (int u = 0; u < 2; ++u) {
      ptx::mbar_init(&sdp_full[u], 1);
      ptx::mbar_init(&pds_full[u], 4 * kCmpWG);
      ptx::mbar_init(&buf_free[u], 1);
    }
    ptx::mbar_init(acc_full, 1);
    ptx::mbar_init(acc_free, 4);
    ptx::fence_mbar_init();
  }
  if (warp == kLoadWarpB) {
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
  const int total_items = kv_item_count(p) * Cfg::kItems;
  // what the item with this index makes
  auto makes_dk = [](int idx) { return kMakes == 3 ? Cfg::kPasses == 1 || (idx & 1) == 0 : kMakes == 1; };
  auto makes_dv = [](int idx) { return kMakes == 3 ? Cfg::kPasses == 1 || (idx & 1) == 1 : kMakes == 2; };

  // Whole warpgroups: four of compute warps, one of the TMA warp, the two MMA warps and an idle warp. The fifth
  // hands registers to the other four. The counts are set inside the role branches, so that the compiler never
  // has to assume the smaller one where the branches meet.
  if (warp >= kEpiWarp0) {
    // ------------------------------------------------------------------------------------------------ epilogue
    // Four warps, one per quarter of the tensor-memory lanes: dK and dV of a finished item go out to global memory
    // while the other roles are already at work on the next item.
    ptx::reg_release_to<kDkdvEpilogueRegs>();
    const int quad = warp & 3;
    const int row = quad * 32 + lane;
    const uint32_t lane_addr = static_cast<uint32_t>(quad * 32) << 16;
    uint32_t n_item = 0;
    for (uint32_t n_sched = 0;; ++n_sched) {
      const int idx = sched_consume<true>(mbox, n_sched, abort_flag);
      if (idx < 0 || idx >= total_items) break;
      const KvItem it = decode_kv_item(p, idx / Cfg::kItems);
      if (!it.valid) continue;
      const int kj = it.k0 + row;
      const int rows_valid = imax(0, imin(32, it.n - (it.k0 + quad * 32)));  // of this warp's 32 key rows
      const int64_t srow = static_cast<int64_t>(it.row0) + it.kh * it.n + kj;
      uint16_t* dk_row = static_cast<uint16_t*>(p.dk) + it.bcoord * p.dk_bs + srow * p.dk_rs + it.hk * p.dk_hs;
      uint16_t* dv_row = static_cast<uint16_t*>(p.dv) + it.bcoord * p.dv_bs + srow * p.dv_rs + it.hk * p.dv_hs;
      if (!ptx::mbar_wait_warp(acc_full, n_item & 1, abort_flag, 62)) break;
      ++n_item;
      ptx::tc_fence_after();
      // dK and dV sit side by side in tensor memory (or the item makes one of them): chunks of 32 columns
      constexpr int kChunks = (Cfg::kPasses == 2 ? 1 : 2) * kHeadDim / 32;
#pragma unroll 1
      for (int gidx = 0; gidx < kChunks; ++gidx) {
        const bool is_dv = Cfg::kPasses == 2 ? makes_dv(idx) : gidx * 32 >= kHeadDim;
        const int col0 = gidx * 32 - (Cfg::kPasses == 1 && is_dv ? kHeadDim : 0);
        uint32_t accv[32];
        ptx::tmem_ld32(tmem + Cfg::kTmemDK + lane_addr + gidx * 32, accv);
        ptx::tmem_wait_ld();
        if (gidx == kChunks - 1) {
          // everything is in registers: the first dV / dK products of the next item may overwrite the accumulators
          ptx::tc_fence_before();
          ptx::mbar_arrive_warp(acc_free);
        }
        // Plain row stores: these four warps are in nobody's way, what counts is that the accumulators are free
        // again before the next item's first dV / dK product is due (a few thousand cycles).
        if (lane < rows_valid) {
          ptx::store_row32<kBf16>(is_dv ? dv_row : dk_row, col0, accv, is_dv ? 1.f : p.softmax_scale, p.head_dim,
                                  p.wide_store != 0);
        }
      }
    }
  } else if (warp >= 4 * kCmpWG) {
  ptx::reg_release_to<kDkdvProducerRegs>();
  if (warp == kLoadWarpB) {
    // ------------------------------------------------------------------------------------------------ producer
    if (lane == 0) {
      uint32_t n_item = 0, gc = 0;
      bool alive = true;
      for (uint32_t n_sched = 0; alive; ++n_sched) {
        const int idx = sched_produce(mbox, n_sched, p.ticket_kv, abort_flag);
        if (idx < 0 || idx >= total_items) break;
        const KvItem it = decode_kv_item(p, idx / Cfg::kItems);
        if (!it.valid) continue;
        const QueryPlan plan = make_query_plan(it.kh, it.k0, it.k1, it.n, bs, kTile);
        const KvSpans spans = make_kv_spans(it, bs);
        if (!ptx::mbar_wait(kv_empty, (n_item & 1) ^ 1, abort_flag, 41)) break;
        ptx::mbar_expect_tx(kv_full, (makes_dk(idx) ? 2 : 1) * T::kTileBytes);
        const int k_row = it.row0 + it.kh * it.n + it.k0;
        load_tile<kHeadDim>(sK, &p.tm_k, kv_full, k_row, it.hk, it.bcoord);
        if (makes_dk(idx)) load_tile<kHeadDim>(sV, &p.tm_v, kv_full, k_row, it.hk, it.bcoord);
        // The loader alone walks the item's geometry. Each sub-step carries a two-word header for the other roles:
        // {bit 0 last sub-step of the item, bit 1 partially masked, bit 2 queries of the keys' own half; first row}.
        // A sub-step is sent when its successor is known, so that the last one can be marked.
        auto emit = [&](const SubStep& st, bool last) -> bool {
          const uint32_t qs = gc % Cfg::kQSlots, ds = gc % Cfg::kDoSlots, ss = gc % Cfg::kStatSlots;
          if (!ptx::mbar_wait(&q_empty[qs], ((gc / Cfg::kQSlots) & 1) ^ 1, abort_flag, 42)) return false;
          uint8_t* stat = sStat + ss * Cfg::kStatBytes;
          volatile int* hdr = reinterpret_cast<volatile int*>(stat + Cfg::kHeaderOffset);
          hdr[0] = (last ? 1 : 0) | (st.cls == kTileMasked ? 2 : 0) | (st.qh == it.kh ? 4 : 0);
          hdr[1] = st.sa;
          ptx::mbar_expect_tx(&stat_full[ss], 2 * kSub * 4);
          const int64_t seg = stat_segment(p, it.b, st.h, st.qh) + st.sa;
          ptx::bulk_load_1d(stat, p.lse2_pad + seg, kSub * 4, &stat_full[ss]);
          ptx::bulk_load_1d(stat + kSub * 4, p.delta_pad + seg, kSub * 4, &stat_full[ss]);
          const int q_row = it.row0 + st.qh * it.n + st.sa;
          ptx::mbar_expect_tx(&q_full[qs], Cfg::kSubTileBytes);
#pragma unroll
          for (int c = 0; c < T::kPanels; ++c) {
            ptx::tma_load_4d(sQ + qs * Cfg::kSubTileBytes + c * Cfg::kSubPanelBytes, &p.tm_q64, &q_full[qs], c * 64, q_row,
                             st.h, it.bcoord);
          }
          if (!ptx::mbar_wait(&do_empty[ds], ((gc / Cfg::kDoSlots) & 1) ^ 1, abort_flag, 43)) return false;
          ptx::mbar_expect_tx(&do_full[ds], Cfg::kSubTileBytes);
#pragma unroll
          for (int c = 0; c < T::kPanels; ++c) {
            ptx::tma_load_4d(sDo + ds * Cfg::kSubTileBytes + c * Cfg::kSubPanelBytes, &p.tm_do64, &do_full[ds], c * 64,
                             q_row, st.h, it.bcoord);
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
        // every valid key tile is seen at least by the queries of its own rows, so there is a last sub-step
        if (alive && have) alive = emit(pend, true);
        ++n_item;
      }
      if (*abort_flag) __nanosleep(100000);
    }
  } else if (warp == kMmaWarpB) {
    // ------------------------------------------------------------------- MMA issuer 1: S^T = K Q^T, dP^T = V dO^T
    // Two warps issue the MMAs of this kernel, one elected lane of them: with the whole warp in waits and loop control the
    // descriptors and counters stay in uniform registers (a single thread in the loop moved them there for every MMA; both
    // kernels of this file, step of 2 x 8192 tokens, 8 heads of 256, 1810 -> 1705 us, of 4 x 4096 tokens, 32/8 heads of 128,
    // deterministic, 1925 -> 1790). The tensor pipe's queue is short, so whatever else an issuing warp does (barrier waits,
    // commits) leaves the pipe idle; with two issuers one's bookkeeping overlaps the
    // other's MMAs. Their only mutual dependency is the S^T / dP^T buffer: sub-step g may overwrite buffer g & 1
    // once dV / dK of sub-step g - 2 have read it (buf_free).
    {
      constexpr int kFmt = kBf16 ? 1 : 0;
      const uint32_t idesc_s = ptx::make_idesc(kTile, kSub, kFmt, false, false);
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
        const KvItem it = decode_kv_item(p, idx / Cfg::kItems);
        if (!it.valid) continue;
        if (!ptx::mbar_wait_warp(kv_full, n_item & 1, abort_flag, 51)) break;
        for (bool last = false; alive && !last; ++g) {
          const uint32_t u = g & 1u, qs = g % Cfg::kQSlots, ds = g % Cfg::kDoSlots, ss = g % Cfg::kStatSlots;
          if (!ptx::mbar_wait_warp(&stat_full[ss], (g / Cfg::kStatSlots) & 1u, abort_flag, 52)) { alive = false; break; }
          last = (ptx::uniform(*reinterpret_cast<const volatile int*>(sStat + ss * Cfg::kStatBytes + Cfg::kHeaderOffset)) & 1) != 0;
          if (!ptx::mbar_wait_warp(&q_full[qs], (g / Cfg::kQSlots) & 1u, abort_flag, 56)) { alive = false; break; }
          if (!ptx::mbar_wait_warp(&buf_free[u], ((g >> 1) & 1u) ^ 1u, abort_flag, 54)) { alive = false; break; }
          if (Cfg::kPasses == 1 &&
              !ptx::mbar_wait_warp(&do_full[ds], (g / Cfg::kDoSlots) & 1u, abort_flag, 58)) { alive = false; break; }
          ptx::tc_fence_after();
          const uint32_t q_off = qs * (Cfg::kSubTileBytes >> 4), do_off = ds * (Cfg::kSubTileBytes >> 4);
          auto product = [&](int kk, uint32_t d_off, uint32_t a_lo, uint32_t b_lo) {
            const uint32_t a_off = ((kk / 4) * T::kPanelBytes + (kk % 4) * 32) >> 4;
            const uint32_t b_off = ((kk / 4) * Cfg::kSubPanelBytes + (kk % 4) * 32) >> 4;
            ptx::umma_ss_f16_lh(tmem + u * 128 + d_off, a_lo + a_off, b_lo + b_off, kHi, idesc_s, kk > 0);
          };
          if (Cfg::kPasses == 1) {
            if (ptx::elect_one()) {
#pragma unroll
              for (int kk = 0; kk < kHeadDim / 16; ++kk) {
                product(kk, 0, k_lo, q_lo + q_off);
                product(kk, 64, v_lo, do_lo + do_off);
              }
            }
          } else {
            if (ptx::elect_one()) {
#pragma unroll
              for (int kk = 0; kk < kHeadDim / 16; ++kk) product(kk, 0, k_lo, q_lo + q_off);
            }
            if (makes_dk(idx)) {
              if (!ptx::mbar_wait_warp(&do_full[ds], (g / Cfg::kDoSlots) & 1u, abort_flag, 58)) { alive = false; break; }
              ptx::tc_fence_after();
              if (ptx::elect_one()) {
#pragma unroll
                for (int kk = 0; kk < kHeadDim / 16; ++kk) product(kk, 64, v_lo, do_lo + do_off);
                ptx::umma_commit(&do_empty[ds]);   // dK does not read dO
              }
            } else {
              if (ptx::elect_one()) ptx::umma_commit(&q_empty[qs]);    // dV does not read Q
            }
          }
          if (ptx::elect_one()) ptx::umma_commit(&sdp_full[u]);
        }
        // K and V are read by these products only: the next item's tiles may load while the last dV / dK products
        // and the epilogue of this item still run
        if (alive && ptx::elect_one()) ptx::umma_commit(kv_empty);
        ++n_item;
      }
    }
  } else if (warp == kMmaWarpB + 1) {
    // ------------------------------------------------------------------- MMA issuer 2: dV += P^T dO, dK += dS^T Q
    {
      constexpr int kFmt = kBf16 ? 1 : 0;
      const uint32_t idesc_g = ptx::make_idesc(kTile, kHeadDim, kFmt, false, true);
      constexpr uint32_t kHi = ptx::smem_desc_hi(1024);
      const uint32_t q_mn = ptx::smem_desc_lo(ptx::smem_u32(sQ), Cfg::kSubPanelBytes);    // MN-major use
      const uint32_t do_mn = ptx::smem_desc_lo(ptx::smem_u32(sDo), Cfg::kSubPanelBytes);
      uint32_t g = 0, n_item_b = 0;
      bool alive = true;
      for (uint32_t n_sched = 0; alive; ++n_sched) {
        const int idx = ptx::uniform(sched_consume<true>(mbox, n_sched, abort_flag));
        if (idx < 0 || idx >= total_items) break;
        const KvItem it = decode_kv_item(p, idx / Cfg::kItems);
        if (!it.valid) continue;
        bool acc = false;
        // the first products of an item overwrite the accumulators: the epilogue warps must have read the last item's
        if (!ptx::mbar_wait_warp(acc_free, (n_item_b & 1u) ^ 1u, abort_flag, 57)) break;
        ++n_item_b;
        for (bool last = false; alive && !last; ++g) {
          const uint32_t u = g & 1u, qs = g % Cfg::kQSlots, ds = g % Cfg::kDoSlots, ss = g % Cfg::kStatSlots;
          if (!ptx::mbar_wait_warp(&stat_full[ss], (g / Cfg::kStatSlots) & 1u, abort_flag, 55)) { alive = false; break; }
          last = (ptx::uniform(*reinterpret_cast<const volatile int*>(sStat + ss * Cfg::kStatBytes + Cfg::kHeaderOffset)) & 1) != 0;
          if (!ptx::mbar_wait_warp(&pds_full[u], (g >> 1) & 1u, abort_flag, 53)) { alive = false; break; }
          // The tiles this thread's products read. Most have landed long ago, but nothing it has waited for so far says so:
          // that the other issuer saw them land reaches this thread only through its products and the compute warps.
          if (makes_dk(idx) &&
              !ptx::mbar_wait_warp(&q_full[qs], (g / Cfg::kQSlots) & 1u, abort_flag, 64)) { alive = false; break; }
          if (makes_dv(idx) &&
              !ptx::mbar_wait_warp(&do_full[ds], (g / Cfg::kDoSlots) & 1u, abort_flag, 59)) { alive = false; break; }
          ptx::tc_fence_after();
          const uint32_t q_off = qs * (Cfg::kSubTileBytes >> 4), do_off = ds * (Cfg::kSubTileBytes >> 4);
          const uint32_t st_t = tmem + u * 128, dpt_t = tmem + u * 128 + 64;
          if (ptx::elect_one()) {
#pragma unroll
            for (int kk = 0; kk < kSub / 16; ++kk) {
              const uint32_t on = (acc || kk > 0) ? 1u : 0u;
              if (makes_dv(idx)) {
                ptx::umma_ts_f16_lh(tmem + Cfg::kTmemDV, st_t + kk * kSubCols, do_mn + do_off + kk * (2048 >> 4), kHi, idesc_g, on);
              }
              if (makes_dk(idx)) {
                ptx::umma_ts_f16_lh(tmem + Cfg::kTmemDK, dpt_t + kk * kSubCols, q_mn + q_off + kk * (2048 >> 4), kHi, idesc_g, on);
              }
            }
            ptx::umma_commit(&buf_free[u]);
            if (makes_dk(idx)) ptx::umma_commit(&q_empty[qs]);
            if (makes_dv(idx)) ptx::umma_commit(&do_empty[ds]);
          }
          acc = true;
        }
        if (!alive) break;
        if (ptx::elect_one()) ptx::umma_commit(acc_full);
      }
    }
  }
  } else {
    ptx::reg_acquire_to<kDkdvComputeRegs>();
    // -------------------------------------------------------------------------------------- softmax backward
    const int wg = warp >> 2;                  // which kSubCols query columns of a sub-tile
    const int quad = warp & 3;
    const int row = quad * 32 + lane;          // key row inside the tile
    const uint32_t lane_addr = static_cast<uint32_t>(quad * 32) << 16;
    uint32_t n_item = 0, gc = 0;
    bool alive = true;
    for (uint32_t n_sched = 0; alive; ++n_sched) {
      const int idx = sched_consume<true>(mbox, n_sched, abort_flag);
      if (idx < 0 || idx >= total_items) break;
      const KvItem it = decode_kv_item(p, idx / Cfg::kItems);
      if (!it.valid) continue;
      const int kj = it.k0 + row;
      // queries that see this thread's key: same-half tiles and (clean keys only) noisy tiles of later blocks
      int same_lo, same_hi, cross_lo, cross_hi;
      query_interval(it.kh, it.kh, kj, it.n, bs, same_lo, same_hi);
      query_interval(0, 1, kj, it.n, bs, cross_lo, cross_hi);
      for (bool last = false; alive && !last;) {
        const uint32_t u = gc & 1u, ss = gc % Cfg::kStatSlots;
        const uint8_t* stage_base = sStat + ss * Cfg::kStatBytes;
        const float* stats = reinterpret_cast<const float*>(stage_base);
        // orders the header and the bulk copies of lse2 / delta before our reads
        if (!ptx::mbar_wait_warp(&stat_full[ss], (gc / Cfg::kStatSlots) & 1u, abort_flag, 60)) { alive = false; break; }
        int2 hdr;
        hdr.x = reinterpret_cast<const volatile int*>(stage_base + Cfg::kHeaderOffset)[0];
        hdr.y = reinterpret_cast<const volatile int*>(stage_base + Cfg::kHeaderOffset)[1];
        last = (hdr.x & 1) != 0;
        // The per-column statistics of this warp's 16 query columns come into registers now, as four 16-byte loads
        // each, while the S^T / dP^T products are still running: scalar loads inside the arithmetic below queue
        // up behind the operand fetches of the MMAs, which keep the shared-memory pipe busy.
        float l2r[kSubCols], dlr[kSubCols];
        {
          const float4* l2v = reinterpret_cast<const float4*>(stats + wg * kSubCols);
          const float4* dlv = reinterpret_cast<const float4*>(stats + kSub + wg * kSubCols);
#pragma unroll
          for (int i = 0; i < kSubCols / 4; ++i) {
            const float4 a = l2v[i], b = dlv[i];
            l2r[4 * i] = a.x; l2r[4 * i + 1] = a.y; l2r[4 * i + 2] = a.z; l2r[4 * i + 3] = a.w;
            dlr[4 * i] = b.x; dlr[4 * i + 1] = b.y; dlr[4 * i + 2] = b.z; dlr[4 * i + 3] = b.w;
          }
        }
        if (!ptx::mbar_wait_warp(&sdp_full[u], (gc >> 1) & 1u, abort_flag, 61)) { alive = false; break; }
        ++gc;
        ptx::tc_fence_after();
        const uint32_t st_t = tmem + u * 128 + lane_addr + wg * kSubCols;
        const uint32_t dpt_t = st_t + 64;
        uint32_t sv[kSubCols], dpv[kSubCols];
        const bool masked = (hdr.x & 2) != 0;
        const int lo = ((hdr.x & 4) ? same_lo : cross_lo) - (hdr.y + wg * kSubCols);
        const int hi = ((hdr.x & 4) ? same_hi : cross_hi) - (hdr.y + wg * kSubCols);
        uint32_t pk_p[kSubCols / 2], pk_ds[kSubCols / 2];
        auto turn = [&](auto p_tag, auto ds_tag) {
          constexpr bool kP = decltype(p_tag)::value, kDs = decltype(ds_tag)::value;
          ptx::tmem_ld16(st_t, sv);
          if (kDs) ptx::tmem_ld16(dpt_t, dpv);
          ptx::tmem_wait_ld();
          if (masked) {
            softmax_backward_cols<kSubCols, kBf16, kSoftcap, true, true, kP, kDs>(sv, dpv, l2r, dlr, 0.f, 0.f, p.scale_log2,
                                                                                  p.softcap_pre, lo, hi, pk_p, pk_ds);
          } else {
            softmax_backward_cols<kSubCols, kBf16, kSoftcap, true, false, kP, kDs>(sv, dpv, l2r, dlr, 0.f, 0.f, p.scale_log2,
                                                                                   p.softcap_pre, 0, 0, pk_p, pk_ds);
          }
          // a warp overwrites only columns it has itself already loaded: its packed P^T / dS^T pieces go to the
          // start of its own kSubCols columns
          if (kP) ptx::tmem_st8(st_t, pk_p);
          if (kDs) ptx::tmem_st8(dpt_t, pk_ds);
        };
        if (Cfg::kPasses == 1) turn(std::true_type{}, std::true_type{});
        else if (makes_dk(idx)) turn(std::false_type{}, std::true_type{});
        else turn(std::true_type{}, std::false_type{});
        ptx::tmem_wait_st();
        ptx::tc_fence_before();
        ptx::mbar_arrive_warp(&pds_full[u]);
      }
      if (!alive) break;
      ++n_item;
    }
  }
  ptx::tc_fence_before();
  __syncthreads();
  if (warp == kLoadWarpB) ptx::tmem_dealloc(tmem, 512);
}

// ------------------------------------------------------------------------------------------------------------
// 3. dQ
// ------------------------------------------------------------------------------------------------------------
struct QItem {
  int b, h, hk, qh, qa, qb, n, row0, bcoord;
  bool valid;
};

__device__ __forceinline__ QItem decode_q_item(const BwdParams& p, int idx) {
  // (sample, head)-major for L2 reuse of K / V; inside a head late query tiles first (they see the most keys).
  QItem it;
  int rem, tiles;
  if (p.vl.base != nullptr) {
    // packed batch: exactly the query tiles that exist, longest sample first, head after head inside a sample
    const VarlenPos pos = varlen_locate(p.vl, idx, 2 * p.heads);
    tiles = pos.units;
    it.b = pos.b;
    it.h = pos.rem / (2 * tiles);
    rem = pos.rem - it.h * (2 * tiles);
  } else {
    const int per_bh = 2 * p.tiles_per_half;
    int bh;
    two_phase_order(idx, per_bh, p.n_long_q, p.batch * p.heads, bh, rem);
    tiles = p.tiles_per_half;
    it.b = bh / p.heads;
    it.h = bh - it.b * p.heads;
  }
  it.qh = rem & 1;
  const int t_rev = rem >> 1;
  it.hk = it.h / (p.heads / p.heads_k);
  const Sample sm = sample_of(p, it.b);
  it.n = sm.n;
  it.row0 = sm.row0;
  it.bcoord = sm.bcoord;
  it.qa = (tiles - 1 - t_rev) * kTile;
  it.valid = it.qa < it.n;
  it.qb = imin(it.qa + kTile, it.n);
  return it;
}

struct QSpans {
  Span half[2];  // key spans of the query tile per key half (0 noisy, 1 clean)
  // selects instead of half[kh]: a run-time index would put the spans in local memory
  __device__ __forceinline__ int classify(int kh, int k0, int keys) const {
    Span s;
    s.lo_first = kh ? half[1].lo_first : half[0].lo_first;
    s.hi_first = kh ? half[1].hi_first : half[0].hi_first;
    s.lo_last = kh ? half[1].lo_last : half[0].lo_last;
    s.hi_last = kh ? half[1].hi_last : half[0].hi_last;
    return s.classify(k0, keys);
  }
};

__device__ __forceinline__ QSpans make_q_spans(const QItem& it, int bs) {
  QSpans sp;
  sp.half[0] = key_span(it.qh, 0, it.qa, it.qb, it.n, bs);
  sp.half[1] = key_span(it.qh, 1, it.qa, it.qb, it.n, bs);
  return sp;
}

template <int kHeadDim, int kStages>
struct DqCfg {
  using T = TileCfg<kHeadDim>;
  // keys per step: 128, or 64 for head dimensions above 128 (Q and dO alone take 128 KB of shared memory there)
  static constexpr int kKeys = kHeadDim > 128 ? 64 : 128;
  static constexpr int kKeyCols = kKeys / kCmpWG;               // key columns per compute warpgroup
  static constexpr int kKvTileBytes = kKeys * kHeadDim * 2;
  static constexpr int kKvPanelBytes = kKeys * 128;
  static constexpr int kSmemBytes = 2 * T::kTileBytes + kStages * kKvTileBytes + 1024 + 512;
  static constexpr int kKSlots = (kStages + 1) / 2;  // K ring; the rest is the V ring
  static constexpr int kVSlots = kStages - kKSlots;
  static_assert(kVSlots >= 1 && kKSlots >= 2, "ring depth");
  __host__ __device__ static constexpr uint32_t k_slot(uint32_t step) { return step % kKSlots; }
  __host__ __device__ static constexpr uint32_t v_slot(uint32_t step) { return kKSlots + step % kVSlots; }
  __host__ __device__ static constexpr uint32_t k_parity(uint32_t step) { return (step / kKSlots) & 1u; }
  __host__ __device__ static constexpr uint32_t v_parity(uint32_t step) { return (step / kVSlots) & 1u; }
  static constexpr int kTmemS = 0, kTmemDP = kKeys, kTmemDS = 2 * kKeys, kTmemDQ = kHeadDim > 128 ? 256 : 384;
  static_assert(kTmemDQ + kHeadDim <= 512 && 2 * kKeys + kKeys / 2 <= kTmemDQ, "tensor memory budget");
};

template <int kHeadDim, int kStages, bool kBf16, bool kSoftcap>
__global__ void __launch_bounds__(kBwdThreads, 1) bwd_dq_kernel(const __grid_constant__ BwdParams p) {
  using Cfg = DqCfg<kHeadDim, kStages>;
  using T = TileCfg<kHeadDim>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sQ = smem;
  uint8_t* sdO = smem + T::kTileBytes;
  uint8_t* sKV = smem + 2 * T::kTileBytes;
  uint64_t* bars = reinterpret_cast<uint64_t*>(sKV + kStages * Cfg::kKvTileBytes);
  uint64_t* q_full = bars;
  uint64_t* q_empty = bars + 1;
  uint64_t* kv_full = bars + 2;
  uint64_t* kv_empty = kv_full + kStages;
  uint64_t* sdp_full = kv_empty + kStages;
  uint64_t* sdp_free = sdp_full + 1;
  uint64_t* ds_full = sdp_free + 1;
  uint64_t* ds_free = ds_full + 1;
  uint64_t* dq_full = ds_free + 1;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(dq_full + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  SchedMailbox* mbox = reinterpret_cast<SchedMailbox*>(reinterpret_cast<uint8_t*>(bars) + 256);

  const int warp = ptx::uniform(static_cast<int>(threadIdx.x >> 5)), lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    *abort_flag = 0;
    sched_init(mbox, 4 * kCmpWG + 2);
    ptx::mbar_init(q_full, 1);
    ptx::mbar_init(q_empty, 1);
    for (int i = 0; i < kStages; ++i) {
      ptx::mbar_init(&kv_full[i], 1);
      ptx::mbar_init(&kv_empty[i], 1);
    }
    ptx::mbar_init(sdp_full, 1);
    ptx::mbar_init(sdp_free, 4 * kCmpWG);
    ptx::mbar_init(ds_full, 4 * kCmpWG);
    ptx::mbar_init(ds_free, 1);
    ptx::mbar_init(dq_full, 1);
    ptx::fence_mbar_init();
  }
  if (warp == kLoadWarpB) {
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
  const int total_items = (p.vl.base != nullptr ? p.vl.base[0] : p.tiles_per_half * p.batch) * 2 * p.heads;

  // Whole warpgroups: four of compute warps, one of the TMA warp, the two MMA warps and an idle warp. The fifth
  // hands registers to the other four. The counts are set inside the role branches, so that the compiler never
  // has to assume the smaller one where the branches meet.
  if (warp >= 4 * kCmpWG) {
  ptx::reg_release_to<kProducerRegs>();
  if (warp == kLoadWarpB) {
    if (lane == 0) {
      uint32_t n_item = 0, slot = 0;
      bool alive = true;
      for (uint32_t n_sched = 0; alive; ++n_sched) {
        const int idx = sched_produce(mbox, n_sched, p.ticket_q, abort_flag);
        if (idx < 0 || idx >= total_items) break;
        const QItem it = decode_q_item(p, idx);
        if (!it.valid) continue;
        const KeyPlan plan = make_key_plan(it.qh, it.qa, it.qb, it.n, bs, Cfg::kKeys);
        const QSpans spans = make_q_spans(it, bs);
        if (!ptx::mbar_wait(q_empty, (n_item & 1) ^ 1, abort_flag, 71)) break;
        ptx::mbar_expect_tx(q_full, 2 * T::kTileBytes);
        const int q_row = it.row0 + it.qh * it.n + it.qa;
        load_tile<kHeadDim>(sQ, &p.tm_q, q_full, q_row, it.h, it.bcoord);
        load_tile<kHeadDim>(sdO, &p.tm_do, q_full, q_row, it.h, it.bcoord);
        for (int s = 0; s < plan.steps() && alive; ++s) {
          int kh, kt;
          plan.step(s, kh, kt);
          if (spans.classify(kh, kt * Cfg::kKeys, Cfg::kKeys) == kTileSkip) continue;
          const int k_row = it.row0 + kh * it.n + kt * Cfg::kKeys;
          // K tiles cycle through slots [0, kKSlots), V tiles through [kKSlots, kStages): a K tile is held until
          // the dQ product of its step, a V tile only until dP, so they need rings of different depth
          for (int which = 0; which < 2; ++which) {
            const uint32_t stage = which == 0 ? Cfg::k_slot(slot) : Cfg::v_slot(slot);
            const uint32_t par = which == 0 ? Cfg::k_parity(slot) : Cfg::v_parity(slot);
            if (!ptx::mbar_wait(&kv_empty[stage], par ^ 1, abort_flag, 72)) { alive = false; break; }
            ptx::mbar_expect_tx(&kv_full[stage], Cfg::kKvTileBytes);
            const CUtensorMap* tm = Cfg::kKeys == 128 ? (which == 0 ? &p.tm_k : &p.tm_v)
                                                      : (which == 0 ? &p.tm_k64 : &p.tm_v64);
#pragma unroll
            for (int c = 0; c < T::kPanels; ++c) {
              ptx::tma_load_4d(sKV + stage * Cfg::kKvTileBytes + c * Cfg::kKvPanelBytes, tm, &kv_full[stage], c * 64,
                               k_row, it.hk, it.bcoord);
            }
          }
          ++slot;
        }
        ++n_item;
      }
      if (*abort_flag) __nanosleep(100000);
    }
  } else if (warp == kMmaWarpB) {
    // ------------------------------------------------------------------ MMA issuer 1: S = Q K^T and dP = dO V^T
    // As in the dK/dV kernel two warps issue MMAs, so that the barrier waits of one overlap the MMAs of the
    // other. They share nothing but the compute warps between them: S / dP of step j + 1 may start as soon as the
    // compute warps have S / dP of step j in registers, whatever the state of dQ.
    {
      constexpr int kFmt = kBf16 ? 1 : 0;
      const uint32_t idesc_s = ptx::make_idesc(kTile, Cfg::kKeys, kFmt, false, false);
      constexpr uint32_t kHi = ptx::smem_desc_hi(1024);
      const uint32_t q_lo = ptx::smem_desc_lo(ptx::smem_u32(sQ), 16);
      const uint32_t do_lo = ptx::smem_desc_lo(ptx::smem_u32(sdO), 16);
      const uint32_t kv_lo_k = ptx::smem_desc_lo(ptx::smem_u32(sKV), 16);
      uint32_t n_item = 0, step = 0;
      bool alive = true;
      for (uint32_t n_sched = 0; alive; ++n_sched) {
        const int idx = ptx::uniform(sched_consume<true>(mbox, n_sched, abort_flag));
        if (idx < 0 || idx >= total_items) break;
        const QItem it = decode_q_item(p, idx);
        if (!it.valid) continue;
        const KeyPlan plan = make_key_plan(it.qh, it.qa, it.qb, it.n, bs, Cfg::kKeys);
        const QSpans spans = make_q_spans(it, bs);
        int active = 0;
        for (int s = 0; s < plan.steps(); ++s) {
          int kh, kt;
          plan.step(s, kh, kt);
          active += spans.classify(kh, kt * Cfg::kKeys, Cfg::kKeys) != kTileSkip;
        }
        if (!ptx::mbar_wait_warp(q_full, n_item & 1, abort_flag, 81)) break;
        ++n_item;
        for (int j = 0; j < active; ++j, ++step) {
          const uint32_t ks = Cfg::k_slot(step), vs = Cfg::v_slot(step);
          if (!ptx::mbar_wait_warp(&kv_full[ks], Cfg::k_parity(step), abort_flag, 83)) { alive = false; break; }
          if (!ptx::mbar_wait_warp(&kv_full[vs], Cfg::v_parity(step), abort_flag, 84)) { alive = false; break; }
          if (!ptx::mbar_wait_warp(sdp_free, (step & 1) ^ 1, abort_flag, 82)) { alive = false; break; }
          ptx::tc_fence_after();
          if (ptx::elect_one()) {
#pragma unroll
            for (int kk = 0; kk < kHeadDim / 16; ++kk) {
              const uint32_t a_off = ((kk / 4) * T::kPanelBytes + (kk % 4) * 32) >> 4;
              const uint32_t b_off = ((kk / 4) * Cfg::kKvPanelBytes + (kk % 4) * 32) >> 4;
              ptx::umma_ss_f16_lh(tmem + Cfg::kTmemS, q_lo + a_off, kv_lo_k + ks * (Cfg::kKvTileBytes >> 4) + b_off, kHi,
                                  idesc_s, kk > 0);
              ptx::umma_ss_f16_lh(tmem + Cfg::kTmemDP, do_lo + a_off, kv_lo_k + vs * (Cfg::kKvTileBytes >> 4) + b_off, kHi,
                                  idesc_s, kk > 0);
            }
            ptx::umma_commit(sdp_full);
            ptx::umma_commit(&kv_empty[vs]);  // V tile no longer needed
          }
        }
        // Q and dO are read by these products only: the tiles of the next item may load while the last dQ
        // product and the epilogue of this one still run
        if (alive && ptx::elect_one()) ptx::umma_commit(q_empty);
      }
    }
  } else if (warp == kMmaWarpB + 1) {
    // ------------------------------------------------------------------------------ MMA issuer 2: dQ += dS K
    {
      constexpr int kFmt = kBf16 ? 1 : 0;
      const uint32_t idesc_g = ptx::make_idesc(kTile, kHeadDim, kFmt, false, true);
      constexpr uint32_t kHi = ptx::smem_desc_hi(1024);
      const uint32_t kv_lo_mn = ptx::smem_desc_lo(ptx::smem_u32(sKV), Cfg::kKvPanelBytes);
      uint32_t step = 0;
      bool alive = true;
      for (uint32_t n_sched = 0; alive; ++n_sched) {
        const int idx = ptx::uniform(sched_consume<true>(mbox, n_sched, abort_flag));
        if (idx < 0 || idx >= total_items) break;
        const QItem it = decode_q_item(p, idx);
        if (!it.valid) continue;
        const KeyPlan plan = make_key_plan(it.qh, it.qa, it.qb, it.n, bs, Cfg::kKeys);
        const QSpans spans = make_q_spans(it, bs);
        int active = 0;
        for (int s = 0; s < plan.steps(); ++s) {
          int kh, kt;
          plan.step(s, kh, kt);
          active += spans.classify(kh, kt * Cfg::kKeys, Cfg::kKeys) != kTileSkip;
        }
        for (int j = 0; j < active; ++j, ++step) {
          const uint32_t ks = Cfg::k_slot(step);
          // the K tile arrived long ago (S of this step used it); this wait only orders our reads after the copy
          if (!ptx::mbar_wait_warp(&kv_full[ks], Cfg::k_parity(step), abort_flag, 86)) { alive = false; break; }
          if (!ptx::mbar_wait_warp(ds_full, step & 1, abort_flag, 85)) { alive = false; break; }
          ptx::tc_fence_after();
          // dQ += dS K: the packed dS pieces of the compute warpgroups lie side by side, 8 columns per 16 keys
          if (ptx::elect_one()) {
#pragma unroll
            for (int kk = 0; kk < Cfg::kKeys / 16; ++kk) {
              ptx::umma_ts_f16_lh(tmem + Cfg::kTmemDQ, tmem + Cfg::kTmemDS + kk * 8,
                                  kv_lo_mn + ks * (Cfg::kKvTileBytes >> 4) + kk * (2048 >> 4), kHi, idesc_g,
                                  (j > 0 || kk > 0) ? 1u : 0u);
            }
            ptx::umma_commit(&kv_empty[ks]);
            ptx::umma_commit(ds_free);
          }
        }
        if (!alive) break;
        if (ptx::elect_one()) ptx::umma_commit(dq_full);
      }
    }
  }
  } else {
    ptx::reg_acquire_to<kComputeRegs>();
    const int wg = warp >> 2;                  // which kCols key columns
    const int quad = warp & 3;
    const int row = quad * 32 + lane;          // query row inside the tile
    const uint32_t lane_addr = static_cast<uint32_t>(quad * 32) << 16;
    uint32_t n_item = 0, cnt = 0, n_sched = 0;
    bool alive = true;

    // What a compute thread keeps of an item. The next item's record is filled while the last dQ product of the
    // current one is still in the tensor pipe, so that its decode and its two statistics loads cost nothing. Two
    // records alternate (no copies: they are meant to stay in registers).
    struct ItemState {
      KeyPlan plan;
      QSpans spans;
      int qh, blk0, blk1;
      int rows_valid;   // of this warp's 32 query rows
      float lse2, delta;
      uint16_t* dst;   // this thread's dQ row
    };
    auto fetch = [&](ItemState& t) -> bool {   // false: no more work (or a wait was abandoned)
      for (;;) {
        const int idx = sched_consume<true>(mbox, n_sched, abort_flag);
        ++n_sched;
        if (idx < 0) alive = false;   // no wait may follow one that was abandoned
        if (idx < 0 || idx >= total_items) return false;
        const QItem it = decode_q_item(p, idx);
        if (!it.valid) continue;
        t.plan = make_key_plan(it.qh, it.qa, it.qb, it.n, bs, Cfg::kKeys);
        t.spans = make_q_spans(it, bs);
        t.qh = it.qh;
        const int r = it.qa + row;
        t.rows_valid = imax(0, imin(32, it.n - (it.qa + quad * 32)));
        const int r_eff = r < it.n ? r : it.n - 1;
        t.blk0 = block_lo(r_eff, bs);
        t.blk1 = imin(t.blk0 + bs, it.n);
        const int64_t seg = stat_segment(p, it.b, it.h, it.qh);
        t.lse2 = p.lse2_pad[seg + r];
        t.delta = p.delta_pad[seg + r];
        const int64_t srow = static_cast<int64_t>(it.row0) + it.qh * it.n + r;
        t.dst = static_cast<uint16_t*>(p.dq) + it.bcoord * p.dq_bs + srow * p.dq_rs + it.h * p.dq_hs;
        return true;
      }
    };

    // One item: its steps, then the next item's record, then the epilogue. Returns whether `nxt` holds an item.
    auto run_item = [&](const ItemState& cur, ItemState& nxt) -> bool {
      for (int s = 0; s < cur.plan.steps() && alive; ++s) {
        int kh, kt;
        cur.plan.step(s, kh, kt);
        constexpr int kKc = Cfg::kKeyCols;
        const int cls = cur.spans.classify(kh, kt * Cfg::kKeys, Cfg::kKeys);
        if (cls == kTileSkip) continue;
        int lo = 0, hi = 0;
        if (cls == kTileMasked) {
          if (cur.qh == 1) { lo = 0; hi = cur.blk1; }
          else if (kh == 1) { lo = 0; hi = cur.blk0; }
          else { lo = cur.blk0; hi = cur.blk1; }
          lo -= kt * Cfg::kKeys + wg * kKc;
          hi -= kt * Cfg::kKeys + wg * kKc;
        }
        if (!ptx::mbar_wait_warp(sdp_full, cnt & 1, abort_flag, 91)) { alive = false; break; }
        ptx::tc_fence_after();
        uint32_t sv[kKc], dpv[kKc];
        if (kKc == 32) {
          ptx::tmem_ld32(tmem + Cfg::kTmemS + lane_addr + wg * kKc, sv);
          ptx::tmem_ld32(tmem + Cfg::kTmemDP + lane_addr + wg * kKc, dpv);
        } else {
          ptx::tmem_ld16(tmem + Cfg::kTmemS + lane_addr + wg * kKc, sv);
          ptx::tmem_ld16(tmem + Cfg::kTmemDP + lane_addr + wg * kKc, dpv);
        }
        ptx::tmem_wait_ld();
        ptx::tc_fence_before();
        ptx::mbar_arrive_warp(sdp_free);
        uint32_t pk_ds[kKc / 2];
        if (cls == kTileMasked) {
          softmax_backward_cols<kKc, kBf16, kSoftcap, false, true, false>(sv, dpv, nullptr, nullptr, cur.lse2, cur.delta,
                                                                          p.scale_log2, p.softcap_pre, lo, hi, nullptr, pk_ds);
        } else {
          softmax_backward_cols<kKc, kBf16, kSoftcap, false, false, false>(sv, dpv, nullptr, nullptr, cur.lse2, cur.delta,
                                                                           p.scale_log2, p.softcap_pre, 0, 0, nullptr, pk_ds);
        }
        if (!ptx::mbar_wait_warp(ds_free, (cnt & 1) ^ 1, abort_flag, 92)) { alive = false; break; }
        ++cnt;
        ptx::tc_fence_after();
        if (kKc == 32) ptx::tmem_st16(tmem + Cfg::kTmemDS + lane_addr + wg * (kKc / 2), pk_ds);
        else ptx::tmem_st8(tmem + Cfg::kTmemDS + lane_addr + wg * (kKc / 2), pk_ds);
        ptx::tmem_wait_st();
        ptx::tc_fence_before();
        ptx::mbar_arrive_warp(ds_full);
      }
      if (!alive) return false;
      const bool have_next = fetch(nxt);
      if (!alive) return false;
      if (!ptx::mbar_wait_warp(dq_full, n_item & 1, abort_flag, 93)) { alive = false; return false; }
      ++n_item;
      ptx::tc_fence_after();
      constexpr int kChunks = kHeadDim / 32;  // 32-column chunks, dealt round-robin to the warpgroups
#pragma unroll
      for (int g0 = 0; g0 < kChunks; g0 += kCmpWG) {
        const int gidx = g0 + wg;
        if (gidx < kChunks) {
          uint32_t acc[32];
          ptx::tmem_ld32(tmem + Cfg::kTmemDQ + lane_addr + gidx * 32, acc);
          ptx::tmem_wait_ld();
          ptx::store_rows32_grouped<kBf16>(cur.dst, p.dq_rs, cur.rows_valid, gidx * 32, acc, p.softmax_scale, p.head_dim);
        }
      }
      ptx::tc_fence_before();
      return have_next;
    };

    ItemState st0, st1;
    bool have = fetch(st0);
    while (have && alive) {
      have = run_item(st0, st1);
      if (!have || !alive) break;
      have = run_item(st1, st0);
    }
  }
  ptx::tc_fence_before();
  __syncthreads();
  if (warp == kLoadWarpB) ptx::tmem_dealloc(tmem, 512);
}

template <int kHeadDim, int kStages, bool kBf16, bool kSoftcap, int kMakes>
int launch_dkdv(const BwdParams& p, int sm_count, cudaStream_t stream) {
  using Cfg = DkdvCfg<kHeadDim, kStages, kMakes>;
  auto kernel = bwd_dkdv_kernel<kHeadDim, kStages, kBf16, kSoftcap, kMakes>;
  static PerDeviceFlags smem_set;
  const int rc = set_dynamic_smem(kernel, Cfg::kSmemBytes, smem_set);
  if (rc) return rc;
  const int items = bwd_item_bound(p, p.heads_k) * Cfg::kItems;
  const int grid = items < sm_count ? items : sm_count;
  return launch_kernel(p.overlap != 0, kernel, grid, Cfg::kThreads, Cfg::kSmemBytes, stream, p);
}

template <int kHeadDim, int kStagesKv, int kStagesQ, bool kBf16, bool kSoftcap>
int launch_bwd_instance(const BwdParams& p, int sm_count, unsigned stages, cudaStream_t stream) {
  if (stages & 2u) {
    int rc;
    if constexpr (kHeadDim > 128) {
      if (p.apart) {
        rc = launch_dkdv<kHeadDim, kStagesKv, kBf16, kSoftcap, 2>(p, sm_count, stream);
        if (rc == FDA_OK) {
          BwdParams q = p;
          q.ticket_kv = p.ticket_kv + 16;   // a counter of its own
          rc = launch_dkdv<kHeadDim, kStagesKv, kBf16, kSoftcap, 1>(q, sm_count, stream);
        }
      } else {
        rc = launch_dkdv<kHeadDim, kStagesKv, kBf16, kSoftcap, 3>(p, sm_count, stream);
      }
    } else {
      rc = launch_dkdv<kHeadDim, kStagesKv, kBf16, kSoftcap, 3>(p, sm_count, stream);
    }
    if (rc) return rc;
  }
  if (stages & 4u) {
    using Cfg = DqCfg<kHeadDim, kStagesQ>;
    auto kernel = bwd_dq_kernel<kHeadDim, kStagesQ, kBf16, kSoftcap>;
    static PerDeviceFlags smem_set;
    int rc = set_dynamic_smem(kernel, Cfg::kSmemBytes, smem_set);
    if (rc) return rc;
    const int items = bwd_item_bound(p, p.heads);
    const int grid = items < sm_count ? items : sm_count;
    return launch_kernel(p.overlap != 0, kernel, grid, kBwdThreads, Cfg::kSmemBytes, stream, p);
  }
  return FDA_OK;
}

template <int kHeadDim, int kStagesKv, int kStagesQ>
int dispatch_bwd(const BwdParams& p, int sm_count, bool bf16, bool softcap, unsigned stages, cudaStream_t stream) {
  if (bf16) {
    return softcap ? launch_bwd_instance<kHeadDim, kStagesKv, kStagesQ, true, true>(p, sm_count, stages, stream)
                   : launch_bwd_instance<kHeadDim, kStagesKv, kStagesQ, true, false>(p, sm_count, stages, stream);
  }
  return softcap ? launch_bwd_instance<kHeadDim, kStagesKv, kStagesQ, false, true>(p, sm_count, stages, stream)
                 : launch_bwd_instance<kHeadDim, kStagesKv, kStagesQ, false, false>(p, sm_count, stages, stream);
}

inline int64_t round_up64(int64_t x, int64_t m) { return (x + m - 1) / m * m; }

}  // namespace

// bwd_fused_sm100.cu
bool bwd_chains_fit(const FdaProblem& pr, int tokens);
size_t bwd_fused_acc_bytes(const FdaProblem& pr);
int64_t bwd_fused_acc_tiles(const FdaProblem& pr);
int bwd_fused_kv_split(const FdaProblem& pr);
size_t bwd_fused_part_bytes(const FdaProblem& pr);
int launch_bwd_fused(const BwdParams& p, int d_round, bool bf16, bool softcap, int sm_count, unsigned stages,
                     cudaStream_t stream);

constexpr int64_t kSmallAccBytes = 32 << 20;

// The single-pass backward adds dQ partials in an order that depends on scheduling and needs head dim <= 128.
bool bwd_single_pass(const FdaProblem& pr) { return pr.deterministic == 0 && pr.head_dim <= 128; }

// Heads wider than 128, split form: dV items in a launch of their own have three dO slots, at the price of a second
// tail and of items that cannot fill each other's gaps. Backward, together / apart, us, heads of 256: 16 x 2000 tokens,
// 8 heads, blocks of 16 820 / 789, 16/8 heads, blocks of 512 1844 / 1721; 4 x 4096, 8 heads 679 / 641, 1 x 16384 2173 /
// 2000. Short ones and those whose longest chain is more than a CTA's share stay together (32 x 512 tokens 246 / 264; 1
// x 16384, 8/2 heads 2360 / 3140).
bool bwd_dv_apart(const FdaProblem& pr) { return pr.head_dim > 128 && bwd_chains_fit(pr, 700); }

// The items that count for overlapped_launches, by what the host knows of the lengths.
bool bwd_overlaps(const FdaProblem& pr, bool single_pass) {
  int64_t items = 0;
  if (single_pass && pr.head_dim > 64) {
    const int64_t tiles = pr.cu_seqlens == nullptr ? (pr.seqlen / 2 + kTile - 1) / kTile * static_cast<int64_t>(pr.batch)
                                                   : pr.total / (2 * kTile) + pr.batch;
    items = tiles * 2 * pr.heads_k * bwd_fused_kv_split(pr);
  }
  return overlapped_launches(pr, items);
}

// Scratch of the split backward: delta_pad then lse2_pad, each batch * heads * 2 * n_pad floats (256-byte aligned
// pieces), then 256 bytes of work counters.
size_t bwd_split_workspace_bytes(const FdaProblem& pr) {
  const int64_t n_pad = round_up64(pr.seqlen / 2 > 0 ? pr.seqlen / 2 : 1, kTile);
  const int64_t one = round_up64(static_cast<int64_t>(pr.batch) * pr.heads * 2 * n_pad * 4, 256);
  // ... and for packed batches the work list (samples longest first, running tile counts)
  return static_cast<size_t>(2 * one + 256) + (pr.cu_seqlens != nullptr ? varlen_list_bytes(pr.batch) : 0);
}

// The single-pass backward keeps its fp32 dQ accumulator behind that, and behind it parts of dK and dV where it makes some.
size_t bwd_workspace_bytes(const FdaProblem& pr) {
  size_t bytes = bwd_split_workspace_bytes(pr);
  if (bwd_single_pass(pr)) {
    bytes += static_cast<size_t>(round_up64(static_cast<int64_t>(bwd_fused_acc_bytes(pr)), 256)) + bwd_fused_part_bytes(pr);
  }
  return bytes;
}

int launch_bwd(const FdaBwdArgs& a, cudaStream_t stream, unsigned stage_mask) {
  const FdaProblem& pr = a.p;
  DeviceInfo info;
  int rc = current_device_info(&info);
  if (rc) return rc;
  if (info.cc_major != 10) return FDA_ERR_ARCH;
  const int d = pr.head_dim;
  const int d_round = d <= 64 ? 64 : (d <= 128 ? 128 : 256);
  const bool varlen = pr.cu_seqlens != nullptr;
  const int64_t rows = varlen ? pr.total : pr.seqlen;
  const int tma_batch = varlen ? 1 : pr.batch;
  const bool fp16 = pr.dtype == FDA_FP16;

  BwdParams p;
  memset(&p, 0, sizeof(p));
  const bool single_pass = bwd_single_pass(pr) && (stage_mask & FDA_BWD_FORCE_SPLIT) == 0;
  p.apart = bwd_dv_apart(pr) ? 1 : 0;
  auto encode = [&](CUtensorMap* map, const FdaTensor& t, int heads, int box_rows) {
    return encode_tile_map(map, t.ptr, 2, false, fp16, d, rows, heads, tma_batch, t.row_stride, t.head_stride,
                           t.batch_stride, 64, box_rows);
  };
  if ((rc = encode(&p.tm_q, a.q, pr.heads, kTile)) || (rc = encode(&p.tm_do, a.dout, pr.heads, kTile)) ||
      (rc = encode(&p.tm_k, a.k, pr.heads_k, kTile)) || (rc = encode(&p.tm_v, a.v, pr.heads_k, kTile))) {
    return rc;
  }
  // 64-row boxes: the dK/dV kernel's query sub-tiles, and the dQ kernel's keys for head dimensions above 128
  if (!single_pass && ((rc = encode(&p.tm_q64, a.q, pr.heads, kSub)) || (rc = encode(&p.tm_do64, a.dout, pr.heads, kSub)))) {
    return rc;
  }
  if (!single_pass && d > 128 && ((rc = encode(&p.tm_k64, a.k, pr.heads_k, 64)) || (rc = encode(&p.tm_v64, a.v, pr.heads_k, 64)))) {
    return rc;
  }
  // the preprocess and the epilogues use 16-byte vector accesses on rows of out / dout / dq / dk / dv
  const FdaTensor* vec[] = {&a.out, &a.dout, &a.dq, &a.dk, &a.dv};
  for (const FdaTensor* t : vec) {
    if ((reinterpret_cast<uintptr_t>(t->ptr) & 15) || (t->row_stride % 8) || (t->head_stride % 8) ||
        (!varlen && (t->batch_stride % 8))) {
      return FDA_ERR_STRIDE;
    }
  }
  p.wide_store = (d % 16 == 0) ? 1 : 0;
  const FdaTensor* grads[] = {&a.dq, &a.dk, &a.dv};
  for (const FdaTensor* t : grads) {
    if ((reinterpret_cast<uintptr_t>(t->ptr) & 31) || (t->row_stride % 16) || (t->head_stride % 16) ||
        (!varlen && (t->batch_stride % 16))) {
      p.wide_store = 0;
    }
  }
  p.out = a.out.ptr;
  p.dout = a.dout.ptr;
  p.dq = a.dq.ptr;
  p.dk = a.dk.ptr;
  p.dv = a.dv.ptr;
  auto set3 = [&](const FdaTensor& t, int64_t& bs_, int64_t& rs_, int64_t& hs_) {
    bs_ = varlen ? 0 : t.batch_stride;
    rs_ = t.row_stride;
    hs_ = t.head_stride;
  };
  set3(a.out, p.o_bs, p.o_rs, p.o_hs);
  set3(a.dout, p.do_bs, p.do_rs, p.do_hs);
  set3(a.dq, p.dq_bs, p.dq_rs, p.dq_hs);
  set3(a.dk, p.dk_bs, p.dk_rs, p.dk_hs);
  set3(a.dv, p.dv_bs, p.dv_rs, p.dv_hs);
  p.lse = a.lse;
  p.cu_seqlens = pr.cu_seqlens;
  p.batch = pr.batch;
  p.seqlen = pr.seqlen;
  p.total = pr.total;
  p.heads = pr.heads;
  p.heads_k = pr.heads_k;
  p.overlap = bwd_overlaps(pr, single_pass) ? 1 : 0;
  p.next_early = pr.sm_margin <= 0 ? 1 : 0;
  p.head_dim = d;
  p.block_size = pr.block_size;
  p.n_pad = static_cast<int>(round_up64(pr.seqlen / 2 > 0 ? pr.seqlen / 2 : 1, kTile));
  p.tiles_per_half = p.n_pad / kTile;
  const int64_t one = round_up64(static_cast<int64_t>(pr.batch) * pr.heads * 2 * p.n_pad * 4, 256);
  p.delta_pad = static_cast<float*>(a.workspace);
  p.lse2_pad = reinterpret_cast<float*>(static_cast<uint8_t*>(a.workspace) + one);
  p.ticket_kv = reinterpret_cast<int*>(static_cast<uint8_t*>(a.workspace) + 2 * one);
  p.ticket_q = p.ticket_kv + 32;
  if (single_pass) {
    if (a.workspace_bytes < bwd_workspace_bytes(pr)) return FDA_ERR_WORKSPACE;
    p.dq_acc = reinterpret_cast<float*>(static_cast<uint8_t*>(a.workspace) + bwd_split_workspace_bytes(pr));
    p.acc_tiles = static_cast<int>(bwd_fused_acc_tiles(pr));
    p.acc_floats = static_cast<int64_t>(bwd_fused_acc_bytes(pr) / 4);
    p.kv_split = bwd_fused_kv_split(pr);
    p.part_floats = static_cast<int64_t>(bwd_fused_part_bytes(pr) / 4);
    if (p.kv_split > 1) p.dkv_part = p.dq_acc + round_up64(p.acc_floats, 64);
  }
  // The work counters are zeroed by whichever kernel runs before the persistent ones anyway.
  if ((stage_mask & 6u) != 0 && !varlen) {
    if (stage_mask & 1u) p.zero_tickets = p.ticket_kv;
    else FDA_CUDA_TRY(cudaMemsetAsync(p.ticket_kv, 0, kTicketInts * 4, stream));
  }
  // The accumulator is zeroed by the preprocess (a stage call of the kernel alone fills it itself): one launch less, and the
  // fill runs beside the loads of O and dO. In front of the kernel / in the preprocess, backward with 16
  // heads of 128: 87.0 / 80.8 us (34 MB), 1163 / 1143 (268 MB); 32/8 heads of 64, 134 MB: 672 / 659.
  // Not where packed samples are much shorter than max_seqlen: most blocks of the preprocess then have nothing but padding to
  // write, and the stores are dear there. 32 samples of 1024 tokens, 32/8 heads of 128 (in front / in the preprocess): 1116 / 1114 us
  // with max_seqlen as it is, 1161 / 1168 with three times that, 1225 / 1256 with four, 1474 / 1537 with eight. (Small
  // accumulators are always filled there: the launch counts for more.)
  const int64_t padded_rows = static_cast<int64_t>(pr.batch) * 2 * p.n_pad, acc_rows = static_cast<int64_t>(p.acc_tiles) * 64;
  if (single_pass && (stage_mask & 3u) == 3u && (padded_rows <= 3 * acc_rows || p.acc_floats * 4 <= kSmallAccBytes)) {
    p.zero_acc16 = p.acc_floats / 4;
  }
  if (varlen) {
    // the work list of the persistent kernels is built on the device (no host synchronisation); every stage call
    // rebuilds it, so stages may be launched one by one
    int* list = reinterpret_cast<int*>(static_cast<uint8_t*>(a.workspace) + 2 * one + 256);
    if (stage_mask & 6u) {
      rc = launch_varlen_prepare(pr.cu_seqlens, pr.batch, kTile, list, p.ticket_kv, stream, p.overlap != 0);
      if (rc) return rc;
    }
    p.vl.base = list;
    p.vl.batch = pr.batch;
  }
  const bool softcap = pr.softcap > 0.f;
  p.softmax_scale = pr.softmax_scale;
  if (softcap) {
    p.scale_log2 = pr.softcap * kLog2e;
    p.softcap_pre = pr.softmax_scale / pr.softcap;
  } else {
    p.scale_log2 = pr.softmax_scale * kLog2e;
    p.softcap_pre = 0.f;
  }
  int sm_count = info.sm_count - (pr.sm_margin > 0 ? pr.sm_margin : 0);
  if (sm_count < 1) sm_count = 1;
  {
    // dK/dV: the noisy key tiles (the second half of the ranks) are short; dQ: the shortest eighth (fractions
    // found by measurement on the benchmark shape); few items per CTA: rank for rank over all of them
    const int per_bh = 2 * p.tiles_per_half;
    const int parts = single_pass ? p.kv_split : 1;
    p.n_long_kv = order_n_long(per_bh, FDA_SHORT8_KV, static_cast<long long>(per_bh) * pr.batch * pr.heads_k * parts, sm_count);
    p.n_long_q = order_n_long(per_bh, FDA_SHORT8_Q, static_cast<long long>(per_bh) * pr.batch * pr.heads, sm_count);
  }
  const bool bf16 = pr.dtype == FDA_BF16;

  if (stage_mask & 1u) {
    const int lanes = d <= 64 ? 8 : (d <= 128 ? 16 : 32);
    const int rows_per_block = 8 * (32 / lanes) * kPreUnroll;
    dim3 grid((p.n_pad + rows_per_block - 1) / rows_per_block, 2 * pr.heads, pr.batch);
    auto pre = [&](auto bf16_tag) {
      constexpr bool kB = decltype(bf16_tag)::value;
      return lanes == 8 ? bwd_preprocess_kernel<kB, 8> : lanes == 16 ? bwd_preprocess_kernel<kB, 16> : bwd_preprocess_kernel<kB, 32>;
    };
    rc = launch_kernel(p.overlap != 0, bf16 ? pre(std::true_type{}) : pre(std::false_type{}), grid, 256, 0, stream, p);
    if (rc) return rc;
  }
  if (single_pass) return launch_bwd_fused(p, d_round, bf16, softcap, sm_count, stage_mask, stream);
  if (d_round == 64) return dispatch_bwd<64, 6, 7>(p, sm_count, bf16, softcap, stage_mask, stream);
  if (d_round == 128) return dispatch_bwd<128, 4, 5>(p, sm_count, bf16, softcap, stage_mask, stream);
  return dispatch_bwd<256, 1, 3>(p, sm_count, bf16, softcap, stage_mask, stream);
}


// ------------------------------------------------------------------------------------------------------------
// Backward without a caller-provided workspace (fda_bwd_noalloc). It always runs the split backward, whose
// scratch (delta, -LSE * log2(e), the two work counters) is small; that scratch lives in this fixed array, which
// every GPU that loads the library holds until the process exits. In host code the array's name is only a
// stand-in for the symbol: the device address is looked up once per device, with that device current, and that
// pointer is what the kernels receive.
// ------------------------------------------------------------------------------------------------------------
static __device__ __align__(256) unsigned char g_bwd_noalloc_scratch[FDA_NOALLOC_SCRATCH_BYTES];

int launch_bwd_noalloc(const FdaBwdArgs& a, cudaStream_t stream) {
  if (bwd_split_workspace_bytes(a.p) > static_cast<size_t>(FDA_NOALLOC_SCRATCH_BYTES)) return FDA_ERR_SCRATCH_LIMIT;
  static std::atomic<void*> scratch_of_device[kMaxCachedDevices];
  int dev = 0;
  FDA_CUDA_TRY(cudaGetDevice(&dev));
  const bool cached = dev >= 0 && dev < kMaxCachedDevices;
  void* ptr = cached ? scratch_of_device[dev].load(std::memory_order_acquire) : nullptr;
  if (ptr == nullptr) {
    FDA_CUDA_TRY(cudaGetSymbolAddress(&ptr, g_bwd_noalloc_scratch));
    if (cached) scratch_of_device[dev].store(ptr, std::memory_order_release);
  }
  FdaBwdArgs with_scratch = a;
  with_scratch.workspace = ptr;
  with_scratch.workspace_bytes = FDA_NOALLOC_SCRATCH_BYTES;
  return launch_bwd(with_scratch, stream, 7u | FDA_BWD_FORCE_SPLIT);
}

int read_status_bwd(int32_t* out4) {
  int zero[4] = {0, 0, 0, 0};
  FDA_CUDA_TRY(cudaMemcpyFromSymbol(out4, g_fda_status, sizeof(int) * 4));
  FDA_CUDA_TRY(cudaMemcpyToSymbol(g_fda_status, zero, sizeof(int) * 4));
  return FDA_OK;
}

}  // namespace fda
