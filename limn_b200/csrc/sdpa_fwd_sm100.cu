// "sdpa" forward for f16/bf16 with hd and hd_v multiples of 8 up to 128, with or without a key mask: TMA-staged tiles,
// tcgen05 MMAs accumulating in tensor memory, online softmax with one thread per query row. The kernels are built for
// head dims 64 and 128; a narrower head runs in the next of the two: TMA fills the columns a row does not have with
// zeros, which add nothing to a score and give zero output columns that are not stored. hd and hd_v may differ for
// the same reason: Q and K are read with hd columns, V with hd_v, and O is stored hd_v wide.
//
// A work item is two consecutive tiles of 128 query rows of one (batch, head) problem; the problem's keys
// and values stream past them in tiles of 128 keys:
//   S_t = Q_t K_j^T          tcgen05.mma, both operands K-major in shared memory, S_t in tensor memory
//   P_t = exp2(S_t - m_t)    128 softmax threads per Q tile, one row each; P_t overwrites S_t as 16-bit
//   O_t += P_t V_j           tcgen05.mma, A = P_t from tensor memory, B = V_j (MN-major) from shared memory
// Two Q tiles per item keep the tensor pipe busy on one while the other is in its softmax.
// (A problem with a single Q tile puts it in both places and deals its key tiles out between them: launch_fwd below.)
// Each output row has exactly one owner and is accumulated in a fixed key order, so two
// runs give the same bits, as the kernel this replaces promises (limn/cuda_emit.py:748-752).
//
// The grid is one CTA per SM. A CTA fetches items from a counter (longest first) until none is left, so
// barriers, tensor memory and descriptors are set up once, and the next item's Q, K and V are on their way
// (and its first scores computed) while the current item's last tile and epilogue are still running.
//
// Warp roles (10 warps): 0-3 softmax/epilogue of Q tile 0, 4-7 of Q tile 1, 8 TMA producer and work
// fetcher, 9 MMA issuer and tensor-memory owner.
//
// Semantics follow the oracle (limn/sdpa.py:91-137): causal keeps key j for row i when
// j <= i; O is rounded once from the fp32 accumulator; L = m + log(l) in natural log.
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <cstdlib>

#include "common.h"
#include "sm100_ptx.cuh"
#include "tensor_map.h"

namespace limn_b200 {
namespace {

using namespace ptx;

constexpr int kTileRows = 128;   // query rows per Q tile, keys per K/V tile
constexpr int kQTiles = 2;       // Q tiles per CTA
// Ten warps work, but the block size decides how the compiler allocates registers in the softmax loop (all sizes
// end at 168 registers; what differs is what is spilled where). Measured on B200 with the elected issue: head dim 128 under a
// causal mask 10 warps, 5 % over 11 and 12 (prefill_4k 0.912, 0.964 and 0.957 ms), without one 10 by 1 and 6 %; head dim 64 10 by 2
// to 5 %; under a key mask at head dim 64 11 (192 padded problems of 500 33.5 us, 34.6 with 12; causal on top 25.3, 25.6), at 128 no
// difference. The spare warps go straight to the final barrier.
template <int D, bool kMask>
constexpr int fwd_threads() {
  return kMask ? (D == 64 ? 352 : 384) : 320;
}
constexpr int kProducerWarp = 8;
constexpr int kMmaWarp = 9;
constexpr uint32_t kTmemCols = 512;
constexpr float kLog2e = 1.4426950408889634f;
constexpr float kRescaleSlack = 8.f;   // log2 units a row maximum may outgrow its reference before O is rescaled
// Of every 8 pairs of scores, how many take exp2 as a polynomial on the FMA pipe instead of on the special-function
// unit. Measured on B200 with the elected issue, as time over that without any: head dim 64 two pairs 0.95 to 0.98 (one 1.0,
// three 1.0), under a key mask two 0.95 but 1.03 with a causal mask on top; head dim 128 without a mask one pair of degree 3 0.96
// (degree 4 or 5 gain nothing), with any mask 1.0 to 1.02. Degree 5 at head dim 64 keeps the log-sum-exp at float32's own
// accuracy, 4e-8 (a cubic in one pair of eight: 1e-7 to 1.6e-6), for 1 % of the time. LIMN_POLY_PAIRS overrides the choice for
// experiments.
template <int D, bool kCausal, bool kMask>
constexpr int poly_pairs_of_8() {
#ifdef LIMN_POLY_PAIRS
  return LIMN_POLY_PAIRS;
#else
  if (D == 64) return kCausal && kMask ? 0 : 2;
  return kCausal || kMask ? 0 : 1;
#endif
}

template <int D, bool kCausal, RowStore kStore>
struct FwdLayout {
  static constexpr int kTileBytes = kTileRows * D * 2;
  static constexpr int kAtomBytes = kTileRows * 128;        // one 64-element-wide column block of a tile
  // K and V rings, each this deep. Shared memory would hold more at head dim 64, but deeper rings are slower there
  // (measured 5: +4 %; 3: +1.5 % once, no difference with the elected issue): two tiles in flight cover the load latency.
  static constexpr int kStages = 2;
  static constexpr int kQOff = 0;
  static constexpr int kKOff = kQOff + kQTiles * kTileBytes;
  static constexpr int kVOff = kKOff + kStages * kTileBytes;
  // Where the epilogue leaves O for the tile store: one 64-column block (128 rows x 128 B) per softmax group, which a
  // group's two blocks take turns in. Used at head dim 128 under a causal mask, where it is worth 2 to 3 %: the two
  // Q tiles of an item end at different times there and each group's stores are on its own critical path. Without
  // a causal mask both groups reach the epilogue together and the hand-overs cost more than the stores did (-1 %
  // at head dim 128, -6 % at 64, measured).
  static constexpr bool kTileStore = D == 128 && kCausal;
  static constexpr int kStageOff = kVOff + kStages * kTileBytes;
  // Without it rows leave as kStore says (see rows_leave).
  static constexpr int kWarpStage = kStore == RowStore::kStaged ? 4096 : 0;  // of each softmax warp, for two 32-column pieces of its rows
  static constexpr int kBarOff = kStageOff + (kTileStore ? kQTiles * kAtomBytes : 8 * kWarpStage);
  static constexpr int kBytes = kBarOff + 512 + 1024;       // room for 64 barriers + slack to align the base to 1024
  // tensor-memory columns
  static constexpr int kSCol = 0;                           // S_t at kSCol + 128 t (P_t overlays its first 64)
  static constexpr int kOCol = 256;                         // O_t at kOCol + D t
};

// barrier indices inside the barrier block
template <int D>
struct FwdBars {
  static constexpr int kS = FwdLayout<D, false, RowStore::kOwn>::kStages;
  static constexpr int q_full = 0;               // + t
  static constexpr int k_full = 2;               // + stage
  static constexpr int k_empty = k_full + kS;
  static constexpr int v_full = k_empty + kS;
  static constexpr int v_empty = v_full + kS;
  static constexpr int s_full = v_empty + kS;    // + t
  static constexpr int p_full = s_full + 2;      // + t
  static constexpr int o_full = p_full + 2;      // + t
  static constexpr int p_half = o_full + 2;      // + t: the first 64 keys' worth of P_t is in place (and O_t rescaled)
  static constexpr int q_empty = p_half + 2;     // + t: the item's last S_t has been computed, Q_t may be replaced
  static constexpr int o_free = q_empty + 2;     // + t: the epilogue has read O_t, the next item may overwrite it
  static constexpr int work_full = o_free + 2;   // + slot: the producer has fetched a work item
  static constexpr int work_empty = work_full + 2;  // + slot: every consumer has read it
  static constexpr int stage_full = work_empty + 2;   // + t: every row of a staging block is written (128 arrivals)
  static constexpr int stage_free = stage_full + 2;   // + t: the tile store has read the block
  static constexpr int merge_full = stage_free + 2;   // shared item: Q tile 1's part of every row is complete (128 arrivals)
  static constexpr int count = merge_full + 1;
};

// Build-time diagnostic (-DLIMN_TRACE): one CTA records clock64() at each step of its pipeline into a
// buffer named by the LIMN_TRACE_PTR environment variable. Compiled out of the shipped library.
#ifdef LIMN_TRACE
#define TRACE_EVENT(code) do { if (blockIdx.x == 7 && lane == 0 && trace_n < 250) { prm.trace[warp * 512 + 2 * trace_n] = clock64(); prm.trace[warp * 512 + 2 * trace_n + 1] = (code); ++trace_n; } } while (0)
#else
#define TRACE_EVENT(code) do {} while (0)
#endif

struct FwdParams {
  long long bh;
#ifdef LIMN_TRACE
  long long* trace;
#endif
  const unsigned short* mask;  // (bh, t_k) key flags in the storage dtype, 0 hides a key; null without a mask
  void* out;
  float* lse;
  unsigned* status;
  unsigned* schedule;  // [0] next work item, [1] CTAs that have finished; both zero between launches
  int group;           // problems per scheduling group (see cta_work)
  int heads;           // problem p is (batch p / heads, head p % heads) in the tensor maps and in `out`
  Strides out_strides; // of O, in elements
  unsigned items;      // work items: bh * q_pairs
  int t_q, t_k;
  int width;        // columns of V and O as they lie in memory (<= D)
  int q_pairs;      // work items per problem
  int kv_tiles;     // ceil(t_k / 128)
  float scale;
};

template <int D, bool kCausal, bool kFp16, bool kMask, bool kShared, RowStore kStore>
__global__ void __launch_bounds__((fwd_threads<D, kMask>()), 1)
sdpa_fwd_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                const __grid_constant__ CUtensorMap map_v, const __grid_constant__ CUtensorMap map_o, const FwdParams prm) {
  using L = FwdLayout<D, kCausal, kStore>;
  using B = FwdBars<D>;
  extern __shared__ unsigned char smem_unaligned[];
  __shared__ uint32_t tmem_slot;
  __shared__ uint32_t abort_flag;
  __shared__ unsigned work_ring[2];
  __shared__ float merge_m[kTileRows], merge_l[kTileRows];  // shared item: from Q tile 1's softmax group to the other

  const uint32_t raw = smem_addr(smem_unaligned);
  const uint32_t base = (raw + 1023u) & ~1023u;
  const uint32_t bars = base + L::kBarOff;
  auto bar = [&](int i) { return bars + 8u * i; };

  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0);  // (the same in every lane, and known to be)
  const int lane = threadIdx.x & 31;

  // ---- which rows a work item covers ----
  struct Item {
    int problem;
    int head, batch;    // the problem's coordinates in the operands
    int q0[kQTiles];    // first query row of each Q tile
    int n_kv[kQTiles];  // key tiles each Q tile consumes
    int n_max;          // the larger of the two
    int loads;          // key tiles the item streams
  };
  auto decode = [&](unsigned index) {
    Item it;
    int slot;
    cta_work(static_cast<int>(index), prm.q_pairs, prm.bh, prm.group, it.problem, slot);
    it.batch = it.problem / prm.heads;
    it.head = it.problem - it.batch * prm.heads;
    const int pair = prm.q_pairs - 1 - slot;  // longest causal rows first
#pragma unroll
    for (int t = 0; t < kQTiles; ++t) {
      it.q0[t] = (pair * kQTiles + t) * kTileRows;
      int n = prm.kv_tiles;
      if (kCausal) n = min(n, pair * kQTiles + t + 1);
      it.n_kv[t] = it.q0[t] < prm.t_q ? n : 0;
    }
    it.loads = max(it.n_kv[0], it.n_kv[1]);
    if (kShared) {
      it.q0[1] = it.q0[0];
      it.n_kv[1] = it.loads / 2;
      it.n_kv[0] = it.loads - it.n_kv[1];
    }
    it.n_max = max(it.n_kv[0], it.n_kv[1]);
    return it;
  };

  // ---- set-up: barriers, tensor memory ----
  if (threadIdx.x == kProducerWarp * 32) {
    for (int i = 0; i < B::count; ++i) {
      unsigned arrivals = 1u;
      if ((i >= B::p_full && i < B::p_full + 2) || (i >= B::p_half && i < B::p_half + 2) || (i >= B::o_free && i < B::o_free + 2) ||
          (i >= B::stage_full && i < B::stage_full + 2) || i == B::merge_full)
        arrivals = 128u;                                           // every thread of a softmax group
      if (i >= B::work_empty && i < B::work_empty + 2) arrivals = 9u;  // the MMA warp and the eight softmax warps
      mbar_init(bar(i), arrivals);
    }
    mbar_init_fence();
    tma_prefetch_descriptor(&map_q);
    tma_prefetch_descriptor(&map_k);
    tma_prefetch_descriptor(&map_v);
  }
  // up to here nothing has touched global memory, so all of it may run under the tail of the kernel before this one
  grid_dependency_wait();
  grid_launch_dependents();
  // What is left of the set-up runs side by side: the status word is read, tensor memory allocated (a block that stands
  // down frees it again), and the producer, which initialised the barriers itself, does not wait for either: its first loads are
  // on their way. A kernel of one tile: 6.0 -> 5.5 us.
  // Whether the block stands down, because an earlier kernel on this device gave up, is decided by thread 0's one reading of
  // the word and holds for all of the block, also when the host clears the word meanwhile: no item is computed, nothing is stored
  // or drawn from the work counter, and the producer's first loads are given time to land at the end.
  if (threadIdx.x == 0) abort_flag = *reinterpret_cast<volatile unsigned*>(prm.status) != kStatusOk;
  if (warp == 0) named_barrier_arrive(kDecided, 64);
  if (warp == kMmaWarp) {
    tmem_alloc(smem_addr(&tmem_slot), kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  if (warp == kProducerWarp) named_barrier_arrive(kSetUp, fwd_threads<D, kMask>());
  else named_barrier_sync(kSetUp, fwd_threads<D, kMask>());
  tc_fence_after_sync();
  const uint32_t tmem = __shfl_sync(0xffffffffu, tmem_slot, 0);

  bool ok = warp == kProducerWarp || !abort_flag;  // (the producer asks once its first loads are out)
#ifdef LIMN_TRACE
  int trace_n = 0;
#endif
  TRACE_EVENT(0);

  // Work items are fetched by the producer and passed to the other warps through a two-entry ring, so
  // the producer can load the next item's Q, K and V while the current item is still being computed.
  // Every role walks the same items in the same order and counts its own barrier phases as it goes.
  auto next_item = [&](unsigned n_item, unsigned& index) {
    const unsigned slot = n_item & 1u;
    if (!mbar_wait(bar(B::work_full + slot), (n_item >> 1) & 1u, prm.status, 0x0400u | slot)) return false;
    index = *reinterpret_cast<volatile unsigned*>(&work_ring[slot]);
    return true;
  };

  if (warp == kProducerWarp) {
    // ================= TMA producer, work fetcher =================
    unsigned q_uses[kQTiles] = {0u, 0u};  // items so far in which Q tile t had rows
    auto publish = [&](unsigned n_item, unsigned index) {
      *reinterpret_cast<volatile unsigned*>(&work_ring[n_item & 1u]) = index;
      mbar_arrive(bar(B::work_full + (n_item & 1u)));
    };
    auto load_q = [&](const Item& item, int t) {
      ++q_uses[t];
      mbar_expect_tx(bar(B::q_full + t), L::kTileBytes);
#pragma unroll
      for (int a = 0; a < D / 64; ++a)
        tma_load_4d(base + L::kQOff + t * L::kTileBytes + a * L::kAtomBytes, &map_q, bar(B::q_full + t), a * 64, item.q0[t], item.head, item.batch);
    };
    auto load_k = [&](const Item& item, int j, int stage) {
      mbar_expect_tx(bar(B::k_full + stage), L::kTileBytes);
#pragma unroll
      for (int a = 0; a < D / 64; ++a)
        tma_load_4d(base + L::kKOff + stage * L::kTileBytes + a * L::kAtomBytes, &map_k, bar(B::k_full + stage), a * 64, j * kTileRows, item.head, item.batch);
    };
    auto load_v = [&](const Item& item, int j, int stage) {
      mbar_expect_tx(bar(B::v_full + stage), L::kTileBytes);
#pragma unroll
      for (int a = 0; a < D / 64; ++a)
        tma_load_4d(base + L::kVOff + stage * L::kTileBytes + a * L::kAtomBytes, &map_v, bar(B::v_full + stage), a * 64, j * kTileRows, item.head, item.batch);
    };
    // a CTA's first item is its own number (no round trip to the counter on the way to the first load); the counter hands out
    // what lies beyond the grid
    if (lane == 0) publish(0u, blockIdx.x);
    Item item = decode(blockIdx.x);
    unsigned step = 0;  // key tiles loaded so far, over all items
    int j = 0;
    if (lane == 0) {
#pragma unroll
      for (int t = 0; t < kQTiles; ++t)
        if (item.n_kv[t] > 0) load_q(item, t);
      for (; j < min(item.loads, L::kStages); ++j, ++step) {  // (as many as have room)
        load_k(item, j, j);
        load_v(item, j, j);
      }
    }
    __syncwarp();
    named_barrier_sync(kDecided, 64);
    if (lane == 0 && !abort_flag) {
      for (unsigned n_item = 1;; ++n_item) {
        for (; j < item.loads && ok; ++j, ++step) {
          const int stage = step % L::kStages;
          const uint32_t wrap = (step / L::kStages) & 1;
          ok = mbar_wait(bar(B::k_empty + stage), wrap ^ 1u, prm.status, 0x0100u | stage);
          if (!ok) break;
          load_k(item, j, stage);
          ok = mbar_wait(bar(B::v_empty + stage), wrap ^ 1u, prm.status, 0x0110u | stage);
          if (!ok) break;
          load_v(item, j, stage);
        }
        const unsigned slot = n_item & 1u;
        if (ok) ok = mbar_wait(bar(B::work_empty + slot), ((n_item >> 1) & 1u) ^ 1u, prm.status, 0x0120u | slot);
        if (!ok) break;
        const unsigned index = gridDim.x + atomicAdd(prm.schedule, 1u);
        publish(n_item, index);
        if (index >= prm.items) break;
        item = decode(index);
#pragma unroll
        for (int t = 0; t < kQTiles; ++t) {
          if (item.n_kv[t] == 0 || !ok) continue;
          ok = mbar_wait(bar(B::q_empty + t), (q_uses[t] & 1u) ^ 1u, prm.status, 0x0130u | t);
          if (ok) load_q(item, t);
        }
        j = 0;
      }
    }
  } else if (warp == kMmaWarp) {
    // ================= MMA issuer =================
    // The warp stays together and one lane of it is elected for each bunch of MMAs: what the instructions take from uniform
    // registers is then computed there. A lane 0 on its own took 240 to 560 clocks to issue four MMAs and the barriers
    // around them, now 130 to 400, and what the issue takes lies in the chain from one tile's probabilities to the next one's
    // scores. Measured, with the set-up below: encoder_2k 0.376 -> 0.350 ms, 64 problems of 2048 x 2048 x 128 without a
    // mask 0.137 -> 0.127, under one 48.3 -> 43.6 us (1024 keys), prefill_4k 0.934 -> 0.911 ms.
    if (ok) {
      constexpr uint32_t idesc_s = mma_idesc(kTileRows, kTileRows, kFp16, false, false);
      constexpr uint32_t idesc_pv = mma_idesc(kTileRows, D, kFp16, false, true);
      // S_t = Q_t K^T over the head dim, 16 elements per instruction
      auto issue_s = [&](int t, int stage) {
        const uint32_t q_lo = desc_lo(base + L::kQOff + t * L::kTileBytes, 0);
        const uint32_t k_lo = desc_lo(base + L::kKOff + stage * L::kTileBytes, 0);
        const uint32_t c = tmem + L::kSCol + t * 128;
        mma_ss_lo<false>(c, q_lo, k_lo, idesc_s);
#pragma unroll
        for (int kk = 1; kk < D / 16; ++kk) {
          constexpr uint32_t kAtom16 = L::kAtomBytes >> 4;
          const uint32_t off = (kk / 4) * kAtom16 + (kk % 4) * 2;  // in 16-byte units
          mma_ss_lo<true>(c, q_lo + off, k_lo + off, idesc_s);
        }
      };
      // O_t += P_t V over the 128 keys of the tile, 16 keys per instruction
      auto issue_pv = [&](int t, int stage, int part, bool first) {
        const uint32_t v_lo = desc_lo(base + L::kVOff + stage * L::kTileBytes, L::kAtomBytes);
        const uint32_t c = tmem + L::kOCol + t * D;
        const uint32_t a = tmem + L::kSCol + t * 128;
#pragma unroll
        for (int kk = 4 * part; kk < 4 * part + 4; ++kk)
          mma_ts_lo(c, a + kk * 8, v_lo + kk * (16 * 128 / 16), idesc_pv, (kk > 0 || !first) ? 1u : 0u);
      };
      unsigned q_uses[kQTiles] = {0u, 0u};  // items finished in which Q tile t had rows
      unsigned tiles[kQTiles] = {0u, 0u};   // key tiles Q tile t has been through, over all items
      unsigned step = 0;                    // key tiles consumed so far, over all items
      auto wait = [&](int i, uint32_t parity, unsigned tag) { return __all_sync(0xffffffffu, mbar_wait(bar(i), parity, prm.status, tag)); };
      for (unsigned n_item = 0; ok; ++n_item) {
        unsigned index;
        ok = __all_sync(0xffffffffu, next_item(n_item, index));
        if (!ok) break;
        index = __shfl_sync(0xffffffffu, index, 0);
        if (elect_one()) mbar_arrive(bar(B::work_empty + (n_item & 1u)));
        __syncwarp();
        if (index >= prm.items) break;
        const Item item = decode(index);
        auto at = [&](int t, int j) { return step + (kShared ? 2 * j + t : j); };  // Q tile t's j-th key tile, over all items
#pragma unroll
        for (int t = 0; t < kQTiles; ++t)
          if (item.n_kv[t] > 0 && ok) ok = wait(B::q_full + t, q_uses[t] & 1u, 0x0200u | t);
        if (!ok) break;
        if (item.n_max > 0) {
#pragma unroll
          for (int t = 0; t < kQTiles; ++t)
            if (item.n_kv[t] > 0 && ok) {
              const unsigned first = at(t, 0);
              const int stage = first % L::kStages;
              ok = wait(B::k_full + stage, (first / L::kStages) & 1, 0x0210u);
              if (!ok) break;
              tc_fence_after_sync();
              // (the S_t region is free: the MMAs run in issue order, and the last one issued for this tile was
              // the product that consumed the P_t stored there)
              if (elect_one()) {
                issue_s(t, stage);
                mma_commit(bar(B::s_full + t));
                if (item.n_kv[t] == 1) mma_commit(bar(B::q_empty + t));
                if (kShared) mma_commit(bar(B::k_empty + stage));
              }
              __syncwarp();
            }
          if (!ok) break;
          if (!kShared && elect_one()) mma_commit(bar(B::k_empty + step % L::kStages));
          __syncwarp();
        }
        for (int j = 0; j < item.n_max && ok; ++j) {
          bool issued_next = false;
#pragma unroll
          for (int t = 0; t < kQTiles; ++t) {
            if (!ok || j >= item.n_kv[t]) continue;
            const unsigned here = at(t, j), then = at(t, j + 1);
            const int stage = here % L::kStages, next = then % L::kStages;
            ok = wait(B::v_full + stage, (here / L::kStages) & 1, 0x0220u | stage);
            if (!ok) break;
            TRACE_EVENT(100 + t);
            const uint32_t phase = tiles[t] & 1u;
            // the product starts on the first 64 keys while the softmax is still on the last 64
            ok = wait(B::p_half + t, phase, 0x0260u | t);
            if (!ok) break;
            // the item's first product overwrites O_t: the previous item's epilogue must have read it
            if (j == 0) ok = wait(B::o_free + t, (q_uses[t] & 1u) ^ 1u, 0x0270u | t);
            if (!ok) break;
            tc_fence_after_sync();
            if (elect_one()) issue_pv(t, stage, 0, j == 0);
            __syncwarp();
            ok = wait(B::p_full + t, phase, 0x0230u | t);
            if (!ok) break;
            TRACE_EVENT(110 + t);
            tc_fence_after_sync();
            const bool last = j + 1 >= item.n_kv[t];
            if (elect_one()) {
              issue_pv(t, stage, 1, j == 0);
              if (last) mma_commit(bar(B::o_full + t));
              if (kShared) mma_commit(bar(B::v_empty + stage));
            }
            __syncwarp();
            TRACE_EVENT(120 + t);
            ++tiles[t];
            if (!last) {
              // the scores can only follow the product that consumed the P_t lying over them; s_full then also
              // tells the softmax that O_t is settled
              ok = wait(B::k_full + next, (then / L::kStages) & 1, 0x0240u | next);
              if (!ok) break;
              tc_fence_after_sync();
              if (elect_one()) {
                issue_s(t, next);
                mma_commit(bar(B::s_full + t));
                if (j + 2 == item.n_kv[t]) mma_commit(bar(B::q_empty + t));
                if (kShared) mma_commit(bar(B::k_empty + next));
              }
              __syncwarp();
              TRACE_EVENT(130 + t);
              issued_next = true;
            }
          }
          if (!ok) break;
          if (!kShared && elect_one()) {
            mma_commit(bar(B::v_empty + (step + j) % L::kStages));
            if (issued_next) mma_commit(bar(B::k_empty + (step + j + 1) % L::kStages));
          }
          __syncwarp();
        }
        step += item.loads;
#pragma unroll
        for (int t = 0; t < kQTiles; ++t)
          if (item.n_kv[t] > 0) ++q_uses[t];
      }
    }
  } else if (warp < kProducerWarp) {
    // ================= softmax + epilogue, one thread per query row =================
    const int t = warp >> 2;
    const int row_in_tile = threadIdx.x & 127;
    const uint32_t lane_base = static_cast<uint32_t>((warp & 3) * 32) << 16;
    const uint32_t t_s = tmem + lane_base + L::kSCol + t * 128;
    const uint32_t t_o = tmem + lane_base + L::kOCol + t * D;
    const float sl2 = prm.scale * kLog2e;
    // m is the score (in raw units) the exponentials are measured against. It only moves when the
    // row maximum has outgrown it by more than kRescaleSlack (in log2 units), so most tiles need no
    // rescaling of O_t; until then probabilities may reach 2^kRescaleSlack, which fp32 sums and
    // 16-bit P carry without loss. The result is the same softmax: L = m * scale + log(l).
    const uint64_t sl2_2 = f2_pack(sl2, sl2);
    unsigned tiles = 0;   // key tiles this group has been through, over all items
    unsigned o_uses = 0;  // items this group has finished
    unsigned stores = 0;  // staging blocks this group has handed to TMA
    unsigned merges = 0;  // shared items so far
    // Key mask: a hidden key is a score of -inf for every row. Each lane fetches four of a tile's 128 flags one tile
    // ahead of their use; a ballot per 32 keys then gives every thread all of them.
    // (the flags stay as loaded until the next tile needs them: a warp issues in order, so turning them into anything
    // right after the load would stall it for the load's latency, every tile)
    auto fetch_flags = [&](int problem, int kv0, unsigned (&out4)[4]) {
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const int key = kv0 + 32 * c + lane;
        out4[c] = key < prm.t_k ? prm.mask[static_cast<long long>(problem) * prm.t_k + key] : 0u;  // past the end: hidden
      }
    };
    for (unsigned n_item = 0; ok; ++n_item) {
    unsigned index;
    ok = __all_sync(0xffffffffu, next_item(n_item, index));
    if (!ok) break;
    __syncwarp();
    if (lane == 0) mbar_arrive(bar(B::work_empty + (n_item & 1u)));
    if (index >= prm.items) break;
    const Item item = decode(index);
    const int problem = item.problem;
    const int n = item.n_kv[t];
    if (n == 0) continue;
    const int row = item.q0[t] + row_in_tile;
    float m = -INFINITY, l = 0.f;
    unsigned flags[4] = {1u, 1u, 1u, 1u};
    auto key0 = [&](int j) { return (kShared ? 2 * j + t : j) * kTileRows; };  // first key of this Q tile's j-th key tile
    if (kMask) fetch_flags(problem, key0(0), flags);
    for (int j = 0; j < n; ++j, ++tiles) {
      // Key mask: which of the tile's 128 keys are hidden, as four ballot words in registers (each lane fetched four
      // of the flags a tile ahead). A tile none of whose keys is hidden (every tile but the last few of a padded
      // batch) is handled like an unmasked one.
      unsigned hid[4] = {0u, 0u, 0u, 0u};
      bool any_hidden = false;
      if (kMask) {
#pragma unroll
        for (int c = 0; c < 4; ++c) hid[c] = __ballot_sync(0xffffffffu, (flags[c] & 0x7fffu) == 0u);
        any_hidden = ((hid[0] | hid[1]) | (hid[2] | hid[3])) != 0u;
        if (j + 1 < n) fetch_flags(problem, key0(j + 1), flags);
      }
      ok = __all_sync(0xffffffffu, mbar_wait(bar(B::s_full + t), tiles & 1u, prm.status, 0x0300u | t));  // warp-uniform: the tensor-memory ops below are warp-wide
      if (!ok) break;
      TRACE_EVENT(2);
      tc_fence_after_sync();
      uint32_t s[4][32];
#pragma unroll
      for (int c = 0; c < 4; ++c) tmem_ld32(t_s + 32 * c, s[c]);
      tmem_ld_wait();
      TRACE_EVENT(3);
      const int kv0 = key0(j);
      const bool diagonal = kCausal && kv0 + kTileRows > item.q0[t];     // some key of this tile is right of some row
      const bool ragged = kv0 + kTileRows > prm.t_k;                // some key of this tile does not exist
      if (diagonal || ragged || (kMask && any_hidden)) {
        int limit = prm.t_k - kv0;                                  // keys [0, limit) of the tile are visible
        if (kCausal) limit = min(limit, row - kv0 + 1);
#pragma unroll
        for (int c = 0; c < 4; ++c)
#pragma unroll
          for (int i = 0; i < 32; ++i)
            if (c * 32 + i >= limit || (kMask && ((hid[c] >> i) & 1u) != 0u)) s[c][i] = 0xff800000u;  // -inf
      }
      float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
      for (int c = 0; c < 4; ++c)
#pragma unroll
        for (int i = 0; i < 32; i += 2) mx4[(i >> 1) & 3] = max3(mx4[(i >> 1) & 3], __uint_as_float(s[c][i]), __uint_as_float(s[c][i + 1]));
      const float mx = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3]));
      // A row may have met nothing but scores of -inf yet, be it that its keys are hidden or that the operands make them so:
      // then mx and m are both -inf, nothing moves, and the exponentials are measured against 0 so that they come out
      // exp2(-inf) = 0 instead of NaN.
      const bool moves = (mx - m) * sl2 > kRescaleSlack;  // true at the first score above -inf, where m is -inf
      float alpha = 1.f;
      if (moves) {
        alpha = exp2_approx((m - mx) * sl2);
        m = mx;
      }
      TRACE_EVENT(4);
      const float shift = m == -INFINITY ? 0.f : -m * sl2;
      const uint64_t shift2 = f2_pack(shift, shift);
      uint64_t sum2[2] = {0ull, 0ull};
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        if (h == 1) {
          // O_t was last written by the PV of tile j-1, which s_full also covers. It is rescaled before any of
          // this tile's P_t is handed over (the product on the first half starts early), at the point where
          // the first half's scores are no longer held in registers.
          if (j > 0 && __any_sync(0xffffffffu, moves)) {
#pragma unroll
            for (int c = 0; c < D / 32; ++c) {
              uint32_t o[32];
              tmem_ld32(t_o + 32 * c, o);
              tmem_ld_wait();
#pragma unroll
              for (int i = 0; i < 32; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * alpha);
              tmem_st32(t_o + 32 * c, o);
            }
          }
        }
        uint32_t packed[32];
#pragma unroll
        for (int cc = 0; cc < 2; ++cc) {
          const int c = 2 * h + cc;
#pragma unroll
          for (int i = 0; i < 32; i += 2) {
            const uint64_t x2 = f2_fma(f2_pack_bits(s[c][i], s[c][i + 1]), sl2_2, shift2);
            float p0, p1;
            if (((i >> 1) & 7) < poly_pairs_of_8<D, kCausal, kMask>()) {
              exp2_poly2<D == 64 ? 5 : 3>(x2, p0, p1);
            } else {
              f2_unpack(x2, p0, p1);
              p0 = exp2_approx(p0);
              p1 = exp2_approx(p1);
            }
            sum2[(i >> 1) & 1] = f2_add(sum2[(i >> 1) & 1], f2_pack(p0, p1));
            packed[cc * 16 + (i >> 1)] = kFp16 ? pack_f16(p0, p1) : pack_bf16(p0, p1);
          }
          if (h == 1 && cc == 0) {
            // the first half's store was issued a chunk of exponentials ago; hand it over
            tmem_st_wait();
            tc_fence_before_sync();
            mbar_arrive(bar(B::p_half + t));
          }
        }
        tmem_st32(t_s + 32 * h, packed);
      }
      TRACE_EVENT(5);
      float sum_a, sum_b, sum_c, sum_d;
      f2_unpack(sum2[0], sum_a, sum_b);
      f2_unpack(sum2[1], sum_c, sum_d);
      l = l * alpha + ((sum_a + sum_b) + (sum_c + sum_d));
      tmem_st_wait();
      TRACE_EVENT(6);
      tc_fence_before_sync();
      mbar_arrive(bar(B::p_full + t));
    }
    if (ok) ok = __all_sync(0xffffffffu, mbar_wait(bar(B::o_full + t), o_uses & 1u, prm.status, 0x0310u | t));
    if (ok) {
      tc_fence_after_sync();
      float from_1 = 0.f;  // shared item: what Q tile 1's part of this row counts relative to this one's (already in l and O_0's factor)
      float keep = 1.f;
      if (kShared) {
        // a group for Q tile 1 leaves its maximum and sum and lets the other one read O_1
        if (t == 1) {
          merge_m[row_in_tile] = m, merge_l[row_in_tile] = l;
          tc_fence_before_sync();
          mbar_arrive(bar(B::merge_full));
          ++o_uses;
          continue;
        }
        ok = __all_sync(0xffffffffu, mbar_wait(bar(B::merge_full), merges & 1u, prm.status, 0x0340u));
        if (!ok) break;
        ++merges;
        tc_fence_after_sync();
        const float m_1 = *const_cast<volatile float*>(&merge_m[row_in_tile]), l_1 = *const_cast<volatile float*>(&merge_l[row_in_tile]);
        const float top = fmaxf(m, m_1);
        // (a part that has seen no visible key has m = -inf and l = 0, and counts nothing)
        // (expf, twice a row: with ex2.approx L was 3 % further from float64 than an unshared row's under a mask at width 128)
        keep = m == -INFINITY ? 0.f : expf((m - top) * prm.scale);
        from_1 = m_1 == -INFINITY ? 0.f : expf((m_1 - top) * prm.scale);
        l = l * keep + l_1 * from_1;
        m = top;
      }
      const float inv = 1.f / l;
      // 32 columns of the row, as they leave (16 bits later)
      auto take = [&](int col, uint32_t (&o)[32]) {
        tmem_ld32(t_o + col, o);
        if (kShared) {
          uint32_t o_1[32];
          tmem_ld32(t_o + D + col, o_1);
          tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < 32; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * keep + __uint_as_float(o_1[i]) * from_1);
        } else {
          tmem_ld_wait();
        }
      };
      auto free_o = [&] {
        tc_fence_before_sync();
        mbar_arrive(bar(B::o_free + t));
        if (kShared) mbar_arrive(bar(B::o_free + 1));
      };
      const long long out_row = static_cast<long long>(problem) * prm.t_q + row;  // in L, which is always dense
      if constexpr (L::kTileStore) {
        // O goes out as tile stores: every thread leaves its row, rounded, in the group's staging block (in the
        // swizzled layout, so the 32 rows of a warp fall on distinct banks), and one thread hands the block to TMA,
        // which writes whole 128-byte rows and leaves out the rows and columns the tensor does not have. (A thread
        // storing its own row in 16-byte pieces costs the load/store unit 32 transactions per instruction.)
        const uint32_t stage = base + L::kStageOff + t * L::kAtomBytes;
        const bool leader = (warp & 3) == 0 && lane == 0;
#pragma unroll
        for (int blk = 0; blk < D / 64 && ok; ++blk, ++stores) {
          // the store before this one has read the block: the thread that issued it says so (waits are bounded,
          // like every wait here: a group whose warps disagree about going on must not hang on one another)
          if (leader) {
            tma_store_wait_read();
            mbar_arrive(bar(B::stage_free + t));
          }
          ok = __all_sync(0xffffffffu, mbar_wait(bar(B::stage_free + t), stores & 1u, prm.status, 0x0320u | t));
          if (!ok) break;
#pragma unroll
          for (int cc = 0; cc < 2; ++cc) {
            uint32_t o[32];
            take(64 * blk + 32 * cc, o);
#pragma unroll
            for (int v4 = 0; v4 < 4; ++v4) {
              uint32_t w[4];
#pragma unroll
              for (int i = 0; i < 4; ++i) {
                const float a = __uint_as_float(o[v4 * 8 + 2 * i]) * inv;
                const float b = __uint_as_float(o[v4 * 8 + 2 * i + 1]) * inv;
                w[i] = kFp16 ? pack_f16(a, b) : pack_bf16(a, b);
              }
              st_shared_v4(swizzled_piece(stage, row_in_tile, cc * 4 + v4), w[0], w[1], w[2], w[3]);
            }
          }
          if (blk == D / 64 - 1) {
            // O_t is in registers or staged: the next item's first product may overwrite it
            free_o();
          }
          fence_async_shared();
          mbar_arrive(bar(B::stage_full + t));
          if (leader) {
            if (mbar_wait(bar(B::stage_full + t), stores & 1u, prm.status, 0x0330u | t)) {
              tma_store_4d(&map_o, stage, 64 * blk, item.q0[t], item.head, item.batch);
              tma_store_commit();
            }
          }
        }
        if (row < prm.t_q) prm.lse[out_row] = m * prm.scale + logf(l);
      } else {
      // (own rows, address by the row / by the warp's first row: 2000 problems of 128 x 80 40.9 / 43.4 us, causal 256 of 256 x 64 13.6 / 13.4)
      if constexpr (kStore == RowStore::kOwn && !kCausal) {
        const long long out_at = item.batch * prm.out_strides.batch + item.head * prm.out_strides.head + row * prm.out_strides.row;
#pragma unroll
        for (int c = 0; c < D / 32; ++c) {
          uint32_t o[32];
          take(32 * c, o);
          if (row < prm.t_q) store_row32<kFp16>(static_cast<unsigned char*>(prm.out) + 2 * (out_at + 32 * c), o, inv, prm.width - 32 * c);
        }
      } else {
        const int top = item.q0[t] + (warp & 3) * 32;  // the warp's first row
        const long long row_bytes = 2 * prm.out_strides.row;
        unsigned char* to = static_cast<unsigned char*>(prm.out) + 2 * (item.batch * prm.out_strides.batch + item.head * prm.out_strides.head) + top * row_bytes;
#pragma unroll
        for (int c = 0; c < D / 32; ++c) {
          uint32_t o[32];
          take(32 * c, o);
          if constexpr (kStore == RowStore::kOwn) {
            if (row < prm.t_q) store_row32<kFp16>(to + lane * row_bytes + 64 * c, o, inv, prm.width - 32 * c);
          } else if (32 * c < prm.width && top < prm.t_q)  // (256 x 2048 x 64 341 us without the second, 335 with it)
            store_rows32<kFp16, kStore>(to + 64 * c, row_bytes, top, prm.t_q, o, inv, prm.width - 32 * c, base + L::kStageOff + warp * L::kWarpStage + (c & 1) * (L::kWarpStage / 2));
        }
      }
      if (row < prm.t_q) prm.lse[out_row] = m * prm.scale + logf(l);
      // O_t is in registers or stored: the next item's first product may overwrite it
      free_o();
      }
      ++o_uses;
    }
    }  // items
    // the last tile store must have read its staging block before the CTA gives its shared memory back
    if (L::kTileStore && (warp & 3) == 0 && lane == 0) tma_store_wait_read();
  }

  // ---- teardown ----
  tc_fence_before_sync();
  __syncthreads();
  if (warp == kMmaWarp) {
    if (abort_flag || *reinterpret_cast<volatile unsigned*>(prm.status) != kStatusOk) {
      // a wait gave up somewhere: give copies and MMAs still in flight time to land before the
      // tensor memory and shared memory they target are released
      for (int i = 0; i < 2000; ++i) __nanosleep(1000);
    }
    tc_fence_after_sync();
    tmem_free(tmem, kTmemCols);
  }
  // the last CTA to leave puts the work counters back to zero for the next launch that is handed this pair
  if (threadIdx.x == 0 && atomicAdd(prm.schedule + 1, 1u) == gridDim.x - 1) {
    prm.schedule[0] = 0u;
    prm.schedule[1] = 0u;
    __threadfence();
  }
}

template <int D, bool kCausal, bool kFp16, bool kMask, bool kShared, RowStore kStore>
int launch_fwd_s(const Problem& p) {
  using L = FwdLayout<D, kCausal, kStore>;
  CUtensorMap map_q, map_k, map_v, map_o;
  const int heads = p.heads > 0 ? p.heads : static_cast<int>(p.bh), batch = static_cast<int>(p.bh / heads);
  if (int rc = make_tile_map(&map_q, p.q, kFp16, batch, heads, p.t_q, p.hd, kTileRows, operand_strides(p, kOpQ, heads, p.t_q, p.hd))) return rc;
  if (int rc = make_tile_map(&map_k, p.k, kFp16, batch, heads, p.t_k, p.hd, kTileRows, operand_strides(p, kOpK, heads, p.t_k, p.hd))) return rc;
  if (int rc = make_tile_map(&map_v, p.v, kFp16, batch, heads, p.t_k, p.hd_v, kTileRows, operand_strides(p, kOpV, heads, p.t_k, p.hd_v))) return rc;
  if (int rc = make_tile_map(&map_o, p.out, kFp16, batch, heads, p.t_q, p.hd_v, kTileRows, operand_strides(p, kOpOut, heads, p.t_q, p.hd_v))) return rc;
  FwdParams prm;
  prm.out = p.out;
  prm.heads = heads;
  prm.out_strides = operand_strides(p, kOpOut, heads, p.t_q, p.hd_v);
  prm.width = p.hd_v;
  if ((prm.out_strides.batch | prm.out_strides.head | prm.out_strides.row) & 7)
    return fail(LIMN_B200_BAD_ARGUMENT, "sdpa: operand strides must be multiples of 8 elements");
  if (reinterpret_cast<uintptr_t>(p.out) & 15u) return fail(LIMN_B200_BAD_ARGUMENT, "sdpa: the output is not 16-byte aligned");
  prm.mask = static_cast<const unsigned short*>(p.mask);
  prm.lse = static_cast<float*>(p.lse_out);
  prm.status = p.status;
  if (prm.status == nullptr)
    if (int rc = status_word(&prm.status)) return rc;
  prm.bh = p.bh;
  prm.t_q = p.t_q, prm.t_k = p.t_k;
  prm.q_pairs = (p.t_q + kQTiles * kTileRows - 1) / (kQTiles * kTileRows);
  prm.kv_tiles = (p.t_k + kTileRows - 1) / kTileRows;
#ifdef LIMN_TRACE
  const char* trace_ptr = getenv("LIMN_TRACE_PTR");
  if (trace_ptr == nullptr) return fail(LIMN_B200_BAD_ARGUMENT, "this is a -DLIMN_TRACE build: set LIMN_TRACE_PTR to the trace buffer's device address");
  prm.trace = reinterpret_cast<long long*>(strtoull(trace_ptr, nullptr, 16));
#endif
  prm.scale = static_cast<float>(p.scale);
  const long long items = p.bh * prm.q_pairs;
  if (items > 0x7fffffffLL) return fail(LIMN_B200_UNSUPPORTED, "sdpa: %lld work items exceed the counter", items);
  prm.items = static_cast<unsigned>(items);
  if (int rc = schedule_words(&prm.schedule)) return rc;
  int sms = 0;
  if (int rc = sm_count(&sms)) return rc;
  prm.group = work_group(p, items, sms);
  const long long ctas = items < sms ? items : sms;  // one CTA per SM (shared and tensor memory allow no more), each fetching items until none is left
  auto kernel = sdpa_fwd_kernel<D, kCausal, kFp16, kMask, kShared, kStore>;
  // the attribute is per device and per kernel instantiation; set it on first use there
  static bool sized[64] = {};
  int device = 0;
  LIMN_CUDA(cudaGetDevice(&device), "asking for the current device");
  if (device >= 0 && device < 64 && !sized[device]) {
    LIMN_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, L::kBytes),
              "sizing shared memory for the sdpa kernel");
    sized[device] = true;
  }
  LIMN_CUDA(launch_overlapped(kernel, dim3(static_cast<unsigned>(ctas)), dim3(fwd_threads<D, kMask>()), L::kBytes, p.stream, map_q, map_k, map_v, map_o, prm),
            "launching the sdpa kernel");
  note_launches(1);
  return LIMN_B200_OK;
}

// How the rows of O leave without a causal mask. A thread's own row, piece by piece, is up to 32 lines of memory an instruction, but an
// instruction touches only the rows there are; exchanging pieces (head dim 128) or going by way of shared memory (64) takes a warp the
// same time whatever number of rows it has, in a chain of its own. So it is a matter of how full the tiles of rows are, of what a row
// has of its kernel's width, and of how far apart rows lie (scattered_rows). Measured on B200, us, own / exchanged or staged, dense rows:
//   128 columns: 700 problems of 32 17.7 / 21.8, of 96 19.0 / 22.2, of 128 19.6 / 20.3; 148 of 160 9.8 / 10.1, of 192 10.2 / 10.2, of 224 10.7 / 10.3, of
//     256 10.8 / 9.9, of 272 18.0 / 18.6, of 384 (64 of them) 11.2 / 10.8
//   80 columns: 700 of 128 17.0 / 18.3, 148 of 160 9.4 / 10.0, of 224 9.8 / 10.2, of 256 9.8 / 9.6, of 320 17.0 / 18.0; 200 of 256 15.3 / 14.8
//   64 columns: 2000 of 64 39.8 / 43.4, of 128 37.2 / 36.3, 148 of 160 8.2 / 8.5, of 224 8.5 / 8.5, of 256 8.2 / 8.1, of 320 15.1 / 15.6, of 512 18.7 / 18.1;
//     under a key mask 192 of 128 10.0 / 10.4, of 500 36.9 / 37.1, 400 of 2000 820 / 843
//   48 columns: 2000 of 64 39.7 / 43.3, 148 of 256 8.1 / 8.2, of 320 14.7 / 15.4, of 512 18.4 / 18.3
// Token-major with 12 heads: 128 columns 204 of 64 9.6 / 10.2, of 128 11.1 / 9.9, of 160 17.1 / 15.6; 64 columns 204 of 64 8.2 / 8.4, of 128 8.7 / 8.0, of 200
//   13.8 / 13.2; under a key mask 192 of 256 14.4 / 12.9. With 5 heads 700 of 100 under a mask 21.7 / 22.9, at 128 columns 24.6 / 26.3.
// Two groups that share the keys, dense: 128 columns 148 of 128 x 512 10.4 / 10.7; 64 columns 200 of 64 x 600 15.4 / 15.5, of 128 x 600 15.8 / 15.7, 700 of 100 x 1500
//   71.8 / 70.4, 16 of 40 x 2463 19.3 / 19.0, masked of 100 x 300 9.0 / 8.8. Under a causal mask at head dim 64 own rows (256 of 256 13.7 / 14.0).
template <int D, bool kMask, bool kShared>
RowStore rows_leave(const Problem& p) {
  constexpr RowStore kLong = D == 128 ? RowStore::kExchanged : RowStore::kStaged;
  const int heads = p.heads > 0 ? p.heads : static_cast<int>(p.bh);
  const long long missing = (kTileRows - p.t_q % kTileRows) % kTileRows, size = 1LL * p.t_q * p.hd_v;  // rows of the last tile; elements
  bool pays;
  if (scattered_rows(operand_strides(p, kOpOut, heads, p.t_q, p.hd_v).row, p.hd_v)) pays = size >= 112 * D;
  else if (D == 128) pays = !kShared && p.t_q > kTileRows && (p.hd_v > 80 ? 3 : 8) * missing < p.t_q;
  else if (kShared) pays = p.hd_v > 48 && (p.t_q >= 96 || p.t_k >= 1024);
  else pays = !kMask && p.hd_v > 48 && size >= 64 * kTileRows && 8 * missing < p.t_q;
  return pays ? kLong : RowStore::kOwn;
}

template <int D, bool kFp16, bool kMask, bool kShared>
int launch_fwd_rows(const Problem& p) {
  if (rows_leave<D, kMask, kShared>(p) == RowStore::kOwn) return launch_fwd_s<D, false, kFp16, kMask, kShared, RowStore::kOwn>(p);
  return launch_fwd_s<D, false, kFp16, kMask, kShared, D == 128 ? RowStore::kExchanged : RowStore::kStaged>(p);
}

// A problem with one Q tile: its tile goes into both places, the even key tiles to the first and the odd ones to the second,
// whose softmax group would be idle otherwise, and the epilogue puts the two parts of every row together. That halves the
// chain of key tiles, which is all there is to such an item. Measured, us without / with: 64 problems of 100 x 1500 keys x 64
// 18.6 / 14.1, 8 of 128 x 4096 x 128 46.9 / 30.7, 192 of 100 x 700 x 64 under a mask 22.8 / 19.0.
// The line, without / with: what sharing costs is a second copy of Q and the merge, so it pays from some number of key tiles on.
//   two tiles at width 128 without a mask, not shared: 1600 of 16 x 160 48.0 / 58.8, 320 15.0 / 16.7, 32 6.8 / 6.9; 32 of 100 x 256 6.9 / 7.3
//   two at width 64, shared: 32 of 16 x 160 6.1 / 5.8, 96 6.5 / 6.8, 320 13.0 / 13.9, 1600 41.3 / 47.6; of 100 rows 6.4 / 6.0, 6.7 / 7.1, 13.9 / 14.2, 44.9 / 48.4
//   two under a mask, shared: width 64 8 to 1600 of 100 x 160 7.3 / 7.1 to 60.7 / 55.9, width 128 8.2 / 8.1 to 71.3 / 64.7
//   three at width 128 (384 keys), shared: 32 of 100 rows 8.3 / 8.3, 320 20.1 / 18.7, 1600 70.1 / 70.4; of 16 rows 7.8 / 7.9, 17.8 / 17.7, 61.0 / 63.4
//   four (512 keys): 9.6 / 9.1, 25.0 / 23.0, 88.0 / 87.3
// It does not depend on how many problems there are: a row's bits must not. (The last, single tile of an odd number of them was
// tried too: a gain of 3 % at head dim 64, a loss of up to 24 % at 128, where the kernel then spills.)
template <int D, bool kCausal, bool kFp16, bool kMask>
int launch_fwd(const Problem& p) {
  if constexpr (kCausal) {  // (a problem of one Q tile has one key tile)
    return launch_fwd_s<D, kCausal, kFp16, kMask, false, RowStore::kOwn>(p);
  } else {
    constexpr int kAlone = (D == 128 && !kMask) ? 2 * kTileRows : kTileRows;  // keys up to which one group takes them all
    if (p.t_q <= kTileRows && p.t_k > kAlone) return launch_fwd_rows<D, kFp16, kMask, true>(p);
    return launch_fwd_rows<D, kFp16, kMask, false>(p);
  }
}

template <int D, bool kMask>
int launch_fwd_m(const Problem& p) {
  const bool fp16 = p.dtype == LIMN_B200_F16;
  if (p.causal) return fp16 ? launch_fwd<D, true, true, kMask>(p) : launch_fwd<D, true, false, kMask>(p);
  return fp16 ? launch_fwd<D, false, true, kMask>(p) : launch_fwd<D, false, false, kMask>(p);
}

template <int D>
int launch_fwd_d(const Problem& p) {
  return p.mask ? launch_fwd_m<D, true>(p) : launch_fwd_m<D, false>(p);
}

}  // namespace

int tcgen05_fwd(const Problem& p) { return (p.hd > 64 || p.hd_v > 64) ? launch_fwd_d<128>(p) : launch_fwd_d<64>(p); }

}  // namespace limn_b200
