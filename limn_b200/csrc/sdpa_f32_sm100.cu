// float32 attention on the tensor cores: head dims up to 128, optional key mask, rectangular t_q x t_k.
//
// float32 has to keep its own width (the reference checks it at 1e-5: tests/test_attention.py:250-255), and the tensor
// cores multiply 8-bit significands in bfloat16. Three of those hold a float32: x = h + m + l, each the bfloat16
// nearest to what the ones before left, 8 + 8 + 8 bits and two signs. A product of two float32 matrices is then the
// sum of six bfloat16 products, h h + (h m + m h) + (m m + h l + l h); what is left out (m l, l m, l l) is 2^-24.3 of it at
// most and 2^-27.5 in the root mean square, about float32's own rounding. The accumulator adds in float32 but truncates,
// so the six are issued smallest first, and no total stays in tensor memory for longer than one tile: every tile's
// product starts from zero and is added to the row's total in registers, rounded to nearest, as the CUDA-core kernels
// (tiled_rows.cuh) do.
//
// What bounds it: six bfloat16 products at 4096 multiply-adds a clock and SM are 683 float32 multiply-adds a clock,
// against 128 on the CUDA cores; the split, the softmax and the running totals stay there and take about as long as the
// MMAs (dQ at head dim 64, clocks a tile: row warps 2 500, MMAs 2 300, splitting warps 3 800 with the loads). Up to head dim 64, and above
// in the forward, a block's warps have roles: row warps (a row to two or four threads: softmax or dS, the split of their operand, the
// totals), splitting warps (the streamed tiles, from global memory to three pieces in shared memory) and one that issues the MMAs;
// they meet at barriers only, a block takes up to 32 items one after the other, and a tile's scores, the products of the one before
// and the split of the ones behind go on at the same time. Items of few tiles, where that has nothing to work on, go to kernels without
// roles (f32_fwd_pair_kernel, f32_bwd_wide_kernel). Measured on B200 (forward / dQ without the row dot / dK and dV, us, causal; before the
// roles; in brackets the CUDA-core kernels): 256 x 256 keys x 64: 31 / 36 / 49, 39 / 54 / 73 (120 / 170 / 217); 6 x 8192 x 32: 225 / 232 / 293, 291 /
// 288 / 388 (1 456 / 1 743 / 2 345); 64 x 1024 x 128: 120 / 214 / 269, 175 / 227 / 293 (796 / 1 105 / 1 805); 64 x 32 x 64: 6.3 / 7.0 / 8.4, 7.4 / 7.0 / 9.1
// (8.7 / 10.4 / 13.0); the row dot beside dQ 8, 5, 20 and 1.1. Against float64, O, dQ, dK and dV are closer than theirs (8192 keys x 32: O 1.4e-7 for 6.1e-7, dQ
// 3.2e-7 for 7.6e-7 in the 2-norm), and so is L (256 x 256 x 64: 2.9e-8 for 3.5e-8; rounding it once is 2.6e-8).
//
// A block owns 128 rows at a time (query rows in the forward and the dQ pass, key rows in the dK/dV pass), one row to each
// tensor-memory lane, and streams the other side in tiles of 64 rows. Operands are loaded
// with ordinary loads (the split has to pass through registers anyway), split and left in shared memory in the
// 128-byte-swizzled layout, or in tensor memory where they are held; probabilities and dS are split in registers and go to tensor
// memory as the A operand.
//
// A non-finite operand would turn up as NaN in places where float32 arithmetic gives an infinity or even a finite
// number (inf - inf in the split, inf * 0 between pieces), and one below about 2^-110 would lose its last bits. The split
// notices both, and a block that met one computes its rows again on the CUDA cores, with the code of the tiled kernels
// there. The kernels without roles leave their loops when they meet one; the others, whose warps run apart, go on to their end first and
// then do the items again (a step whose every block does, forward / dQ / dK and dV, us: 6 x 8192 x 32 1 446 / 1 970 / 2 560, the tiled kernels
// alone 1 340 / 1 790 / 2 410; one row to a warp took 57 900 / 52 000 / 59 500). Going through an item's barriers without its work, once it is
// known to be done again, took 1 341 us in the forward, and 3 to 10 % more in calls with ordinary operands: more code in the loops.
#include <algorithm>
#include <cmath>
#include <cstdint>

#include "common.h"
#include "sm100_ptx.cuh"
#include "tiled_rows.cuh"

namespace limn_b200 {
namespace {

using namespace ptx;

constexpr int kRows = 128;    // rows a block owns
constexpr int kStream = 64;   // rows of a streamed tile
constexpr unsigned kFull = 0xffffffffu;
// dS goes to the tensor cores this much larger: its third piece is then a bfloat16 wherever dS is a float32, however small
// the gradients (an overflow shows in the split or in the sums, which are divided by it again).
constexpr float kDsUp = 65536.f;
constexpr int kPieceCols = kStream / 2;  // tensor-memory columns of one 16-bit piece of a (kRows x kStream) matrix

struct Params {
  const float *q, *k, *v, *mask, *dout, *lse_in, *delta;
  float *out, *lse_out, *dq, *dk, *dv;
  unsigned* status;
  long long bh;
  int slots, group;  // row tiles per problem; problems scheduled side by side
  int t_q, t_k, hd, hd_v, causal;
  float scale, ds_scale, c_hi, c_lo;  // ds_scale = scale * kDsUp; c_hi + c_lo = scale * log2(e), c_lo > 0
  bool wide_out;  // the results take 16-byte stores
};

// ---- x = h + m + l for two floats at a time ----
// What an operand's split shows. Of a float32 of ordinary size the second remainder has eight bits at most and is its own
// third piece, so the low half of its word is zero. It is not for an infinity or a NaN (the remainder is the NaN 0x7fffffff) and for
// a number so small (below about 2^-110) that pieces fall under bfloat16's 2^-133 and bits would be lost. Weights (P and dS) are
// not looked at one by one: one that is not finite makes a NaN of its row's sums, where it is noticed.
struct Check {
  uint32_t words = 0;  // all second remainders of operands
  bool sums = false;   // a sum was not finite
  __device__ __forceinline__ bool bad() const { return (words & 0xffffu) != 0u || sums; }
};
// The middle piece is left as -m, the way the subtractions give it, and the products with one of it turn its sign round
// (piece_minus). Both remainders are exact. Eight clocks a pair and scheduler; with the pieces unpacked to float32 and a packed FMA
// for each remainder it was eleven.
template <bool kOperand>
__device__ __forceinline__ void split_pair(uint64_t x, uint32_t& h, uint32_t& m, uint32_t& l, Check& check) {
  float a, b;
  f2_unpack(x, a, b);
  h = pack_bf16(a, b);
  a = sub_bf16_lo(h, a), b = sub_bf16_hi(h, b);  // h - x
  m = pack_bf16(a, b);
  a = sub_bf16_lo(m, a), b = sub_bf16_hi(m, b);  // x - h - m
  l = pack_bf16(a, b);
  if (kOperand) check.words |= __float_as_uint(a) | __float_as_uint(b);
}

template <int N>
__device__ __forceinline__ void tmem_ld(uint32_t addr, uint32_t (&r)[N]) {
  if constexpr (N == 32) tmem_ld32(addr, r);
  else if constexpr (N == 16) tmem_ld16(addr, r);
  else tmem_ld8(addr, r);
}
template <int N>
__device__ __forceinline__ void tmem_st(uint32_t addr, const uint32_t (&r)[N]) {
  if constexpr (N == 16) tmem_st16(addr, r);
  else if constexpr (N == 8) tmem_st8(addr, r);
  else tmem_st4(addr, r);
}

// Eight consecutive floats, those from `left` on zero (they are not there). kWide: the width is a multiple of 4 and the base 16-byte
// aligned. Predicated loads over zeroed registers, in assembly so that they stay that: written as a choice between the
// loaded value and zero they became a load and a select, which waits for the load where it was issued.
template <bool kWide>
__device__ __forceinline__ void load8(float (&x)[8], const float* at, int left) {
#pragma unroll
  for (int i = 0; i < 8; i += 4) {
    if constexpr (kWide) {
      asm volatile(
          "{\n\t.reg .pred p;\n\tsetp.gt.s32 p, %5, 0;\n\t"
          "mov.f32 %0, 0f00000000;\n\tmov.f32 %1, 0f00000000;\n\tmov.f32 %2, 0f00000000;\n\tmov.f32 %3, 0f00000000;\n\t"
          "@p ld.global.v4.f32 {%0, %1, %2, %3}, [%4];\n\t}"
          : "=&f"(x[i]), "=&f"(x[i + 1]), "=&f"(x[i + 2]), "=&f"(x[i + 3])
          : "l"(at + i), "r"(left - i));
    } else {
#pragma unroll
      for (int e = i; e < i + 4; ++e)
        asm volatile("{\n\t.reg .pred p;\n\tsetp.gt.s32 p, %2, 0;\n\tmov.f32 %0, 0f00000000;\n\t@p ld.global.f32 %0, [%1];\n\t}"
                     : "=&f"(x[e])
                     : "l"(at + e), "r"(left - e));
    }
  }
}

template <bool kWide>
__device__ __forceinline__ void load8(float (&x)[8], const float* src, int row, int rows, int col, int width) {
  load8<kWide>(x, src + static_cast<long long>(row) * width + col, row < rows ? width - col : 0);
}

// Rows [first, first + R) of a (rows, width) matrix into three bfloat16 pieces in shared memory: piece p, column block a
// of 64 at dst + (p * kAtoms + a) * R * 128, 128-byte rows, 128-byte swizzle.
template <int HD, int R, int kThreads, bool kWide>
struct Stage {
  static constexpr int kAtoms = HD > 64 ? 2 : 1;
  static constexpr int kChunks = HD / 8;
  static constexpr int kTurns = R * kChunks / kThreads;
  static constexpr uint32_t kPiece = kAtoms * R * 128;
  static constexpr uint32_t kBytes = 3 * kPiece;
  static_assert(R * kChunks % kThreads == 0 || R * kChunks < kThreads, "whole turns");
  static constexpr int kLoops = kTurns > 0 ? kTurns : 1;

  float x[kLoops][8];

  __device__ __forceinline__ void load(const float* src, int first, int rows, int width) {
#pragma unroll
    for (int n = 0; n < kLoops; ++n) {
      const int e = threadIdx.x + n * kThreads;
      if (kTurns == 0 && e >= R * kChunks) break;
      load8<kWide>(x[n], src, first + e / kChunks, rows, (e % kChunks) * 8, width);
    }
  }
  __device__ __forceinline__ void store(uint32_t dst, Check& check) {
#pragma unroll
    for (int n = 0; n < kLoops; ++n) {
      const int e = threadIdx.x + n * kThreads;
      if (kTurns == 0 && e >= R * kChunks) break;
      const int r = e / kChunks, chunk = e % kChunks;
      uint32_t h[4], m[4], l[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) split_pair<true>(f2_pack(x[n][2 * i], x[n][2 * i + 1]), h[i], m[i], l[i], check);
      const uint32_t at = swizzled_piece(dst + (chunk / 8) * R * 128, r, chunk % 8);
      st_shared_v4(at, h[0], h[1], h[2], h[3]);
      st_shared_v4(at + kPiece, m[0], m[1], m[2], m[3]);
      st_shared_v4(at + 2 * kPiece, l[0], l[1], l[2], l[3]);
    }
  }
};

// The six products in the order they are added, smallest first.
__device__ __host__ constexpr int piece_a(int i) { return (0x001102 >> (4 * i)) & 0xf; }  // l h m m h h
__device__ __host__ constexpr int piece_b(int i) { return (0x010120 >> (4 * i)) & 0xf; }  // h l m h m h
__device__ __host__ constexpr bool piece_minus(int i) { return (piece_a(i) == 1) != (piece_b(i) == 1); }

// D (kRows x kStream) = A (kRows x HD) B^T (kStream x HD), both with the contraction dim contiguous. A lies in shared
// memory (a0 its address) or in tensor memory (a0 its column, pieces HD / 2 columns apart). Columns past the head dim are
// zero on both sides. Fully unrolled over compile-time offsets: one thread issues every MMA of the block, and with a
// loop over the steps it took 115 clocks an MMA instead of the 32 the tensor cores need.
// kTwo: the last half of the largest products goes to a second accumulator, kStream columns of it at d2, so that a score
// takes no more than four truncated additions at its full size at head dim 128 either.
template <int HD, bool kTmemA, bool kTwo = false>
__device__ __forceinline__ void issue_scores(uint32_t d, uint32_t a0, uint32_t b0, uint32_t d2 = 0) {
  constexpr uint32_t kPieceA = (HD > 64 ? 2 : 1) * kRows * 128, kPieceB = (HD > 64 ? 2 : 1) * kStream * 128;
  const uint32_t a_lo = kTmemA ? a0 : desc_lo(a0, 0), b_lo = desc_lo(b0, 0);
#pragma unroll
  for (int i = 0; i < 6; ++i) {
    const uint32_t idesc = mma_idesc(kRows, kStream, false, false, false, piece_minus(i));
#pragma unroll
    for (int s = 0; s < HD / 16; ++s) {
      const uint32_t b = b_lo + piece_b(i) * (kPieceB / 16) + (s / 4) * (kStream * 128 / 16) + (s % 4) * 2;
      const bool second = kTwo && i == 5 && s >= HD / 32;
      const bool starts = (i == 0 && s == 0) || (second && s == HD / 32);
      const uint32_t to = second ? d2 : d;
      if constexpr (kTmemA) {
        mma_ts_lo(to, a_lo + piece_a(i) * (HD / 2) + s * 8, b, idesc, starts ? 0u : 1u);
      } else {
        const uint32_t a = a_lo + piece_a(i) * (kPieceA / 16) + (s / 4) * (kRows * 128 / 16) + (s % 4) * 2;
        if (starts) mma_ss_lo<false>(to, a, b, idesc);
        else mma_ss_lo<true>(to, a, b, idesc);
      }
    }
  }
}

// D (kRows x HD) = W (kRows x kStream, pieces in tensor memory) X (kStream x HD, rows streamed).
template <int HD>
__device__ __forceinline__ void issue_weigh(uint32_t d, uint32_t w0, uint32_t x0) {
  constexpr uint32_t kPiece = (HD > 64 ? 2 : 1) * kStream * 128;
  const uint32_t x_lo = desc_lo(x0, kStream * 128);
#pragma unroll
  for (int i = 0; i < 6; ++i) {
    const uint32_t idesc = mma_idesc(kRows, HD, false, false, true, piece_minus(i));
#pragma unroll
    for (int s = 0; s < kStream / 16; ++s)
      mma_ts_lo(d, w0 + piece_a(i) * kPieceCols + s * 8, x_lo + piece_b(i) * (kPiece / 16) + s * (16 * 128 / 16), idesc, i > 0 || s > 0);
  }
}

// N numbers of one row, split, to tensor memory at `at` (pieces kPieceCols columns apart).
template <int N>
__device__ __forceinline__ void hand_over(uint32_t at, const uint64_t (&w)[N / 2]) {
  uint32_t h[N / 2], m[N / 2], l[N / 2];
  Check none;
#pragma unroll
  for (int i = 0; i < N / 2; ++i) split_pair<false>(w[i], h[i], m[i], l[i], none);
  tmem_st<N / 2>(at, h);
  tmem_st<N / 2>(at + kPieceCols, m);
  tmem_st<N / 2>(at + 2 * kPieceCols, l);
}

// The N columns from `col` on of a warp's 32 rows from `first` on, a row to a thread, into a matrix of (rows, width), rows exchanged
// for pieces (a block's 128 x 64 results took 2 000 to 6 000 clocks without).
template <int N>
__device__ __forceinline__ void store_rows(float* dst, const uint64_t (&acc)[N / 2], int first, int rows, int col, int width, bool wide) {
  if (first >= rows) return;  // (the whole warp; dK and dV of 700 problems of 16 x 72 59.4 us without, 58.1 with it)
  const int lane = static_cast<int>(lane_id());
  if (wide) {
    constexpr int B = N / 4 < 4 ? N / 4 : 4;
    const int top = first + (lane & ~(B - 1)), at = col + 4 * (lane & (B - 1));
#pragma unroll
    for (int set = 0; set < N / 4; set += B) {
      uint32_t x[B][4];
#pragma unroll
      for (int i = 0; i < B; ++i)
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          float a, b;
          f2_unpack(acc[2 * (set + i) + c], a, b);
          x[i][2 * c] = __float_as_uint(a), x[i][2 * c + 1] = __float_as_uint(b);
        }
      swap_rows_for_pieces<B>(x);
#pragma unroll
      for (int r = 0; r < B; ++r)
        if (top + r < rows && at + 4 * set < width)
          *reinterpret_cast<uint4*>(dst + static_cast<long long>(top + r) * width + at + 4 * set) = make_uint4(x[r][0], x[r][1], x[r][2], x[r][3]);
    }
  } else if (first + lane < rows) {
    float* row = dst + static_cast<long long>(first + lane) * width;
#pragma unroll
    for (int i = 0; i < N; ++i) {
      float x[2];
      f2_unpack(acc[i / 2], x[0], x[1]);
      if (col + i < width) row[col + i] = x[i & 1];
    }
  }
}

// ---- the rows of a block whose operands do not split, on the CUDA cores (tiled_rows.cuh): each 256 threads of the block
// take 64 rows at a time. Streamed tiles are as long as the block's shared memory allows for all its groups together. ----
template <int HD, Op kOp, int kGroups, uint32_t kBytes>
constexpr int again_tile() {
  constexpr uint32_t kShare = kBytes / kGroups & ~15u;
  if (HD <= 64 && tiled::shared_bytes<HD, 64>(kOp) <= kShare) return 64;
  if (tiled::shared_bytes<HD, 32>(kOp) <= kShare) return 32;
  return 16;
}
template <int HD, Op kOp, int kGroups, uint32_t kBytes, bool kWide>
__device__ __noinline__ void rows_again(const Params& g, long long b, int first, unsigned char* shared) {
  constexpr int BN = again_tile<HD, kOp, kGroups, kBytes>();
  constexpr uint32_t kShare = kBytes / kGroups & ~15u;
  static_assert(tiled::shared_bytes<HD, BN>(kOp) <= kShare, "shared memory");
  tiled::Args a = {};
  a.q = g.q, a.k = g.k, a.v = g.v, a.mask = g.mask, a.dout = g.dout, a.lse_in = g.lse_in, a.delta = g.delta;
  a.out = g.out, a.dq = g.dq, a.dk = g.dk, a.dv = g.dv, a.lse_out = g.lse_out;
  a.t_q = g.t_q, a.t_k = g.t_k, a.hd = g.hd, a.hd_v = g.hd_v, a.causal = g.causal, a.scale = g.scale;
  a.wide_qk = a.wide_v = kWide;
  const int group = threadIdx.x / tiled::kThreads, thread = threadIdx.x % tiled::kThreads;
  float* mine = reinterpret_cast<float*>(shared + group * kShare);
  auto sync = [group] { asm volatile("bar.sync %0, %1;" ::"r"(1 + group), "n"(tiled::kThreads) : "memory"); };
  const int owned = kOp == Op::BwdKV ? g.t_k : g.t_q;
  for (int at = first + group * tiled::kBM; at < min(first + kRows, owned); at += kGroups * tiled::kBM) {
    if constexpr (kOp == Op::Fwd) tiled::fwd_rows<float, HD, BN>(a, b, at, mine, thread, sync);
    else if constexpr (kOp == Op::BwdQ) tiled::bwd_q_rows<float, HD, BN>(a, b, at, mine, thread, sync);
    else tiled::bwd_kv_rows<float, HD, BN>(a, b, at, mine, thread, sync);
    sync();  // its shared memory has been read
  }
}

// ---- block set-up (of the kernels without roles) and teardown ----
// False: an earlier kernel on this device gave up on a wait, take no work. Every barrier expects one arrival.
template <int kCols, int kBars>
__device__ __forceinline__ bool set_up(const Params& g, uint32_t* slot, uint32_t* abort_flag, uint64_t* bars, uint32_t& tmem) {
  if (threadIdx.x == 0) {
#pragma unroll
    for (int i = 0; i < kBars; ++i) mbar_init(smem_addr(bars + i), 1);
    mbar_init_fence();
  }
  grid_dependency_wait();
  if (threadIdx.x == 0) *abort_flag = *reinterpret_cast<volatile unsigned*>(g.status) != kStatusOk;
  __syncthreads();
  if (*abort_flag) return false;
  if (threadIdx.x < 32) {
    tmem_alloc(smem_addr(slot), kCols);
    tmem_relinquish();
    tc_fence_before_sync();
  }
  __syncthreads();
  tc_fence_after_sync();
  grid_launch_dependents();
  tmem = __shfl_sync(kFull, *slot, 0);
  return true;
}
template <int kCols, int kWarp = 0>
__device__ __forceinline__ void tear_down(const Params& g, uint32_t tmem) {
  tc_fence_before_sync();
  __syncthreads();
  if (threadIdx.x / 32 == kWarp) {
    if (*reinterpret_cast<volatile unsigned*>(g.status) != kStatusOk) {
      // a wait gave up somewhere: give MMAs still in flight time to land before their memory is released
      for (int i = 0; i < 2000; ++i) __nanosleep(1000);
    }
    tc_fence_after_sync();
    tmem_free(tmem, kCols);
  }
}

// One float a row of the tile that starts at j0, zero beyond the end: thread i < kStream has row i's.
__device__ __forceinline__ float row_value(const float* from, int j0, int rows, int thread = threadIdx.x) {
  const int j = j0 + thread;
  float x;  // (as in load8: nothing waits for it here)
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %2, 0;\n\tmov.f32 %0, 0f00000000;\n\t@p ld.global.f32 %0, [%1];\n\t}"
               : "=&f"(x)
               : "l"(from + j), "r"(thread < kStream && j < rows ? 1u : 0u));
  return x;
}
// The hidden keys of a tile (flag 0, keys past the end among them) as two words in shared memory, bit set = hidden.
__device__ __forceinline__ void post_hidden(uint32_t* words, float flag, int thread = threadIdx.x) {
  if (thread < kStream) {
    const unsigned hid = __ballot_sync(kFull, flag == 0.f);
    if ((thread & 31) == 0) words[thread >> 5] = hid;
  }
}
// ... and the part of them a thread with columns [group * N, group * N + N) needs.
template <int N>
__device__ __forceinline__ uint32_t my_hidden(const uint32_t* words, int group) {
  if constexpr (N == 32) return words[group];
  else return words[group >> 1] >> (16 * (group & 1));
}

__device__ __forceinline__ uint32_t align_1024(uint32_t addr) { return (addr + 1023u) & ~1023u; }

// log2(e) in two parts: minus a log-sum-exp in log2 units, as hi + lo
__device__ __forceinline__ void to_minus_log2(const float lse, float& hi, float& lo) {
  constexpr float kHi = 1.44269502f, kLo = 1.92596303e-8f;
  hi = -(lse * kHi);
  lo = -(fmaf(lse, kHi, hi) + lse * kLo);
}

// What both backward kernels do with the scores of a row: P = 2^(s c - L), kDsUp dS = P (dP - delta) scale kDsUp, 0 where
// unseen.
// `hi`, `lo`, `delta` give minus a column's L (in log2 units) and minus its delta; a row's own ones repeated in the dQ pass.
template <int CW, typename Columns>
__device__ __forceinline__ void weigh_scores(const Params& g, const uint32_t (&s)[CW], const uint32_t (&dp)[CW], uint32_t unseen,
                                             Columns columns, uint64_t (&p)[CW / 2], uint64_t (&ds)[CW / 2]) {
  const uint64_t c_hi = f2_pack(g.c_hi, g.c_hi), c_lo = f2_pack(g.c_lo, g.c_lo), scale = f2_pack(g.ds_scale, g.ds_scale);
#pragma unroll
  for (int c = 0; c < CW / 2; ++c) {
    uint64_t hi, lo, delta;
    columns(2 * c, hi, lo, delta);
    const uint64_t s2 = f2_pack_bits(s[2 * c], s[2 * c + 1]);
    const uint64_t x = f2_add(f2_fma(s2, c_hi, hi), f2_fma(s2, c_lo, lo));
    float a, b;
    f2_unpack(x, a, b);
    p[c] = f2_pack(exp2_approx(a), exp2_approx(b));
    ds[c] = f2_mul(f2_mul(p[c], f2_add(delta, f2_pack_bits(dp[2 * c], dp[2 * c + 1]))), scale);
  }
  if (unseen != 0u) {  // (dS too: delta of a row with no key is NaN)
#pragma unroll
    for (int c = 0; c < CW / 2; ++c) {
      float a, b;
      f2_unpack(p[c], a, b);
      p[c] = f2_pack((unseen >> (2 * c)) & 1u ? 0.f : a, (unseen >> (2 * c + 1)) & 1u ? 0.f : b);
      f2_unpack(ds[c], a, b);
      ds[c] = f2_pack((unseen >> (2 * c)) & 1u ? 0.f : a, (unseen >> (2 * c + 1)) & 1u ? 0.f : b);
    }
  }
}

// The sums over dS at their own size again, and whether they are finite: one is not where one of them overflowed at kDsUp times
// its size, and a whole row is not where a P or a dS of it was not (dS is P times something, and the products of a piece that is
// infinite are infinite or NaN for every column).
template <int N>
__device__ __forceinline__ void settle(uint64_t (&acc)[N], Check& check) {
  uint64_t zero = 0;
#pragma unroll
  for (int c = 0; c < N; ++c) {
    zero = f2_fma(acc[c], 0ull, zero);
    acc[c] = f2_mul(acc[c], f2_pack(1.f / kDsUp, 1.f / kDsUp));
  }
  float a, b;
  f2_unpack(zero, a, b);
  check.sums |= !(a == 0.f && b == 0.f);
}

// The columns of a thread's CW that its row does not see: outside [from, to), as bits.
template <int CW>
__device__ __forceinline__ uint32_t outside(int from, int to) {
  uint32_t unseen = 0;
  if (from > 0) unseen |= from >= CW ? kFull : (1u << from) - 1u;
  if (to < CW) unseen |= to <= 0 ? kFull : ~((1u << to) - 1u);
  return unseen;
}

// ---- the kernels that work in roles: row warps, splitting warps, one issuing warp ----
// Two or four row threads to a row take scores out of tensor memory, turn them into weights, split those and sum a tile's products; the
// splitting warps bring the streamed operands into shared memory in pieces, a few tiles ahead; the issuing warp issues every MMA.
// The roles meet at mbarriers whose waits are bounded; no barrier of the block stands inside their loops, so a warp that gave up on a
// wait cannot hang the others. A block goes through several work items: the splitting warps run ahead into the next item while the
// row warps end this one.
template <int kGroups>
struct Roles {  // kGroups threads to a row, the other warps by what registers are left
  static constexpr int kRowWarps = 4 * kGroups, kSplitWarps = kGroups == 4 ? 3 : 7, kIssuer = kRowWarps + kSplitWarps;
  static constexpr int kRowThreads = 32 * kRowWarps, kSplitThreads = 32 * kSplitWarps, kThreads = 32 * (kIssuer + 1);
};
constexpr int kAgainGroups = 2;                  // of tiled::kThreads of a block's threads, whatever their roles, for items done again on the CUDA cores
constexpr int kMostItems = 32;                   // work items of a block: each has a bit of a word

// Work item `k` of this block. Blocks take turns, there and back: items are in the order of their length under a causal mask, and a
// block that got a long one in one turn gets a short one in the next.
__device__ __forceinline__ bool work_item(const Params& g, int k, int& problem, int& slot) {
  const long long grid = gridDim.x, within = (k & 1) ? grid - 1 - blockIdx.x : blockIdx.x, index = k * grid + within;
  if (k >= kMostItems || index >= g.bh * g.slots) return false;
  cta_work(static_cast<int>(index), g.slots, g.bh, g.group, problem, slot);
  return true;
}

// What the splitting warps carry from global memory to pieces in shared memory, half a streamed tile (one operand) at a time, and in
// registers meanwhile: a thread that has split one of its eighths of a row loads the next half's in its place.
template <int HD, int kThreads, bool kWide>
struct Carry {
  static constexpr int kChunks = HD / 8, kStep = kThreads / kChunks;  // rows from one turn to the next
  static constexpr int kTurns = (kStream + kStep - 1) / kStep;
  static constexpr int kHalves = kTurns > 3 ? 1 : 2;  // that a thread's registers hold: with two, each operand's next tile is under way
  static constexpr uint32_t kPiece = (HD > 64 ? 2 : 1) * kStream * 128, kTile = 3 * kPiece;
  static constexpr int kPeriod = kStep % 4 == 0 ? 2 : 4;  // turns after which the swizzle is the same again
  static_assert(kThreads % kChunks == 0 && kStep % 2 == 0, "a thread keeps its columns");
  float x[kTurns][8];
  int row, column;    // of the first turn
  uint32_t where[kPeriod];  // of the turns' pieces in a tile, less the rows between them

  __device__ __forceinline__ void set_up(int thread) {
    row = thread / kChunks, column = thread % kChunks * 8;
#pragma unroll
    for (int n = 0; n < kPeriod; ++n) where[n] = swizzled_piece(column / 64 * (kStream * 128), row + n * kStep, column / 8 % 8) - n * kStep * 128;
  }
  __device__ __forceinline__ bool has(int n) const { return n * kStep + kStep <= kStream || n * kStep + row < kStream; }
  // The rows of a half that starts with row `first` of a (rows, width) matrix.
  struct Source {
    const float* at;
    int rows, width;  // rows from this thread's first one on
  };
  __device__ __forceinline__ Source source(const float* src, int first, int rows, int width) const {
    return {src + static_cast<long long>(first + row) * width + column, rows - first - row, width};
  }
  __device__ __forceinline__ void load(int n, const Source& s) {
    if (has(n)) load8<kWide>(x[n], s.at + n * kStep * s.width, n * kStep < s.rows ? s.width - column : 0);
  }
  __device__ __forceinline__ void load_all(const Source& s) {
#pragma unroll
    for (int n = 0; n < kTurns; ++n) load(n, s);
  }
  // This half to the tile at dst, the next one's rows to registers.
  __device__ __forceinline__ void store_and_load(uint32_t dst, Check& check, const Source& next) {
#pragma unroll
    for (int n = 0; n < kTurns; ++n) {
      if (has(n)) {  // (whole warps have it or not)
        uint32_t h[4], m[4], l[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) split_pair<true>(f2_pack(x[n][2 * i], x[n][2 * i + 1]), h[i], m[i], l[i], check);
        const uint32_t to = dst + where[n % kPeriod] + n * kStep * 128;
        st_shared_v4(to, h[0], h[1], h[2], h[3]);
        st_shared_v4(to + kPiece, m[0], m[1], m[2], m[3]);
        st_shared_v4(to + 2 * kPiece, l[0], l[1], l[2], l[3]);
        load(n, next);
      }
    }
  }
};

__device__ __forceinline__ void warp_arrives(uint32_t bar) {
  __syncwarp();
  if (lane_id() == 0) mbar_arrive(bar);
}
// Every lane waits, and the warp goes on together: false for all of it if one of them gave up. The case that the barrier is through is
// four instructions. kCall: the other one is a call (6 x 8192 x 32 causal: the dQ pass 236 us with calls and 252 without, the
// forward 250 and 238).
__device__ __noinline__ bool warp_waits_on(uint32_t bar, uint32_t parity, unsigned* status, unsigned tag) {
  return __all_sync(kFull, mbar_wait(bar, parity, status, tag));
}
template <bool kCall>
__device__ __forceinline__ bool warp_waits(uint32_t bar, uint32_t parity, unsigned* status, unsigned tag) {
  uint32_t through;
  asm volatile(
      "{\n\t"
      ".reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "vote.sync.all.pred p, p, 0xffffffff;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t"
      "}\n"
      : "=r"(through)
      : "r"(bar), "r"(parity)
      : "memory");
  if (through != 0) return true;
  return kCall ? warp_waits_on(bar, parity, status, tag) : __all_sync(kFull, mbar_wait(bar, parity, status, tag)) != 0;
}

// 16 bytes (4, where rows are not whole 16-byte pieces) from global to shared memory without registers; zero where `left` <= 0.
template <bool kWide>
__device__ __forceinline__ void copy_async16(uint32_t dst, const float* src, int left) {
  if constexpr (kWide) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(left > 0 ? 16 : 0) : "memory");
  } else {
#pragma unroll
    for (int i = 0; i < 4; ++i)
      asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst + 4 * i), "l"(left > i ? src + i : src), "r"(left > i ? 4 : 0) : "memory");
  }
}
__device__ __forceinline__ void copy_async_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// Where a row warp's part of a held operand (its 32 rows, its group's OW columns) waits, as float32, for its turn in tensor
// memory: only that warp touches it. 16-byte piece p of row r; eight rows' pieces lie on distinct banks.
template <int OW>
__device__ __forceinline__ uint32_t held_piece(uint32_t at, int r, int p) {
  constexpr int kPieces = OW / 4;  // of a row
  static_assert(kPieces == 8 || kPieces == 4 || kPieces == 2, "a row's part is 32 to 128 bytes");
  const int where = kPieces == 8 ? p ^ (r & 7) : kPieces == 4 ? p ^ ((r >> 1) & 3) : p ^ ((r >> 2) & 1);
  return at + static_cast<uint32_t>(r * kPieces + where) * 16u;
}
template <int OW, bool kWide>
__device__ __forceinline__ void fetch_held(uint32_t at, const float* src, int first, int rows, int col, int width) {
  constexpr int kPieces = OW / 4;
  const int lane = static_cast<int>(lane_id());
#pragma unroll
  for (int n = 0; n < kPieces; ++n) {
    const int e = lane + 32 * n, r = e / kPieces, p = e % kPieces;
    const bool there = first + r < rows;
    const int c = col + 4 * p;
    copy_async16<kWide>(held_piece<OW>(at, r, p), there && c < width ? src + static_cast<long long>(first + r) * width + c : src, there ? width - c : 0);
  }
}
// ... and from there, split, to this thread's lane of tensor memory at column `to` (pieces HD / 2 columns apart).
template <int HD, int OW>
__device__ __forceinline__ void place_held(uint32_t to, uint32_t at, Check& check) {
  const int lane = static_cast<int>(lane_id());
#pragma unroll
  for (int c = 0; c < OW; c += OW < 16 ? OW : 16) {  // (16 columns at a time)
    constexpr int N = OW < 16 ? OW : 16;
    float x[N];
#pragma unroll
    for (int p = 0; p < N / 4; ++p)
      asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
                   : "=f"(x[4 * p]), "=f"(x[4 * p + 1]), "=f"(x[4 * p + 2]), "=f"(x[4 * p + 3])
                   : "r"(held_piece<OW>(at, lane, c / 4 + p)) : "memory");
    uint32_t h[N / 2], m[N / 2], l[N / 2];
#pragma unroll
    for (int e = 0; e < N / 2; ++e) split_pair<true>(f2_pack(x[2 * e], x[2 * e + 1]), h[e], m[e], l[e], check);
    if constexpr (N == 16) {
      tmem_st8(to + c / 2, h), tmem_st8(to + c / 2 + HD / 2, m), tmem_st8(to + c / 2 + HD, l);
    } else {
      tmem_st4(to + c / 2, h), tmem_st4(to + c / 2 + HD / 2, m), tmem_st4(to + c / 2 + HD, l);
    }
  }
}

// A work item: `tiles` tiles of the streamed rows from `begin` on for the own rows from `first` on of problem b.
struct Item {
  long long b;
  int first, begin, tiles;
};

// The barriers the roles meet at come in rings of kRing, tile t's at t % kRing: whoever waits for a tile's is never more than a round
// behind. What has to be there for a bunch of MMAs arrives on one barrier, whoever brings it: the issuing warp's waits are time in
// which the tensor cores run dry (their queue is six MMAs, 200 clocks, and filling it again takes as long).
constexpr int kRing = 4;
__device__ __forceinline__ uint32_t ring_bar(uint32_t first, int t) { return first + 8 * (static_cast<uint32_t>(t) % kRing); }
__device__ __forceinline__ uint32_t ring_parity(int t) { return static_cast<uint32_t>(t) / kRing & 1u; }

// The splitting warps' way through a block's items: tile after tile of the two streamed operands into the places of theirs (consecutive
// ones from tiles0 and tiles1 on). The place of operand r is free again when the tile that had it has arrived at the ring free_r; a
// tile there is an arrival at the ring there_r. `carry` holds the first half already. load_rows(item, row) fetches what goes with a
// tile's rows, post_rows(tile) leaves it in shared memory before the first operand is there. Returns the items in which something does not
// split.
template <int HD, int kThreads, bool kWide, int kPlaces0, int kPlaces1, bool kCall, typename Items, typename Source0, typename Source1, typename LoadRows, typename PostRows>
__device__ __forceinline__ uint32_t split_streams(Carry<HD, kThreads, kWide> (&carry)[Carry<HD, kThreads, kWide>::kHalves], Item it, bool more, Items item, Source0 stream0, Source1 stream1, int streamed, int width0,
                                                  int width1, uint32_t free0, uint32_t free1, uint32_t there0, uint32_t there1, uint32_t tiles0,
                                                  uint32_t tiles1, unsigned* status, bool& ok, LoadRows load_rows, PostRows post_rows) {
  static_assert(kPlaces0 <= kRing && kPlaces1 <= kRing, "a barrier for each");
  constexpr uint32_t kTile = Carry<HD, kThreads, kWide>::kTile;
  constexpr bool kDeep = Carry<HD, kThreads, kWide>::kHalves == 2;
  uint32_t again = 0;
  int t = 0;
  if (more) load_rows(it, it.begin);
  for (int k = 0; ok && more; ++k) {
    Check check;
    Item next = it;
    more = item(k + 1, next);
    for (int j = 0; j < it.tiles; ++j, ++t) {
      const int x0 = it.begin + j * kStream, place0 = t % kPlaces0, place1 = t % kPlaces1;
      if (t >= kPlaces0) ok = ok && warp_waits<kCall>(ring_bar(free0, t - kPlaces0), ring_parity(t - kPlaces0), status, 0x0b30u);
      if (!ok) break;
      post_rows(t);
      const bool last = j + 1 == it.tiles;
      const Item& then = last ? next : it;
      const int x1 = last ? next.begin : x0 + kStream, rows = last && !more ? 0 : streamed;  // 0: nothing left to load
      if constexpr (kDeep) carry[0].store_and_load(tiles0 + place0 * kTile, check, carry[0].source(stream0(then), x1, rows, width0));
      else carry[0].store_and_load(tiles0 + place0 * kTile, check, carry[0].source(stream1(it), x0, streamed, width1));
      fence_async_shared();
      warp_arrives(ring_bar(there0, t));
      if (t >= kPlaces1) ok = ok && warp_waits<kCall>(ring_bar(free1, t - kPlaces1), ring_parity(t - kPlaces1), status, 0x0b31u);
      if (!ok) break;
      if (rows > 0) load_rows(then, x1);
      if constexpr (kDeep) carry[1].store_and_load(tiles1 + place1 * kTile, check, carry[1].source(stream1(then), x1, rows, width1));
      else carry[0].store_and_load(tiles1 + place1 * kTile, check, carry[0].source(stream0(then), x1, rows, width0));
      fence_async_shared();
      warp_arrives(ring_bar(there1, t));
    }
    if (check.bad()) again |= 1u << k;
    it = next;
  }
  return again;
}

// The same with one place for each operand, the next tile's first operand before this tile's second: its place is free as soon as the
// tile has been scored, the other's only when the tile before it has been weighed. (The order of the other function would leave the
// tensor cores waiting for both.)
template <int HD, int kThreads, bool kWide, bool kCall, typename Items, typename Source0, typename Source1, typename LoadRows, typename PostRows>
__device__ __forceinline__ uint32_t split_streams_one(Carry<HD, kThreads, kWide>& carry, const Item& start, bool any, Items item, Source0 stream0, Source1 stream1, int streamed,
                                                      int width0, int width1, uint32_t free0, uint32_t free1, uint32_t there0, uint32_t there1, uint32_t tile0,
                                                      uint32_t tile1, unsigned* status, bool& ok, LoadRows load_rows, PostRows post_rows) {
  struct Cursor {
    Item it;
    int k, j;
    bool there;
  };
  auto advance = [&](Cursor& c) {
    if (++c.j < c.it.tiles) return;
    c.j = 0;
    c.there = item(++c.k, c.it);
  };
  auto first_row = [](const Cursor& c) { return c.it.begin + c.j * kStream; };
  uint32_t again = 0;
  Cursor a = {start, 0, 0, any}, b = a;  // the tile whose first operand is due, and the one before it
  if (any) load_rows(a.it, first_row(a));
  for (int t = 0; ok && (a.there || t > 0); ++t) {
    Cursor next = a;
    if (a.there) {
      advance(next);
      if (t > 0) ok = warp_waits<kCall>(ring_bar(free0, t - 1), ring_parity(t - 1), status, 0x0b30u);
      if (!ok) break;
      post_rows(t);
      if (next.there) load_rows(next.it, first_row(next));
      Check check;
      if (t > 0) carry.store_and_load(tile0, check, carry.source(stream1(b.it), first_row(b), streamed, width1));
      else carry.store_and_load(tile0, check, next.there ? carry.source(stream0(next.it), first_row(next), streamed, width0) : carry.source(stream1(a.it), first_row(a), streamed, width1));
      fence_async_shared();
      warp_arrives(ring_bar(there0, t));
      if (check.bad()) again |= 1u << a.k;
    }
    if (t > 0) {
      if (t > 1) ok = warp_waits<kCall>(ring_bar(free1, t - 2), ring_parity(t - 2), status, 0x0b31u);
      if (!ok) break;
      Check check;
      carry.store_and_load(tile1, check, next.there ? carry.source(stream0(next.it), first_row(next), streamed, width0) : carry.source(stream1(a.it), first_row(a), a.there ? streamed : 0, width1));
      fence_async_shared();
      warp_arrives(ring_bar(there1, t - 1));
      if (check.bad()) again |= 1u << b.k;
    }
    if (!a.there) break;
    b = a, a = next;
  }
  return again;
}

// A row's share of its columns by the row's total (tiled_rows.cuh says how, and when that is exact): a warp with a row of another kind
// divides. A division by itself is a chain with a branch for each column, and a column of zeros, as a width below the kernel's has
// them, takes its slow side. Measured, a division a column -> so: 256 x 256 x 64 causal 33.9 -> 31.4 us, 64 x 1024 x 128 127 -> 121, 2048 x 128 x 40
// 123.8 -> 78.2, 2048 x 192 x 100 512 -> 398, 6 x 8192 x 32 225 either way.
template <int N>
__device__ __forceinline__ void divide_row(uint64_t (&x)[N], float total) {
  float largest = 0.f;
#pragma unroll
  for (int c = 0; c < N; ++c) {
    float x0, x1;
    f2_unpack(x[c], x0, x1);
    largest = max3(largest, fabsf(x0), fabsf(x1));
  }
  if (__all_sync(kFull, tiled::by_reciprocal(largest, total))) {
    constexpr float kUp = tiled::kQuotientUp;
    const float r = __frcp_rn(total);
    const uint64_t first = f2_pack(r * kUp, r * kUp), less = f2_pack(-r, -r), total2 = f2_pack(total, total), up = f2_pack(-kUp, -kUp), down = f2_pack(1.f / kUp, 1.f / kUp);
#pragma unroll
    for (int c = 0; c < N; ++c) {
      const uint64_t minus_x = f2_mul(x[c], up);
      uint64_t q = f2_mul(x[c], first);
      q = f2_fma(f2_fma(q, total2, minus_x), less, q);
      x[c] = f2_mul(f2_fma(f2_fma(q, total2, minus_x), less, q), down);
    }
  } else {
#pragma unroll
    for (int c = 0; c < N; ++c) {
      float x0, x1;
      f2_unpack(x[c], x0, x1);
      x[c] = f2_pack(x0 / total, x1 / total);
    }
  }
}

// ---- forward ----
template <int HD>
struct Fwd {
  // tensor memory: scores (above head dim 64 in two parts, see issue_scores), the pieces of P, a tile's product, and the pieces of Q
  // where there is room
  static constexpr bool kTwo = HD > 64, kHeldT = HD <= 64;
  static constexpr uint32_t kS = 0, kS2 = kStream, kP = kTwo ? 2 * kStream : kStream, kO = kP + 3 * kPieceCols, kHeldCol = kO + HD;
  static constexpr int kCols = 512;
  static_assert(kHeldCol + (kHeldT ? 3 * HD / 2 : 0) <= kCols, "tensor memory");
  // Threads to a row: eight row warps and seven splitting ones. With sixteen and three, 256 x 512 x 64 takes 125 us for 105, 6 x 8192 x 32
  // causal 237 for 225: what a warp spends on a tile whatever its width, and on the row maxima, is spent half as often.
  static constexpr int kGroups = 2;
  static constexpr int kShares = HD > 64 ? 2 : 1;  // of a thread in its row's denominator: sums of 16 columns above head dim 64 (0.6 % nearer to float64), of 32 below
  static constexpr int kPlaces0 = HD > 64 ? 1 : 3, kPlaces1 = HD > 64 ? 1 : 3;  // of K and of V
  static constexpr uint32_t kTile = 3 * (HD > 64 ? 2 : 1) * kStream * 128;
  static constexpr uint32_t kHeldPiece = (HD > 64 ? 2 : 1) * kRows * 128;
  static constexpr uint32_t kTile0 = 0, kTile1 = kPlaces0 * kTile, kHeld = kTile1 + kPlaces1 * kTile;
  static constexpr uint32_t kBytes = kHeld + (kHeldT ? kRows * HD * 4 : 3 * kHeldPiece) + 1024;
};

template <int HD, bool kWide>
__global__ void __launch_bounds__(Roles<Fwd<HD>::kGroups>::kThreads, 1) f32_fwd_kernel(const __grid_constant__ Params g) {
  using L = Fwd<HD>;
  using W = Roles<L::kGroups>;
  constexpr int G = L::kGroups, CW = kStream / G, OW = HD / G;
  extern __shared__ __align__(16) unsigned char raw[];
  // A tile's hidden keys come with K, whose place is free again when the tile has been scored, before the row warps are done with it:
  // they have twice as many places (five would do: the row warps are in the tile after next by then).
  constexpr int kHiddenPlaces = 2 * kRing;
  __shared__ uint32_t slot, abort_flag, again_all, hidden[kHiddenPlaces][2];
  // kGo: a tile can be scored (its K is there, the scores before it have been read, Q is there). kReady: it can be weighed (P is there,
  // V is there). kScored, kWeighed: the tensor cores have done it.
  enum { kGo = 0, kReady = kRing, kScored = 2 * kRing, kWeighed = 3 * kRing, kBars = 4 * kRing };
  __shared__ __align__(8) uint64_t bars[kBars];
  __shared__ float exchange[2][G * L::kShares][kRows];
  const int warp = __shfl_sync(kFull, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
#pragma unroll
    for (int i = 0; i < kBars; ++i)
      mbar_init(smem_addr(bars + i), i < kScored ? W::kRowWarps + W::kSplitWarps : 1);
    mbar_init_fence();
    again_all = 0;
  }
  auto place = [](int t, int places) { return t % places; };
  auto ring = [&](int which, int t) { return ring_bar(smem_addr(bars + which), t); };
  const uint32_t base = align_1024(smem_addr(raw));
  auto tile0_at = [&](int t) { return base + L::kTile0 + place(t, L::kPlaces0) * L::kTile; };
  auto tile1_at = [&](int t) { return base + L::kTile1 + place(t, L::kPlaces1) * L::kTile; };
  auto item = [&](int k, Item& it) {
    int problem = 0, at = 0;
    if (!work_item(g, k, problem, at)) return false;
    it.b = problem;
    it.first = (g.slots - 1 - at) * kRows;  // long causal rows first
    it.begin = 0;
    it.tiles = ((g.causal ? min(g.t_k, it.first + kRows) : g.t_k) + kStream - 1) / kStream;
    return true;
  };
  const int group = warp >> 2, quarter = warp & 3, row = quarter * 32 + lane;
  const uint32_t raw_q = base + L::kHeld + warp * (32 * OW * 4);
  auto fetch = [&](const Item& it) {
    if constexpr (L::kHeldT) fetch_held<OW, kWide>(raw_q, g.q + it.b * g.t_q * g.hd, it.first + quarter * 32, g.t_q, group * OW, g.hd);
  };
  auto keys = [&](const Item& it) { return g.k + it.b * g.t_k * g.hd; };
  auto values = [&](const Item& it) { return g.v + it.b * g.t_k * g.hd_v; };

  Item it;
  const bool any = item(0, it);
  grid_dependency_wait();
  if (warp == W::kIssuer) {
    tmem_alloc(smem_addr(&slot), L::kCols);
    tmem_relinquish();
  }
  if (threadIdx.x == 0) abort_flag = *reinterpret_cast<volatile unsigned*>(g.status) != kStatusOk;
  // the first operands set out before the block is set up
  using Carried = Carry<HD, W::kSplitThreads, kWide>;
  Carried carry[Carried::kHalves];
#pragma unroll
  for (int h = 0; h < Carried::kHalves; ++h) carry[h].set_up(threadIdx.x - W::kRowThreads);
  if (any && warp < W::kRowWarps) {
    fetch(it);
  } else if (any && warp < W::kIssuer) {
    carry[0].load_all(carry[0].source(keys(it), 0, g.t_k, g.hd));
    if (Carried::kHalves > 1) carry[Carried::kHalves - 1].load_all(carry[0].source(values(it), 0, g.t_k, g.hd_v));
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem = __shfl_sync(kFull, slot, 0);
  bool ok = true;
  uint32_t again = 0;  // items in which this thread met something that does not split
  if (abort_flag) {
    // an earlier kernel on this device gave up on a wait: take no work
    copy_async_wait();
  } else if (warp == W::kIssuer) {
    // ================= issuing warp: it stays together and elects a lane for each bunch of MMAs =================
    grid_launch_dependents();
    int t = 0;  // tiles so far
    auto weigh = [&](int t) {
      ok = ok && warp_waits<false>(ring(kReady, t), ring_parity(t), g.status, 0x0a11u);
      if (!ok) return;
      tc_fence_after_sync();
      if (elect_one()) {
        issue_weigh<HD>(tmem + L::kO, tmem + L::kP, tile1_at(t));
        mma_commit(ring(kWeighed, t));
      }
      __syncwarp();
    };
    for (int k = 0; ok && item(k, it); ++k) {
      for (int j = 0; ok && j < it.tiles; ++j, ++t) {
        ok = warp_waits<false>(ring(kGo, t), ring_parity(t), g.status, 0x0a10u);
        if (!ok) break;
        tc_fence_after_sync();
        if (elect_one()) {
          issue_scores<HD, L::kHeldT, L::kTwo>(tmem + L::kS, L::kHeldT ? tmem + L::kHeldCol : base + L::kHeld, tile0_at(t), tmem + L::kS2);
          mma_commit(ring(kScored, t));
        }
        __syncwarp();
        if (j > 0) weigh(t - 1);
      }
      if (ok) weigh(t - 1);
    }
  } else if (warp >= W::kRowWarps) {
    // ================= splitting warps =================
    const int thread = threadIdx.x - W::kRowThreads;
    float flag = 0.f;
    auto load_rows = [&](const Item& it, int x0) {
      if (g.mask) flag = row_value(g.mask + it.b * g.t_k, x0, g.t_k, thread);
    };
    auto post_rows = [&](int t) {
      if (g.mask) post_hidden(hidden[t % kHiddenPlaces], flag, thread);
    };
    if constexpr (L::kPlaces0 > 1)
      again = split_streams<HD, W::kSplitThreads, kWide, L::kPlaces0, L::kPlaces1, false>(
          carry, it, any, item, keys, values, g.t_k, g.hd, g.hd_v, ring(kScored, 0), ring(kWeighed, 0), ring(kGo, 0), ring(kReady, 0), base + L::kTile0, base + L::kTile1,
          g.status, ok, load_rows, post_rows);
    else
      again = split_streams_one<HD, W::kSplitThreads, kWide, false>(carry[0], it, any, item, keys, values, g.t_k, g.hd, g.hd_v, ring(kScored, 0), ring(kWeighed, 0),
                                                                    ring(kGo, 0), ring(kReady, 0), base + L::kTile0, base + L::kTile1, g.status, ok, load_rows, post_rows);
  } else if (any) {
    // ================= row warps =================
    // A warp that gave up on a wait waits for nothing any more but goes through its tiles like the others: the two warps that share
    // rows meet at a barrier in each.
    const uint32_t lanes = tmem + (static_cast<uint32_t>(quarter * 32) << 16);
    auto meet = [&] { named_barrier_sync(1 + quarter, 32 * G); };
    auto put_held = [&](const Item& it, int k) {  // Q of item k, to where the MMAs read it
      Check check;
      if constexpr (L::kHeldT) {  // (it has been fetched)
        copy_async_wait();
        __syncwarp();
        place_held<HD, OW>(lanes + L::kHeldCol + group * (OW / 2), raw_q, check);
        tmem_st_wait();
        tc_fence_before_sync();
      } else {
        constexpr int kChunks = HD / 8, kStep = W::kRowThreads / kChunks, kAtOnce = 4;
        const int r = threadIdx.x / kChunks, chunk = threadIdx.x % kChunks;
        const float* q = g.q + it.b * g.t_q * g.hd;
#pragma unroll
        for (int n = 0; n < kRows / kStep; n += kAtOnce) {
          float x[kAtOnce][8];
#pragma unroll
          for (int u = 0; u < kAtOnce; ++u) load8<kWide>(x[u], q, it.first + r + (n + u) * kStep, g.t_q, 8 * chunk, g.hd);
#pragma unroll
          for (int u = 0; u < kAtOnce; ++u) {
            uint32_t h[4], m[4], l[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) split_pair<true>(f2_pack(x[u][2 * i], x[u][2 * i + 1]), h[i], m[i], l[i], check);
            const uint32_t to = swizzled_piece(base + L::kHeld + chunk / 8 * (kRows * 128), r + (n + u) * kStep, chunk % 8);
            st_shared_v4(to, h[0], h[1], h[2], h[3]);
            st_shared_v4(to + L::kHeldPiece, m[0], m[1], m[2], m[3]);
            st_shared_v4(to + 2 * L::kHeldPiece, l[0], l[1], l[2], l[3]);
          }
        }
        fence_async_shared();
      }
      if (check.bad()) again |= 1u << k;
    };
    put_held(it, 0);
    warp_arrives(ring(kGo, 0));
    const uint64_t c_hi = f2_pack(g.c_hi, g.c_hi), c_lo = f2_pack(g.c_lo, g.c_lo);
    int t = 0;
    for (int k = 0;; ++k) {
      const int i = it.first + row;
      float denom[L::kShares] = {};
      float top = -INFINITY, shift = 0.f;  // row maximum (raw scores); shift = top * c, in log2 units
      float shrink = 0.f;                               // what the sums so far are multiplied with when the last tile's product comes
      uint64_t acc[OW / 2];
#pragma unroll
      for (int c = 0; c < OW / 2; ++c) acc[c] = 0;
      auto gather_product = [&](int t) {  // of tile t
        ok = ok && warp_waits<false>(ring(kWeighed, t), ring_parity(t), g.status, 0x0a22u);
        tc_fence_after_sync();
        const uint64_t shrink2 = f2_pack(shrink, shrink);
        constexpr int N = OW > 32 ? 16 : OW;  // columns at a time
#pragma unroll
        for (int part = 0; part < OW; part += N) {
          uint32_t o[N];
          tmem_ld<N>(lanes + L::kO + group * OW + part, o);
          tmem_ld_wait();
#pragma unroll
          for (int c = 0; c < N / 2; ++c) acc[part / 2 + c] = f2_fma(acc[part / 2 + c], shrink2, f2_pack_bits(o[2 * c], o[2 * c + 1]));
        }
      };
      Item next = it;
      bool more = false;
      for (int j = 0; j < it.tiles; ++j, ++t) {
        const int j0 = j * kStream;
        if (g.mask) ok = ok && warp_waits<false>(ring(kGo, t), ring_parity(t), g.status, 0x0a20u);  // (its hidden keys)
        ok = ok && warp_waits<false>(ring(kScored, t), ring_parity(t), g.status, 0x0a21u);
        tc_fence_after_sync();
        uint32_t s[CW];
        tmem_ld<CW>(lanes + L::kS + group * CW, s);
        if constexpr (L::kTwo) {
#pragma unroll
          for (int part = 0; part < CW; part += 16) {
            uint32_t more_s[16];
            tmem_ld<16>(lanes + L::kS2 + group * CW + part, more_s);
            tmem_ld_wait();
#pragma unroll
            for (int c = 0; c < 16; ++c) s[part + c] = __float_as_uint(__uint_as_float(s[part + c]) + __uint_as_float(more_s[c]));
          }
        }
        if (j == 0) {
          more = item(k + 1, next);
          if (more) fetch(next);
        }
        tmem_ld_wait();
        tc_fence_before_sync();
        if (j + 1 < it.tiles) warp_arrives(ring(kGo, t + 1));
        int limit = g.t_k - j0;
        if (g.causal) limit = min(limit, i - j0 + 1);
        limit -= group * CW;
        uint32_t unseen = limit >= CW ? 0u : limit <= 0 ? kFull : ~((1u << limit) - 1u);
        if (g.mask) unseen |= my_hidden<CW>(hidden[t % kHiddenPlaces], group);
        if (unseen != 0u) {
#pragma unroll
          for (int c = 0; c < CW; ++c)
            if ((unseen >> c) & 1u) s[c] = 0xff800000u;
        }
        float tile_top = -INFINITY;
#pragma unroll
        for (int c = 0; c < CW; c += 2) tile_top = max3(tile_top, __uint_as_float(s[c]), __uint_as_float(s[c + 1]));
        exchange[t & 1][group][row] = tile_top;
        meet();
        float raised = top;
#pragma unroll
        for (int c = 0; c < G; ++c) raised = fmaxf(raised, exchange[t & 1][c][row]);
        const float moved = raised == -INFINITY ? 0.f : raised * g.c_hi;
        const float less = top == -INFINITY ? 0.f : exp2_approx(shift - moved);  // nothing gathered yet: nothing to rescale
        top = raised, shift = moved;
        const uint64_t minus_shift = f2_pack(-shift, -shift);
        uint64_t w[CW / 2];
        uint64_t sum[L::kShares] = {};
#pragma unroll
        for (int c = 0; c < CW / 2; ++c) {
          const uint64_t s2 = f2_pack_bits(s[2 * c], s[2 * c + 1]);
          float x0, x1;
          f2_unpack(f2_fma(s2, c_lo, f2_fma(s2, c_hi, minus_shift)), x0, x1);
          w[c] = f2_pack(exp2_approx(x0), exp2_approx(x1));
          sum[c * L::kShares / (CW / 2)] = f2_add(sum[c * L::kShares / (CW / 2)], w[c]);
        }
#pragma unroll
        for (int c = 0; c < L::kShares; ++c) {
          float sum0, sum1;
          f2_unpack(sum[c], sum0, sum1);
          denom[c] = fmaf(denom[c], less, sum0 + sum1);  // this thread's shares; they meet after the last tile
        }
        if (j > 0) gather_product(t - 1);
        shrink = less;
        // (the product of the tile before has been gathered, so its P has been read)
        hand_over<CW>(lanes + L::kP + group * (CW / 2), w);
        tmem_st_wait();
        tc_fence_before_sync();
        warp_arrives(ring(kReady, t));
      }
      if (more) {
        put_held(next, k + 1);
        warp_arrives(ring(kGo, t));
      }
      gather_product(t - 1);
      tc_fence_before_sync();
#pragma unroll
      for (int c = 0; c < L::kShares; ++c) {
        if (!(denom[c] < INFINITY)) again |= 1u << k;
        exchange[t & 1][group * L::kShares + c][row] = denom[c];
      }
      meet();
      float total = 0.f;
#pragma unroll
      for (int c = 0; c < G * L::kShares; ++c) total += exchange[t & 1][c][row];
      meet();  // (the next item's first maxima may go there)
      if (ok) {
        divide_row(acc, total);  // 0/0 = NaN for a row with no key, as the oracle has it
        store_rows<OW>(g.out + it.b * g.t_q * g.hd_v, acc, it.first + quarter * 32, g.t_q, group * OW, g.hd_v, g.wide_out);
        // once per row, so in double: L is then as good as its sum
        if (group == 0 && i < g.t_q)
          g.lse_out[it.b * g.t_q + i] =
              top == -INFINITY ? -INFINITY : static_cast<float>(shift * 0.69314718055994530942 + log(static_cast<double>(total)));
      }
      if (!more) break;
      it = next;
    }
  }
  __syncwarp();
  if (again != 0) atomicOr(&again_all, again);
  tc_fence_before_sync();
  ok = __syncthreads_and(ok);
  if (ok && again_all != 0 && !abort_flag && threadIdx.x < kAgainGroups * tiled::kThreads) {
    for (uint32_t left = again_all; left != 0; left &= left - 1)
      if (item(__ffs(static_cast<int>(left)) - 1, it)) rows_again<HD, Op::Fwd, kAgainGroups, L::kBytes, kWide>(g, it.b, it.first, raw);
  }
  tear_down<L::kCols, W::kIssuer>(g, tmem);
}

// ---- forward of short problems: two blocks of 256 threads to an SM, no roles ----
// The same sums in the same order, everything by all of a block's threads, one thing after the other. An item of one key tile is a chain of
// latencies whichever way the work is shared out; here an SM has two of them at once, and a block is ready sooner.
template <int HD, bool kWide>
struct FwdPair {
  static constexpr int kGroups = 2, kThreads = kRows * kGroups;
  using Held = Stage<HD, kRows, kThreads, kWide>;
  using Tile = Stage<HD, kStream, kThreads, kWide>;
  static constexpr uint32_t kQ = 0, kK = Held::kBytes, kV = kK + Tile::kBytes, kBytes = kV + Tile::kBytes + 1024;
  static constexpr uint32_t kS = 0, kP = kStream, kO = kP + 3 * kPieceCols;
  static constexpr int kCols = 256;
  static_assert(kO + HD <= kCols, "tensor memory");
};

template <int HD, bool kWide>
__global__ void __launch_bounds__(FwdPair<HD, kWide>::kThreads, 2) f32_fwd_pair_kernel(const __grid_constant__ Params g) {
  using L = FwdPair<HD, kWide>;
  constexpr int G = L::kGroups, CW = kStream / G, OW = HD / G;
  extern __shared__ __align__(16) unsigned char raw[];
  __shared__ uint32_t slot, abort_flag, hidden[2][2];
  __shared__ __align__(8) uint64_t bars[2];
  __shared__ float exchange[G][kRows];
  uint32_t tmem;
  if (!set_up<L::kCols, 2>(g, &slot, &abort_flag, bars, tmem)) return;
  const uint32_t base = align_1024(smem_addr(raw));
  const uint32_t scored = smem_addr(bars), weighed = smem_addr(bars + 1);
  const int warp = threadIdx.x >> 5, group = warp >> 2;
  const int row = (warp & 3) * 32 + (threadIdx.x & 31);
  const uint32_t lanes = tmem + (static_cast<uint32_t>((warp & 3) * 32) << 16);
  const bool issues = __shfl_sync(kFull, warp, 0) == 0;  // the warp that issues, one lane of it elected per bunch

  int problem, at;
  cta_work(blockIdx.x, g.slots, g.bh, g.group, problem, at);
  const int first = (g.slots - 1 - at) * kRows;  // long causal rows first
  const long long b = problem;
  const float* k = g.k + b * g.t_k * g.hd;
  const float* v = g.v + b * g.t_k * g.hd_v;
  const float* mask = g.mask ? g.mask + b * g.t_k : nullptr;
  const int tiles = ((g.causal ? min(g.t_k, first + kRows) : g.t_k) + kStream - 1) / kStream;
  const int i = first + row;
  auto score = [&] {
    if (issues && elect_one()) {
      tc_fence_after_sync();
      issue_scores<HD, false>(tmem + L::kS, base + L::kQ, base + L::kK);
      mma_commit(scored);
    }
  };

  Check check;
  typename L::Tile stage_k, stage_v;
  stage_k.load(k, 0, g.t_k, g.hd);
  {
    typename L::Held stage_q;
    stage_q.load(g.q + b * g.t_q * g.hd, first, g.t_q, g.hd);
    stage_q.store(base + L::kQ, check);
  }
  stage_k.store(base + L::kK, check);
  if (mask) post_hidden(hidden[0], row_value(mask, 0, g.t_k));
  fence_async_shared();
  __syncthreads();
  score();
  stage_v.load(v, 0, g.t_k, g.hd_v);
  stage_v.store(base + L::kV, check);
  fence_async_shared();

  float top = -INFINITY, shift = 0.f, denom = 0.f;  // row maximum (raw scores); shift = top * c, in log2 units
  uint64_t acc[OW / 2];
#pragma unroll
  for (int c = 0; c < OW / 2; ++c) acc[c] = 0;
  const uint64_t c_hi = f2_pack(g.c_hi, g.c_hi), c_lo = f2_pack(g.c_lo, g.c_lo);
  bool ok = true;
  for (int j = 0; j < tiles; ++j) {
    const int j0 = j * kStream;
    const bool more = j + 1 < tiles;
    ok &= mbar_wait(scored, j & 1, g.status, 0x0a00u);
    tc_fence_after_sync();
    uint32_t s[CW];
    tmem_ld<CW>(lanes + L::kS + group * CW, s);
    tmem_ld_wait();
    int limit = g.t_k - j0;
    if (g.causal) limit = min(limit, i - j0 + 1);
    limit -= group * CW;
    uint32_t unseen = limit >= CW ? 0u : limit <= 0 ? kFull : ~((1u << limit) - 1u);
    if (mask) unseen |= my_hidden<CW>(hidden[j & 1], group);
    if (unseen != 0u) {
#pragma unroll
      for (int c = 0; c < CW; ++c)
        if ((unseen >> c) & 1u) s[c] = 0xff800000u;
    }
    float tile_top = -INFINITY;
#pragma unroll
    for (int c = 0; c < CW; c += 2) tile_top = max3(tile_top, __uint_as_float(s[c]), __uint_as_float(s[c + 1]));
    exchange[group][row] = tile_top;
    __syncthreads();
    float raised = top;
#pragma unroll
    for (int c = 0; c < G; ++c) raised = fmaxf(raised, exchange[c][row]);
    const float moved = raised == -INFINITY ? 0.f : raised * g.c_hi;
    const float shrink = top == -INFINITY ? 0.f : exp2_approx(shift - moved);  // nothing gathered yet: nothing to rescale
    top = raised, shift = moved;
    const uint64_t minus_shift = f2_pack(-shift, -shift);
    uint64_t w[CW / 2];
    uint64_t sum = 0;
#pragma unroll
    for (int c = 0; c < CW / 2; ++c) {
      const uint64_t s2 = f2_pack_bits(s[2 * c], s[2 * c + 1]);
      float x0, x1;
      f2_unpack(f2_fma(s2, c_lo, f2_fma(s2, c_hi, minus_shift)), x0, x1);
      w[c] = f2_pack(exp2_approx(x0), exp2_approx(x1));
      sum = f2_add(sum, w[c]);
    }
    float sum0, sum1;
    f2_unpack(sum, sum0, sum1);
    denom = fmaf(denom, shrink, sum0 + sum1);  // this thread's share; the shares meet after the last tile
    check.sums |= !(denom < INFINITY);
    hand_over<CW>(lanes + L::kP + group * (CW / 2), w);
    tmem_st_wait();
    tc_fence_before_sync();
    if (!__syncthreads_and(ok && !check.bad())) break;  // (nothing is in flight here)
    if (issues && elect_one()) {
      tc_fence_after_sync();
      issue_weigh<HD>(tmem + L::kO, tmem + L::kP, base + L::kV);
      mma_commit(weighed);
    }
    if (more) {
      // K's place has been read (the scores are there) and so have the scores themselves
      stage_k.load(k, j0 + kStream, g.t_k, g.hd);
      const float flag = mask ? row_value(mask, j0 + kStream, g.t_k) : 0.f;
      stage_k.store(base + L::kK, check);
      if (mask) post_hidden(hidden[(j + 1) & 1], flag);
      fence_async_shared();
      __syncthreads();
      score();
      stage_v.load(v, j0 + kStream, g.t_k, g.hd_v);
    }
    ok &= mbar_wait(weighed, j & 1, g.status, 0x0a01u);
    tc_fence_after_sync();
    uint32_t o[OW];
    tmem_ld<OW>(lanes + L::kO + group * OW, o);
    tmem_ld_wait();
    tc_fence_before_sync();
    const uint64_t shrink2 = f2_pack(shrink, shrink);
#pragma unroll
    for (int c = 0; c < OW / 2; ++c) acc[c] = f2_fma(acc[c], shrink2, f2_pack_bits(o[2 * c], o[2 * c + 1]));
    if (more) {
      stage_v.store(base + L::kV, check);  // the weighing has read the tile before this one
      fence_async_shared();
    }
  }
  exchange[group][row] = denom;  // (every read of the maxima lies before a barrier of the block)
  ok = __syncthreads_and(ok);
  const bool bad = __syncthreads_or(check.bad());
  if (ok && bad) {
    rows_again<HD, Op::Fwd, 1, L::kBytes, kWide>(g, b, first, raw);
  } else if (ok) {
    float total = 0.f;
#pragma unroll
    for (int c = 0; c < G; ++c) total += exchange[c][row];
    divide_row(acc, total);  // 0/0 = NaN for a row with no key, as the oracle has it
    store_rows<OW>(g.out + b * g.t_q * g.hd_v, acc, first + (warp & 3) * 32, g.t_q, group * OW, g.hd_v, g.wide_out);
    // once per row, so in double: L is then as good as its sum
    if (group == 0 && i < g.t_q)
      g.lse_out[b * g.t_q + i] = top == -INFINITY ? -INFINITY : static_cast<float>(shift * 0.69314718055994530942 + log(static_cast<double>(total)));
  }
  tear_down<L::kCols>(g, tmem);
}

// ---- backward at head dims up to 64: dQ for 128 query rows, or dK and dV for 128 key rows ----
// A tile's scores are computed while the row warps are at the tile before it, and its products are gathered while the next tile's
// are: a row warp comes to each of its waits with the answer there, as long as the tensor cores keep up.
template <int HD, bool kKV>
struct Bwd {
  // tensor memory: scores, dP, the pieces of dS and (dK/dV) of P, a tile's products, and the held operands if they fit:
  // they are the A side of the scores, an MMA then only reads the streamed tile from shared memory (whose bandwidth
  // bounds it at 48 clocks with both there, for 32)
  static constexpr uint32_t kS = 0, kDp = kStream, kDs = 2 * kStream, kP = kDs + 3 * kPieceCols;
  static constexpr uint32_t kOut0 = kKV ? kP + 3 * kPieceCols : kP, kOut1 = kOut0 + HD, kHeldCol = kKV ? kOut1 + HD : kOut1;
  static constexpr bool kHeldT = kHeldCol + 3 * HD <= 512;
  static constexpr int kCols = 512;
  // shared memory: places for the first streamed operand, which the products need, and for the second; the held operands, in
  // pieces or, where those are in tensor memory, as the next item's float32. The first operand has three places: with two, a tile
  // could not be brought in before the products of the tile two before it were done.
  static constexpr int kPlaces0 = 3, kPlaces1 = HD > 32 && kKV ? 2 : 3;
  // The scores against the first operand do not wait for the second, dP does. (Measured, us, without -> with: dQ 6 x 8192 x 32 causal
  // 236 -> 232, 256 x 512 x 64 147 -> 144; dK and dV at head dim 64, whose second operand has two places and comes late, 187 -> 175
  // there; at head dim 32 one wait less is better: 303 and 318.)
  static constexpr bool kLate1 = !kKV || HD > 32;
  static constexpr uint32_t kTile = 3 * kStream * 128, kHeldPieces = 3 * kRows * 128, kHeldRaw = kRows * HD * 4;
  static constexpr uint32_t kTile0 = 0, kTile1 = kPlaces0 * kTile, kHeld0 = kTile1 + kPlaces1 * kTile, kHeld1 = kHeld0 + (kHeldT ? kHeldRaw : kHeldPieces);
  static constexpr uint32_t kBytes = kHeld1 + (kHeldT ? kHeldRaw : kHeldPieces) + 1024;
};

// kGroups threads to a row (and the split of the warps that goes with it): the same bits either way. Two are faster in dQ up to head dim 32
// where a block has one item of several tiles (2 x 128 x 32 7.7 us for 8.3, 64 x 128 8.6 for 8.9, 2 x 8192 152 for 156), as the splitting warps have it ready
// sooner; four in the long run (6 x 8192 x 32 causal 233 for 239) and at head dim 64 (64 x 128 x 64 11.5 for 12.1, 16 x 600 x 64 23.4 for
// 26.8, 256 x 512 x 64 143 for 150). All of them spill: with four threads to a row and 96 registers 76 to 152 bytes are stored and 56 to 140
// loaded again a thread, with two and 128 up to 36; of the forwards those above head dim 64, 184 and 216. That is not in the tile loops: 16
// causal problems of 2048 x 64 execute 25 000 local loads and 13 000 stores in dQ (of 31.8 M instructions), 9 600 and 12 800 in dK and dV (43.9 M).
template <int HD, bool kKV, bool kWide, int kGroups>
__global__ void __launch_bounds__(Roles<kGroups>::kThreads, 1) f32_bwd_kernel(const __grid_constant__ Params g) {
  using L = Bwd<HD, kKV>;
  using W = Roles<kGroups>;
  using Held = Stage<HD, kRows, W::kRowThreads, kWide>;
  constexpr int CW = kStream / kGroups, OW = HD / kGroups;
  extern __shared__ __align__(16) unsigned char raw[];
  __shared__ uint32_t slot, abort_flag, again_all, hidden[kRing][2];
  // kGo: a tile can be scored (both its operands are there, the scores before it have been read, the held operands are there).
  // kReady: it can be weighed (P and dS are there). kScored, kWeighed: the tensor cores have done it (kHalfWeighed: dV's part). kGoOn: the
  // second operand is there, where it is waited for by itself.
  enum { kGo = 0, kReady = kRing, kScored = 2 * kRing, kWeighed = 3 * kRing, kHalfWeighed = 4 * kRing, kGoOn = 5 * kRing, kBars = 6 * kRing };
  __shared__ __align__(8) uint64_t bars[kBars];
  __shared__ __align__(16) float lse_hi[kKV ? kRing : 1][kStream], lse_lo[kKV ? kRing : 1][kStream], deltas[kKV ? kRing : 1][kStream];
  const int warp = __shfl_sync(kFull, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
#pragma unroll
    for (int i = 0; i < kBars; ++i)
      mbar_init(smem_addr(bars + i), i < kReady ? W::kRowWarps + (L::kLate1 ? 1 : 2) * W::kSplitWarps : i < kScored ? W::kRowWarps : i < kGoOn ? 1 : W::kSplitWarps);
    mbar_init_fence();
    again_all = 0;
  }
  auto place = [](int t, int places) { return t % places; };
  auto ring = [&](int which, int t) { return ring_bar(smem_addr(bars + which), t); };
  const uint32_t base = align_1024(smem_addr(raw));
  auto tile0_at = [&](int t) { return base + L::kTile0 + place(t, L::kPlaces0) * L::kTile; };
  auto tile1_at = [&](int t) { return base + L::kTile1 + place(t, L::kPlaces1) * L::kTile; };

  // the held pair (against which the tiles are scored) and the streamed pair
  const int owned = kKV ? g.t_k : g.t_q, streamed = kKV ? g.t_q : g.t_k;
  auto item = [&](int k, Item& it) {
    int problem = 0, at = 0;
    if (!work_item(g, k, problem, at)) return false;
    it.b = problem;
    it.first = (kKV ? at : g.slots - 1 - at) * kRows;  // the longest causal streams first
    it.begin = kKV && g.causal ? it.first : 0;
    const int end = !kKV && g.causal ? min(streamed, it.first + kRows) : streamed;
    it.tiles = (end - it.begin + kStream - 1) / kStream;
    return true;
  };
  auto held0 = [&](const Item& it) { return (kKV ? g.k : g.q) + it.b * owned * g.hd; };
  auto held1 = [&](const Item& it) { return (kKV ? g.v : g.dout) + it.b * owned * g.hd_v; };
  auto stream0 = [&](const Item& it) { return (kKV ? g.q : g.k) + it.b * streamed * g.hd; };
  auto stream1 = [&](const Item& it) { return (kKV ? g.dout : g.v) + it.b * streamed * g.hd_v; };

  // a row warp's part of the held operands
  const int group = warp >> 2, quarter = warp & 3, row = quarter * 32 + lane;
  const uint32_t raw0 = base + L::kHeld0 + warp * (32 * OW * 4), raw1 = base + L::kHeld1 + warp * (32 * OW * 4);
  auto fetch = [&](const Item& it) {
    fetch_held<OW, kWide>(raw0, held0(it), it.first + quarter * 32, owned, group * OW, g.hd);
    fetch_held<OW, kWide>(raw1, held1(it), it.first + quarter * 32, owned, group * OW, g.hd_v);
  };

  // the held operands of an item into L2, a 128-byte line to a thread
  auto prefetch_held = [&](const Item& it) {
    constexpr int kLines = HD / 32;
    const int e = threadIdx.x, r = it.first + (e % (kRows * kLines)) / kLines, c = (e % kLines) * 32;
    const bool second = e >= kRows * kLines;
    const int width = second ? g.hd_v : g.hd;
    if (e < 2 * kRows * kLines && r < owned && c < width)
      asm volatile("prefetch.global.L2 [%0];" ::"l"((second ? held1(it) : held0(it)) + static_cast<long long>(r) * width + c));
  };

  Item it;
  const bool any = item(0, it);
  grid_dependency_wait();
  if (warp == W::kIssuer) {
    tmem_alloc(smem_addr(&slot), L::kCols);
    tmem_relinquish();
  }
  if (threadIdx.x == 0) abort_flag = *reinterpret_cast<volatile unsigned*>(g.status) != kStatusOk;
  // the first operands set out before the block is set up
  using Carried = Carry<HD, W::kSplitThreads, kWide>;
  Carried carry[Carried::kHalves];
#pragma unroll
  for (int h = 0; h < Carried::kHalves; ++h) carry[h].set_up(threadIdx.x - W::kRowThreads);
  if (any && warp < W::kRowWarps) {
    if (L::kHeldT) fetch(it);
  } else if (any && warp < W::kIssuer) {
    carry[0].load_all(carry[0].source(stream0(it), it.begin, streamed, g.hd));
    if (Carried::kHalves > 1) carry[Carried::kHalves - 1].load_all(carry[0].source(stream1(it), it.begin, streamed, g.hd_v));
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem = __shfl_sync(kFull, slot, 0);
  bool ok = true;
  uint32_t again = 0;  // items in which this thread met something that does not split
  if (abort_flag) {
    // an earlier kernel on this device gave up on a wait: take no work
    copy_async_wait();
  } else if (warp == W::kIssuer) {
    // ================= issuing warp: it stays together and elects a lane for each bunch of MMAs =================
    grid_launch_dependents();
    int t = 0;  // tiles so far
    auto weigh = [&](int t) {
      ok = ok && warp_waits<true>(ring(kReady, t), ring_parity(t), g.status, 0x0b11u);
      if (!ok) return;
      tc_fence_after_sync();
      if (elect_one()) {
        if (kKV) {
          issue_weigh<HD>(tmem + L::kOut1, tmem + L::kP, tile1_at(t));
          mma_commit(ring(kHalfWeighed, t));
        }
        issue_weigh<HD>(tmem + L::kOut0, tmem + L::kDs, tile0_at(t));
        mma_commit(ring(kWeighed, t));
      }
      __syncwarp();
    };
    for (int k = 0; ok && item(k, it); ++k) {
      for (int j = 0; ok && j < it.tiles; ++j, ++t) {
        ok = warp_waits<true>(ring(kGo, t), ring_parity(t), g.status, 0x0b10u);
        if (!ok) break;
        tc_fence_after_sync();
        if (L::kLate1) {
          if (elect_one()) issue_scores<HD, L::kHeldT>(tmem + L::kS, L::kHeldT ? tmem + L::kHeldCol : base + L::kHeld0, tile0_at(t));
          __syncwarp();
          ok = warp_waits<true>(ring(kGoOn, t), ring_parity(t), g.status, 0x0b14u);
          if (!ok) break;
          tc_fence_after_sync();
        }
        if (elect_one()) {
          if (!L::kLate1) issue_scores<HD, L::kHeldT>(tmem + L::kS, L::kHeldT ? tmem + L::kHeldCol : base + L::kHeld0, tile0_at(t));
          issue_scores<HD, L::kHeldT>(tmem + L::kDp, L::kHeldT ? tmem + L::kHeldCol + 3 * HD / 2 : base + L::kHeld1, tile1_at(t));
          mma_commit(ring(kScored, t));
        }
        __syncwarp();
        if (j > 0) weigh(t - 1);
      }
      if (ok) weigh(t - 1);
    }
  } else if (warp >= W::kRowWarps) {
    // ================= splitting warps =================
    const int thread = threadIdx.x - W::kRowThreads;
    float row_a = 0.f, row_b = 0.f;  // dK/dV: L and delta of a query row; dQ: a key's flag
    again = split_streams<HD, W::kSplitThreads, kWide, L::kPlaces0, L::kPlaces1, true>(
        carry, it, any, item, stream0, stream1, streamed, g.hd, g.hd_v, ring(kWeighed, 0), ring(kKV ? kHalfWeighed : kScored, 0), ring(kGo, 0), ring(L::kLate1 ? kGoOn : kGo, 0), base + L::kTile0, base + L::kTile1, g.status, ok,
        [&](const Item& it, int x0) {
          if (kKV) {
            row_a = row_value(g.lse_in + it.b * g.t_q, x0, streamed, thread);
            row_b = row_value(g.delta + it.b * g.t_q, x0, streamed, thread);
          } else if (g.mask) {
            row_a = row_value(g.mask + it.b * g.t_k, x0, streamed, thread);
          }
        },
        [&](int t) {
          const int place = t % kRing;
          if (kKV) {
            if (thread < kStream) {
              float hi, lo;
              to_minus_log2(row_a, hi, lo);
              lse_hi[place][thread] = hi;
              lse_lo[place][thread] = lo;
              deltas[place][thread] = -row_b;
            }
          } else if (g.mask) {
            post_hidden(hidden[place], row_a, thread);
          }
        });
  } else if (any) {
    // ================= row warps =================
    const uint32_t lanes = tmem + (static_cast<uint32_t>(quarter * 32) << 16);
    // the held operands of item k, which have been fetched, to where the MMAs read them
    auto put_held = [&](const Item& it, int k) {
      Check check;
      if constexpr (L::kHeldT) {
        copy_async_wait();
        __syncwarp();
        place_held<HD, OW>(lanes + L::kHeldCol + group * (OW / 2), raw0, check);
        place_held<HD, OW>(lanes + L::kHeldCol + 3 * HD / 2 + group * (OW / 2), raw1, check);
        tmem_st_wait();
        tc_fence_before_sync();
      } else {
        Held stage0, stage1;
        stage0.load(held0(it), it.first, owned, g.hd);
        stage1.load(held1(it), it.first, owned, g.hd_v);
        stage0.store(base + L::kHeld0, check);
        stage1.store(base + L::kHeld1, check);
        fence_async_shared();
      }
      if (check.bad()) again |= 1u << k;
    };
    put_held(it, 0);
    warp_arrives(ring(kGo, 0));
    int t = 0;
    for (int k = 0;; ++k) {
      const int mine = it.first + row;  // this thread's row
      float my_hi = 0.f, my_lo = 0.f, my_delta = 0.f;  // dQ: of this thread's row
      bool live = mine < owned;
      if constexpr (kKV) {
        if (live && g.mask) live = g.mask[it.b * g.t_k + mine] != 0.f;
      } else if (live) {
        to_minus_log2(g.lse_in[it.b * g.t_q + mine], my_hi, my_lo);
        my_delta = -g.delta[it.b * g.t_q + mine];
      }
      uint64_t acc0[OW / 2], acc1[OW / 2];  // dQ, or dK and dV
#pragma unroll
      for (int c = 0; c < OW / 2; ++c) acc0[c] = acc1[c] = 0;
      auto gather = [&](uint32_t from, uint64_t(&acc)[OW / 2]) {
        uint32_t o[OW];
        tmem_ld<OW>(lanes + from + group * OW, o);
        tmem_ld_wait();
#pragma unroll
        for (int c = 0; c < OW / 2; ++c) acc[c] = f2_add(acc[c], f2_pack_bits(o[2 * c], o[2 * c + 1]));
      };
      auto gather_products = [&](int t) {  // of tile t
        ok = ok && warp_waits<true>(ring(kWeighed, t), ring_parity(t), g.status, 0x0b22u);
        if (!ok) return;
        tc_fence_after_sync();
        if (kKV) gather(L::kOut1, acc1);
        gather(L::kOut0, acc0);
      };
      Item next = it;
      bool more = false;
      for (int j = 0; j < it.tiles; ++j, ++t) {
        const int x0 = it.begin + j * kStream;
        if (kKV || g.mask) ok = ok && warp_waits<true>(ring(kGo, t), ring_parity(t), g.status, 0x0b20u);  // (what goes with its rows)
        ok = ok && warp_waits<true>(ring(kScored, t), ring_parity(t), g.status, 0x0b21u);
        if (!ok) break;
        tc_fence_after_sync();
        uint32_t s[CW], dp[CW];
        tmem_ld<CW>(lanes + L::kS + group * CW, s);
        tmem_ld<CW>(lanes + L::kDp + group * CW, dp);
        if (j == 0) {  // (every warp has put its held operands in place: the tile has been scored)
          more = item(k + 1, next);
          if (more && L::kHeldT) fetch(next);
          else if (more) prefetch_held(next);
        }
        tmem_ld_wait();
        tc_fence_before_sync();
        if (j + 1 < it.tiles) warp_arrives(ring(kGo, t + 1));
        int from = 0, to = streamed - x0 - group * CW;
        if (g.causal) {
          if (kKV) from = mine - x0 - group * CW;
          else to = min(to, mine - x0 - group * CW + 1);
        }
        uint32_t unseen = outside<CW>(from, live ? to : 0);
        if (!kKV && g.mask) unseen |= my_hidden<CW>(hidden[t % kRing], group);
        uint64_t p[CW / 2], ds[CW / 2];
        weigh_scores<CW>(g, s, dp, unseen, [&](int c, uint64_t& hi, uint64_t& lo, uint64_t& delta) {
          if (kKV) {
            hi = *reinterpret_cast<const uint64_t*>(&lse_hi[t % kRing][group * CW + c]);
            lo = *reinterpret_cast<const uint64_t*>(&lse_lo[t % kRing][group * CW + c]);
            delta = *reinterpret_cast<const uint64_t*>(&deltas[t % kRing][group * CW + c]);
          } else {
            hi = f2_pack(my_hi, my_hi), lo = f2_pack(my_lo, my_lo), delta = f2_pack(my_delta, my_delta);
          }
        }, p, ds);
        if (j > 0) gather_products(t - 1);
        if (!ok) break;
        // (the products of the tile before have been gathered, so its P and dS have been read)
        hand_over<CW>(lanes + L::kDs + group * (CW / 2), ds);
        if (kKV) hand_over<CW>(lanes + L::kP + group * (CW / 2), p);
        tmem_st_wait();
        tc_fence_before_sync();
        warp_arrives(ring(kReady, t));
      }
      if (!ok) break;
      if (more) {
        put_held(next, k + 1);
        warp_arrives(ring(kGo, t));
      }
      gather_products(t - 1);
      if (!ok) break;
      tc_fence_before_sync();
      Check check;
      settle(acc0, check);
      if (check.bad()) again |= 1u << k;
      const int top = it.first + quarter * 32;
      if (kKV) {
        store_rows<OW>(g.dk + it.b * owned * g.hd, acc0, top, owned, group * OW, g.hd, g.wide_out);
        store_rows<OW>(g.dv + it.b * owned * g.hd_v, acc1, top, owned, group * OW, g.hd_v, g.wide_out);
      } else {
        store_rows<OW>(g.dq + it.b * owned * g.hd, acc0, top, owned, group * OW, g.hd, g.wide_out);
      }
      if (!more) break;
      it = next;
    }
    copy_async_wait();
  }
  __syncwarp();
  if (again != 0) atomicOr(&again_all, again);
  tc_fence_before_sync();
  ok = __syncthreads_and(ok);
  if (ok && again_all != 0 && !abort_flag && threadIdx.x < kAgainGroups * tiled::kThreads) {
    for (uint32_t left = again_all; left != 0; left &= left - 1)
      if (item(__ffs(static_cast<int>(left)) - 1, it))
        rows_again<HD, kKV ? Op::BwdKV : Op::BwdQ, kAgainGroups, L::kBytes, kWide>(g, it.b, it.first, raw);
  }
  tear_down<L::kCols, W::kIssuer>(g, tmem);
}

// ---- backward at head dims above 64, and of items of one tile (one_tile) ----
// Above 64 two held operands and two streamed tiles do not fit in shared memory: the first held operand lies in tensor memory, the
// streamed tiles have one buffer, and a tile's products are written over the scores they came from. What is left to run
// side by side is little, so the row warps also issue. An item of one tile has nothing to run side by side.
template <int HD, bool kWide>
struct BwdWide {
  static constexpr int kGroups = 4;
  static constexpr int kThreads = kRows * kGroups;
  using Held = Stage<HD, kRows, kThreads, kWide>;
  using Tile = Stage<HD, kStream, kThreads, kWide>;
  static constexpr uint32_t kHeld1 = 0, kTile0 = Held::kBytes, kTile1 = kTile0 + Tile::kBytes;
  // (up to head dim 64 as much as the kernel with roles has, so that items done again on the CUDA cores stream the same tiles)
  static constexpr uint32_t kBytes = HD <= 64 ? std::min(Bwd<HD, false>::kBytes, Bwd<HD, true>::kBytes) : kTile1 + Tile::kBytes + 1024;
  static_assert(kTile1 + Tile::kBytes + 1024 <= kBytes, "shared memory");
  static constexpr uint32_t kS = 0, kDp = kStream, kDs = 2 * kStream, kP = kDs + 3 * kPieceCols, kHeldT = kP + 3 * kPieceCols;
  static constexpr uint32_t kOut = 0;
  static constexpr int kCols = 512;
  static_assert(kHeldT + 3 * HD / 2 <= kCols && kOut + HD <= kDs, "tensor memory");
};

template <int HD, bool kKV, bool kWide>
__global__ void __launch_bounds__(BwdWide<HD, kWide>::kThreads, 1) f32_bwd_wide_kernel(const __grid_constant__ Params g) {
  using L = BwdWide<HD, kWide>;
  constexpr int G = L::kGroups, CW = kStream / G, OW = HD / G;
  extern __shared__ __align__(16) unsigned char raw[];
  __shared__ uint32_t slot, abort_flag, hidden[2];
  __shared__ __align__(8) uint64_t bars[3];
  __shared__ __align__(16) float lse_hi[kStream], lse_lo[kStream], deltas[kStream];  // dK/dV: of the streamed rows
  uint32_t tmem;
  if (!set_up<L::kCols, 3>(g, &slot, &abort_flag, bars, tmem)) return;
  const uint32_t base = align_1024(smem_addr(raw));
  const uint32_t scored = smem_addr(bars), weighed0 = smem_addr(bars + 1), weighed1 = smem_addr(bars + 2);
  const int warp = threadIdx.x >> 5, group = warp >> 2;
  const int row = (warp & 3) * 32 + (threadIdx.x & 31);
  const uint32_t lanes = tmem + (static_cast<uint32_t>((warp & 3) * 32) << 16);
  const bool issues = __shfl_sync(kFull, warp, 0) == 0;  // the warp that issues, one lane of it elected per bunch

  int problem, at;
  cta_work(blockIdx.x, g.slots, g.bh, g.group, problem, at);
  const int first = (kKV ? at : g.slots - 1 - at) * kRows;  // the longest causal streams first
  const long long b = problem;
  // the held pair (against which the tiles are scored) and the streamed pair
  const int owned = kKV ? g.t_k : g.t_q, streamed = kKV ? g.t_q : g.t_k;
  const float* held0 = (kKV ? g.k : g.q) + b * owned * g.hd;
  const float* held1 = (kKV ? g.v : g.dout) + b * owned * g.hd_v;
  const float* stream0 = (kKV ? g.q : g.k) + b * streamed * g.hd;
  const float* stream1 = (kKV ? g.dout : g.v) + b * streamed * g.hd_v;
  const float* mask = g.mask ? g.mask + b * g.t_k : nullptr;
  const int begin = kKV && g.causal ? first : 0;
  const int end = !kKV && g.causal ? min(streamed, first + kRows) : streamed;
  const int n = (end - begin + kStream - 1) / kStream;
  const int mine = first + row;  // this thread's row

  Check check;
  // the streamed tile j, and what goes with its rows
  auto stage_tile = [&](int j) {
    const int x0 = begin + j * kStream;
    typename L::Tile tile0, tile1;
    tile0.load(stream0, x0, streamed, g.hd);
    tile1.load(stream1, x0, streamed, g.hd_v);
    if (kKV) {
      const float lse = row_value(g.lse_in + b * g.t_q, x0, streamed), delta = row_value(g.delta + b * g.t_q, x0, streamed);
      if (threadIdx.x < kStream) {
        float hi, lo;
        to_minus_log2(lse, hi, lo);
        lse_hi[threadIdx.x] = hi;
        lse_lo[threadIdx.x] = lo;
        deltas[threadIdx.x] = -delta;
        check.sums |= !(lse < INFINITY);  // (its weights are not finite, which would only be seen in the sums)
      }
    } else if (mask) {
      post_hidden(hidden, row_value(mask, x0, streamed));
    }
    tile0.store(base + L::kTile0, check);
    tile1.store(base + L::kTile1, check);
    fence_async_shared();
  };
  auto issue_tile = [&]() {
    tc_fence_after_sync();
    issue_scores<HD, true>(tmem + L::kS, tmem + L::kHeldT, base + L::kTile0);
    issue_scores<HD, false>(tmem + L::kDp, base + L::kHeld1, base + L::kTile1);
    mma_commit(scored);
  };

  float my_hi = 0.f, my_lo = 0.f, my_delta = 0.f;  // dQ: of this thread's row
  bool live = mine < owned;
  {
    float x[OW / 8][8];
#pragma unroll
    for (int c = 0; c < OW / 8; ++c) load8<kWide>(x[c], held0, mine, owned, group * OW + 8 * c, g.hd);
    typename L::Held stage1;
    stage1.load(held1, first, owned, g.hd_v);
    uint32_t h[OW / 2], m[OW / 2], l[OW / 2];
#pragma unroll
    for (int e = 0; e < OW / 2; ++e) split_pair<true>(f2_pack(x[e / 4][2 * (e % 4)], x[e / 4][2 * (e % 4) + 1]), h[e], m[e], l[e], check);
    const uint32_t to = lanes + L::kHeldT + group * (OW / 2);
    tmem_st<OW / 2>(to, h);
    tmem_st<OW / 2>(to + HD / 2, m);
    tmem_st<OW / 2>(to + HD, l);
    tmem_st_wait();
    tc_fence_before_sync();
    if constexpr (kKV) {
      if (live && mask) live = mask[mine] != 0.f;
    } else if (live) {
      to_minus_log2(g.lse_in[b * g.t_q + mine], my_hi, my_lo);
      my_delta = -g.delta[b * g.t_q + mine];
    }
    stage1.store(base + L::kHeld1, check);
  }
  stage_tile(0);  // (fences the held rows too)
  __syncthreads();
  if (issues && elect_one()) issue_tile();

  uint64_t acc0[OW / 2], acc1[OW / 2];  // dQ, or dV and dK
#pragma unroll
  for (int c = 0; c < OW / 2; ++c) acc0[c] = acc1[c] = 0;
  auto gather = [&](uint64_t(&acc)[OW / 2]) {
    tc_fence_after_sync();
    uint32_t o[OW];
    tmem_ld<OW>(lanes + L::kOut + group * OW, o);
    tmem_ld_wait();
    tc_fence_before_sync();
#pragma unroll
    for (int c = 0; c < OW / 2; ++c) acc[c] = f2_add(acc[c], f2_pack_bits(o[2 * c], o[2 * c + 1]));
  };
  bool ok = true;
  for (int j = 0; j < n; ++j) {
    const int x0 = begin + j * kStream;
    ok &= mbar_wait(scored, j & 1, g.status, 0x0b00u);
    tc_fence_after_sync();
    uint32_t s[CW], dp[CW];
    tmem_ld<CW>(lanes + L::kS + group * CW, s);
    tmem_ld<CW>(lanes + L::kDp + group * CW, dp);
    tmem_ld_wait();
    int from = 0, to = streamed - x0 - group * CW;
    if (g.causal) {
      if (kKV) from = mine - x0 - group * CW;
      else to = min(to, mine - x0 - group * CW + 1);
    }
    uint32_t unseen = outside<CW>(from, live ? to : 0);
    if (!kKV && mask) unseen |= my_hidden<CW>(hidden, group);
    uint64_t p[CW / 2], ds[CW / 2];
    weigh_scores<CW>(g, s, dp, unseen, [&](int c, uint64_t& hi, uint64_t& lo, uint64_t& delta) {
      if (kKV) {
        hi = *reinterpret_cast<const uint64_t*>(&lse_hi[group * CW + c]);
        lo = *reinterpret_cast<const uint64_t*>(&lse_lo[group * CW + c]);
        delta = *reinterpret_cast<const uint64_t*>(&deltas[group * CW + c]);
      } else {
        hi = f2_pack(my_hi, my_hi), lo = f2_pack(my_lo, my_lo), delta = f2_pack(my_delta, my_delta);
      }
    }, p, ds);
    hand_over<CW>(lanes + L::kDs + group * (CW / 2), ds);
    if (kKV) hand_over<CW>(lanes + L::kP + group * (CW / 2), p);
    tmem_st_wait();
    tc_fence_before_sync();
    if (!__syncthreads_and(ok && !check.bad())) break;  // (nothing is in flight here)
    if (issues && elect_one()) {
      tc_fence_after_sync();
      issue_weigh<HD>(tmem + L::kOut, tmem + (kKV ? L::kP : L::kDs), base + (kKV ? L::kTile1 : L::kTile0));
      mma_commit(weighed0);
    }
    ok &= mbar_wait(weighed0, j & 1, g.status, 0x0b01u);
    gather(acc0);
    if (kKV) {
      if (!__syncthreads_and(ok)) break;
      if (issues && elect_one()) {
        tc_fence_after_sync();
        issue_weigh<HD>(tmem + L::kOut, tmem + L::kDs, base + L::kTile0);
        mma_commit(weighed1);
      }
      ok &= mbar_wait(weighed1, j & 1, g.status, 0x0b02u);
      gather(acc1);
    }
    if (j + 1 < n) {
      stage_tile(j + 1);
      if (!__syncthreads_and(ok)) break;
      if (issues && elect_one()) issue_tile();
    }
  }
  if (kKV) settle(acc1, check);
  else settle(acc0, check);
  ok = __syncthreads_and(ok);
  const bool bad = __syncthreads_or(check.bad());
  if (ok && bad) {
    rows_again<HD, kKV ? Op::BwdKV : Op::BwdQ, L::kThreads / tiled::kThreads, L::kBytes, kWide>(g, b, first, raw);
  } else if (ok) {
    const int top = first + (warp & 3) * 32;
    if (kKV) {
      store_rows<OW>(g.dv + b * owned * g.hd_v, acc0, top, owned, group * OW, g.hd_v, g.wide_out);
      store_rows<OW>(g.dk + b * owned * g.hd, acc1, top, owned, group * OW, g.hd, g.wide_out);
    } else {
      store_rows<OW>(g.dq + b * owned * g.hd, acc0, top, owned, group * OW, g.hd, g.wide_out);
    }
  }
  tear_down<L::kCols>(g, tmem);
}

bool aligned(const void* x) { return (reinterpret_cast<uintptr_t>(x) & 15u) == 0; }  // (null is)

// Forwards up to head dim 64 in f32_fwd_pair_kernel: those of one key tile that have a block for two SMs out of three and up to four for each,
// and those of up to five tiles that have one to two blocks to an SM, which it holds all at once where the other kernel takes two rounds.
// Measured on B200, us, here / in roles:
//   16 x 16 x 32: 16 problems 5.0 / 5.1, 100 5.1 / 5.7, 148 5.1 / 6.0, 149 6.4 / 8.3, 296 6.8 / 8.8, 400 10.7 / 11.4, 592 12.8 / 14.4, 5000 97 / 105
//   64 x 64 x 32: 16 5.1 / 5.0, 100 5.2 / 5.7, 148 5.2 / 6.0, 149 6.5 / 8.1, 296 7.1 / 8.6, 400 11.0 / 11.2, 592 13.0 / 14.1, 700 16.8 / 16.8, 5000 109 / 103
//   64 x 64 x 64: 16 6.2 / 6.3, 100 6.3 / 7.0, 149 7.9 / 10.5, 296 8.7 / 11.1, 592 16.1 / 18.5, 5000 146 / 143; 1000 of 300 x 64 94 / 89
//   128 x 128 x 32: 148 7.3 / 7.1, 149 9.0 / 10.6, 296 9.7 / 11.1, 297 14.6 / 14.1; 64 x 320 x 32: 149 15.7 / 17.5, 296 16.5 / 17.9
//   64 x 100 x 64: 148 8.9 / 8.6, 149 11.3 / 13.4, 296 11.9 / 13.9, 297 18.3 / 17.8; 64 x 320 x 64: 149 20.6 / 21.8, 222 22.0 / 22.1; 100 x 448 x 64: 222 29.0 / 28.2
bool two_to_an_sm(const Problem& p, long long blocks, int sms) {
  if (p.t_k <= kStream) return 3 * blocks > 2LL * sms && blocks <= 4LL * sms;
  return p.t_k <= 5 * kStream && blocks > sms && blocks <= 2LL * sms;
}

// Backward passes up to head dim 64 in the kernel without roles: one tile of streamed rows, one block to a problem and at most one to an SM.
// Measured on B200, us, here / in roles, by own x streamed rows x width:
//   dQ: 16 x 16 x 64 1 problem 7.7 / 8.5, 148 8.4 / 8.7; 64 x 64 x 64 1 8.5 / 8.5, 148 9.2 / 9.3; 100 x 64 x 64 100 10.0 / 9.4; 100 x 64 x 40 1 8.4 / 8.5, 148 9.2 / 9.7;
//     16 x 16 x 32 1 6.3 / 6.6, 148 6.8 / 6.9; 32 x 32 x 32 1 6.3 / 6.5, 100 6.7 / 7.0; 64 x 64 x 32 1 6.5 / 6.5, 148 7.3 / 7.1; 64 x 64 x 16 100 6.6 / 6.9, 148 6.9 / 6.9
//   dK and dV: 16 x 16 x 32 64 6.4 / 6.4, 100 6.4 / 6.6, 148 6.4 / 7.0; 64 x 64 x 32 64 6.7 / 6.7, 148 6.8 / 7.2; 100 x 64 x 32 148 7.3 / 7.6; 64 x 64 x 64 64 8.9 / 8.6,
//     100 9.0 / 9.0, 148 9.0 / 9.3
//   rows that are not whole 16-byte pieces: dQ 16 x 16 x 25 1 7.1 / 8.0, 148 7.4 / 8.6; 128 x 64 x 50 64 15.3 / 16.5; dK and dV 16 x 16 x 25 1 6.3 / 7.0, 100 x 64 x 30 148 11.9 / 12.6
bool one_tile(Op op, const Problem& p, bool wide, int sms) {
  const int widest = p.hd > p.hd_v ? p.hd : p.hd_v, owned = op == Op::BwdQ ? p.t_q : p.t_k, streamed = op == Op::BwdQ ? p.t_k : p.t_q;
  if (streamed > kStream || owned > kRows || p.bh > sms) return false;
  if (!wide) return true;
  if (op == Op::BwdKV) return 3 * p.bh > 2LL * sms;
  if (widest > 32) return owned <= 64 || widest <= 40;
  return owned <= 64 && (widest <= 24 || (owned <= 32 && streamed <= 32));
}

// A problem's bits do not depend on which kernel it comes to, on the CUDA cores either.
template <int HD, bool kWide>
constexpr bool same_tiles_again() {
  return again_tile<HD, Op::Fwd, 1, FwdPair<HD, kWide>::kBytes>() == again_tile<HD, Op::Fwd, kAgainGroups, Fwd<HD>::kBytes>() &&
         again_tile<HD, Op::BwdQ, kAgainGroups, BwdWide<HD, kWide>::kBytes>() == again_tile<HD, Op::BwdQ, kAgainGroups, Bwd<HD, false>::kBytes>() &&
         again_tile<HD, Op::BwdKV, kAgainGroups, BwdWide<HD, kWide>::kBytes>() == again_tile<HD, Op::BwdKV, kAgainGroups, Bwd<HD, true>::kBytes>();
}
static_assert(same_tiles_again<32, true>() && same_tiles_again<32, false>() && same_tiles_again<64, true>() && same_tiles_again<64, false>());

template <int HD, bool kWide>
int launch_sized(Op op, const Problem& p) {
  Params g = {};
  auto in = [](const void* x) { return static_cast<const float*>(x); };
  g.q = in(p.q), g.k = in(p.k), g.v = in(p.v), g.mask = in(p.mask), g.dout = in(p.dout), g.lse_in = in(p.lse_in), g.delta = in(p.delta);
  g.out = static_cast<float*>(p.out), g.lse_out = static_cast<float*>(p.lse_out);
  g.dq = static_cast<float*>(p.dq), g.dk = static_cast<float*>(p.dk), g.dv = static_cast<float*>(p.dv);
  g.status = p.status;
  if (g.status == nullptr)
    if (int rc = status_word(&g.status)) return rc;
  g.bh = p.bh;
  g.slots = ((op == Op::BwdKV ? p.t_k : p.t_q) + kRows - 1) / kRows;
  g.t_q = p.t_q, g.t_k = p.t_k, g.hd = p.hd, g.hd_v = p.hd_v, g.causal = p.causal ? 1 : 0;
  g.scale = static_cast<float>(p.scale);
  g.ds_scale = g.scale * kDsUp;
  // The additions that make up a score truncate, which takes 4e-8 (one of them, head dims up to 16) to 11e-8 (eight) of it
  // on average; 8e-8 is put back here. Measured against float64 at 22 shapes, 2-norm, without -> with: L 3.6e-8 -> 2.9e-8 and O
  // 1.25e-7 -> 1.02e-7 at 256 x 256 x 64, dQ 4.4e-7 -> 3.9e-7 at 500 x 64 x 128, none worse (4e-8 and 12e-8 do less).
  const double c = static_cast<double>(g.scale) * 1.4426950408889634 * (1.0 + 8e-8);
  g.c_hi = static_cast<float>(c);
  if (g.c_hi > c) g.c_hi = nextafterf(g.c_hi, 0.f);
  g.c_lo = static_cast<float>(c - g.c_hi);
  if (!(g.c_lo > 0.f)) g.c_lo = 1e-37f;  // a score of -inf has to stay one
  g.wide_out = p.hd % 4 == 0 && p.hd_v % 4 == 0;
  if (op == Op::Fwd) g.wide_out = g.wide_out && aligned(p.out);
  else g.wide_out = g.wide_out && aligned(p.dq) && aligned(p.dk) && aligned(p.dv);
  const long long blocks = p.bh * g.slots;
  int sms = 0;
  if (int rc = sm_count(&sms)) return rc;
  g.group = work_group(p, blocks, sms);
  void (*kernel)(const Params) = nullptr;
  uint32_t shared = 0, threads = 0;
  long long grid = blocks;
  const bool two = HD <= 32 && op == Op::BwdQ && blocks <= sms;  // threads to a row (see f32_bwd_kernel)
  bool roles = true;
  const bool pair = HD <= 64 && op == Op::Fwd && two_to_an_sm(p, blocks, sms);
  const bool alone = HD <= 64 && op != Op::Fwd && one_tile(op, p, kWide, sms);
  if (pair) {
    if constexpr (HD <= 64) kernel = f32_fwd_pair_kernel<HD, kWide>, shared = FwdPair<HD, kWide>::kBytes, threads = FwdPair<HD, kWide>::kThreads;
    roles = false;
  } else if (op == Op::Fwd) {
    kernel = f32_fwd_kernel<HD, kWide>, shared = Fwd<HD>::kBytes, threads = Roles<Fwd<HD>::kGroups>::kThreads;
  } else if constexpr (HD > 64) {
    using B = BwdWide<HD, kWide>;
    kernel = op == Op::BwdQ ? f32_bwd_wide_kernel<HD, false, kWide> : f32_bwd_wide_kernel<HD, true, kWide>;
    shared = B::kBytes, threads = B::kThreads;
    roles = false;
  } else if (alone) {
    using B = BwdWide<HD, kWide>;
    kernel = op == Op::BwdQ ? f32_bwd_wide_kernel<HD, false, kWide> : f32_bwd_wide_kernel<HD, true, kWide>;
    shared = B::kBytes, threads = B::kThreads;
    roles = false;
  } else if (op == Op::BwdQ) {
    kernel = f32_bwd_kernel<HD, false, kWide, 4>, shared = Bwd<HD, false>::kBytes, threads = Roles<4>::kThreads;
    if constexpr (HD <= 32)
      if (two) kernel = f32_bwd_kernel<HD, false, kWide, 2>, threads = Roles<2>::kThreads;
  } else {
    kernel = f32_bwd_kernel<HD, true, kWide, 4>, shared = Bwd<HD, true>::kBytes, threads = Roles<4>::kThreads;
  }
  if (roles) {
    // every SM has its block, and they are done together: as many blocks to an SM one after the other as the limit on a
    // block's items asks for
    const long long turn = static_cast<long long>(sms) * kMostItems;
    grid = std::min(blocks, sms * ((blocks + turn - 1) / turn));
  }
  // the attribute is per device and per kernel instantiation; set it on first use there
  const int which = alone ? 4 + static_cast<int>(op) : pair ? 4 : two ? 3 : static_cast<int>(op);
  static bool sized[64][7] = {};
  int device = 0;
  LIMN_CUDA(cudaGetDevice(&device), "asking for the current device");
  if (device < 0 || device >= 64 || !sized[device][which]) {
    LIMN_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(shared)),
              "sizing shared memory for a float32 sdpa kernel");
    if (device >= 0 && device < 64) sized[device][which] = true;
  }
  LIMN_CUDA(launch_overlapped(kernel, dim3(static_cast<unsigned>(grid)), dim3(threads), shared, p.stream, g),
            "launching a float32 sdpa kernel");
  note_launches(1);
  return LIMN_B200_OK;
}

// Many short problems are better off in the tiled CUDA-core kernels: with both sides inside one 64-row tile half of a block's
// 128 rows are empty, a head dim below the kernel's width is padding, and a block's fixed cost is all there is, while several
// of their 256-thread blocks share an SM. Measured on B200 as time here over time there, 16 x 16 / 32 x 32 / 64 x 64 rows:
//   forward  8: 1.23-1.35 / 1.20-1.29 / 1.09-1.19; 16: 1.14-1.23 / 1.11-1.18 / 1.03-1.10; 24: 1.08-1.14 / 1.05-1.10 / 0.97-0.99;
//            32: 1.03-1.05 / 0.99-1.02 / 0.86-0.94; 40: 0.7-0.95; 72: 1.1-1.36 / 1.0-1.3 / 0.63-0.77; 100: 1.04-1.26 / 0.97-1.2 /
//            0.55-0.72; 128: 0.98-1.18 / 0.88-1.13 / 0.51-0.68
//   dQ       8: 0.88-1.25; 16: 0.67-1.13; 24: 0.58-1.0; 32: 0.56-0.93; 72: 1.31-1.46 / 1.09-1.34 / 0.6-0.8; 100: 1.16-1.27 / 1.02-1.18 /
//            0.56-0.7; 128: 1.05-1.13 / 0.89-1.08 / 0.53-0.66
//   dK, dV   8, up to 256 problems 0.94-1.07 and beyond 0.85-0.97 / 0.85-0.94 / 0.76-0.85; 16: 0.8-0.98 / 0.77-0.95 / 0.59-0.88; 24 and 32:
//            0.48-0.9; 72: 0.83-1.01; more: 0.35-0.9
// At head dim 64 all three gain here (0.4-0.96), and so does everything at 128 problems, one block to an SM, and from 65 rows on. What
// is nearer to float64 on one side stays there: the forward at up to 24 with at most two problems to an SM here, the backward at up to 24
// there (2-norm, here over there, the worst of 13 to 19 shapes: widths 24 and 24 dV 1.05; 24 and 8 dQ 1.09, dK 1.05; 8 and 24 dQ 1.06; 16 and 8 dK 1.05; from 25 on 0.55
// to 0.88, whatever the other width) but for dK and dV at 16 and 16 with 32 queries or more (0.82-0.99).
bool short_rows(Op op, const Problem& p) {
  if (p.t_q > 64 || p.t_k > 64) return false;
  int sms = 0;
  if (sm_count(&sms) != LIMN_B200_OK || p.bh <= sms) return false;
  const int widest = p.hd > p.hd_v ? p.hd : p.hd_v;
  if (widest > 64) return op == Op::Fwd ? p.t_k <= 32 : op == Op::BwdQ && p.t_k <= (widest <= 100 ? 32 : 16);
  if (op == Op::Fwd) return widest <= 24 && p.bh > 2LL * sms;
  if (widest > 24) return false;
  if (widest > 16) return p.bh > 4LL * sms && (op == Op::BwdQ || p.t_q <= 32);
  return op == Op::BwdQ || (p.bh > 3LL * sms && (p.hd < 16 || p.hd_v < 16 || p.t_q < 32));
}

}  // namespace

bool f32_split_serves(Op op, const Problem& p) {
  if (p.dtype != LIMN_B200_F32 || p.hd > 128 || p.hd_v > 128) return false;
  if (p.layout != LIMN_B200_BHTD || p.strided) return false;
  if (p.t_q < 16 || p.t_k < 16) return false;  // most of a 128 x 64 tile would be idle
  // row maxima are taken before scaling, and the scale is folded into exp2 in two parts
  const float scale = static_cast<float>(p.scale);
  if (!(scale > 1e-20f && scale < 1e20f)) return false;
  const long long rows = op == Op::BwdKV ? p.t_k : p.t_q;
  return p.bh * ((rows + kRows - 1) / kRows) <= 0x7fffffffLL && !short_rows(op, p);
}

int f32_split_launch(Op op, const Problem& p) {
  const int widest = p.hd > p.hd_v ? p.hd : p.hd_v;
  const bool wide = p.hd % 4 == 0 && p.hd_v % 4 == 0 && aligned(p.q) && aligned(p.k) && aligned(p.v) && aligned(p.dout);
  if (widest <= 32) return wide ? launch_sized<32, true>(op, p) : launch_sized<32, false>(op, p);
  if (widest <= 64) return wide ? launch_sized<64, true>(op, p) : launch_sized<64, false>(op, p);
  return wide ? launch_sized<128, true>(op, p) : launch_sized<128, false>(op, p);
}

}  // namespace limn_b200
