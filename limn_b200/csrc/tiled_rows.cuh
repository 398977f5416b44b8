// The rows of a float32 (or 16-bit, widened) attention problem on the CUDA cores: 256 threads own 64 rows and stream the
// other side through shared memory in tiles of BN rows. The kernels of sdpa_general_tiled.cu are these functions and
// nothing else; the float32 tensor-core kernels (sdpa_f32_sm100.cu) call them for blocks whose operands do not split.
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <cmath>
#include <cstdint>

#include "common.h"

namespace limn_b200 {
namespace tiled {

constexpr int kThreads = 256;  // of a group of threads that works on one block of rows
constexpr int kBM = 64;   // rows a block owns
constexpr int kPad = 4;   // floats of padding per shared-memory row: keeps float4 reads of 16 rows on distinct banks

template <typename T>
__device__ __forceinline__ float widen(T x);
template <>
__device__ __forceinline__ float widen<float>(float x) { return x; }
template <>
__device__ __forceinline__ float widen<__half>(__half x) { return __half2float(x); }
template <>
__device__ __forceinline__ float widen<__nv_bfloat16>(__nv_bfloat16 x) { return __bfloat162float(x); }

template <typename T>
__device__ __forceinline__ T narrow(float x);
template <>
__device__ __forceinline__ float narrow<float>(float x) { return x; }
template <>
__device__ __forceinline__ __half narrow<__half>(float x) { return __float2half_rn(x); }
template <>
__device__ __forceinline__ __nv_bfloat16 narrow<__nv_bfloat16>(float x) { return __float2bfloat16_rn(x); }

// Rows [first, first + R) of a (rows, width) matrix into dst[R][HD + kPad] as float; rows past the matrix and
// columns past `width` become zero, so the products below may run over whole tiles.
template <typename T, int HD, int R>
__device__ __forceinline__ void stage(float* dst, const T* src, int first, int rows, int width, bool wide, int thread) {
  constexpr int LD = HD + kPad;
  constexpr int V = 16 / sizeof(T);  // elements per 16-byte piece
  if (wide) {                        // width is a whole number of pieces and the base is 16-byte aligned
    constexpr int per_row = HD / V;
    for (int e = thread; e < R * per_row; e += kThreads) {
      const int r = e / per_row, c = (e - r * per_row) * V;
      float x[V];
      if (first + r < rows && c < width) {
        const uint4 raw = *reinterpret_cast<const uint4*>(src + static_cast<long long>(first + r) * width + c);
        const T* t = reinterpret_cast<const T*>(&raw);
#pragma unroll
        for (int i = 0; i < V; ++i) x[i] = widen<T>(t[i]);
      } else {
#pragma unroll
        for (int i = 0; i < V; ++i) x[i] = 0.f;
      }
#pragma unroll
      for (int i = 0; i < V; i += 4)
        *reinterpret_cast<float4*>(dst + r * LD + c + i) = make_float4(x[i], x[i + 1], x[i + 2], x[i + 3]);
    }
  } else {
    for (int e = thread; e < R * HD; e += kThreads) {
      const int r = e / HD, c = e - r * HD;
      dst[r * LD + c] = (first + r < rows && c < width) ? widen<T>(src[static_cast<long long>(first + r) * width + c]) : 0.f;
    }
  }
}

// acc[a][b] += sum_d A[row0 + a][d] * B[col0 + 16 b][d] for d < depth (a multiple of 4)
template <int LD, int NB>
__device__ __forceinline__ void dot_tiles(float (&acc)[4][NB], const float* a_rows, const float* b_rows, int depth) {
  for (int d = 0; d < depth; d += 4) {
    float4 av[4], bv[NB];
#pragma unroll
    for (int a = 0; a < 4; ++a) av[a] = *reinterpret_cast<const float4*>(a_rows + a * LD + d);
#pragma unroll
    for (int b = 0; b < NB; ++b) bv[b] = *reinterpret_cast<const float4*>(b_rows + b * 16 * LD + d);
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
      for (int b = 0; b < NB; ++b) {
        acc[a][b] = fmaf(av[a].x, bv[b].x, acc[a][b]);
        acc[a][b] = fmaf(av[a].y, bv[b].y, acc[a][b]);
        acc[a][b] = fmaf(av[a].z, bv[b].z, acc[a][b]);
        acc[a][b] = fmaf(av[a].w, bv[b].w, acc[a][b]);
      }
  }
}

// Columns of the head dim one thread owns in the second product: NV = HD / 16 of them, as NV / VW vectors of VW
// consecutive floats, vector c of thread tx starting at column c * 16 * VW + tx * VW.
template <int HD>
struct Cols {
  static constexpr int NV = HD / 16;
  static constexpr int VW = NV < 4 ? NV : 4;
  static constexpr int NC = NV / VW;
  __device__ static __forceinline__ int at(int tx, int i) { return (i / VW) * 16 * VW + tx * VW + (i % VW); }
};

// acc[a][i] += sum_j W[row0 + a][j] * X[j][col(i)] for j < BN
template <int HD, int BN>
__device__ __forceinline__ void weigh_rows(float (&acc)[4][HD / 16], const float* w_rows, const float* x, int tx) {
  using C = Cols<HD>;
  constexpr int LD = HD + kPad, LP = BN + kPad;
#pragma unroll 2
  for (int j = 0; j < BN; j += 4) {
    float4 w4[4];
#pragma unroll
    for (int a = 0; a < 4; ++a) w4[a] = *reinterpret_cast<const float4*>(w_rows + a * LP + j);
#pragma unroll
    for (int jj = 0; jj < 4; ++jj) {
      float xv[C::NV];
#pragma unroll
      for (int c = 0; c < C::NC; ++c) {
        const float* from = x + (j + jj) * LD + c * 16 * C::VW + tx * C::VW;
        if constexpr (C::VW == 4) {
          const float4 t = *reinterpret_cast<const float4*>(from);
          xv[c * 4] = t.x, xv[c * 4 + 1] = t.y, xv[c * 4 + 2] = t.z, xv[c * 4 + 3] = t.w;
        } else if constexpr (C::VW == 2) {
          const float2 t = *reinterpret_cast<const float2*>(from);
          xv[c * 2] = t.x, xv[c * 2 + 1] = t.y;
        } else {
          xv[c] = *from;
        }
      }
#pragma unroll
      for (int a = 0; a < 4; ++a) {
        const float w = jj == 0 ? w4[a].x : jj == 1 ? w4[a].y : jj == 2 ? w4[a].z : w4[a].w;
#pragma unroll
        for (int i = 0; i < C::NV; ++i) acc[a][i] = fmaf(w, xv[i], acc[a][i]);
      }
    }
  }
}

// the rows this thread owns of a block's result, written where they are real
template <typename T, int HD>
__device__ __forceinline__ void store_rows(T* dst, const float (&acc)[4][HD / 16], long long first_row, int rows_here,
                                           int width, int ty, int tx) {
  using C = Cols<HD>;
#pragma unroll
  for (int a = 0; a < 4; ++a) {
    const int r = ty * 4 + a;
    if (r >= rows_here) continue;
#pragma unroll
    for (int i = 0; i < C::NV; ++i) {
      const int col = C::at(tx, i);
      if (col < width) dst[(first_row + r) * width + col] = narrow<T>(acc[a][i]);
    }
  }
}

__device__ __forceinline__ float group_max(float x) {  // over the 16 threads that share a row
#pragma unroll
  for (int off = 8; off > 0; off >>= 1) x = fmaxf(x, __shfl_xor_sync(0xffffffffu, x, off));
  return x;
}
__device__ __forceinline__ float group_sum(float x) {
#pragma unroll
  for (int off = 8; off > 0; off >>= 1) x += __shfl_xor_sync(0xffffffffu, x, off);
  return x;
}

// A row's columns by its total, every quotient rounded to nearest from one reciprocal and two corrections. (Markstein 1990: with the correctly
// rounded reciprocal, a quotient within an ulp and its exact remainder, the corrected quotient is the correctly rounded one; the first
// correction gives the quotient within an ulp.) The remainder q total - x is a multiple of ulp(q) ulp(total), which is a float32 for totals from 1/2 if
// q is from 2^-102: so columns go up by 2^64 first and quotients down again, and a row of columns too large for that, or of another total,
// divides. (A quotient below 2^-126 is rounded twice, to 24 bits and to those that it has.) With that sign of the remainder a zero keeps its own.
constexpr float kQuotientUp = 0x1p64f;
__device__ __forceinline__ bool by_reciprocal(float largest, float total) { return total >= 0.5f && total < 0x1p40f && largest < 0x1p60f; }

struct Args {
  const void *q, *k, *v, *mask, *dout;
  const float *lse_in, *delta;
  void *out, *dq, *dk, *dv;
  float* lse_out;
  int t_q, t_k, hd, hd_v, causal;
  float scale;
  bool wide_qk, wide_v;  // 16-byte loads are safe for (q, k) and for (v, dO)
};

// ---- forward: O and L for 64 query rows (oracle: limn/sdpa.py:114-137) ----
template <typename T, int HD, int BN, typename Sync>
__device__ __forceinline__ void fwd_rows(const Args& g, long long b, int i0, float* shared, int thread, Sync sync) {
  constexpr int LD = HD + kPad, LP = BN + kPad, NB = BN / 16, NV = HD / 16;
  float* qs = shared;
  float* ks = qs + kBM * LD;
  float* vs = ks + BN * LD;
  float* ps = vs + BN * LD;
  const int tx = thread & 15, ty = thread >> 4;
  const T* q = static_cast<const T*>(g.q) + b * g.t_q * g.hd;
  const T* k = static_cast<const T*>(g.k) + b * g.t_k * g.hd;
  const T* v = static_cast<const T*>(g.v) + b * g.t_k * g.hd_v;
  const T* mask = g.mask ? static_cast<const T*>(g.mask) + b * g.t_k : nullptr;
  const int depth = (g.hd + 3) & ~3;

  stage<T, HD, kBM>(qs, q, i0, g.t_q, g.hd, g.wide_qk, thread);
  float top[4], denom[4], acc[4][NV];
#pragma unroll
  for (int a = 0; a < 4; ++a) {
    top[a] = -INFINITY, denom[a] = 0.f;
#pragma unroll
    for (int i = 0; i < NV; ++i) acc[a][i] = 0.f;
  }
  const int keys_end = g.causal ? min(g.t_k, i0 + kBM) : g.t_k;
  for (int j0 = 0; j0 < keys_end; j0 += BN) {
    sync();  // the tile before this one has been read by everyone
    stage<T, HD, BN>(ks, k, j0, g.t_k, g.hd, g.wide_qk, thread);
    stage<T, HD, BN>(vs, v, j0, g.t_k, g.hd_v, g.wide_v, thread);
    bool open[NB];
#pragma unroll
    for (int c = 0; c < NB; ++c) {
      const int j = j0 + tx + 16 * c;
      open[c] = j < g.t_k && (!mask || widen<T>(mask[j]) != 0.f);
    }
    sync();
    float s[4][NB];
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
      for (int c = 0; c < NB; ++c) s[a][c] = 0.f;
    dot_tiles<LD, NB>(s, qs + ty * 4 * LD, ks + tx * LD, depth);
#pragma unroll
    for (int a = 0; a < 4; ++a) {
      const int i = i0 + ty * 4 + a;
      float tile_top = -INFINITY;
#pragma unroll
      for (int c = 0; c < NB; ++c) {
        const bool seen = open[c] && (!g.causal || j0 + tx + 16 * c <= i);
        s[a][c] = seen ? s[a][c] * g.scale : -INFINITY;
        tile_top = fmaxf(tile_top, s[a][c]);
      }
      const float raised = fmaxf(top[a], group_max(tile_top));
      // as long as no key is visible the weights are taken against 0: exp(-inf), and NaN for a NaN score
      const float base = raised == -INFINITY ? 0.f : raised;
      const float shrink = expf(top[a] - base);  // exp(-inf) = 0 on the first visible tile
#pragma unroll
      for (int c = 0; c < NB; ++c) s[a][c] = expf(s[a][c] - base);
      float added = 0.f;
#pragma unroll
      for (int c = 0; c < NB; ++c) {
        added += s[a][c];
        ps[(ty * 4 + a) * LP + tx + 16 * c] = s[a][c];
      }
      denom[a] = denom[a] * shrink + added;  // this thread's share; the shares meet after the last tile
#pragma unroll
      for (int i2 = 0; i2 < NV; ++i2) acc[a][i2] *= shrink;
      top[a] = raised;
    }
    sync();
    weigh_rows<HD, BN>(acc, ps + ty * 4 * LP, vs, tx);
  }
  const int rows_here = min(kBM, g.t_q - i0);
#pragma unroll
  for (int a = 0; a < 4; ++a) {
    const float total = group_sum(denom[a]);
    // (head dims above 32 take 0.88 to 0.97 of the time that divisions do, up to 32, two columns a thread, 0.99 to 1.04)
    float largest = 0.f;
#pragma unroll
    for (int i = 0; i < NV; ++i) largest = fmaxf(largest, fabsf(acc[a][i]));
    if (NV > 2 && by_reciprocal(largest, total)) {
      const float r = __frcp_rn(total);
#pragma unroll
      for (int i = 0; i < NV; ++i) {
        const float x = acc[a][i] * kQuotientUp;
        float q = x * r;
        q = fmaf(fmaf(q, total, -x), -r, q);
        acc[a][i] = fmaf(fmaf(q, total, -x), -r, q) * (1.f / kQuotientUp);
      }
    } else {
#pragma unroll
      for (int i = 0; i < NV; ++i) acc[a][i] = acc[a][i] / total;  // 0/0 = NaN for a row with no key, as the oracle has it
    }
    const int r = ty * 4 + a;
    if (tx == 0 && r < rows_here) g.lse_out[b * g.t_q + i0 + r] = top[a] + logf(total);
  }
  store_rows<T, HD>(static_cast<T*>(g.out), acc, b * g.t_q + i0, rows_here, g.hd_v, ty, tx);
}

// ---- dQ for 64 query rows (oracle: limn/sdpa.py:157-170) ----
template <typename T, int HD, int BN, typename Sync>
__device__ __forceinline__ void bwd_q_rows(const Args& g, long long b, int i0, float* shared, int thread, Sync sync) {
  constexpr int LD = HD + kPad, LP = BN + kPad, NB = BN / 16, NV = HD / 16;
  float* qs = shared;
  float* dos = qs + kBM * LD;
  float* ks = dos + kBM * LD;
  float* vs = ks + BN * LD;
  float* ss = vs + BN * LD;
  const int tx = thread & 15, ty = thread >> 4;
  const T* q = static_cast<const T*>(g.q) + b * g.t_q * g.hd;
  const T* k = static_cast<const T*>(g.k) + b * g.t_k * g.hd;
  const T* v = static_cast<const T*>(g.v) + b * g.t_k * g.hd_v;
  const T* dout = static_cast<const T*>(g.dout) + b * g.t_q * g.hd_v;
  const T* mask = g.mask ? static_cast<const T*>(g.mask) + b * g.t_k : nullptr;
  const int depth = (g.hd + 3) & ~3, depth_v = (g.hd_v + 3) & ~3;

  stage<T, HD, kBM>(qs, q, i0, g.t_q, g.hd, g.wide_qk, thread);
  stage<T, HD, kBM>(dos, dout, i0, g.t_q, g.hd_v, g.wide_v, thread);
  float row_lse[4], row_delta[4], acc[4][NV];
#pragma unroll
  for (int a = 0; a < 4; ++a) {
    const int i = i0 + ty * 4 + a;
    row_lse[a] = i < g.t_q ? g.lse_in[b * g.t_q + i] : 0.f;
    row_delta[a] = i < g.t_q ? g.delta[b * g.t_q + i] : 0.f;
#pragma unroll
    for (int c = 0; c < NV; ++c) acc[a][c] = 0.f;
  }
  const int keys_end = g.causal ? min(g.t_k, i0 + kBM) : g.t_k;
  for (int j0 = 0; j0 < keys_end; j0 += BN) {
    sync();
    stage<T, HD, BN>(ks, k, j0, g.t_k, g.hd, g.wide_qk, thread);
    stage<T, HD, BN>(vs, v, j0, g.t_k, g.hd_v, g.wide_v, thread);
    bool open[NB];
#pragma unroll
    for (int c = 0; c < NB; ++c) {
      const int j = j0 + tx + 16 * c;
      open[c] = j < g.t_k && (!mask || widen<T>(mask[j]) != 0.f);
    }
    sync();
    float s[4][NB], dp[4][NB];
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
      for (int c = 0; c < NB; ++c) s[a][c] = 0.f, dp[a][c] = 0.f;
    dot_tiles<LD, NB>(s, qs + ty * 4 * LD, ks + tx * LD, depth);
    dot_tiles<LD, NB>(dp, dos + ty * 4 * LD, vs + tx * LD, depth_v);
#pragma unroll
    for (int a = 0; a < 4; ++a) {
      const int i = i0 + ty * 4 + a;
#pragma unroll
      for (int c = 0; c < NB; ++c) {
        const bool seen = open[c] && i < g.t_q && (!g.causal || j0 + tx + 16 * c <= i);
        const float p = seen ? expf(s[a][c] * g.scale - row_lse[a]) : 0.f;
        ss[(ty * 4 + a) * LP + tx + 16 * c] = seen ? p * (dp[a][c] - row_delta[a]) * g.scale : 0.f;
      }
    }
    sync();
    weigh_rows<HD, BN>(acc, ss + ty * 4 * LP, ks, tx);
  }
  store_rows<T, HD>(static_cast<T*>(g.dq), acc, b * g.t_q + i0, min(kBM, g.t_q - i0), g.hd, ty, tx);
}

// ---- dK and dV for 64 key rows (oracle: limn/sdpa.py:190-203) ----
template <typename T, int HD, int BN, typename Sync>
__device__ __forceinline__ void bwd_kv_rows(const Args& g, long long b, int j0, float* shared, int thread, Sync sync) {
  constexpr int LD = HD + kPad, LP = BN + kPad, NB = BN / 16, NV = HD / 16;
  float* ks = shared;
  float* vs = ks + kBM * LD;
  float* qs = vs + kBM * LD;
  float* dos = qs + BN * LD;
  float* pt = dos + BN * LD;
  float* dst = pt + kBM * LP;
  float* lse_s = dst + kBM * LP;
  float* delta_s = lse_s + BN;
  const int tx = thread & 15, ty = thread >> 4;
  const T* q = static_cast<const T*>(g.q) + b * g.t_q * g.hd;
  const T* k = static_cast<const T*>(g.k) + b * g.t_k * g.hd;
  const T* v = static_cast<const T*>(g.v) + b * g.t_k * g.hd_v;
  const T* dout = static_cast<const T*>(g.dout) + b * g.t_q * g.hd_v;
  const T* mask = g.mask ? static_cast<const T*>(g.mask) + b * g.t_k : nullptr;
  const int depth = (g.hd + 3) & ~3, depth_v = (g.hd_v + 3) & ~3;

  stage<T, HD, kBM>(ks, k, j0, g.t_k, g.hd, g.wide_qk, thread);
  stage<T, HD, kBM>(vs, v, j0, g.t_k, g.hd_v, g.wide_v, thread);
  bool live[4];
  float acc_k[4][NV], acc_v[4][NV];
#pragma unroll
  for (int a = 0; a < 4; ++a) {
    const int j = j0 + ty * 4 + a;
    live[a] = j < g.t_k && (!mask || widen<T>(mask[j]) != 0.f);
#pragma unroll
    for (int c = 0; c < NV; ++c) acc_k[a][c] = 0.f, acc_v[a][c] = 0.f;
  }
  const int first = g.causal ? (j0 / BN) * BN : 0;  // the first query tile that sees one of these keys
  for (int i0 = first; i0 < g.t_q; i0 += BN) {
    sync();
    stage<T, HD, BN>(qs, q, i0, g.t_q, g.hd, g.wide_qk, thread);
    stage<T, HD, BN>(dos, dout, i0, g.t_q, g.hd_v, g.wide_v, thread);
    if (thread < BN) {
      const int i = i0 + thread;
      lse_s[thread] = i < g.t_q ? g.lse_in[b * g.t_q + i] : 0.f;
      delta_s[thread] = i < g.t_q ? g.delta[b * g.t_q + i] : 0.f;
    }
    sync();
    float s[4][NB], dp[4][NB];
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
      for (int c = 0; c < NB; ++c) s[a][c] = 0.f, dp[a][c] = 0.f;
    dot_tiles<LD, NB>(s, ks + ty * 4 * LD, qs + tx * LD, depth);
    dot_tiles<LD, NB>(dp, vs + ty * 4 * LD, dos + tx * LD, depth_v);
#pragma unroll
    for (int a = 0; a < 4; ++a) {
      const int j = j0 + ty * 4 + a;
#pragma unroll
      for (int c = 0; c < NB; ++c) {
        const int ii = tx + 16 * c, i = i0 + ii;
        const bool seen = live[a] && i < g.t_q && (!g.causal || j <= i);
        const float p = seen ? expf(s[a][c] * g.scale - lse_s[ii]) : 0.f;
        pt[(ty * 4 + a) * LP + ii] = p;
        dst[(ty * 4 + a) * LP + ii] = seen ? p * (dp[a][c] - delta_s[ii]) * g.scale : 0.f;
      }
    }
    sync();
    weigh_rows<HD, BN>(acc_v, pt + ty * 4 * LP, dos, tx);
    weigh_rows<HD, BN>(acc_k, dst + ty * 4 * LP, qs, tx);
  }
  const int rows_here = min(kBM, g.t_k - j0);
  store_rows<T, HD>(static_cast<T*>(g.dk), acc_k, b * g.t_k + j0, rows_here, g.hd, ty, tx);
  store_rows<T, HD>(static_cast<T*>(g.dv), acc_v, b * g.t_k + j0, rows_here, g.hd_v, ty, tx);
}

template <int HD, int BN>
constexpr size_t shared_bytes(Op op) {
  constexpr size_t LD = HD + kPad, LP = BN + kPad;
  switch (op) {
    case Op::Fwd: return sizeof(float) * ((kBM + 2 * BN) * LD + kBM * LP);
    case Op::BwdQ: return sizeof(float) * ((2 * kBM + 2 * BN) * LD + kBM * LP);
    case Op::BwdKV: return sizeof(float) * ((2 * kBM + 2 * BN) * LD + 2 * kBM * LP + 2 * BN);
  }
  return 0;
}

}  // namespace tiled
}  // namespace limn_b200
