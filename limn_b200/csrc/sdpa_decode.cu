// "sdpa" forward for decode shapes: a handful of query rows against a long run of keys, no causal mask (causal needs
// t_q == t_k), with or without a key mask, hd and hd_v multiples of 8 up to 128: t_q <= 4 in f16/bf16 (more rows go to
// the tensor cores), t_q < 16 in float32 (in chunks of 4 rows, K and V of the later chunks from L2). This is the step of
// a kv cache: one new token reads every slot filled so far (the reference tests the shape at
// tests/test_attention.py:385-396 and serves it with the same one-thread-per-query-row kernel as everything else,
// limn/cuda_emit.py:921-965, which leaves all but t_q threads of a block idle).
//
// The work is reading K and V once; the arithmetic is a few flops per byte, so tensor cores have nothing to add and
// the 128-row MMA tile of the prefill kernel would spend 127 of its 128 rows on nothing. Here one CTA of 16 warps
// owns one (batch, head) problem. D / 8 lanes share a key (each holds 8 of its elements, one 16-byte load in 16-bit
// storage and two in float32), so a warp reads 2, 4 or 8 consecutive keys at a time; every group of lanes walks its own
// subsequence of the keys, four at a time (two in float32: the same bytes in flight, and the same registers, which is
// what keeps two CTAs on an SM) with all loads of K and V issued before the first is used, and keeps an
// online softmax of its own per query row: a running maximum, a denominator and 8 accumulator elements per lane. The
// groups of a warp are merged with shuffles, the 16 warps through shared memory, always in the same order, so two runs
// give the same bits. A batch too small to fill the GPU with one CTA per problem gets a thread-block cluster of up
// to 8 CTAs per problem instead: the CTAs of a cluster deal the problem's keys out among themselves, leave their results in
// CTA 0's shared memory (distributed shared memory, no scratch in global memory), and CTA 0 folds them in rank
// order. A call of a single request is launch and latency: the kernel is launched under the one before it, the flags of a
// pass's keys are fetched beside the keys, and the shares are pushed (a store and one cluster barrier) where CTA 0 used to
// read them one after the other: 8 problems of 1 999 keys x 64 in float32 6.7 -> 5.7 us. Semantics as the oracle's (limn/sdpa.py:91-137): a hidden key contributes exactly 0, a row with
// no visible key is NaN with L = -inf, O is rounded once from fp32, L = m + log(l) in natural log.
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "common.h"
#include "sm100_ptx.cuh"
#include "tensor_map.h"

namespace limn_b200 {
namespace {

constexpr int kWarps = 16;
constexpr int kThreads = kWarps * 32;
constexpr int kMaxRows = 4;          // query rows a CTA carries
constexpr int kMaxSplit = 8;         // CTAs of a cluster
constexpr int kMaxRowsF32 = 15;      // float32 problems up to here come in chunks of kMaxRows
enum Kind { kF16, kBF16, kF32 };     // storage of Q, K, V, the mask and O
template <Kind kKind>
struct Storage {
  static constexpr int kBytes = kKind == kF32 ? 4 : 2;
  static constexpr int kUnroll = kKind == kF32 ? 2 : 4;  // keys a group of lanes has in flight
  static constexpr int kLoads = kKind == kF32 ? 2 : 1;   // 16-byte loads that hold a lane's 8 elements
};
constexpr float kLog2e = 1.4426950408889634f;

struct DecodeParams {
  const void* q;
  const void* k;
  const void* v;
  const void* mask;  // (bh, t_k) flags in the storage dtype, 0 hides a key; null without a mask
  void* out;
  float* lse;
  int heads;  // problem p is (batch p / heads, head p % heads)
  Strides q_strides, k_strides, v_strides, o_strides;  // in elements
  int t_q, t_k;
  int pieces, pieces_v;  // groups of 8 columns a row of Q and K, and of V and O, really has (<= D / 8)
  int chunks;            // CTAs (or clusters) that share a problem's query rows: ceil(t_q / R)
  float scale;
  int split;  // CTAs per problem (the cluster size): 1, 2, 4 or 8
};

// ---- thread-block cluster: rank, barrier, a peer CTA's shared memory ----
__device__ __forceinline__ unsigned cluster_rank() {
  unsigned r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
// to CTA 0's copy of *mine
__device__ __forceinline__ void store_at_first(float* mine, float value) {
  unsigned local = static_cast<unsigned>(__cvta_generic_to_shared(mine)), remote;
  asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(remote) : "r"(local));
  asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(remote), "f"(value) : "memory");
}

template <Kind kKind>
struct Raw8 {  // a lane's 8 elements as loaded
  uint4 part[Storage<kKind>::kLoads];
};
template <Kind kKind>
__device__ __forceinline__ Raw8<kKind> load8(const unsigned char* at) {
  Raw8<kKind> raw;
#pragma unroll
  for (int i = 0; i < Storage<kKind>::kLoads; ++i) raw.part[i] = reinterpret_cast<const uint4*>(at)[i];
  return raw;
}
template <Kind kKind>
__device__ __forceinline__ void widen8(const Raw8<kKind>& raw, float (&f)[8]) {
#pragma unroll
  for (int p = 0; p < Storage<kKind>::kLoads; ++p) {
    const uint32_t w[4] = {raw.part[p].x, raw.part[p].y, raw.part[p].z, raw.part[p].w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      if (kKind == kF32) {
        f[4 * p + i] = __uint_as_float(w[i]);
      } else if (kKind == kF16) {
        const float2 pair = __half22float2(*reinterpret_cast<const __half2*>(&w[i]));
        f[2 * i] = pair.x, f[2 * i + 1] = pair.y;
      } else {
        f[2 * i] = __uint_as_float(w[i] << 16), f[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
      }
    }
  }
}
template <Kind kKind>
__device__ __forceinline__ bool key_visible(const void* flags, int key) {
  if (kKind == kF32) return (static_cast<const uint32_t*>(flags)[key] & 0x7fffffffu) != 0;
  return (static_cast<const unsigned short*>(flags)[key] & 0x7fffu) != 0;
}

// Fold the running softmax (m_b, l_b, acc_b) into (m_a, l_a, acc_a). Scores are in raw units; sl2 = scale * log2 e.
__device__ __forceinline__ void merge(float& m_a, float& l_a, float (&acc_a)[8], float m_b, float l_b, const float (&acc_b)[8], float sl2) {
  const float m = fmaxf(m_a, m_b);
  // a side that has seen no visible key has m = -inf and l = 0: its factor must be 0, not exp2(-inf + inf)
  const float fa = m_a == -INFINITY ? 0.f : exp2f((m_a - m) * sl2);
  const float fb = m_b == -INFINITY ? 0.f : exp2f((m_b - m) * sl2);
  l_a = l_a * fa + l_b * fb;
#pragma unroll
  for (int i = 0; i < 8; ++i) acc_a[i] = acc_a[i] * fa + acc_b[i] * fb;
  m_a = m;
}

// Two CTAs per SM where the registers allow it (one or two query rows), so that every problem of a batch of a few
// hundred is resident at once and the problems share HBM instead of queueing for SMs.
template <int D, Kind kKind, bool kMask, int R>
__global__ void __launch_bounds__(kThreads, R <= 2 ? 2 : 1) sdpa_decode_kernel(const DecodeParams prm) {
  constexpr int kLanesPerKey = D / 8;           // 16, 8 or 4
  constexpr int kGroups = 32 / kLanesPerKey;    // keys a warp reads side by side: 2, 4 or 8
  constexpr int kBytes = Storage<kKind>::kBytes, kUnroll = Storage<kKind>::kUnroll;
  __shared__ float part_m[kWarps][R], part_l[kWarps][R];
  __shared__ float part_acc[kWarps][R][D];
  __shared__ float peer_m[kMaxSplit - 1][R], peer_l[kMaxSplit - 1][R], peer_o[kMaxSplit - 1][R][D];  // in CTA 0: the other CTAs' shares

  static_assert(R * D <= kThreads, "a thread folds one output element");
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int group = lane / kLanesPerKey, gl = lane % kLanesPerKey;
  const int split = prm.split;
  const unsigned rank = split > 1 ? cluster_rank() : 0u;
  if (split > 1) cluster_arrive();  // (a peer's shared memory may be written once the peer has started)
  const int unit = blockIdx.x / split;  // chunks of a problem are neighbours: they read its keys out of L2 together
  const int problem = unit / prm.chunks;
  const int row0 = (unit - problem * prm.chunks) * R;
  const int batch = problem / prm.heads, head = problem - batch * prm.heads;
  const float sl2 = prm.scale * kLog2e;

  const unsigned char* q_base = static_cast<const unsigned char*>(prm.q) + (batch * prm.q_strides.batch + head * prm.q_strides.head) * kBytes;
  const unsigned char* k_base = static_cast<const unsigned char*>(prm.k) + (batch * prm.k_strides.batch + head * prm.k_strides.head) * kBytes;
  const unsigned char* v_base = static_cast<const unsigned char*>(prm.v) + (batch * prm.v_strides.batch + head * prm.v_strides.head) * kBytes;
  const long long k_row = prm.k_strides.row * kBytes, v_row = prm.v_strides.row * kBytes;  // bytes between keys
  const void* flags = kMask ? static_cast<const unsigned char*>(prm.mask) + static_cast<long long>(problem) * prm.t_k * kBytes : nullptr;
  // Lanes beyond a row's columns (a head narrower than D) read the row's first piece again: what they make of K is
  // replaced by zero (their q is zero too, but an infinity in K times that is NaN), and what they gather of V is never stored.
  const bool real = gl < prm.pieces;
  const int k_at = (real ? gl : 0) * 8 * kBytes, v_at = (gl < prm.pieces_v ? gl : 0) * 8 * kBytes;

  // up to here nothing has touched global memory, so all of it may run under the tail of the kernel before this one
  ptx::grid_dependency_wait();
  ptx::grid_launch_dependents();

  // this lane's 8 elements of every query row
  float q[R][8];
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const long long row = min(row0 + r, prm.t_q - 1);  // a last chunk's missing rows repeat the last one and are not stored
    widen8<kKind>(load8<kKind>(q_base + row * prm.q_strides.row * kBytes + k_at), q[r]);
    if (!real) {
#pragma unroll
      for (int i = 0; i < 8; ++i) q[r][i] = 0.f;
    }
  }

  float m[R], l[R], acc[R][8];
#pragma unroll
  for (int r = 0; r < R; ++r) {
    m[r] = -INFINITY, l[r] = 0.f;
#pragma unroll
    for (int i = 0; i < 8; ++i) acc[r][i] = 0.f;
  }

  // keys are dealt out so that the groups of a warp, and the warps of the CTA, read consecutive keys together
  constexpr int kPerPass = kWarps * kUnroll * kGroups;
  for (int first = rank * kPerPass; first < prm.t_k; first += split * kPerPass) {
    Raw8<kKind> k_raw[kUnroll], v_raw[kUnroll];
    int key[kUnroll];
#pragma unroll
    for (int u = 0; u < kUnroll; ++u) {
      key[u] = first + (u * kWarps + warp) * kGroups + group;
      const int at = min(key[u], prm.t_k - 1);  // past the end: read the last key again, its score is discarded below
      k_raw[u] = load8<kKind>(k_base + at * k_row + k_at);
    }
#pragma unroll
    for (int u = 0; u < kUnroll; ++u) {
      const int at = min(key[u], prm.t_k - 1);
      v_raw[u] = load8<kKind>(v_base + at * v_row + v_at);
    }
    // (the flags too before anything waits for a load)
    bool seen[kUnroll];
#pragma unroll
    for (int u = 0; u < kUnroll; ++u) seen[u] = !kMask || key_visible<kKind>(flags, min(key[u], prm.t_k - 1));
    const bool ragged = first + kPerPass > prm.t_k;  // some of this pass's slots lie past the end
    float s[R][kUnroll];
#pragma unroll
    for (int u = 0; u < kUnroll; ++u) {
      float kf[8];
      widen8<kKind>(k_raw[u], kf);
      bool visible = key[u] < prm.t_k;
      // a key that does not exist has no V: the last key's would meet a weight of 0, and 0 * inf is NaN. In float32 a
      // hidden key's V does not count either (as in the one-row-per-warp kernel), so the empty slots of a cache may hold
      // anything; in 16 bits it does, as in the tensor-core kernels and the oracle, where 0 * NaN is NaN.
      if (ragged && !visible) v_raw[u] = Raw8<kKind>{};
      if (kMask && visible) {
        visible = seen[u];
        if (kKind == kF32 && !visible) v_raw[u] = Raw8<kKind>{};
      }
#pragma unroll
      for (int r = 0; r < R; ++r) {
        float dot = 0.f;
#pragma unroll
        for (int i = 0; i < 8; ++i) dot = fmaf(q[r][i], kf[i], dot);
        dot = real ? dot : 0.f;
#pragma unroll
        for (int step = kLanesPerKey / 2; step > 0; step >>= 1) dot += __shfl_xor_sync(0xffffffffu, dot, step);
        s[r][u] = visible ? dot : -INFINITY;
      }
    }
#pragma unroll
    for (int r = 0; r < R; ++r) {
      float mx = s[r][0];
#pragma unroll
      for (int u = 1; u < kUnroll; ++u) mx = fmaxf(mx, s[r][u]);
      const float m_new = fmaxf(m[r], mx);  // (passes a NaN by: the weight below has it)
      // as long as nothing is visible the weights are taken against 0: exp2(-inf), and NaN for a NaN score
      const float base = m_new == -INFINITY ? 0.f : m_new;
      const float alpha = exp2f((m[r] - base) * sl2);  // 0 while m is -inf
      m[r] = m_new;
      float p[kUnroll], sum = 0.f;
#pragma unroll
      for (int u = 0; u < kUnroll; ++u) {
        p[u] = exp2f((s[r][u] - base) * sl2);
        sum += p[u];
      }
      l[r] = l[r] * alpha + sum;
#pragma unroll
      for (int i = 0; i < 8; ++i) acc[r][i] *= alpha;
#pragma unroll
      for (int u = 0; u < kUnroll; ++u) {
        float vf[8];
        widen8<kKind>(v_raw[u], vf);
#pragma unroll
        for (int i = 0; i < 8; ++i) acc[r][i] = fmaf(p[u], vf[i], acc[r][i]);
      }
    }
  }

  // ---- the groups of a warp (lanes gl, gl + kLanesPerKey, ... hold the same 8 elements) ----
#pragma unroll
  for (int r = 0; r < R; ++r) {
#pragma unroll
    for (int step = kLanesPerKey; step < 32; step <<= 1) {
      const float m_b = __shfl_xor_sync(0xffffffffu, m[r], step), l_b = __shfl_xor_sync(0xffffffffu, l[r], step);
      float acc_b[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) acc_b[i] = __shfl_xor_sync(0xffffffffu, acc[r][i], step);
      // both partners compute the same sum in the same order: the lower one keeps (a, b), the upper one (b, a),
      // and addition commutes, so every lane ends with identical values
      if (lane & step) {
        float m_a = m_b, l_a = l_b;
        merge(m_a, l_a, acc_b, m[r], l[r], acc[r], sl2);
        m[r] = m_a, l[r] = l_a;
#pragma unroll
        for (int i = 0; i < 8; ++i) acc[r][i] = acc_b[i];
      } else {
        merge(m[r], l[r], acc[r], m_b, l_b, acc_b, sl2);
      }
    }
    if (group == 0) {
      if (gl == 0) part_m[warp][r] = m[r], part_l[warp][r] = l[r];
#pragma unroll
      for (int i = 0; i < 8; ++i) part_acc[warp][r][gl * 8 + i] = acc[r][i];
    }
  }
  __syncthreads();

  // ---- the 16 warps: thread (r, d) folds them in warp order; the CTAs of a cluster leave their shares with CTA 0, which
  // folds those in rank order. One element per thread, rounded once. ----
  if (split > 1) cluster_wait();  // every CTA of the cluster has started
  const int r = threadIdx.x / D, d = threadIdx.x - r * D;
  const bool mine = threadIdx.x < R * D;
  float m_tot = -INFINITY, l_tot = 0.f, o = 0.f;
  if (mine) {
#pragma unroll
    for (int w = 0; w < kWarps; ++w) m_tot = fmaxf(m_tot, part_m[w][r]);
#pragma unroll
    for (int w = 0; w < kWarps; ++w) {
      const float f = part_m[w][r] == -INFINITY ? 0.f : exp2f((part_m[w][r] - m_tot) * sl2);
      l_tot = fmaf(part_l[w][r], f, l_tot);
      o = fmaf(part_acc[w][r][d], f, o);
    }
    if (rank > 0) {
      store_at_first(&peer_o[rank - 1][r][d], o);
      if (d == 0) store_at_first(&peer_m[rank - 1][r], m_tot), store_at_first(&peer_l[rank - 1][r], l_tot);
    }
  }
  if (split > 1) {
    cluster_arrive();
    cluster_wait();  // (also in the CTAs that are done: none may leave before the barrier is complete)
    if (rank > 0) return;
  }
  const int row = row0 + r;
  if (!mine || row >= prm.t_q) return;
  for (int c = 1; c < split; ++c) {
    const float m_c = peer_m[c - 1][r], l_c = peer_l[c - 1][r], o_c = peer_o[c - 1][r][d];
    const float m_new = fmaxf(m_tot, m_c);
    const float fa = m_tot == -INFINITY ? 0.f : exp2f((m_tot - m_new) * sl2);
    const float fc = m_c == -INFINITY ? 0.f : exp2f((m_c - m_new) * sl2);
    l_tot = l_tot * fa + l_c * fc;
    o = o * fa + o_c * fc;
    m_tot = m_new;
  }
  const float value = o / l_tot;  // 0 / 0 = NaN for a row with no visible key, as the oracle gives
  unsigned char* dst = static_cast<unsigned char*>(prm.out) +
                       (batch * prm.o_strides.batch + head * prm.o_strides.head + static_cast<long long>(row) * prm.o_strides.row + d) * kBytes;
  if (d < prm.pieces_v * 8) {
    if (kKind == kF32) *reinterpret_cast<float*>(dst) = value;
    else if (kKind == kF16) *reinterpret_cast<__half*>(dst) = __float2half_rn(value);
    else *reinterpret_cast<__nv_bfloat16*>(dst) = __float2bfloat16_rn(value);
  }
  if (d == 0) {  // in float32 once per row in double: L is then as good as its sum
    const long long to = static_cast<long long>(problem) * prm.t_q + row;
    if (kKind == kF32) prm.lse[to] = static_cast<float>(static_cast<double>(m_tot) * prm.scale + log(static_cast<double>(l_tot)));
    else prm.lse[to] = m_tot * prm.scale + logf(l_tot);
  }
}

template <int D, Kind kKind, bool kMask, int R>
int launch_one(const Problem& p, DecodeParams& prm) {
  prm.chunks = (p.t_q + R - 1) / R;
  // One CTA per problem fills the GPU from a few hundred problems on (two CTAs fit an SM). Below that, 2, 4 or 8
  // CTAs share a problem, as long as each still has a full pass of keys (16 warps x the keys a warp has in flight).
  int sms = 0;
  if (int rc = sm_count(&sms)) return rc;
  constexpr int per_pass = kWarps * Storage<kKind>::kUnroll * (32 / (D / 8));
  const long long units = p.bh * prm.chunks;
  int split = 1;
  while (split < kMaxSplit && units * split * 2 <= 2LL * sms && (p.t_k + per_pass - 1) / per_pass >= split * 2) split *= 2;
  prm.split = split;
  if (units * split > 0x7fffffffLL) return fail(LIMN_B200_UNSUPPORTED, "sdpa: %lld problems need more blocks than one grid holds", p.bh);
  cudaLaunchConfig_t config = {};
  config.gridDim = dim3(static_cast<unsigned>(units * split));
  config.blockDim = dim3(kThreads);
  config.stream = p.stream;
  cudaLaunchAttribute attribute[2];
  attribute[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attribute[1].val.programmaticStreamSerializationAllowed = 1;
  attribute[0].id = cudaLaunchAttributeClusterDimension;
  attribute[0].val.clusterDim.x = static_cast<unsigned>(split);
  attribute[0].val.clusterDim.y = 1;
  attribute[0].val.clusterDim.z = 1;
  config.attrs = attribute;
  config.numAttrs = 2;
  const DecodeParams& as_launched = prm;
  LIMN_CUDA(cudaLaunchKernelEx(&config, sdpa_decode_kernel<D, kKind, kMask, R>, as_launched), "launching the sdpa decode kernel");
  note_launches(1);
  return LIMN_B200_OK;
}

template <int D, Kind kKind, bool kMask>
int launch_rows(const Problem& p, DecodeParams& prm) {
  switch (p.t_q) {
    case 1: return launch_one<D, kKind, kMask, 1>(p, prm);
    case 2: return launch_one<D, kKind, kMask, 2>(p, prm);
    case 3: return launch_one<D, kKind, kMask, 3>(p, prm);
    default: return launch_one<D, kKind, kMask, 4>(p, prm);
  }
}

template <int D, Kind kKind>
int launch_kind(const Problem& p, DecodeParams& prm) {
  return p.mask ? launch_rows<D, kKind, true>(p, prm) : launch_rows<D, kKind, false>(p, prm);
}

template <int D>
int launch_d(const Problem& p, DecodeParams& prm) {
  switch (p.dtype) {
    case LIMN_B200_F16: return launch_kind<D, kF16>(p, prm);
    case LIMN_B200_BF16: return launch_kind<D, kBF16>(p, prm);
    default: return launch_kind<D, kF32>(p, prm);
  }
}

}  // namespace

bool decode_serves(Op op, const Problem& p) {
  if (op != Op::Fwd || p.causal) return false;  // (causal needs t_q == t_k: a prefill shape, however short)
  if (p.dtype == LIMN_B200_F64) return false;
  if (p.hd > 128 || p.hd % 8 != 0 || p.hd_v > 128 || p.hd_v % 8 != 0) return false;
  if (p.t_q > (p.dtype == LIMN_B200_F32 ? kMaxRowsF32 : kMaxRows)) return false;
  if (p.dtype == LIMN_B200_F32 && (p.strided || p.layout != LIMN_B200_BHTD)) return false;  // dense only in float32
  if (!(p.scale > 0.0) || p.bh > 0x7fffffffLL) return false;
  // 16-byte loads: aligned bases (a null pointer is refused before this is asked in earnest)
  const uintptr_t bases = reinterpret_cast<uintptr_t>(p.q) | reinterpret_cast<uintptr_t>(p.k) | reinterpret_cast<uintptr_t>(p.v);
  return (bases & 15u) == 0;
}

int decode_launch(const Problem& p) {
  DecodeParams prm;
  prm.q = p.q, prm.k = p.k, prm.v = p.v;
  prm.mask = p.mask;
  prm.out = p.out, prm.lse = static_cast<float*>(p.lse_out);
  prm.heads = p.heads > 0 ? p.heads : static_cast<int>(p.bh);
  prm.q_strides = operand_strides(p, kOpQ, prm.heads, p.t_q, p.hd);
  prm.k_strides = operand_strides(p, kOpK, prm.heads, p.t_k, p.hd);
  prm.v_strides = operand_strides(p, kOpV, prm.heads, p.t_k, p.hd_v);
  prm.o_strides = operand_strides(p, kOpOut, prm.heads, p.t_q, p.hd_v);
  {
    const long long all = prm.q_strides.batch | prm.q_strides.head | prm.q_strides.row | prm.k_strides.batch | prm.k_strides.head |
                          prm.k_strides.row | prm.v_strides.batch | prm.v_strides.head | prm.v_strides.row;
    if (all & 7) return fail(LIMN_B200_BAD_ARGUMENT, "sdpa: operand strides must be multiples of 8 elements");
  }
  prm.t_q = p.t_q, prm.t_k = p.t_k;
  prm.pieces = p.hd / 8, prm.pieces_v = p.hd_v / 8;
  prm.scale = static_cast<float>(p.scale);
  const int widest = p.hd > p.hd_v ? p.hd : p.hd_v;
  if (widest <= 32) return launch_d<32>(p, prm);
  return widest <= 64 ? launch_d<64>(p, prm) : launch_d<128>(p, prm);
}

}  // namespace limn_b200
