// Tiled SIMT fused-attention kernels: float32, float16 and bfloat16 storage computed in float32 on the
// CUDA cores, head dims up to 256, optional key mask, rectangular t_q x t_k. They serve what the tensor-core
// kernels leave (head dims that are no multiple of 8 in 16 bits, head dims above 128, float32 with a scale that is
// not positive) whenever the problem is large enough to fill a tile; the one-row-per-warp kernels in
// sdpa_general.cu keep float64, wider heads and short sequences.
//
// Shape of the work: a block of 256 threads owns 64 rows (query rows in the forward and the dQ pass, key rows
// in the dK/dV pass) and streams the other side through shared memory in tiles of BN rows (64, 32 or 16 of them
// for head dims up to 64, 128 or 256). Every tile is two small matrix products on a 16 x 16 thread grid: scores
// (rows x streamed rows, contraction over the head dim, a 4 x BN/16 micro-tile per thread read from shared memory
// as float4), then, after the scores went through shared memory, the update of the rows' totals (contraction
// over the streamed rows, 4 x HD/16 per thread). Each total has one owner and a fixed summation order, no float
// is added atomically: two runs give the same bits, as the reference's kernels promise
// (limn/cuda_emit.py:748-752).
#include "tiled_rows.cuh"

namespace limn_b200 {
namespace {

using namespace tiled;

// Which block of rows a block of threads owns: the ones with the longest causal streams first.
template <typename T, int HD, int BN, Op kOp>
__global__ void __launch_bounds__(kThreads) tiled_kernel(const Args g, int tiles) {
  extern __shared__ __align__(16) float shared[];
  const long long b = blockIdx.x / tiles;
  const int at = static_cast<int>(blockIdx.x - b * tiles);
  auto sync = [] { __syncthreads(); };
  if constexpr (kOp == Op::Fwd) fwd_rows<T, HD, BN>(g, b, (tiles - 1 - at) * kBM, shared, threadIdx.x, sync);
  else if constexpr (kOp == Op::BwdQ) bwd_q_rows<T, HD, BN>(g, b, (tiles - 1 - at) * kBM, shared, threadIdx.x, sync);
  else bwd_kv_rows<T, HD, BN>(g, b, at * kBM, shared, threadIdx.x, sync);
}

template <typename T, int HD, int BN>
int launch_sized(Op op, const Problem& p) {
  const int owned = op == Op::BwdKV ? p.t_k : p.t_q;
  Args g = {};
  g.q = p.q, g.k = p.k, g.v = p.v, g.mask = p.mask, g.dout = p.dout;
  g.lse_in = static_cast<const float*>(p.lse_in), g.delta = static_cast<const float*>(p.delta);
  g.out = p.out, g.dq = p.dq, g.dk = p.dk, g.dv = p.dv, g.lse_out = static_cast<float*>(p.lse_out);
  const int tiles = (owned + kBM - 1) / kBM;
  g.t_q = p.t_q, g.t_k = p.t_k, g.hd = p.hd, g.hd_v = p.hd_v, g.causal = p.causal ? 1 : 0;
  g.scale = static_cast<float>(p.scale);
  constexpr int piece = 16 / sizeof(T);
  auto aligned = [](const void* x) { return x == nullptr || (reinterpret_cast<uintptr_t>(x) & 15u) == 0; };
  g.wide_qk = p.hd % piece == 0 && aligned(p.q) && aligned(p.k);
  g.wide_v = p.hd_v % piece == 0 && aligned(p.v) && aligned(p.dout);
  const long long blocks = p.bh * tiles;
  if (blocks > 0x7fffffffLL) return fail(LIMN_B200_UNSUPPORTED, "sdpa: %lld row tiles need more blocks than one grid holds", blocks);
  const size_t shared = shared_bytes<HD, BN>(op);
  void (*kernel)(const Args, int) = op == Op::Fwd    ? tiled_kernel<T, HD, BN, Op::Fwd>
                                    : op == Op::BwdQ ? tiled_kernel<T, HD, BN, Op::BwdQ>
                                                     : tiled_kernel<T, HD, BN, Op::BwdKV>;
  if (shared > 48 * 1024)
    LIMN_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(shared)),
              "sizing shared memory for a tiled sdpa kernel");
  kernel<<<dim3(static_cast<unsigned>(blocks)), dim3(kThreads), shared, p.stream>>>(g, tiles);
  LIMN_CUDA(cudaGetLastError(), "launching a tiled sdpa kernel");
  note_launches(1);
  return LIMN_B200_OK;
}

template <typename T>
int launch_typed(Op op, const Problem& p) {
  const int widest = p.hd > p.hd_v ? p.hd : p.hd_v;
  if (widest <= 32) return launch_sized<T, 32, 64>(op, p);
  if (widest <= 64) return launch_sized<T, 64, 64>(op, p);
  if (widest <= 128) return launch_sized<T, 128, 32>(op, p);
  return launch_sized<T, 256, 16>(op, p);
}

}  // namespace

bool general_tiled_serves(Op, const Problem& p) {
  if (p.dtype == LIMN_B200_F64 || p.hd > 256 || p.hd_v > 256) return false;
  if (p.layout != LIMN_B200_BHTD || p.strided) return false;
  return p.t_q >= 16 && p.t_k >= 16;  // shorter sides leave most of a 64-row tile idle: one row per warp is better
}

int general_tiled_launch(Op op, const Problem& p) {
  switch (p.dtype) {
    case LIMN_B200_F32: return launch_typed<float>(op, p);
    case LIMN_B200_F16: return launch_typed<__half>(op, p);
    case LIMN_B200_BF16: return launch_typed<__nv_bfloat16>(op, p);
  }
  return fail(LIMN_B200_BAD_ARGUMENT, "sdpa: dtype code %d is not served by the tiled kernels", p.dtype);
}

}  // namespace limn_b200
