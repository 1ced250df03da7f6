// Tensor-core engine: the table of (query tile, key tile) pairs whose probabilities are all exactly zero.
//
// The history term F[i, j] never decreases with the query index i, so for a key tile that many later queries have
// selected against, every logit of a far query tile sits hundreds of units below its row maximum and ex2 (which
// flushes results below 2^-126 to zero) returns exactly 0 for the whole tile: the tile adds nothing to the output,
// to the row sums, or to any gradient.  Such a tile can be left out without changing a single bit of the result.
// The reference computes every causal tile (src/selective_attention/kernels.py:100-160); this is an option on top.
//
// Bound used, in log2 units, for query tile mi and key tile nj < mi of row n = (b, h):
//     z[i, j] - m[i]  <=  c1 |q_i| (|k_j| + |k_i|) - log2e * F[i, j]
// because z[i, j] = c1 q_i.k_j - log2e F[i, j], and the row maximum m[i] is at least the diagonal logit
// z[i, i] = c1 q_i.k_i (no query before i selects against key i, so F[i, i] = 0) >= -c1 |q_i| |k_i|; the row's
// log-sum-exp, which the backward subtracts, is at least m[i].  F[i, j] >= carry[mi][j], the selection key j has
// received from the queries before tile mi.  With Qn, Kn the largest row norms of a tile and Fmin the smallest
// carry over the key tile, the tile is dead when
//     c1 Qn[mi] (Kn[nj] + Kn[mi]) - log2e Fmin[mi][nj]  <  -kDeadMargin,
// kDeadMargin = 150 leaving 24 units beyond the flush threshold for the rounding of the bf16 products and sums.
// Tiles holding an exempt key (F = 0 there) are never dead; the diagonal tile is always kept.
#include <float.h>

#include "sa_tc_host.cuh"
#include "sa_tc_ptx.cuh"

namespace sa {
namespace tc {
namespace {

constexpr int kTile = 128;
constexpr float kDeadMargin = 150.f;

// Largest row norm of each 128-row tile of q (z = 0) and k (z = 1): one block per (tile, row n, tensor), D / 8 lanes per
// token, so that a warp's load is contiguous, and eight (D = 128: sixteen) of them in flight a thread.  Bound by HBM; with a
// thread per token 16 heads of T = 16384 took 21 us.  Tiles are counted in absolute positions; the query tensor
// starts at position q_offset (a prefill that continues from a cache), the key tensor at 0.
template <int D>
__global__ void __launch_bounds__(kTile) tile_norms_kernel(const __nv_bfloat16* __restrict__ q, RowLayout q_rows,
                                                           const __nv_bfloat16* __restrict__ k, RowLayout k_rows,
                                                           int heads, int seq, int ntiles, int q_offset,
                                                           float* __restrict__ qn, float* __restrict__ kn) {
  constexpr int kLanes = D / 8, kRows = kTile / kLanes, kPasses = kTile / kRows;
  const int tile = blockIdx.x, n = blockIdx.y, which = blockIdx.z;
  const int b = n / heads, h = n - b * heads;
  const int lane = threadIdx.x % kLanes, t0 = tile * kTile + threadIdx.x / kLanes;
  uint4 v[kPasses];
#pragma unroll
  for (int u = 0; u < kPasses; ++u) {
    const int t = t0 + u * kRows;
    v[u] = make_uint4(0u, 0u, 0u, 0u);
    if (t < seq && (which == 1 || t >= q_offset))
      v[u] = *reinterpret_cast<const uint4*>((which == 0 ? q + q_rows.at(b, h, t - q_offset) : k + k_rows.at(b, h, t)) + lane * 8);
  }
  float m = 0.f;                                                  // of the squares
#pragma unroll
  for (int u = 0; u < kPasses; ++u) {
    const uint32_t w[4] = {v[u].x, v[u].y, v[u].z, v[u].w};
    float ss = 0.f;
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float lo = __uint_as_float(w[e] << 16), hi = __uint_as_float(w[e] & 0xffff0000u);
      ss = fmaf(lo, lo, fmaf(hi, hi, ss));
    }
#pragma unroll
    for (int o = kLanes / 2; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    m = fmaxf(m, ss);
  }
#pragma unroll
  for (int o = 16; o >= kLanes; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
  __shared__ float part[4];
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = m;
  __syncthreads();
  if (threadIdx.x == 0)
    (which == 0 ? qn : kn)[(int64_t)n * ntiles + tile] = sqrtf(fmaxf(fmaxf(part[0], part[1]), fmaxf(part[2], part[3])));
}

// alive[n][mi][nj] for nj <= mi: one block per (query tile mi >= mi_first, 16 key tiles, sequence b); a warp takes every fourth
// of them, finds the smallest carry over its 128 keys, and its lanes write the verdict for the heads of the sequence.
// (Bound by latency; with a query tile's key tiles all in one block T = 16384 took 20 us.)
constexpr int kTableChunk = 16;
__global__ void __launch_bounds__(kTile) tile_table_kernel(const float* __restrict__ carry, const float* __restrict__ qn,
                                                           const float* __restrict__ kn, int heads, int seq, int ntiles,
                                                           int mi_first, float c1, uint8_t* __restrict__ alive) {
  const int mi = mi_first + blockIdx.x, b = blockIdx.z, nj0 = blockIdx.y * kTableChunk;
  if (nj0 > mi) return;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const float* carry_row = carry + ((int64_t)b * (ntiles + 1) + mi) * seq;
  float fmin[kTableChunk / 4];
#pragma unroll
  for (int u = 0; u < kTableChunk / 4; ++u) {
    fmin[u] = FLT_MAX;
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const int nj = nj0 + warp + 4 * u, j = nj * kTile + c * 32 + lane;
      if (nj <= mi && j < seq) fmin[u] = fminf(fmin[u], carry_row[j]);
    }
  }
#pragma unroll
  for (int u = 0; u < kTableChunk / 4; ++u) {
    const int nj = nj0 + warp + 4 * u;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) fmin[u] = fminf(fmin[u], __shfl_xor_sync(0xffffffffu, fmin[u], o));
    if (nj > mi) continue;
    for (int h = lane; h < heads; h += 32) {
      const int64_t n = (int64_t)b * heads + h;
      const float bound = c1 * qn[n * ntiles + mi] * (kn[n * ntiles + nj] + kn[n * ntiles + mi]) - kLog2e * fmin[u];
      alive[(n * ntiles + mi) * ntiles + nj] = (nj == mi || !(bound < -kDeadMargin)) ? 1 : 0;
    }
  }
}

}  // namespace

// Skipping is offered for bf16 operands at head_dim 64 / 128 up to 1024 tiles (the forward keeps a tile's list of live
// key tiles in shared memory) and 65535 rows (the norms have them on grid.y).
size_t tile_table_bytes(const Problem& p) {
  const int64_t ntiles = (p.seq + kTile - 1) / kTile;
  if (p.dtype != SA_BF16 || (p.head_dim != 64 && p.head_dim != 128) || ntiles > 1024 || p.damp != SA_DAMP_NONE) return 0;
  const int64_t nrows = (int64_t)p.batch * p.heads;
  if (nrows > 65535) return 0;
  const int64_t table = (nrows * ntiles * ntiles + 255) & ~(int64_t)255;
  return (size_t)(table + 2 * nrows * ntiles * 4);
}


int build_tile_table(const Problem& p, const float* carry, cudaStream_t s) {
  const int ntiles = (p.seq + kTile - 1) / kTile;
  const int64_t nrows = (int64_t)p.batch * p.heads;
  if (tile_table_bytes(p) == 0 || p.tile_table == nullptr) return SA_ERR_UNSUPPORTED;
  uint8_t* alive = static_cast<uint8_t*>(p.tile_table);
  float* qn = reinterpret_cast<float*>(alive + ((nrows * ntiles * ntiles + 255) & ~(int64_t)255));
  float* kn = qn + nrows * ntiles;
  const RowLayout q_rows{p.q.sb, p.q.sh, p.q.st}, k_rows{p.k.sb, p.k.sh, p.k.st};
  const dim3 gn(ntiles, (unsigned)nrows, 2);
  count_launch();
  if (p.head_dim == 64)
    tile_norms_kernel<64><<<gn, kTile, 0, s>>>(static_cast<const __nv_bfloat16*>(p.q.ptr), q_rows,
                                               static_cast<const __nv_bfloat16*>(p.k.ptr), k_rows, p.heads, p.seq, ntiles,
                                               p.q_offset, qn, kn);
  else
    tile_norms_kernel<128><<<gn, kTile, 0, s>>>(static_cast<const __nv_bfloat16*>(p.q.ptr), q_rows,
                                                static_cast<const __nv_bfloat16*>(p.k.ptr), k_rows, p.heads, p.seq, ntiles,
                                                p.q_offset, qn, kn);
  SA_CUDA_CHECK(cudaGetLastError());
  count_launch();
  const int mi_first = p.q_offset / kTile;                // a continued prefill computes the query tiles from here on
  tile_table_kernel<<<dim3(ntiles - mi_first, (ntiles + kTableChunk - 1) / kTableChunk, p.batch), kTile, 0, s>>>(carry, qn, kn, p.heads, p.seq, ntiles, mi_first,
                                                                       p.scale * kLog2e, alive);
  SA_CUDA_CHECK(cudaGetLastError());
  return SA_OK;
}

}  // namespace tc
}  // namespace sa
