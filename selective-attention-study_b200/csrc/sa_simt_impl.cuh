// CUDA-core (fp32 FFMA) engine of the Selective Attention operator.
//
// Exact fp32 products ("ieee"), every supported head_dim and dtype, any sequence length.  It is the
// accuracy path behind the fp32 parity bar and the path for shapes the tensor-core engine does not take.
//
// Four kernels mirror the structure of the operator (reference: src/selective_attention/kernels.py):
//   colsum   one (32 queries, 64 keys) tile of the selection logits each: the sum per key          (:111-138)
//   scan     the running sum per key across the query blocks, in place (-> carry), and the totals
//   forward  per 32-query block of one head, online softmax over 64-key tiles of (L_h - F)          (:140-194)
//   backward per 32-key block of one head, query blocks last to first; dV, dK in registers; dQ and the
//            head-0 selection gradients through fp32 reductions                                      (:196-268)
//
// Register tiles.  128 threads as 8 x 16; a thread owns 4 rows (4 ty ..) of a tile and the columns tx + 16 c, or 4 rows and
// D / 16 output columns (256 threads with 2 rows each, 1.5 loads a FMA more, took 17 % longer).  Operands sit in shared
// memory as fp32 rows of D + 4 floats (consecutive rows start 4 banks apart, so eight rows of a 16-byte load do not
// conflict) and are read 16 bytes at a time along the contraction: 8 loads for 64 FMAs.  The contraction index runs upwards
// in every product, one FMA after the other.
// What bounds it: FFMA issue and the shared-memory loads that feed it, at about the same rate; with few (batch, head) rows
// the longest walk.  With one load per FMA operand and thread, and the selection pass on T / 64 blocks, the case
// B = 2, H = 4, T = 1024, D = 64 took 153 + 403 + 859 us (selection, forward, backward); this form takes 15 + 134 + 339 us.
//
// A head that is its own selector (head 0, unless the selector comes from outside) has its selection logits already, and
// since Q0 = Q, K0 = K its two gradient paths add before the products: dK += (dz + g)^T Q, dQ += (dz + g) K.
#pragma once
#include "sa_common.cuh"

namespace sa {
namespace simt {

constexpr int kThreads = 128;
constexpr int kQ = 32;         // query rows per tile (== kSimtCarryRows)
constexpr int kKF = 64;        // keys per tile, selection and forward kernels
constexpr int kKB = 32;        // keys per block, backward kernel
constexpr int kRows = 4;       // rows of a 32-row tile that a thread owns
constexpr int kGroups = kQ / kRows;

template <typename T>
__device__ __forceinline__ const T* row_ptr(const Strided& s, int b, int h) {
  return static_cast<const T*>(s.ptr) + b * s.sb + h * s.sh;
}

// ROWS rows of D elements from token t0 on, on their way to dst[ROWS][D + 4] as fp32, zero past seq.  fetch() has all of a
// thread's loads in flight at once; between fetch() and store() they are covered by whatever is computed there.
// `vec`: four elements at a time.
template <typename T, int D, int ROWS>
struct Tile {
  static constexpr int C = D / 4, N = (ROWS * C + kThreads - 1) / kThreads;
  struct alignas(4 * sizeof(T)) Quad { T e[4]; };
  Quad x[N];
  __device__ __forceinline__ void fetch(const T* base, int64_t st, int t0, int seq, bool vec) {
#pragma unroll
    for (int u = 0; u < N; ++u) {
      const int idx = threadIdx.x + u * kThreads, r = idx / C, c = (idx - r * C) * 4, t = t0 + r;
#pragma unroll
      for (int e = 0; e < 4; ++e) x[u].e[e] = from_float<T>(0.f);
      if (t >= seq || r >= ROWS) continue;
      const T* src = base + (int64_t)t * st + c;
      if (vec) {
        x[u] = *reinterpret_cast<const Quad*>(src);
      } else {
#pragma unroll
        for (int e = 0; e < 4; ++e) x[u].e[e] = src[e];
      }
    }
  }
  __device__ __forceinline__ void store(float* dst) const {
#pragma unroll
    for (int u = 0; u < N; ++u) {
      const int idx = threadIdx.x + u * kThreads, r = idx / C, c = (idx - r * C) * 4;
      if (r < ROWS)
        *reinterpret_cast<float4*>(dst + r * (D + 4) + c) =
            make_float4(to_float<T>(x[u].e[0]), to_float<T>(x[u].e[1]), to_float<T>(x[u].e[2]), to_float<T>(x[u].e[3]));
    }
  }
};
// Whether the next tiles' elements are held in registers during the products of the tile at hand.
template <typename T, int D> constexpr bool kAhead = D * (int)sizeof(T) <= 256;

template <typename T, int D, int ROWS>
__device__ __forceinline__ void load_tile(float* dst, const T* base, int64_t st, int t0, int seq, bool vec) {
  Tile<T, D, ROWS> x;
  x.fetch(base, st, t0, seq, vec);
  x.store(dst);
}

__device__ __forceinline__ float4 ld4(const float* p) { return *reinterpret_cast<const float4*>(p); }

// acc[u][c] += a[4 ty + u] . b[tx + 16 c] over D, in order
template <int D, int NC>
__device__ __forceinline__ void dot_rows(float (&acc)[kRows][NC], const float* a, const float* b, int ty, int tx) {
  const float* ar = a + (ty * kRows) * (D + 4);
  const float* br = b + tx * (D + 4);
#pragma unroll 4
  for (int d = 0; d < D; d += 4) {
    float4 x[kRows], y[NC];
#pragma unroll
    for (int u = 0; u < kRows; ++u) x[u] = ld4(ar + u * (D + 4) + d);
#pragma unroll
    for (int c = 0; c < NC; ++c) y[c] = ld4(br + 16 * c * (D + 4) + d);
#pragma unroll
    for (int u = 0; u < kRows; ++u)
#pragma unroll
      for (int c = 0; c < NC; ++c) {
        acc[u][c] = fmaf(x[u].x, y[c].x, acc[u][c]);
        acc[u][c] = fmaf(x[u].y, y[c].y, acc[u][c]);
        acc[u][c] = fmaf(x[u].z, y[c].z, acc[u][c]);
        acc[u][c] = fmaf(x[u].w, y[c].w, acc[u][c]);
      }
  }
}

// The D / 16 output columns of a thread: in fours (D = 128: 4 tx .. and 64 + 4 tx ..), or 2 tx, 2 tx + 1, or tx.
template <int CD>
__device__ __forceinline__ void load_cols(const float* row, int tx, float (&x)[CD]) {
  if constexpr (CD >= 4) {
#pragma unroll
    for (int f = 0; f < CD / 4; ++f) {
      const float4 v = ld4(row + 64 * f + 4 * tx);
      x[4 * f] = v.x; x[4 * f + 1] = v.y; x[4 * f + 2] = v.z; x[4 * f + 3] = v.w;
    }
  } else if constexpr (CD == 2) {
    const float2 v = *reinterpret_cast<const float2*>(row + 2 * tx);
    x[0] = v.x; x[1] = v.y;
  } else {
    x[0] = row[tx];
  }
}
// dst += x: fp32 reductions in global memory, as wide as the columns are contiguous
template <int CD>
__device__ __forceinline__ void reduce_cols(float* row, int tx, const float (&x)[CD], float scale) {
  if constexpr (CD >= 4) {
#pragma unroll
    for (int f = 0; f < CD / 4; ++f)
      asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(row + 64 * f + 4 * tx), "f"(x[4 * f] * scale),
                   "f"(x[4 * f + 1] * scale), "f"(x[4 * f + 2] * scale), "f"(x[4 * f + 3] * scale)
                   : "memory");
  } else if constexpr (CD == 2) {
    asm volatile("red.global.add.v2.f32 [%0], {%1, %2};" ::"l"(row + 2 * tx), "f"(x[0] * scale), "f"(x[1] * scale) : "memory");
  } else {
    atomicAdd(row + tx, x[0] * scale);
  }
}
template <int CD>
__device__ __forceinline__ int col_of(int tx, int c) { return CD >= 4 ? 64 * (c >> 2) + 4 * tx + (c & 3) : CD * tx + c; }

// acc[u][:] += sum_j w[4 ty + u][j] rows[j][:] over N rows j, w with row stride WS
template <int D, int N, int WS, int CD>
__device__ __forceinline__ void weighted_rows(float (&acc)[kRows][CD], const float* w, const float* rows, int ty, int tx) {
  const float* wr = w + (ty * kRows) * WS;
#pragma unroll 2
  for (int j = 0; j < N; j += 4) {
    float4 x[kRows];
#pragma unroll
    for (int u = 0; u < kRows; ++u) x[u] = ld4(wr + u * WS + j);
#pragma unroll
    for (int v = 0; v < 4; ++v) {
      float y[CD];
      load_cols<CD>(rows + (j + v) * (D + 4), tx, y);
#pragma unroll
      for (int u = 0; u < kRows; ++u) {
        const float xv = v == 0 ? x[u].x : v == 1 ? x[u].y : v == 2 ? x[u].z : x[u].w;
#pragma unroll
        for (int c = 0; c < CD; ++c) acc[u][c] = fmaf(xv, y[c], acc[u][c]);
      }
    }
  }
}

// ---------------------------------------------------------------------------------------------------
// selection: grid (key tiles of 64, query blocks of 32, batch); carry[b][block][key] <- the block's sum per key
// ---------------------------------------------------------------------------------------------------
template <typename T, int D>
__global__ void __launch_bounds__(kThreads) colsum_kernel(Problem p, float* __restrict__ carry, int nblocks, bool vec) {
  extern __shared__ __align__(16) float smem[];
  float* k0s = smem;                       // [64][D + 4]
  float* q0s = k0s + kKF * (D + 4);        // [32][D + 4]
  float* part = q0s + kQ * (D + 4);        // [8][64]
  const int j0 = blockIdx.x * kKF, rb = blockIdx.y, b = blockIdx.z, m0 = rb * kQ;
  if (m0 + kQ <= j0) return;               // all keys of the tile come after all its queries
  load_tile<T, D, kKF>(k0s, row_ptr<T>(p.k0, b, 0), p.k0.st, j0, p.seq, vec);
  load_tile<T, D, kQ>(q0s, row_ptr<T>(p.q0, b, 0), p.q0.st, m0, p.seq, vec);
  __syncthreads();
  const int ty = threadIdx.x >> 4, tx = threadIdx.x & 15;
  float acc[kRows][4] = {};
  dot_rows<D, 4>(acc, q0s, k0s, ty, tx);
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    const int j = j0 + tx + 16 * c;
    float sum = 0.f;
#pragma unroll
    for (int u = 0; u < kRows; ++u) {
      const int i = m0 + ty * kRows + u;
      const float l0 = acc[u][c] * p.scale;
      sum += ((j < i) && (j >= p.exempt) && (i < p.seq) && (l0 > 0.f)) ? l0 : 0.f;
    }
    part[ty * kKF + tx + 16 * c] = sum;
  }
  __syncthreads();
  const int j = j0 + threadIdx.x;
  if (threadIdx.x < kKF && j < p.seq) {
    float sum = 0.f;
#pragma unroll
    for (int g = 0; g < kGroups; ++g) sum += part[g * kKF + threadIdx.x];
    carry[((int64_t)b * nblocks + rb) * p.seq + j] = sum;
  }
}

// One thread per key: exclusive prefix over the query blocks from the key's own on, in place, and the total.
static __global__ void __launch_bounds__(128) scan_kernel(float* __restrict__ carry, float* __restrict__ total, int seq, int nblocks) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x, b = blockIdx.y;
  if (j >= seq) return;
  float* col = carry + (int64_t)b * nblocks * seq + j;
  float run = 0.f;
  int rb = (j & ~(kKF - 1)) / kQ;          // the first block whose tile with this key was computed
  for (; rb + 8 <= nblocks; rb += 8) {
    float x[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) x[u] = col[(int64_t)(rb + u) * seq];
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      col[(int64_t)(rb + u) * seq] = run;
      run += x[u];
    }
  }
  for (; rb < nblocks; ++rb) {
    const float x = col[(int64_t)rb * seq];
    col[(int64_t)rb * seq] = run;
    run += x;
  }
  total[(int64_t)b * seq + j] = run;
}

// ---------------------------------------------------------------------------------------------------
// forward: grid (query tiles of 32 [heaviest first], batch * heads)
// ---------------------------------------------------------------------------------------------------
template <typename T, int D>
__global__ void __launch_bounds__(kThreads) forward_kernel(Problem p, const float* __restrict__ carry,
                                                           float* __restrict__ out, float* __restrict__ lse2,
                                                           int nblocks, bool vec) {
  extern __shared__ __align__(16) float smem[];
  constexpr int P = D + 4, W = kKF + 4, CD = D / 16;
  float* qs = smem;                        // [32][P]
  float* q0s = qs + kQ * P;
  float* ks = q0s + kQ * P;                // [64][P]
  float* k0s = ks + kKF * P;
  float* vs = k0s + kKF * P;
  float* ps = vs + kKF * P;                // [32][W] exp2 tile
  float* gs = ps + kQ * W;                 // [8][64]: selection of a row group, at [group][tx][c]

  const int mi = gridDim.x - 1 - blockIdx.x;
  const int n = blockIdx.y;
  const int b = n / p.heads, h = n - b * p.heads;
  const int m0 = mi * kQ;
  const bool self = h == 0 && !p.external_selector;
  const T* kh = row_ptr<T>(p.k, b, h);
  const T* vh = row_ptr<T>(p.v, b, h);
  const T* k0 = row_ptr<T>(p.k0, b, 0);
  load_tile<T, D, kQ>(qs, row_ptr<T>(p.q, b, h), p.q.st, m0, p.seq, vec);
  if (!self) load_tile<T, D, kQ>(q0s, row_ptr<T>(p.q0, b, 0), p.q0.st, m0, p.seq, vec);

  const int ty = threadIdx.x >> 4, tx = threadIdx.x & 15;
  float damp[kRows];
#pragma unroll
  for (int u = 0; u < kRows; ++u) {
    const int i = m0 + ty * kRows + u;
    damp[u] = 1.f;
    if (p.damp == SA_DAMP_LINEAR) damp[u] = fminf(1.f, (float)p.train_len / (float)(i + 1));
    if (p.damp == SA_DAMP_SQRT) damp[u] = fminf(1.f, sqrtf((float)p.train_len / (float)(i + 1)));
  }
  float run_max[kRows], run_den[kRows], acc[kRows][CD] = {};
#pragma unroll
  for (int u = 0; u < kRows; ++u) run_max[u] = -INFINITY, run_den[u] = 0.f;
  const float* carry_row = carry + ((int64_t)b * nblocks + mi) * p.seq;
  const int last_key = min(m0 + kQ, p.seq);  // keys < last_key can be visible

  Tile<T, D, kKF> tk, tk0, tv;
  float hist[4], next_hist[4];
  auto fetch = [&](int n0) {
    tk.fetch(kh, p.k.st, n0, p.seq, vec);
    if (!self) tk0.fetch(k0, p.k0.st, n0, p.seq, vec);
    tv.fetch(vh, p.v.st, n0, p.seq, vec);
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const int j = n0 + tx + 16 * c;
      next_hist[c] = (j < last_key) ? carry_row[j] : 0.f;
    }
  };
  if (kAhead<T, D>) fetch(0);
  for (int n0 = 0; n0 < last_key; n0 += kKF) {
    if (!kAhead<T, D>) fetch(n0);
    __syncthreads();
    tk.store(ks);
    if (!self) tk0.store(k0s);
    tv.store(vs);
#pragma unroll
    for (int c = 0; c < 4; ++c) hist[c] = next_hist[c];
    __syncthreads();
    if (kAhead<T, D> && n0 + kKF < last_key) fetch(n0 + kKF);
    float z[kRows][4] = {}, sel[kRows][4] = {};
    dot_rows<D, 4>(z, qs, ks, ty, tx);
    if (!self) dot_rows<D, 4>(sel, q0s, k0s, ty, tx);
    float before[4];
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const int j = n0 + tx + 16 * c;
      float sum = 0.f;
#pragma unroll
      for (int u = 0; u < kRows; ++u) {          // sel becomes the exclusive prefix inside the row group
        const int i = m0 + ty * kRows + u;
        const float l0 = (self ? z[u][c] : sel[u][c]) * p.scale;
        const bool gate = (j < i) && (j >= p.exempt) && (i < p.seq) && (l0 > 0.f);
        sel[u][c] = sum;
        sum += gate ? l0 : 0.f;
      }
      before[c] = sum;
    }
    *reinterpret_cast<float4*>(gs + ty * kKF + tx * 4) = make_float4(before[0], before[1], before[2], before[3]);
    __syncthreads();
#pragma unroll
    for (int c = 0; c < 4; ++c) before[c] = 0.f;
    for (int g = 0; g < ty; ++g) {
      const float4 x = ld4(gs + g * kKF + tx * 4);
      before[0] += x.x; before[1] += x.y; before[2] += x.z; before[3] += x.w;
    }
#pragma unroll
    for (int u = 0; u < kRows; ++u) {
      const int i = m0 + ty * kRows + u;
      float tile_max = -INFINITY;
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const int j = n0 + tx + 16 * c;
        const bool causal = (j <= i) && (i < p.seq);
        const float f = (hist[c] + (before[c] + sel[u][c])) * damp[u];
        z[u][c] = causal ? (z[u][c] * p.scale - f) * kLog2e : -INFINITY;
        tile_max = fmaxf(tile_max, z[u][c]);
      }
#pragma unroll
      for (int s = 1; s < 16; s <<= 1) tile_max = fmaxf(tile_max, __shfl_xor_sync(0xffffffffu, tile_max, s));
      const float new_max = fmaxf(run_max[u], tile_max);
      const float alpha = (new_max == -INFINITY) ? 1.f : exp2f(run_max[u] - new_max);
      float sum = 0.f;
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const float e = (z[u][c] == -INFINITY) ? 0.f : exp2f(z[u][c] - new_max);
        ps[(ty * kRows + u) * W + tx + 16 * c] = e;
        sum += e;
      }
      run_den[u] = run_den[u] * alpha + sum;  // this thread's columns only; the rows are added up at the end
      run_max[u] = new_max;
#pragma unroll
      for (int c = 0; c < CD; ++c) acc[u][c] *= alpha;
    }
    __syncwarp();                             // a row's 16 threads are in one warp: its P row is read by them alone
    weighted_rows<D, kKF, W, CD>(acc, ps, vs, ty, tx);
  }
#pragma unroll
  for (int u = 0; u < kRows; ++u) {
#pragma unroll
    for (int s = 1; s < 16; s <<= 1) run_den[u] += __shfl_xor_sync(0xffffffffu, run_den[u], s);
    const int i = m0 + ty * kRows + u;
    if (i >= p.seq) continue;
    const float inv = 1.f / run_den[u];
    float* orow = out + ((int64_t)n * p.seq + i) * D;
#pragma unroll
    for (int c = 0; c < CD; ++c) orow[col_of<CD>(tx, c)] = acc[u][c] * inv;
    if (tx == 0) lse2[(int64_t)n * p.seq + i] = run_max[u] + log2f(run_den[u]);
  }
}

// ---------------------------------------------------------------------------------------------------
// backward: grid (key blocks of 32, batch * heads); query blocks last to first
// ---------------------------------------------------------------------------------------------------
template <typename T, int D>
__global__ void __launch_bounds__(kThreads) backward_kernel(
    Problem p, const float* __restrict__ lse2, const float* __restrict__ carry, const float* __restrict__ dbar,
    const float* __restrict__ d_out, float* __restrict__ dq_acc, float* __restrict__ dk_acc,
    float* __restrict__ dq0, float* __restrict__ dk0, T* __restrict__ dv, int nblocks, bool vec) {
  extern __shared__ __align__(16) float smem[];
  constexpr int P = D + 4, W = kKB + 4, CD = D / 16;
  float* ks = smem;                 // [32][P] keys of this head
  float* vs = ks + kKB * P;
  float* k0s = vs + kKB * P;
  float* qs = k0s + kKB * P;        // [32][P] query tile of this head
  float* q0s = qs + kQ * P;
  float* dos = q0s + kQ * P;
  float* as = dos + kQ * P;         // [32 queries][W] attention
  float* zs = as + kQ * W;          // [32][W] dz; a head that is its own selector: dz + g
  float* gs = zs + kQ * W;          // [32][W] g
  float* gsel = gs + kQ * W;        // [8][32] selection of a row group, at [group][tx][c]
  float* gdz = gsel + kGroups * kKB;   // [8][32] dz of a row group
  float* lse_s = gdz + kGroups * kKB;  // [32]
  float* dbar_s = lse_s + kQ;          // [32]

  const int kb = blockIdx.x;
  const int n = blockIdx.y;
  const int b = n / p.heads, h = n - b * p.heads;
  const int j0 = kb * kKB;
  const bool self = h == 0 && !p.external_selector;
  const T* qh = row_ptr<T>(p.q, b, h);
  const T* q0 = row_ptr<T>(p.q0, b, 0);
  const float* doh = d_out + (int64_t)n * p.seq * D;
  const bool vec_do = (reinterpret_cast<uintptr_t>(d_out) & 15) == 0;
  load_tile<T, D, kKB>(ks, row_ptr<T>(p.k, b, h), p.k.st, j0, p.seq, vec);
  load_tile<T, D, kKB>(vs, row_ptr<T>(p.v, b, h), p.v.st, j0, p.seq, vec);
  if (!self) load_tile<T, D, kKB>(k0s, row_ptr<T>(p.k0, b, 0), p.k0.st, j0, p.seq, vec);

  const int ty = threadIdx.x >> 4, tx = threadIdx.x & 15;   // 4 rows 4 ty .. (queries, or keys of the accumulators)
  float dk_r[kRows][CD] = {}, dv_r[kRows][CD] = {}, dk0_r[kRows][CD] = {};
  float suffix[2] = {0.f, 0.f};     // sum of dz over queries in later tiles, keys tx and tx + 16

  Tile<T, D, kQ> tq, tq0;
  Tile<float, D, kQ> tdo;
  float next_lse = 0.f, next_dbar = 0.f, next_hist[2];
  auto fetch = [&](int rb) {
    const int m0 = rb * kQ;
    tq.fetch(qh, p.q.st, m0, p.seq, vec);
    if (!self) tq0.fetch(q0, p.q0.st, m0, p.seq, vec);
    tdo.fetch(doh, D, m0, p.seq, vec_do);
    if (threadIdx.x < kQ) {
      const int t = m0 + threadIdx.x;
      next_lse = (t < p.seq) ? lse2[(int64_t)n * p.seq + t] : 0.f;
      next_dbar = (t < p.seq) ? dbar[(int64_t)n * p.seq + t] : 0.f;
    }
    const float* carry_row = carry + ((int64_t)b * nblocks + rb) * p.seq;
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      const int j = j0 + tx + 16 * c;
      next_hist[c] = (j < p.seq && j < m0 + kQ) ? carry_row[j] : 0.f;
    }
  };
  if (kAhead<T, D>) fetch(nblocks - 1);
  for (int rb = nblocks - 1; rb >= 0 && rb * kQ + kQ > j0; --rb) {
    const int m0 = rb * kQ;
    if (!kAhead<T, D>) fetch(rb);
    __syncthreads();
    tq.store(qs);
    if (!self) tq0.store(q0s);
    tdo.store(dos);
    if (threadIdx.x < kQ) {
      lse_s[threadIdx.x] = next_lse;
      dbar_s[threadIdx.x] = next_dbar;
    }
    const float hist[2] = {next_hist[0], next_hist[1]};
    __syncthreads();
    if (kAhead<T, D> && rb > 0 && rb * kQ > j0) fetch(rb - 1);

    float aff[kRows][2] = {}, sel[kRows][2] = {}, dov[kRows][2] = {};
    dot_rows<D, 2>(aff, qs, ks, ty, tx);
    if (!self) dot_rows<D, 2>(sel, q0s, k0s, ty, tx);
    dot_rows<D, 2>(dov, dos, vs, ty, tx);
    unsigned gates = 0u;
    float before[2];
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      const int j = j0 + tx + 16 * c;
      float sum = 0.f;
#pragma unroll
      for (int u = 0; u < kRows; ++u) {          // sel becomes the exclusive prefix inside the row group
        const int i = m0 + ty * kRows + u;
        const float l0 = (self ? aff[u][c] : sel[u][c]) * p.scale;
        const bool gate = (j < i) && (j >= p.exempt) && (i < p.seq) && (l0 > 0.f);
        gates |= (gate ? 1u : 0u) << (u * 2 + c);
        sel[u][c] = sum;
        sum += gate ? l0 : 0.f;
      }
      before[c] = sum;
    }
    *reinterpret_cast<float2*>(gsel + ty * kKB + tx * 2) = make_float2(before[0], before[1]);
    __syncthreads();
    before[0] = before[1] = 0.f;
    for (int g = 0; g < ty; ++g) {
      const float2 x = *reinterpret_cast<const float2*>(gsel + g * kKB + tx * 2);
      before[0] += x.x; before[1] += x.y;
    }
    float dz[kRows][2], dz_sum[2] = {0.f, 0.f};
#pragma unroll
    for (int u = 0; u < kRows; ++u) {
      const int r = ty * kRows + u, i = m0 + r;
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        const int j = j0 + tx + 16 * c;
        const bool causal = (j <= i) && (i < p.seq);
        float attn = 0.f;
        dz[u][c] = 0.f;
        if (causal) {
          attn = exp2f((aff[u][c] * p.scale - (hist[c] + (before[c] + sel[u][c]))) * kLog2e - lse_s[r]);
          dz[u][c] = attn * (dov[u][c] - dbar_s[r]);
        }
        as[r * W + tx + 16 * c] = attn;
        dz_sum[c] += dz[u][c];
      }
    }
    *reinterpret_cast<float2*>(gdz + ty * kKB + tx * 2) = make_float2(dz_sum[0], dz_sum[1]);
    __syncthreads();
    float later[2] = {suffix[0], suffix[1]};
    for (int g = kGroups - 1; g >= 0; --g) {
      const float2 x = *reinterpret_cast<const float2*>(gdz + g * kKB + tx * 2);
      if (g > ty) { later[0] += x.x; later[1] += x.y; }
      suffix[0] += x.x; suffix[1] += x.y;
    }
#pragma unroll
    for (int u = kRows - 1; u >= 0; --u) {
      const int r = ty * kRows + u;
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        const float g = ((gates >> (u * 2 + c)) & 1u) ? -later[c] : 0.f;
        later[c] += dz[u][c];
        zs[r * W + tx + 16 * c] = self ? dz[u][c] + g : dz[u][c];
        if (!self) gs[r * W + tx + 16 * c] = g;
      }
    }
    __syncthreads();

    // key rows: dV += A^T dO, dK += Z^T Q, dK0 += G^T Q0
#pragma unroll 2
    for (int r = 0; r < kQ; ++r) {
      const float4 a = ld4(as + r * W + ty * kRows), z = ld4(zs + r * W + ty * kRows);
      const float av[kRows] = {a.x, a.y, a.z, a.w}, zv[kRows] = {z.x, z.y, z.z, z.w};
      float y[CD];
      load_cols<CD>(dos + r * P, tx, y);
#pragma unroll
      for (int u = 0; u < kRows; ++u)
#pragma unroll
        for (int c = 0; c < CD; ++c) dv_r[u][c] = fmaf(av[u], y[c], dv_r[u][c]);
      load_cols<CD>(qs + r * P, tx, y);
#pragma unroll
      for (int u = 0; u < kRows; ++u)
#pragma unroll
        for (int c = 0; c < CD; ++c) dk_r[u][c] = fmaf(zv[u], y[c], dk_r[u][c]);
      if (!self) {
        const float4 g = ld4(gs + r * W + ty * kRows);
        const float gv[kRows] = {g.x, g.y, g.z, g.w};
        load_cols<CD>(q0s + r * P, tx, y);
#pragma unroll
        for (int u = 0; u < kRows; ++u)
#pragma unroll
          for (int c = 0; c < CD; ++c) dk0_r[u][c] = fmaf(gv[u], y[c], dk0_r[u][c]);
      }
    }
    // query rows: dQ += Z K, dQ0 += G K0, reduced across the key blocks in global memory
    {
      float x[kRows][CD] = {};
      weighted_rows<D, kKB, W, CD>(x, zs, ks, ty, tx);
#pragma unroll
      for (int u = 0; u < kRows; ++u)
        if (m0 + ty * kRows + u < p.seq) reduce_cols<CD>(dq_acc + ((int64_t)n * p.seq + m0 + ty * kRows + u) * D, tx, x[u], p.scale);
    }
    if (!self) {
      float x[kRows][CD] = {};
      weighted_rows<D, kKB, W, CD>(x, gs, k0s, ty, tx);
#pragma unroll
      for (int u = 0; u < kRows; ++u)
        if (m0 + ty * kRows + u < p.seq) reduce_cols<CD>(dq0 + ((int64_t)b * p.seq + m0 + ty * kRows + u) * D, tx, x[u], p.scale);
    }
  }
#pragma unroll
  for (int u = 0; u < kRows; ++u) {
    const int j = j0 + ty * kRows + u;
    if (j >= p.seq) continue;
    float* dk_row = dk_acc + ((int64_t)n * p.seq + j) * D;
    T* dv_row = dv + ((int64_t)n * p.seq + j) * D;
#pragma unroll
    for (int c = 0; c < CD; ++c) {
      dk_row[col_of<CD>(tx, c)] = dk_r[u][c] * p.scale;
      dv_row[col_of<CD>(tx, c)] = from_float<T>(dv_r[u][c]);
    }
    if (!self) reduce_cols<CD>(dk0 + ((int64_t)b * p.seq + j) * D, tx, dk0_r[u], p.scale);
  }
}

template <int D> constexpr size_t colsum_smem() { return sizeof(float) * ((kKF + kQ) * (D + 4) + kGroups * kKF); }
template <int D> constexpr size_t forward_smem() {
  return sizeof(float) * ((2 * kQ + 3 * kKF) * (D + 4) + kQ * (kKF + 4) + kGroups * kKF);
}
template <int D> constexpr size_t backward_smem() {
  return sizeof(float) * ((3 * kKB + 3 * kQ) * (D + 4) + 3 * kQ * (kKB + 4) + 2 * kGroups * kKB + 2 * kQ);
}

// Four consecutive elements of every row start at a 16-byte (fp32) or 8-byte boundary.
inline bool vector_rows(const Problem& p) {
  const int64_t es = p.dtype == SA_F32 ? 4 : 2;
  for (const Strided* s : {&p.q, &p.k, &p.v, &p.q0, &p.k0})
    if ((reinterpret_cast<uintptr_t>(s->ptr) | (uintptr_t)(s->sb * es) | (uintptr_t)(s->sh * es) | (uintptr_t)(s->st * es)) & (4 * es - 1))
      return false;
  return true;
}

// The selection pass: carry checkpoints every 32 queries and the per-key totals.
template <typename T, int D>
int carry_impl(const Problem& p, float* carry, float* total, cudaStream_t s) {
  const int nb = (p.seq + kQ - 1) / kQ;
  SA_CUDA_CHECK(allow_smem(colsum_kernel<T, D>, colsum_smem<D>()));
  count_launch();
  colsum_kernel<T, D><<<dim3((p.seq + kKF - 1) / kKF, nb, p.batch), kThreads, colsum_smem<D>(), s>>>(p, carry, nb, vector_rows(p));
  SA_CUDA_CHECK(cudaGetLastError());
  count_launch();
  scan_kernel<<<dim3((p.seq + 127) / 128, p.batch), 128, 0, s>>>(carry, total, p.seq, nb);
  SA_CUDA_CHECK(cudaGetLastError());
  return SA_OK;
}

template <typename T, int D>
int forward_impl(const Problem& p, float* out, float* lse2, float* carry, float* total, cudaStream_t s) {
  if (int st = carry_impl<T, D>(p, carry, total, s)) return st;
  const int nb = (p.seq + kQ - 1) / kQ;
  SA_CUDA_CHECK(allow_smem(forward_kernel<T, D>, forward_smem<D>()));
  count_launch();
  forward_kernel<T, D><<<dim3(nb, p.batch * p.heads), kThreads, forward_smem<D>(), s>>>(p, carry, out, lse2, nb, vector_rows(p));
  SA_CUDA_CHECK(cudaGetLastError());
  return SA_OK;
}

template <typename T, int D>
int backward_impl(const Problem& p, const float* lse2, const float* carry, const float* dbar, const float* d_out,
                  float* dq_acc, float* dk_acc, float* dq0, float* dk0, void* dv, cudaStream_t s) {
  const int nb = (p.seq + kQ - 1) / kQ;
  SA_CUDA_CHECK(allow_smem(backward_kernel<T, D>, backward_smem<D>()));
  count_launch();
  backward_kernel<T, D><<<dim3((p.seq + kKB - 1) / kKB, p.batch * p.heads), kThreads, backward_smem<D>(), s>>>(
      p, lse2, carry, dbar, d_out, dq_acc, dk_acc, dq0, dk0, static_cast<T*>(dv), nb, vector_rows(p));
  SA_CUDA_CHECK(cudaGetLastError());
  return SA_OK;
}

template <typename T>
int forward_by_dim(const Problem& p, float* out, float* lse2, float* carry, float* total, cudaStream_t s) {
  switch (p.head_dim) {
    case 16: return forward_impl<T, 16>(p, out, lse2, carry, total, s);
    case 32: return forward_impl<T, 32>(p, out, lse2, carry, total, s);
    case 64: return forward_impl<T, 64>(p, out, lse2, carry, total, s);
    case 128: return forward_impl<T, 128>(p, out, lse2, carry, total, s);
  }
  return SA_ERR_UNSUPPORTED;
}

template <typename T>
int carry_by_dim(const Problem& p, float* carry, float* total, cudaStream_t s) {
  switch (p.head_dim) {
    case 16: return carry_impl<T, 16>(p, carry, total, s);
    case 32: return carry_impl<T, 32>(p, carry, total, s);
    case 64: return carry_impl<T, 64>(p, carry, total, s);
    case 128: return carry_impl<T, 128>(p, carry, total, s);
  }
  return SA_ERR_UNSUPPORTED;
}

template <typename T>
int backward_by_dim(const Problem& p, const float* lse2, const float* carry, const float* dbar, const float* d_out,
                    float* dq_acc, float* dk_acc, float* dq0, float* dk0, void* dv, cudaStream_t s) {
  switch (p.head_dim) {
    case 16: return backward_impl<T, 16>(p, lse2, carry, dbar, d_out, dq_acc, dk_acc, dq0, dk0, dv, s);
    case 32: return backward_impl<T, 32>(p, lse2, carry, dbar, d_out, dq_acc, dk_acc, dq0, dk0, dv, s);
    case 64: return backward_impl<T, 64>(p, lse2, carry, dbar, d_out, dq_acc, dk_acc, dq0, dk0, dv, s);
    case 128: return backward_impl<T, 128>(p, lse2, carry, dbar, d_out, dq_acc, dk_acc, dq0, dk0, dv, s);
  }
  return SA_ERR_UNSUPPORTED;
}

}  // namespace simt
}  // namespace sa
