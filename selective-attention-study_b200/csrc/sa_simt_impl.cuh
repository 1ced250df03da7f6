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
// Work split of forward and backward.  A team is 256 threads in two groups of 128, 8 x 16; a CTA has one team or two.
//   logits    each group forms half of the contraction of the whole tile, 4 rows x 4 (backward 2) columns a thread, and hands
//             the other group its half of the columns, so that what follows has one group for each half of the columns
//   forward   a group has the softmax state and the output of its own 32 keys of every tile; a second team takes every other
//             key tile; the two or four are merged at the end, and nothing else crosses groups
//   backward  a second team takes every other query tile and shares the sums of dz per key, the one thing that is carried from
//             tile to tile; key gradients: 4 x 4 a thread for any D, so 128 / D sets of threads take the queries in turn and
//             are added up at the end; dQ and the selector's dQ0: a group each
// Operands sit in shared memory as fp32 rows of D + 4 floats (consecutive rows start 4 banks apart) and are read 16 bytes at a
// time; two FMAs an instruction, along the contraction in the logits (even and odd elements apart), else along the columns.
// What bounds it: shared-memory loads (71 % of their rate in backward at D = 32) and FMAs at about the same rate; with few
// (batch, head) rows the longest walk.  us for selection, forward, backward, at first / 128 threads a CTA, one FMA an
// instruction / now:  (2, 4, 1024, 64) fp32  153, 403, 859 / 15, 134, 339 / 14, 78, 160;  (4, 8, 1000, 32) fp16 now 12, 170, 290.
//
// A head that is its own selector (head 0, unless the selector comes from outside) has its selection logits already, and
// since Q0 = Q, K0 = K its two gradient paths add before the products: dK += (dz + g)^T Q, dQ += (dz + g) K.
#pragma once
#include "sa_common.cuh"

namespace sa {
namespace simt {

constexpr int kTeam = 256;     // forward and backward: a CTA is two teams (forward, D = 128: one) of two groups of 128
constexpr int kSelThreads = 128;
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
template <typename T, int D, int ROWS, int THREADS = kTeam>
struct Tile {
  static constexpr int C = D / 4, N = (ROWS * C + THREADS - 1) / THREADS;
  struct alignas(4 * sizeof(T)) Quad { T e[4]; };
  Quad x[N];
  __device__ __forceinline__ void fetch(int id, const T* base, int64_t st, int t0, int seq, bool vec) {
#pragma unroll
    for (int u = 0; u < N; ++u) {
      const int idx = id + u * THREADS, r = idx / C, c = (idx - r * C) * 4, t = t0 + r;
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
  __device__ __forceinline__ void store(int id, float* dst) const {
#pragma unroll
    for (int u = 0; u < N; ++u) {
      const int idx = id + u * THREADS, r = idx / C, c = (idx - r * C) * 4;
      if (r < ROWS)
        *reinterpret_cast<float4*>(dst + r * (D + 4) + c) =
            make_float4(to_float<T>(x[u].e[0]), to_float<T>(x[u].e[1]), to_float<T>(x[u].e[2]), to_float<T>(x[u].e[3]));
    }
  }
};
template <typename T, int D, int ROWS, int THREADS>
__device__ __forceinline__ void load_tile(float* dst, const T* base, int64_t st, int t0, int seq, bool vec) {
  Tile<T, D, ROWS, THREADS> x;
  x.fetch(threadIdx.x, base, st, t0, seq, vec);
  x.store(threadIdx.x, dst);
}

// Thread `id` of a grid of X columns: neighbouring lanes take two rows of one column.  A 16-byte shared-memory load takes 2 cycles
// a warp where lanes l and l ^ 1 (or l ^ 2) read the same address, and 4 where only l and l ^ 16 do, however few the addresses.
template <int X> __device__ __forceinline__ int col_of(int id) { return (id >> 1) % X; }
template <int X> __device__ __forceinline__ int row_of(int id) { return (id & 1) | (id / (2 * X) << 1); }

__device__ __forceinline__ float4 ld4(const float* p) { return *reinterpret_cast<const float4*>(p); }

// Two fp32 FMAs in one instruction: 118 FMAs a cycle and SM measured, where the single one reaches 85.
using f32x2 = unsigned long long;
__device__ __forceinline__ f32x2 pack2(float lo, float hi) {
  f32x2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ float2 unpack2(f32x2 x) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(x));
  return r;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
  f32x2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ ulonglong2 ld4x2(const float* p) { return *reinterpret_cast<const ulonglong2*>(p); }
__device__ __forceinline__ void team_sync(int team) { asm volatile("bar.sync %0, 256;" ::"r"(1 + team) : "memory"); }
__device__ __forceinline__ void group_sync(int group) { asm volatile("bar.sync %0, 128;" ::"r"(3 + group) : "memory"); }

// acc[u][c] = a[4 ty + u] . row tx + 16 c of `own` (the first half of the columns) or `other`, over DN elements: the even and the
// odd ones each in order, then their sum
template <int D, int DN, int NC>
__device__ __forceinline__ void dot_rows(float (&acc)[kRows][NC], const float* a, const float* own, const float* other, int ty, int tx) {
  const float* ar = a + (ty * kRows) * (D + 4);
  const float* b0 = own + tx * (D + 4);
  const float* b1 = other + tx * (D + 4);
  f32x2 sum[kRows][NC];
#pragma unroll
  for (int u = 0; u < kRows; ++u)
#pragma unroll
    for (int c = 0; c < NC; ++c) sum[u][c] = 0ull;
#pragma unroll 4
  for (int d = 0; d < DN; d += 4) {
    ulonglong2 x[kRows], y[NC];
#pragma unroll
    for (int u = 0; u < kRows; ++u) x[u] = ld4x2(ar + u * (D + 4) + d);
#pragma unroll
    for (int c = 0; c < NC; ++c) y[c] = ld4x2((c < NC / 2 ? b0 + 16 * c * (D + 4) : b1 + 16 * (c - NC / 2) * (D + 4)) + d);
#pragma unroll
    for (int u = 0; u < kRows; ++u)
#pragma unroll
      for (int c = 0; c < NC; ++c) {
        sum[u][c] = fma2(x[u].x, y[c].x, sum[u][c]);
        sum[u][c] = fma2(x[u].y, y[c].y, sum[u][c]);
      }
  }
#pragma unroll
  for (int u = 0; u < kRows; ++u)
#pragma unroll
    for (int c = 0; c < NC; ++c) {
      const float2 v = unpack2(sum[u][c]);
      acc[u][c] = v.x + v.y;
    }
}

// CD neighbouring output columns of one row (CD = 8: two runs of four, 64 columns apart).
template <int CD>
struct Cols {
  f32x2 p[CD / 2];
  __device__ __forceinline__ void zero() {
#pragma unroll
    for (int k = 0; k < CD / 2; ++k) p[k] = 0ull;
  }
  __device__ __forceinline__ void load(const float* row, int tx) {
    if constexpr (CD == 2) {
      p[0] = *reinterpret_cast<const f32x2*>(row + 2 * tx);
    } else {
#pragma unroll
      for (int f = 0; f < CD / 4; ++f) {
        const ulonglong2 v = ld4x2(row + 64 * f + 4 * tx);
        p[2 * f] = v.x; p[2 * f + 1] = v.y;
      }
    }
  }
  __device__ __forceinline__ void add(f32x2 w, const Cols& y) {
#pragma unroll
    for (int k = 0; k < CD / 2; ++k) p[k] = fma2(w, y.p[k], p[k]);
  }
  __device__ __forceinline__ void scale(float a) {
    const f32x2 aa = pack2(a, a);
#pragma unroll
    for (int k = 0; k < CD / 2; ++k) p[k] = fma2(aa, p[k], 0ull);
  }
  __device__ __forceinline__ float get(int c) const {
    const float2 v = unpack2(p[c >> 1]);
    return (c & 1) ? v.y : v.x;
  }
};
template <>
struct Cols<1> {
  float p;
  __device__ __forceinline__ void zero() { p = 0.f; }
  __device__ __forceinline__ void load(const float* row, int tx) { p = row[tx]; }
  __device__ __forceinline__ void add(f32x2 w, const Cols& y) { p = fmaf(unpack2(w).x, y.p, p); }
  __device__ __forceinline__ void scale(float a) { p *= a; }
  __device__ __forceinline__ float get(int) const { return p; }
};
template <int CD>
__device__ __forceinline__ int out_col(int tx, int c) { return CD >= 4 ? 64 * (c >> 2) + 4 * tx + (c & 3) : CD * tx + c; }
__device__ __forceinline__ void reduce4(float* dst, float4 x) {
  asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(dst), "f"(x.x), "f"(x.y), "f"(x.z), "f"(x.w) : "memory");
}

// acc[u] += sum_j w[R y + u][j] rows[j][columns of x] over N rows j, w with row stride WS
template <int D, int N, int WS, int R, int CD>
__device__ __forceinline__ void weighted_rows(Cols<CD> (&acc)[R], const float* w, const float* rows, int y, int x) {
  const float* wr = w + (y * R) * WS;
#pragma unroll 2
  for (int j = 0; j < N; j += 4) {
    float4 a[R];
#pragma unroll
    for (int u = 0; u < R; ++u) a[u] = ld4(wr + u * WS + j);
#pragma unroll
    for (int v = 0; v < 4; ++v) {
      Cols<CD> b;
      b.load(rows + (j + v) * (D + 4), x);
#pragma unroll
      for (int u = 0; u < R; ++u) {
        const float av = v == 0 ? a[u].x : v == 1 ? a[u].y : v == 2 ? a[u].z : a[u].w;
        acc[u].add(pack2(av, av), b);
      }
    }
  }
}

// ---------------------------------------------------------------------------------------------------
// selection: grid (key tiles of 64, query blocks of 32, batch); carry[b][block][key] <- the block's sum per key
// ---------------------------------------------------------------------------------------------------
template <typename T, int D>
__global__ void __launch_bounds__(kSelThreads) colsum_kernel(Problem p, float* __restrict__ carry, int nblocks, bool vec) {
  extern __shared__ __align__(16) float smem[];
  float* k0s = smem;                       // [64][D + 4]
  float* q0s = k0s + kKF * (D + 4);        // [32][D + 4]
  float* part = q0s + kQ * (D + 4);        // [8][64]
  const int j0 = blockIdx.x * kKF, rb = blockIdx.y, b = blockIdx.z, m0 = rb * kQ;
  if (m0 + kQ <= j0) return;               // all keys of the tile come after all its queries
  load_tile<T, D, kKF, kSelThreads>(k0s, row_ptr<T>(p.k0, b, 0), p.k0.st, j0, p.seq, vec);
  load_tile<T, D, kQ, kSelThreads>(q0s, row_ptr<T>(p.q0, b, 0), p.q0.st, m0, p.seq, vec);
  __syncthreads();
  const int ty = row_of<16>(threadIdx.x), tx = col_of<16>(threadIdx.x);
  float acc[kRows][4];
  dot_rows<D, D, 4>(acc, q0s, k0s, k0s + 32 * (D + 4), ty, tx);
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
template <int D> constexpr int kForwardTeamFloats = 3 * kKF * (D + 4) + kQ * (kKF + 4) + kGroups * kKF + 4 * kTeam * 4;

template <typename T, int D, int TEAMS>
__global__ void __launch_bounds__(kTeam * TEAMS, TEAMS == 1 && D < 128 ? 2 : 1) forward_kernel(Problem p, const float* __restrict__ carry,
                                                                             float* __restrict__ out, float* __restrict__ lse2,
                                                                             int nblocks, bool vec) {
  extern __shared__ __align__(16) float smem[];
  constexpr int P = D + 4, W = kKF + 4, CD = D / 16, kThreads = kTeam * TEAMS;
  const int team = threadIdx.x / kTeam, id = threadIdx.x % kTeam, grp = id >> 7, ty = row_of<16>(id & 127), tx = col_of<16>(id);
  float* qs = smem;                        // [32][P]
  float* q0s = qs + kQ * P;
  float* ks = q0s + kQ * P + team * kForwardTeamFloats<D>;    // [64][P], from here on a team's own
  float* k0s = ks + kKF * P;
  float* vs = k0s + kKF * P;
  float* ps = vs + kKF * P;                // [32][W] exp2 tile
  float* gs = ps + kQ * W;                 // [2][8][16][2]: selection of a row group
  float4* ex = reinterpret_cast<float4*>(gs + kGroups * kKF);    // [4][256]: the products' other half, for the other group

  const int rows = p.batch * p.heads, mi = nblocks - 1 - (int)blockIdx.x / rows, n = (int)blockIdx.x % rows;
  const int b = n / p.heads, h = n - b * p.heads;
  const int m0 = mi * kQ;
  const bool self = h == 0 && !p.external_selector;
  const T* kh = row_ptr<T>(p.k, b, h);
  const T* vh = row_ptr<T>(p.v, b, h);
  const T* k0 = row_ptr<T>(p.k0, b, 0);
  load_tile<T, D, kQ, kThreads>(qs, row_ptr<T>(p.q, b, h), p.q.st, m0, p.seq, vec);
  if (!self) load_tile<T, D, kQ, kThreads>(q0s, row_ptr<T>(p.q0, b, 0), p.q0.st, m0, p.seq, vec);

  float damp[kRows];
#pragma unroll
  for (int u = 0; u < kRows; ++u) {
    const int i = m0 + ty * kRows + u;
    damp[u] = 1.f;
    if (p.damp == SA_DAMP_LINEAR) damp[u] = fminf(1.f, (float)p.train_len / (float)(i + 1));
    if (p.damp == SA_DAMP_SQRT) damp[u] = fminf(1.f, sqrtf((float)p.train_len / (float)(i + 1)));
  }
  // A group keeps the running maximum, the denominator and the sums of its own 32 keys of every tile.
  float run_max[kRows], run_den[kRows];
  Cols<CD> acc[kRows];
#pragma unroll
  for (int u = 0; u < kRows; ++u) run_max[u] = -INFINITY, run_den[u] = 0.f, acc[u].zero();
  const float* carry_row = carry + ((int64_t)b * nblocks + mi) * p.seq;
  const int last_key = min(m0 + kQ, p.seq);  // keys < last_key can be visible

  // The next tile's keys are on their way while the values are weighted, the values while the products run.
  Tile<T, D, kKF> tk, tk0, tv;
  float hist[2], next_hist[2];
  auto fetch = [&](int n0) {
    tk.fetch(id, kh, p.k.st, n0, p.seq, vec);
    if (!self) tk0.fetch(id, k0, p.k0.st, n0, p.seq, vec);
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      const int j = n0 + 32 * grp + tx + 16 * c;
      next_hist[c] = (j < last_key) ? carry_row[j] : 0.f;
    }
  };
  fetch(team * kKF);
  __syncthreads();
  for (int n0 = team * kKF; n0 < last_key; n0 += TEAMS * kKF) {
    team_sync(team);
    tk.store(id, ks);
    if (!self) tk0.store(id, k0s);
#pragma unroll
    for (int c = 0; c < 2; ++c) hist[c] = next_hist[c];
    tv.fetch(id, vh, p.v.st, n0, p.seq, vec);
    team_sync(team);
    float z[kRows][2], sel[kRows][2];
    {
      const int d0 = grp * (D / 2), own = 32 * grp * P + d0, other = 32 * (1 - grp) * P + d0;
      float t[kRows][4];
      auto product = [&](float (&mine)[kRows][2], const float* a, const float* k, float4* to) {
        dot_rows<D, D / 2, 4>(t, a + d0, k + own, k + other, ty, tx);
#pragma unroll
        for (int u = 0; u < kRows; ++u) mine[u][0] = t[u][0], mine[u][1] = t[u][1];
        to[id] = make_float4(t[0][2], t[0][3], t[1][2], t[1][3]);
        to[kTeam + id] = make_float4(t[2][2], t[2][3], t[3][2], t[3][3]);
      };
      product(z, qs, ks, ex);
      if (!self) product(sel, q0s, k0s, ex + 2 * kTeam);
      tv.store(id, vs);
      team_sync(team);
      auto join = [&](float (&mine)[kRows][2], const float4* from) {
        const float4 x = from[id ^ 128], y = from[kTeam + (id ^ 128)];
        mine[0][0] += x.x; mine[0][1] += x.y; mine[1][0] += x.z; mine[1][1] += x.w;
        mine[2][0] += y.x; mine[2][1] += y.y; mine[3][0] += y.z; mine[3][1] += y.w;
      };
      join(z, ex);
      if (!self) join(sel, ex + 2 * kTeam);
    }
    if (n0 + TEAMS * kKF < last_key) fetch(n0 + TEAMS * kKF);
    float before[2];
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      const int j = n0 + 32 * grp + tx + 16 * c;
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
    float* gsel = gs + grp * (kGroups * 32) + tx * 2;
    *reinterpret_cast<float2*>(gsel + ty * 32) = make_float2(before[0], before[1]);
    group_sync(2 * team + grp);
    before[0] = before[1] = 0.f;
    for (int g = 0; g < ty; ++g) {
      const float2 x = *reinterpret_cast<const float2*>(gsel + g * 32);
      before[0] += x.x; before[1] += x.y;
    }
#pragma unroll
    for (int u = 0; u < kRows; ++u) {
      const int i = m0 + ty * kRows + u;
      float tile_max = -INFINITY;
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        const int j = n0 + 32 * grp + tx + 16 * c;
        const bool causal = (j <= i) && (i < p.seq);
        const float f = (hist[c] + (before[c] + sel[u][c])) * damp[u];
        z[u][c] = causal ? (z[u][c] * p.scale - f) * kLog2e : -INFINITY;
        tile_max = fmaxf(tile_max, z[u][c]);
      }
#pragma unroll
      for (int s = 2; s < 32; s <<= 1) tile_max = fmaxf(tile_max, __shfl_xor_sync(0xffffffffu, tile_max, s));
      const float new_max = fmaxf(run_max[u], tile_max);
      const float alpha = (new_max == -INFINITY) ? 1.f : exp2f(run_max[u] - new_max);
      float sum = 0.f;
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        const float e = (z[u][c] == -INFINITY) ? 0.f : exp2f(z[u][c] - new_max);
        ps[(ty * kRows + u) * W + 32 * grp + tx + 16 * c] = e;
        sum += e;
      }
      run_den[u] = run_den[u] * alpha + sum;  // this thread's columns only; the rows are added up at the end
      run_max[u] = new_max;
      acc[u].scale(alpha);
    }
    __syncwarp();                             // a group's P row is written and read by the 16 threads of one warp alone
    weighted_rows<D, 32, W, kRows, CD>(acc, ps + 32 * grp, vs + 32 * grp * P, ty, tx);
  }
  // the groups' sums, at a common maximum: group g > 0 hands over [32][D], then maxima [32] and denominators [32]
  __syncthreads();
  const int g = threadIdx.x >> 7;
  constexpr int kHanded = kQ * (D + 2);
#pragma unroll
  for (int u = 0; u < kRows; ++u) {
#pragma unroll
    for (int s = 2; s < 32; s <<= 1) run_den[u] += __shfl_xor_sync(0xffffffffu, run_den[u], s);
    const int r = ty * kRows + u;
    if (g > 0) {
      float* to = smem + (g - 1) * kHanded;
#pragma unroll
      for (int c = 0; c < CD; ++c) to[r * D + out_col<CD>(tx, c)] = acc[u].get(c);
      if (tx == 0) to[kQ * D + r] = run_max[u], to[kQ * D + kQ + r] = run_den[u];
    }
  }
  __syncthreads();
  if (g > 0) return;
#pragma unroll
  for (int u = 0; u < kRows; ++u) {
    const int r = ty * kRows + u, i = m0 + r;
    if (i >= p.seq) continue;
    float top = run_max[u];                                     // finite: a visible row sees key 0, which is group 0's
#pragma unroll
    for (int k = 0; k < 2 * TEAMS - 1; ++k) top = fmaxf(top, smem[k * kHanded + kQ * D + r]);
    const float a = exp2f(run_max[u] - top);
    float den = run_den[u] * a, y[CD];
#pragma unroll
    for (int c = 0; c < CD; ++c) y[c] = acc[u].get(c) * a;
#pragma unroll
    for (int k = 0; k < 2 * TEAMS - 1; ++k) {
      const float* from = smem + k * kHanded;
      const float o = exp2f(from[kQ * D + r] - top);
      den += from[kQ * D + kQ + r] * o;
#pragma unroll
      for (int c = 0; c < CD; ++c) y[c] += from[r * D + out_col<CD>(tx, c)] * o;
    }
    const float inv = 1.f / den;
    float* orow = out + ((int64_t)n * p.seq + i) * D;
#pragma unroll
    for (int c = 0; c < CD; ++c) orow[out_col<CD>(tx, c)] = y[c] * inv;
    if (tx == 0) lse2[(int64_t)n * p.seq + i] = top + log2f(den);
  }
}

// ---------------------------------------------------------------------------------------------------
// backward: grid (key blocks of 32, batch * heads); query blocks last to first
// ---------------------------------------------------------------------------------------------------
// dst rows += scale * w rows, R rows and 4 columns a thread, `id` counting the threads
template <int D, int R>
__device__ __forceinline__ void query_grads(const float* w, const float* rows, float* dst, int left, float scale, int id) {
  const int x = col_of<D / 4>(id), y = row_of<D / 4>(id);
  if (y * R >= kQ) return;
  Cols<4> acc[R];
#pragma unroll
  for (int u = 0; u < R; ++u) acc[u].zero();
  weighted_rows<D, kKB, kKB + 4, R, 4>(acc, w, rows, y, x);
#pragma unroll
  for (int u = 0; u < R; ++u)
    if (y * R + u < left)
      reduce4(dst + (int64_t)(y * R + u) * D + 4 * x, make_float4(acc[u].get(0) * scale, acc[u].get(1) * scale,
                                                                  acc[u].get(2) * scale, acc[u].get(3) * scale));
}

template <int D> constexpr int kBackwardTeamFloats = 3 * kQ * (D + 4) + 3 * kQ * (kKB + 4) + 3 * kTeam * 4 + kGroups * kKB + 2 * kQ;

template <typename T, int D, int TEAMS>
__global__ void __launch_bounds__(kTeam * TEAMS, 2 / TEAMS) backward_kernel(
    Problem p, const float* __restrict__ lse2, const float* __restrict__ carry, const float* __restrict__ dbar,
    const float* __restrict__ d_out, float* __restrict__ dq_acc, float* __restrict__ dk_acc,
    float* __restrict__ dq0, float* __restrict__ dk0, T* __restrict__ dv, int nblocks, bool vec) {
  extern __shared__ __align__(16) float smem[];
  constexpr int P = D + 4, W = kKB + 4;
  const int team = threadIdx.x / kTeam, id = threadIdx.x % kTeam;
  float* ks = smem;                 // [32][P] keys of this head
  float* vs = ks + kKB * P;
  float* k0s = vs + kKB * P;
  float* gdz = k0s + kKB * P;       // [2][row groups of all teams][32] dz of a row group, by the parity of the step
  float* qs = gdz + 2 * TEAMS * kGroups * kKB + team * kBackwardTeamFloats<D>;   // [32][P] query tile of this head, from here on a team's own
  float* q0s = qs + kQ * P;
  float* dos = q0s + kQ * P;
  float* as = dos + kQ * P;         // [32 queries][W] attention
  float* zs = as + kQ * W;          // [32][W] dz; a head that is its own selector: dz + g
  float* gs = zs + kQ * W;          // [32][W] g
  float4* ex = reinterpret_cast<float4*>(gs + kQ * W);   // [3][256]: the products' other half, for the other group
  float* gsel = gs + kQ * W + 3 * kTeam * 4;             // [8][32] selection of a row group
  float* lse_s = gsel + kGroups * kKB; // [32]
  float* dbar_s = lse_s + kQ;          // [32]

  const int heads_all = p.batch * p.heads, kb = (int)blockIdx.x / heads_all, n = (int)blockIdx.x % heads_all;
  const int b = n / p.heads, h = n - b * p.heads;
  const int j0 = kb * kKB;
  const bool self = h == 0 && !p.external_selector;
  const T* qh = row_ptr<T>(p.q, b, h);
  const T* q0 = row_ptr<T>(p.q0, b, 0);
  const float* doh = d_out + (int64_t)n * p.seq * D;
  const bool vec_do = (reinterpret_cast<uintptr_t>(d_out) & 15) == 0;
  load_tile<T, D, kKB, kTeam * TEAMS>(ks, row_ptr<T>(p.k, b, h), p.k.st, j0, p.seq, vec);
  load_tile<T, D, kKB, kTeam * TEAMS>(vs, row_ptr<T>(p.v, b, h), p.v.st, j0, p.seq, vec);
  if (!self) load_tile<T, D, kKB, kTeam * TEAMS>(k0s, row_ptr<T>(p.k0, b, 0), p.k0.st, j0, p.seq, vec);

  // logits: 4 queries 4 ty .. and key col of a thread, of which its group forms half of the contraction
  const int grp = id >> 7, ty = row_of<16>(id & 127), tx = col_of<16>(id), col = 16 * grp + tx;
  const int j = j0 + col;
  // key gradients: D / 4 queries of every tile (`part`), 4 keys 4 ky .. and 4 columns 4 kx ..
  constexpr int kParts = 128 / D, kPartRows = kQ / kParts;
  const int part = id / (2 * D), ky = row_of<D / 4>(id % (2 * D)), kx = col_of<D / 4>(id);
  Cols<4> dk_r[kRows], dv_r[kRows], dk0_r[kRows];
#pragma unroll
  for (int u = 0; u < kRows; ++u) dk_r[u].zero(), dv_r[u].zero(), dk0_r[u].zero();
  float suffix = 0.f;               // sum of dz over queries in later tiles

  Tile<T, D, kQ> tq, tq0;
  Tile<float, D, kQ> tdo;
  float next_lse = 0.f, next_dbar = 0.f, next_hist;
  auto fetch = [&](int rb) {
    const int m0 = rb * kQ;
    tq.fetch(id, qh, p.q.st, m0, p.seq, vec);
    if (!self) tq0.fetch(id, q0, p.q0.st, m0, p.seq, vec);
    tdo.fetch(id, doh, D, m0, p.seq, vec_do);
    if (id < kQ) {
      const int t = m0 + id;
      next_lse = (t < p.seq) ? lse2[(int64_t)n * p.seq + t] : 0.f;
      next_dbar = (t < p.seq) ? dbar[(int64_t)n * p.seq + t] : 0.f;
    }
    next_hist = (j < p.seq && j < m0 + kQ) ? carry[((int64_t)b * nblocks + rb) * p.seq + j] : 0.f;
  };
  // A query tile for each team in a step, last to first: team 0 takes the later one.
  if (nblocks - 1 - team >= kb) fetch(nblocks - 1 - team);
  __syncthreads();
  for (int rb = nblocks - 1 - team, step = 0; rb + team >= kb; rb -= TEAMS, ++step) {
    if (rb < kb) {                  // an odd number of tiles: team 1 has none in the last step
      __syncthreads();
      break;
    }
    const int m0 = rb * kQ;
    team_sync(team);
    tq.store(id, qs);
    if (!self) tq0.store(id, q0s);
    tdo.store(id, dos);
    if (id < kQ) {
      lse_s[id] = next_lse;
      dbar_s[id] = next_dbar;
    }
    const float hist = next_hist;
    team_sync(team);

    float aff[kRows], sel[kRows], dov[kRows];
    {
      const int d0 = grp * (D / 2), own = 16 * grp * P + d0, other = 16 * (1 - grp) * P + d0;
      auto product = [&](float (&mine)[kRows], const float* a, const float* k, float4* to) {
        float t[kRows][2];
        dot_rows<D, D / 2, 2>(t, a + d0, k + own, k + other, ty, tx);
#pragma unroll
        for (int u = 0; u < kRows; ++u) mine[u] = t[u][0];
        to[id] = make_float4(t[0][1], t[1][1], t[2][1], t[3][1]);
      };
      product(aff, qs, ks, ex);
      if (!self) product(sel, q0s, k0s, ex + kTeam);
      product(dov, dos, vs, ex + 2 * kTeam);
      team_sync(team);
      auto join = [&](float (&mine)[kRows], const float4* from) {
        const float4 x = from[id ^ 128];
        mine[0] += x.x; mine[1] += x.y; mine[2] += x.z; mine[3] += x.w;
      };
      join(aff, ex);
      if (!self) join(sel, ex + kTeam);
      join(dov, ex + 2 * kTeam);
    }
    unsigned gates = 0u;
    float sum = 0.f;
#pragma unroll
    for (int u = 0; u < kRows; ++u) {            // sel becomes the exclusive prefix inside the row group
      const int i = m0 + ty * kRows + u;
      const float l0 = (self ? aff[u] : sel[u]) * p.scale;
      const bool gate = (j < i) && (j >= p.exempt) && (i < p.seq) && (l0 > 0.f);
      gates |= (gate ? 1u : 0u) << u;
      sel[u] = sum;
      sum += gate ? l0 : 0.f;
    }
    gsel[ty * kKB + col] = sum;
    group_sync(2 * team + grp);
    float before = 0.f;
    for (int g = 0; g < ty; ++g) before += gsel[g * kKB + col];
    float dz[kRows], dz_sum = 0.f;
#pragma unroll
    for (int u = 0; u < kRows; ++u) {
      const int r = ty * kRows + u, i = m0 + r;
      const bool causal = (j <= i) && (i < p.seq);
      float attn = 0.f;
      dz[u] = 0.f;
      if (causal) {
        attn = exp2f((aff[u] * p.scale - (hist + (before + sel[u]))) * kLog2e - lse_s[r]);
        dz[u] = attn * (dov[u] - dbar_s[r]);
      }
      as[r * W + col] = attn;
      dz_sum += dz[u];
    }
    const int order = (TEAMS - 1 - team) * kGroups + ty;        // of the step's row groups, first query first
    float* dz_groups = gdz + (step & 1) * (TEAMS * kGroups * kKB);
    dz_groups[order * kKB + col] = dz_sum;
    if constexpr (TEAMS == 1) group_sync(grp); else __syncthreads();
    float later = suffix;
    const int first = TEAMS == 2 && rb == kb && team == 0 ? kGroups : 0;      // without a tile of team 1
#pragma unroll 8
    for (int g = TEAMS * kGroups - 1; g >= first; --g) {
      const float x = dz_groups[g * kKB + col];
      if (g > order) later += x;
      suffix += x;
    }
#pragma unroll
    for (int u = kRows - 1; u >= 0; --u) {
      const int r = ty * kRows + u;
      const float g = ((gates >> u) & 1u) ? -later : 0.f;
      later += dz[u];
      zs[r * W + col] = self ? dz[u] + g : dz[u];
      if (!self) gs[r * W + col] = g;
    }
    team_sync(team);
    if (rb - TEAMS >= kb) fetch(rb - TEAMS);            // covered by the products below

    // key rows: dV += A^T dO, dK += Z^T Q, dK0 += G^T Q0
    auto key_grads = [&](Cols<4> (&acc)[kRows], const float* w, const float* rows, int r) {
      const float4 a = ld4(w + r * W + ky * kRows);
      Cols<4> y;
      y.load(rows + r * P, kx);
      acc[0].add(pack2(a.x, a.x), y);
      acc[1].add(pack2(a.y, a.y), y);
      acc[2].add(pack2(a.z, a.z), y);
      acc[3].add(pack2(a.w, a.w), y);
    };
#pragma unroll 4
    for (int r = part * kPartRows; r < (part + 1) * kPartRows; ++r) {
      key_grads(dv_r, as, dos, r);
      key_grads(dk_r, zs, qs, r);
      if (!self) key_grads(dk0_r, gs, q0s, r);
    }
    // query rows: dQ += Z K, dQ0 += G K0, reduced across the key blocks in global memory
    float* dq_tile = dq_acc + ((int64_t)n * p.seq + m0) * D;
    float* dq0_tile = dq0 + ((int64_t)b * p.seq + m0) * D;
    if (self) {
      query_grads<D, (D >= 64 ? D / 32 : 1)>(zs, ks, dq_tile, p.seq - m0, p.scale, id);
    } else if constexpr (D == 128) {
      query_grads<D, 4>(zs, ks, dq_tile, p.seq - m0, p.scale, id);
      query_grads<D, 4>(gs, k0s, dq0_tile, p.seq - m0, p.scale, id);
    } else {                                    // one product a group
      query_grads<D, D / 16>(grp ? gs : zs, grp ? k0s : ks, grp ? dq0_tile : dq_tile, p.seq - m0, p.scale, id & 127);
    }
  }
  // the parts' sums of a key row, over the tiles' place in shared memory: [parts of all teams][32][D]
  auto finish = [&](const Cols<4> (&acc)[kRows], auto&& out) {
    __syncthreads();
#pragma unroll
    for (int u = 0; u < kRows; ++u)
      *reinterpret_cast<float4*>(smem + ((team * kParts + part) * kKB + ky * kRows + u) * D + 4 * kx) =
          make_float4(acc[u].get(0), acc[u].get(1), acc[u].get(2), acc[u].get(3));
    __syncthreads();
    for (int idx = threadIdx.x; idx < kKB * D / 4; idx += kTeam * TEAMS) {
      const int r = idx / (D / 4), c = idx % (D / 4) * 4;
      if (j0 + r >= p.seq) break;
      float4 x = ld4(smem + r * D + c);
#pragma unroll
      for (int k = 1; k < TEAMS * kParts; ++k) {
        const float4 y = ld4(smem + (k * kKB + r) * D + c);
        x.x += y.x; x.y += y.y; x.z += y.z; x.w += y.w;
      }
      out(j0 + r, c, x);
    }
  };
  auto scaled = [&](float4 x) { return make_float4(x.x * p.scale, x.y * p.scale, x.z * p.scale, x.w * p.scale); };
  finish(dk_r, [&](int t, int c, float4 x) {
    const float4 y = scaled(x);
    float* dst = dk_acc + ((int64_t)n * p.seq + t) * D + c;
    dst[0] = y.x; dst[1] = y.y; dst[2] = y.z; dst[3] = y.w;
  });
  finish(dv_r, [&](int t, int c, float4 x) {
    T* dst = dv + ((int64_t)n * p.seq + t) * D + c;
    dst[0] = from_float<T>(x.x); dst[1] = from_float<T>(x.y); dst[2] = from_float<T>(x.z); dst[3] = from_float<T>(x.w);
  });
  if (!self) finish(dk0_r, [&](int t, int c, float4 x) { reduce4(dk0 + ((int64_t)b * p.seq + t) * D + c, scaled(x)); });
}

template <int D> constexpr size_t colsum_smem() { return sizeof(float) * ((kKF + kQ) * (D + 4) + kGroups * kKF); }
template <int D, int TEAMS> constexpr size_t forward_smem() { return sizeof(float) * (2 * kQ * (D + 4) + TEAMS * kForwardTeamFloats<D>); }
template <int D, int TEAMS> constexpr size_t backward_smem() {
  return sizeof(float) * (3 * kKB * (D + 4) + TEAMS * (2 * kGroups * kKB + kBackwardTeamFloats<D>));
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
  colsum_kernel<T, D><<<dim3((p.seq + kKF - 1) / kKF, nb, p.batch), kSelThreads, colsum_smem<D>(), s>>>(p, carry, nb, vector_rows(p));
  SA_CUDA_CHECK(cudaGetLastError());
  count_launch();
  scan_kernel<<<dim3((p.seq + 127) / 128, p.batch), 128, 0, s>>>(carry, total, p.seq, nb);
  SA_CUDA_CHECK(cudaGetLastError());
  return SA_OK;
}

template <typename T, int D, int TEAMS>
int launch_forward(const Problem& p, const float* carry, float* out, float* lse2, cudaStream_t s) {
  const int nb = (p.seq + kQ - 1) / kQ;
  constexpr size_t smem = forward_smem<D, TEAMS>();
  SA_CUDA_CHECK(allow_smem(forward_kernel<T, D, TEAMS>, smem));
  count_launch();
  forward_kernel<T, D, TEAMS><<<(unsigned)nb * (unsigned)(p.batch * p.heads), kTeam * TEAMS, smem, s>>>(p, carry, out, lse2, nb, vector_rows(p));
  SA_CUDA_CHECK(cudaGetLastError());
  return SA_OK;
}

template <typename T, int D, int TEAMS>
int launch_backward(const Problem& p, const float* lse2, const float* carry, const float* dbar, const float* d_out,
                    float* dq_acc, float* dk_acc, float* dq0, float* dk0, void* dv, cudaStream_t s) {
  const int nb = (p.seq + kQ - 1) / kQ;
  constexpr size_t smem = backward_smem<D, TEAMS>();
  SA_CUDA_CHECK(allow_smem(backward_kernel<T, D, TEAMS>, smem));
  count_launch();
  backward_kernel<T, D, TEAMS><<<(unsigned)nb * (unsigned)(p.batch * p.heads), kTeam * TEAMS, smem, s>>>(
      p, lse2, carry, dbar, d_out, dq_acc, dk_acc, dq0, dk0, static_cast<T*>(dv), nb, vector_rows(p));
  SA_CUDA_CHECK(cudaGetLastError());
  return SA_OK;
}

// Two teams a CTA and one CTA an SM where one-team CTAs, two an SM, would all be resident at once: the hardware then pairs them
// as it likes, and the fullest SM had twice the mean.  (B, H, T, D) = (2, 4, 1024, 64) takes 76 + 160 us with two teams, 110 +
// 235 us with one.  With more CTAs than that the SMs that finish early take the rest, and teams without a common barrier are
// the faster ones: 292 + 540 against 328 + 588 us at (4, 8, 1000, 64), 192 + 345 against 209 + 363 us at (1, 12, 1280, 64).
inline bool two_teams(const Problem& p) {
  return (int64_t)p.batch * p.heads * ((p.seq + kQ - 1) / kQ) <= 2 * kSms;
}

template <typename T, int D>
int forward_impl(const Problem& p, float* out, float* lse2, float* carry, float* total, cudaStream_t s) {
  if (int st = carry_impl<T, D>(p, carry, total, s)) return st;
  if constexpr (D < 128)                     // a second team's tiles do not fit at D = 128
    if (two_teams(p)) return launch_forward<T, D, 2>(p, carry, out, lse2, s);
  return launch_forward<T, D, 1>(p, carry, out, lse2, s);
}

template <typename T, int D>
int backward_impl(const Problem& p, const float* lse2, const float* carry, const float* dbar, const float* d_out,
                  float* dq_acc, float* dk_acc, float* dq0, float* dk0, void* dv, cudaStream_t s) {
  if constexpr (D < 128)                     // two CTAs do not fit on an SM at D = 128
    if (!two_teams(p)) return launch_backward<T, D, 1>(p, lse2, carry, dbar, d_out, dq_acc, dk_acc, dq0, dk0, dv, s);
  return launch_backward<T, D, 2>(p, lse2, carry, dbar, d_out, dq_acc, dk_acc, dq0, dk0, dv, s);
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
