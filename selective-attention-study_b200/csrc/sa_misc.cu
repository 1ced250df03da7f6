// Bandwidth-bound helpers of the Selective Attention operator (sm_100a):
//   dbar      dbar[row] = sum_d dO[row, d] * out[row, d]   (reference: src/selective_attention/kernels.py:635-636)
//   row stats the tensor-core engine's form of it: -lse2 and -dbar in blocks, dO in bf16, zeroed accumulators
//   fold/cast dq = cast(dq_acc + [head 0] dq0)            (reference: kernels.py:662-666)
//   decode    one cached decode step                       (reference: src/selective_attention/mixers.py:115-130)
#include <type_traits>

#include "sa_common.cuh"
#include "sa_tc_host.cuh"
#include "sa_tc_ptx.cuh"

namespace sa {
namespace {

// ---- dbar (CUDA-core engine) ------------------------------------------------------------------------
// A group of D / 4 consecutive lanes owns one row; every lane handles 4 consecutive elements.
template <typename TDO, int D>
__global__ void __launch_bounds__(256) dbar_kernel(const float* __restrict__ out, const TDO* __restrict__ d_out,
                                                   int64_t rows, float* __restrict__ dbar, float* __restrict__ d_out_f32) {
  constexpr int kLanes = D / 4;
  const int64_t gid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t row = gid / kLanes;
  const int lane = (int)(gid % kLanes);
  float sum = 0.f;
  if (row < rows) {
    const int64_t off = row * D + lane * 4;
    float4 o = *reinterpret_cast<const float4*>(out + off);
    float g[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) g[e] = to_float<TDO>(d_out[off + e]);
    sum = g[0] * o.x + g[1] * o.y + g[2] * o.z + g[3] * o.w;
    if (d_out_f32 != nullptr) *reinterpret_cast<float4*>(d_out_f32 + off) = make_float4(g[0], g[1], g[2], g[3]);
  }
#pragma unroll
  for (int s = kLanes / 2; s > 0; s >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, s);
  if (row < rows && lane == 0) dbar[row] = sum;
}

template <typename TDO>
int dbar_by_dim(const float* out, const void* d_out, int64_t rows, int head_dim, float* dbar, float* d_out_f32, cudaStream_t s) {
  const unsigned blocks = (unsigned)((rows * (head_dim / 4) + 255) / 256);
  const TDO* g = static_cast<const TDO*>(d_out);
  ProfileScope prof(SA_KERNEL_DBAR, s);
  switch (head_dim) {
    case 16: count_launch(), dbar_kernel<TDO, 16><<<blocks, 256, 0, s>>>(out, g, rows, dbar, d_out_f32); break;
    case 32: count_launch(), dbar_kernel<TDO, 32><<<blocks, 256, 0, s>>>(out, g, rows, dbar, d_out_f32); break;
    case 64: count_launch(), dbar_kernel<TDO, 64><<<blocks, 256, 0, s>>>(out, g, rows, dbar, d_out_f32); break;
    case 128: count_launch(), dbar_kernel<TDO, 128><<<blocks, 256, 0, s>>>(out, g, rows, dbar, d_out_f32); break;
    default: return SA_ERR_UNSUPPORTED;
  }
  SA_CUDA_CHECK(cudaGetLastError());
  return SA_OK;
}

// ---- row statistics (tensor-core engine) -------------------------------------------------------------
// One pass over out and dO: dbar = sum_d dO * out, the bf16 copy of dO where the caller's is not one the TMA can read,
// and the zeros that the backward kernel's reductions start from (dq_acc, and dk0 / dq0 for the selecting head).  What the
// backward kernel wants per query, -lse2 and -dbar, goes out as blocks of 64 queries, [row n][block][-lse2 x 64, -dbar x 64]
// with blocks up to the end of the last 128-query tile (-inf and 0 there: such a query has P = 0), so that a 64-query half
// takes its statistics in one 512-byte bulk copy whatever the sequence length.
// Bound by memory: reads 4 + sizeof(dO) and writes 4 (+ 2) bytes an element; a separate memset of the same zeros cost a
// launch and nothing less.
template <typename TDO, int D>
__global__ void __launch_bounds__(256) row_stats_kernel(const float* __restrict__ out, const TDO* __restrict__ d_out,
                                                        RowLayout in_rows, bool vec, const float* __restrict__ lse2,
                                                        float* __restrict__ stats, __nv_bfloat16* __restrict__ d_out_low,
                                                        float* __restrict__ dq_acc, float* __restrict__ zero_a,
                                                        float* __restrict__ zero_b, int heads, int seq, int padded,
                                                        int64_t rows) {
  constexpr int kLanes = D / 4;
  const int64_t gid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t row = gid / kLanes;               // (n, padded query index)
  const int lane = (int)(gid % kLanes);
  if (row >= rows) return;                         // whole groups of lanes leave together: rows * kLanes threads work
  const int n = (int)(row / padded), t = (int)(row - (int64_t)n * padded);
  const int b = n / heads, h = n - b * heads;
  float sum = 0.f;
  if (t < seq) {
    const int64_t off = ((int64_t)n * seq + t) * D + lane * 4;
    const TDO* src = d_out + in_rows.at(b, h, t) + lane * 4;
    const float4 o = *reinterpret_cast<const float4*>(out + off);
    TDO raw[4];
    if (vec) {
      if constexpr (sizeof(TDO) == 4) *reinterpret_cast<float4*>(raw) = *reinterpret_cast<const float4*>(src);
      else *reinterpret_cast<uint2*>(raw) = *reinterpret_cast<const uint2*>(src);
    } else {
#pragma unroll
      for (int e = 0; e < 4; ++e) raw[e] = src[e];
    }
    float g[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) g[e] = to_float<TDO>(raw[e]);
    sum = g[0] * o.x + g[1] * o.y + g[2] * o.z + g[3] * o.w;
    if (d_out_low != nullptr)
      *reinterpret_cast<uint2*>(d_out_low + off) = make_uint2(tc::pack_bf16(g[0], g[1]), tc::pack_bf16(g[2], g[3]));
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    *reinterpret_cast<float4*>(dq_acc + off) = zero;
    if (h == 0) {
      const int64_t off0 = ((int64_t)b * seq + t) * D + lane * 4;
      if (zero_a != nullptr) *reinterpret_cast<float4*>(zero_a + off0) = zero;
      if (zero_b != nullptr) *reinterpret_cast<float4*>(zero_b + off0) = zero;
    }
  }
#pragma unroll
  for (int s = kLanes / 2; s > 0; s >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, s);
  if (lane == 0) {
    float* block = stats + ((int64_t)n * (padded >> 6) + (t >> 6)) * 128 + (t & 63);
    block[0] = (t < seq) ? -lse2[(int64_t)n * seq + t] : -INFINITY;
    block[64] = (t < seq) ? -sum : 0.f;
  }
}

// ---- fold + cast ------------------------------------------------------------------------------------
// Eight elements a thread: two or four 16-byte loads in flight and one 16-byte store (bf16, fp16) where dst allows it.
template <typename T>
__global__ void __launch_bounds__(256) fold_cast_kernel(const float* __restrict__ acc, const float* __restrict__ acc0,
                                                        T* __restrict__ dst, int heads, int64_t per_head,
                                                        int64_t total8, bool vec, RowLayout dst_rows, int head_dim) {
  const int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= total8) return;
  const int64_t e = idx * 8;
  const int64_t row = e / per_head;           // (batch, head) row
  const int64_t within = e - row * per_head;
  const int b = (int)(row / heads), h = (int)(row - (int64_t)b * heads);
  float x[8];
  *reinterpret_cast<float4*>(x) = *reinterpret_cast<const float4*>(acc + e);
  *reinterpret_cast<float4*>(x + 4) = *reinterpret_cast<const float4*>(acc + e + 4);
  if (h == 0 && acc0 != nullptr) {
    const float* z = acc0 + (int64_t)b * per_head + within;
    float y[8];
    *reinterpret_cast<float4*>(y) = *reinterpret_cast<const float4*>(z);
    *reinterpret_cast<float4*>(y + 4) = *reinterpret_cast<const float4*>(z + 4);
#pragma unroll
    for (int u = 0; u < 8; ++u) x[u] += y[u];
  }
  const int64_t t = within / head_dim;
  T* out = dst + dst_rows.at(b, h, t) + (within - t * head_dim);
  T w[8];
#pragma unroll
  for (int u = 0; u < 8; ++u) w[u] = from_float<T>(x[u]);
  if (vec) {
#pragma unroll
    for (int u = 0; u < (int)sizeof(T) / 2; ++u) reinterpret_cast<uint4*>(out)[u] = reinterpret_cast<const uint4*>(w)[u];
  } else {
#pragma unroll
    for (int u = 0; u < 8; ++u) out[u] = w[u];
  }
}

// ---- decode -----------------------------------------------------------------------------------------
constexpr int kDecThreads = 128;
constexpr int kDecSplitMin = 128;             // keys per CTA: a multiple of 128, at least 128
constexpr int kDecLiveSplit = 1024;           // with key norms
constexpr int kDecSplitsMax = 256;            // of a long cache: more would make the merge long
constexpr int kDecCtasPerSm = 4;              // attend CTAs resident per SM (48 KB of stages each)

// Keys per CTA for `t` cached keys and `rows` = batch * heads query rows: the grid is about one full wave of
// resident CTAs, so no SM is left with a straggler and the combine pass stays short.  With 512 keys at least, 96 rows of
// 1,500 keys were 288 CTAs of three ring refills each and took 13.9 us; with 256 they fill the wave.
static int decode_target_splits(int rows) { return max(1, min(kSms * kDecCtasPerSm / rows, kDecSplitsMax)); }
static int decode_split_keys(int t, int rows) {
  const int target_splits = decode_target_splits(rows);
  const int keys = (t + target_splits - 1) / target_splits;
  return (keys + kDecSplitMin - 1) / kDecSplitMin * kDecSplitMin;
}
// The most key ranges that a step over up to `t` keys can have, with key norms or without.
static int decode_splits_max(int t, int rows) {
  return max(min(decode_target_splits(rows), (t + kDecSplitMin - 1) / kDecSplitMin), (t + kDecLiveSplit - 1) / kDecLiveSplit);
}

// 16-byte load of 8 (bf16 / fp16) or two 16-byte loads of 8 fp32 elements, converted to fp32.
template <typename T>
__device__ __forceinline__ void load8(const T* p, float (&x)[8]) {
  if constexpr (sizeof(T) == 2) {
    const uint4 raw = *reinterpret_cast<const uint4*>(p);
    const T* h = reinterpret_cast<const T*>(&raw);
#pragma unroll
    for (int e = 0; e < 8; ++e) x[e] = to_float<T>(h[e]);
  } else {
    const float4 a = *reinterpret_cast<const float4*>(p);
    const float4 c = *reinterpret_cast<const float4*>(p + 4);
    x[0] = a.x; x[1] = a.y; x[2] = a.z; x[3] = a.w; x[4] = c.x; x[5] = c.y; x[6] = c.z; x[7] = c.w;
  }
}

// 16-byte load of 8 (bf16 / fp16) or two 16-byte loads of 8 fp32 elements from shared memory, converted to fp32.
template <typename T>
__device__ __forceinline__ void load8_shared(const uint8_t* p, float (&x)[8]) {
  load8<T>(reinterpret_cast<const T*>(p), x);
}

constexpr int kDecStages = 3;                   // stages of 8 KB of K + 8 KB of V
constexpr int kDecStageBytes = 8192;            // per tensor
constexpr size_t kDecSmemBytes = (size_t)kDecStages * 2 * kDecStageBytes + 128;
constexpr int kDecMaxLive = 512;                // stages (of 8 KB) of a CTA's key range when dead stages are left out
constexpr float kDecDeadMargin = 150.f;         // binades below the newest key's logit at which a key counts as dead

// Merges the per-split partial softmaxes of one query row; called by all 128 threads of a CTA.  The global
// maximum is found first so that the weighted sums over splits have no serial dependence: warp w folds splits
// w, w + 4, ... (lane l owns output columns l, l + 32, ...), then the four warps are added through shared memory.
// The partials were written by other CTAs: they are read past the L1 cache.
template <typename TY>
__device__ __forceinline__ void decode_combine_row(const float* prow, TY* yrow, int splits, int D,
                                                   float (*part)[128 + 1], float* red) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  float m = -INFINITY;
  for (int s = threadIdx.x; s < splits; s += 128) m = fmaxf(m, __ldcg(prow + (int64_t)s * (D + 2) + D));
  red[threadIdx.x] = m;
  __syncthreads();
  for (int st = 64; st > 0; st >>= 1) {
    if (threadIdx.x < st) red[threadIdx.x] = fmaxf(red[threadIdx.x], red[threadIdx.x + st]);
    __syncthreads();
  }
  m = red[0];
  float den = 0.f, num[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 4
  for (int s = warp; s < splits; s += 4) {
    const float* p = prow + (int64_t)s * (D + 2);
    const float c = exp2f(__ldcg(p + D) - m);
    den = fmaf(__ldcg(p + D + 1), c, den);
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int d = lane + 32 * u;
      if (d < D) num[u] = fmaf(__ldcg(p + d), c, num[u]);
    }
  }
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    const int d = lane + 32 * u;
    if (d < D) part[warp][d] = num[u];
  }
  if (lane == 0) part[warp][128] = den;
  __syncthreads();
  const int d = threadIdx.x;
  if (d < D) {
    const float nn = part[0][d] + part[1][d] + part[2][d] + part[3][d];
    const float dd = part[0][128] + part[1][128] + part[2][128] + part[3][128];
    yrow[d] = from_float<TY>(nn / dd);
  }
}

// grid = batch * heads * splits CTAs (a row's splits are neighbours).  One thread streams the CTA's keys of K and V through a ring of shared-memory
// stages with bulk copies, kDecStages - 1 stages (32 KB) ahead of the arithmetic, so the bytes in flight do not
// depend on how the arithmetic is scheduled.  A group of D / 8 lanes owns every (128 / lanes)-th key of a stage
// and keeps its own running maximum, denominator and weighted sum (one pass, rescaled when its maximum grows);
// the groups are merged at the end.
//
// LIVE (optional, needs the per-key norms `knorm`): the history term of a key only grows, so most of a long cache
// can be dead for the new query -- its weight exp2(z - m) is below 2^-150 and adds nothing to fp32 sums of order one.
// A key is dead when  c1 |q| |k_j| - log2e selected[j]  <  z_new - 150, z_new being the logit of the newest key (its
// history term is zero, and the row maximum is at least that).  A CTA first marks the 64-key stages of its range that
// hold a live key (it reads 8 bytes per key for that instead of the 2 x 128 or 256 of K and V) and then streams
// only those.  The CTAs of a selecting head stay dense: the new query's selection is needed for every key.
template <typename T, typename TY, int D, bool LIVE>
__global__ void __launch_bounds__(kDecThreads) decode_attend_kernel(
    const T* __restrict__ q1, const T* __restrict__ k1, const T* __restrict__ v1, T* kc, T* vc, float* selected,
    float* __restrict__ partial, float* __restrict__ sel_new, int heads, int groups, int t, int capacity,
    int exempt, float scale, int split_keys, tc::WaitCtx status, TY* __restrict__ y, unsigned int* __restrict__ row_tickets, unsigned int* __restrict__ split_tickets, int splits,
    float* knorm) {
  constexpr int kLanes = D / 8;                                   // lanes per key
  constexpr int kGroups = kDecThreads / kLanes;                   // keys the CTA covers per step
  constexpr int kRowBytes = D * (int)sizeof(T);
  constexpr int kStageKeys = kDecStageBytes / kRowBytes;
  constexpr int kPer = kStageKeys / kGroups;                      // keys per group per stage (4, fp32: 2)
  static_assert(kPer >= 1 && kPer * kGroups == kStageKeys, "stage layout");
  // Launched while the step before is still running (programmatic stream serialization); its results from here on.
  asm volatile("griddepcontrol.launch_dependents;");
  asm volatile("griddepcontrol.wait;" ::: "memory");
  extern __shared__ uint8_t dec_smem_raw[];
  uint8_t* ring = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(dec_smem_raw) + 127) & ~uintptr_t(127));
  __shared__ uint64_t full[kDecStages];
  __shared__ float red[kDecThreads];
  __shared__ float gmax[kGroups];
  __shared__ float accs[kGroups][D];
  __shared__ float part[4][128 + 1];
  __shared__ unsigned int ticket_s[2];
  __shared__ uint16_t live_s[LIVE ? kDecMaxLive : 1];             // LIVE: the stages of this CTA's range that hold a live key
  __shared__ unsigned int live_bits[LIVE ? kDecMaxLive / 32 : 1];
  __shared__ int live_n_s;

  const int n = (int)(blockIdx.x / (unsigned)splits), split = (int)(blockIdx.x % (unsigned)splits);
  const int b = n / heads, h = n - b * heads;
  const int per = heads / groups, g = h / per;
  const bool selector = (h - g * per) == 0;
  const int c0 = split * split_keys, c1 = min(t, c0 + split_keys);
  const int n_stages = (c1 - c0 + kStageKeys - 1) / kStageKeys;
  const int grp = threadIdx.x / kLanes, lane = threadIdx.x % kLanes;
  const uint8_t* kb = reinterpret_cast<const uint8_t*>(kc + (int64_t)n * capacity * D);
  const uint8_t* vb = reinterpret_cast<const uint8_t*>(vc + (int64_t)n * capacity * D);

  // The range that ends with the newest key: that key and value come from k1, v1, and this CTA writes them to the cache (in a
  // launch of their own the append took 1.6 us of a 13 us step, and the launch as much on the host).
  const bool tail = c1 == t;
  const int c_mem = tail ? t - 1 : c1;                            // keys below come from the cache
  const bool sparse = LIVE && !selector;                          // this CTA leaves out dead stages
  auto stage_of = [&](int it) { return sparse ? (int)live_s[it] : it; };
  auto issue = [&](int it) {                                      // thread 0 only; `it` counts the stages this CTA streams
    const int st = it;
    const int j0 = c0 + stage_of(it) * kStageKeys;
    const uint32_t bytes = (uint32_t)(min(kStageKeys, c_mem - j0) * kRowBytes);      // 0: the newest key alone
    uint8_t* dst = ring + (size_t)(st % kDecStages) * 2 * kDecStageBytes;
    uint64_t* bar = &full[st % kDecStages];
    tc::mbar_expect_tx(bar, 2 * bytes);
    if (bytes == 0) return;
    tc::bulk_load(dst, kb + (int64_t)j0 * kRowBytes, bytes, bar);
    tc::bulk_load(dst + kDecStageBytes, vb + (int64_t)j0 * kRowBytes, bytes, bar);
  };
  float qv[8];
  load8<T>(q1 + (int64_t)n * D + lane * 8, qv);
  const float* selb = selected + ((int64_t)b * groups + g) * capacity;
  float* selnb = sel_new + ((int64_t)b * groups + g) * t;
  int n_iter = n_stages;
  if (knorm != nullptr && tail) {                                 // the newest key's norm
    float kx[8], ss = 0.f;
    load8<T>(k1 + (int64_t)n * D + lane * 8, kx);
#pragma unroll
    for (int e = 0; e < 8; ++e) ss = fmaf(kx[e], kx[e], ss);
#pragma unroll
    for (int sft = kLanes / 2; sft > 0; sft >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, sft);
    if (threadIdx.x == 0) knorm[(int64_t)n * capacity + t - 1] = sqrtf(ss);
  }
  if (sparse) {
    // |q| and the newest key's logit, by every group of lanes (each holds the whole of q between its lanes)
    float kx[8], ss = 0.f, dot = 0.f;
    load8<T>(k1 + (int64_t)n * D + lane * 8, kx);
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      ss = fmaf(qv[e], qv[e], ss);
      dot = fmaf(qv[e], kx[e], dot);
    }
#pragma unroll
    for (int sft = kLanes / 2; sft > 0; sft >>= 1) {
      ss += __shfl_xor_sync(0xffffffffu, ss, sft);
      dot += __shfl_xor_sync(0xffffffffu, dot, sft);
    }
    const float thr = (dot * scale - selb[t - 1]) * kLog2e - kDecDeadMargin;
    const float cq = scale * kLog2e * sqrtf(ss);
    const float* kn = knorm + (int64_t)n * capacity;
    for (int w = threadIdx.x; w < (n_stages + 31) / 32; w += kDecThreads) live_bits[w] = 0u;
    __syncthreads();
    constexpr int kAhead = 4;                                      // independent loads in flight per thread
    for (int base = c0 + threadIdx.x; base < c1; base += kDecThreads * kAhead) {
      float nrm[kAhead], sel[kAhead];
#pragma unroll
      for (int u = 0; u < kAhead; ++u) {
        const int j = base + u * kDecThreads;
        nrm[u] = (j < c_mem) ? __ldcg(kn + j) : 0.f;
        sel[u] = (j < c1) ? __ldcg(selb + j) : 0.f;
      }
#pragma unroll
      for (int u = 0; u < kAhead; ++u) {
        const int j = base + u * kDecThreads;
        if (j < c1 && (j == t - 1 || cq * nrm[u] - kLog2e * sel[u] >= thr)) {
          const int st = (j - c0) / kStageKeys;
          atomicOr(&live_bits[st >> 5], 1u << (st & 31));
        }
      }
    }
    __syncthreads();
    if (threadIdx.x < 32) {                                        // compact the marked stages, in order
      int count = 0;
      for (int w0 = 0; w0 < (n_stages + 31) / 32; w0 += 32) {
        const int w = w0 + threadIdx.x;
        const unsigned int bits = (w < (n_stages + 31) / 32) ? live_bits[w] : 0u;
        int mine = __popc(bits), before = mine;
#pragma unroll
        for (int sft = 1; sft < 32; sft <<= 1) {
          const int v = __shfl_up_sync(0xffffffffu, before, sft);
          if ((int)threadIdx.x >= sft) before += v;
        }
        const int total = __shfl_sync(0xffffffffu, before, 31);
        int pos = count + before - mine;
        for (unsigned int rest = bits; rest != 0u; rest &= rest - 1u) live_s[pos++] = (uint16_t)(w * 32 + __ffs(rest) - 1);
        count += total;
      }
      if (threadIdx.x == 0) live_n_s = count;
    }
    __syncthreads();
    n_iter = live_n_s;
  }
  if (threadIdx.x == 0) {
    for (int st = 0; st < kDecStages; ++st) tc::mbar_init(&full[st], 1);
    tc::mbar_init_fence();
    for (int st = 0; st < min(kDecStages - 1, n_iter); ++st) issue(st);
  }
  __syncthreads();                                                // barriers initialised before anyone waits

  float m = -INFINITY, den = 0.f, acc[8];
#pragma unroll
  for (int e = 0; e < 8; ++e) acc[e] = 0.f;
  for (int st = 0; st < n_iter; ++st) {
    const int j0 = c0 + stage_of(st) * kStageKeys;
    float sv[kPer];
#pragma unroll
    for (int u = 0; u < kPer; ++u) {                              // the history sums arrive while the stage is awaited
      const int j = j0 + u * kGroups + grp;
      sv[u] = (j < c1) ? selb[j] : 0.f;
    }
    // the slot that stage st + kDecStages - 1 uses was read in iteration st - 1; every thread is past it
    if (threadIdx.x == 0 && st + kDecStages - 1 < n_iter) issue(st + kDecStages - 1);
    tc::mbar_wait(&full[st % kDecStages], (st / kDecStages) & 1, status, 600);
    if (tail && st == n_iter - 1) {                               // the newest key and value: into their rows of the stage and the cache
      constexpr int kChunks = kRowBytes / 16;
      if (threadIdx.x < 2 * kChunks) {
        const bool val = threadIdx.x >= kChunks;
        const int c = (int)threadIdx.x - (val ? kChunks : 0);
        const uint4 x = reinterpret_cast<const uint4*>((val ? v1 : k1) + (int64_t)n * D)[c];
        reinterpret_cast<uint4*>(ring + ((size_t)(st % kDecStages) * 2 + (val ? 1 : 0)) * kDecStageBytes + (t - 1 - j0) * kRowBytes)[c] = x;
        reinterpret_cast<uint4*>((val ? vc : kc) + ((int64_t)n * capacity + t - 1) * D)[c] = x;
      }
      __syncthreads();
    }
    const uint8_t* ks = ring + (size_t)(st % kDecStages) * 2 * kDecStageBytes;
    const uint8_t* vs = ks + kDecStageBytes;

    float z[kPer];
#pragma unroll
    for (int u = 0; u < kPer; ++u) {
      float kx[8];
      load8_shared<T>(ks + (u * kGroups + grp) * kRowBytes + lane * 8 * (int)sizeof(T), kx);
      float dot = 0.f;
#pragma unroll
      for (int e = 0; e < 8; ++e) dot = fmaf(qv[e], kx[e], dot);
      z[u] = dot;
    }
#pragma unroll
    for (int u = 0; u < kPer; ++u) {
#pragma unroll
      for (int sft = kLanes / 2; sft > 0; sft >>= 1) z[u] += __shfl_xor_sync(0xffffffffu, z[u], sft);
    }
    float mx = m;
#pragma unroll
    for (int u = 0; u < kPer; ++u) {
      const int j = j0 + u * kGroups + grp;
      const float raw = z[u] * scale;
      if (j < c1) {
        if (selector && lane == 0) selnb[j] = (j >= exempt && j != t - 1 && raw > 0.f) ? raw : 0.f;
        z[u] = (raw - sv[u]) * kLog2e;
      } else {
        z[u] = -INFINITY;                                         // past the end: the stage holds no data there
      }
      mx = fmaxf(mx, z[u]);
    }
    if (mx > m) {                                                 // the group's maximum grew: rescale its sums
      const float c = exp2f(m - mx);                              // m = -inf on the first keys: c = 0
      den *= c;
#pragma unroll
      for (int e = 0; e < 8; ++e) acc[e] *= c;
      m = mx;
    }
#pragma unroll
    for (int u = 0; u < kPer; ++u) {
      if (z[u] != -INFINITY) {
        const float w = exp2f(z[u] - m);
        float vx[8];
        load8_shared<T>(vs + (u * kGroups + grp) * kRowBytes + lane * 8 * (int)sizeof(T), vx);
        den += w;
#pragma unroll
        for (int e = 0; e < 8; ++e) acc[e] = fmaf(w, vx[e], acc[e]);
      }
    }
    __syncthreads();                                              // stage read by everyone: its slot may be refilled
  }

  // merge the groups: common maximum, then rescaled sums
  if (lane == 0) gmax[grp] = m;
  __syncthreads();
  float cta_max = -INFINITY;
#pragma unroll 4
  for (int gg = 0; gg < kGroups; ++gg) cta_max = fmaxf(cta_max, gmax[gg]);
  const float c = (m == -INFINITY) ? 0.f : exp2f(m - cta_max);   // a group that saw no key contributes nothing
#pragma unroll
  for (int e = 0; e < 8; ++e) accs[grp][lane * 8 + e] = acc[e] * c;
  red[threadIdx.x] = (lane == 0) ? den * c : 0.f;
  __syncthreads();
  for (int sft = kDecThreads / 2; sft > 0; sft >>= 1) {
    if (threadIdx.x < sft) red[threadIdx.x] += red[threadIdx.x + sft];
    __syncthreads();
  }
  float* prow = partial + ((int64_t)n * splits + split) * (D + 2);
  for (int d = threadIdx.x; d < D; d += kDecThreads) {
    float sum = 0.f;
    for (int gg = 0; gg < kGroups; ++gg) sum += accs[gg][d];
    prow[d] = sum;
  }
  if (threadIdx.x == 0) {
    prow[D] = cta_max;
    prow[D + 1] = red[0];
  }

  // The last CTA of a query row merges the row's partials into y; the last of the `per` heads that share a
  // history vector to finish a key range adds the new selection of that range to it (every reader is done).
  __threadfence();                                                // partials and sel_new visible before the ticket
  __syncthreads();
  if (threadIdx.x == 0) {
    ticket_s[0] = atomicAdd(&row_tickets[n], 1u);
    ticket_s[1] = atomicAdd(&split_tickets[((int64_t)b * groups + g) * splits + split], 1u);
  }
  __syncthreads();
  const bool last_of_row = ticket_s[0] == (unsigned)splits - 1;
  const bool last_of_range = ticket_s[1] == (unsigned)per - 1;
  if (!last_of_row && !last_of_range) return;
  __threadfence();
  if (threadIdx.x == 0) {                                          // zero again for the next step
    if (last_of_row) row_tickets[n] = 0u;
    if (last_of_range) split_tickets[((int64_t)b * groups + g) * splits + split] = 0u;
  }
  if (last_of_range) {
    float* sel_rw = selected + ((int64_t)b * groups + g) * capacity;
    constexpr int kBatch = 8;                                     // independent loads in flight per thread
    for (int base = c0 + threadIdx.x; base < c1; base += kDecThreads * kBatch) {
      float old_v[kBatch], new_v[kBatch];
#pragma unroll
      for (int u = 0; u < kBatch; ++u) {
        const int j = base + u * kDecThreads;
        old_v[u] = (j < c1) ? __ldcg(sel_rw + j) : 0.f;
        new_v[u] = (j < c1) ? __ldcg(selnb + j) : 0.f;
      }
#pragma unroll
      for (int u = 0; u < kBatch; ++u) {
        const int j = base + u * kDecThreads;
        if (j < c1) sel_rw[j] = old_v[u] + new_v[u];
      }
    }
  }
  if (last_of_row)
    decode_combine_row(partial + (int64_t)n * splits * (D + 2), y + (int64_t)n * D, splits, D, part, red);
}

template <typename T, typename TY, int D, bool LIVE>
int launch_attend(unsigned grid, cudaStream_t s, const T* q, const T* k1, const T* v1, T* kc, T* vc, float* selected, float* partial,
                  float* sel_new, int heads, int groups, int t, int capacity, int exempt, int split_keys,
                  const tc::WaitCtx& status, TY* y, unsigned int* row_tickets, unsigned int* split_tickets, int splits,
                  float* knorm) {
  auto kernel = decode_attend_kernel<T, TY, D, LIVE>;
  SA_CUDA_CHECK(allow_smem(kernel, kDecSmemBytes));
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t config{};
  config.gridDim = dim3(grid);
  config.blockDim = dim3(kDecThreads);
  config.dynamicSmemBytes = kDecSmemBytes;
  config.stream = s;
  config.attrs = &attr;
  config.numAttrs = 1;
  count_launch();
  SA_CUDA_CHECK(cudaLaunchKernelEx(&config, kernel, q, k1, v1, kc, vc, selected, partial, sel_new, heads, groups, t, capacity, exempt,
                                   1.0f / sqrtf((float)D), split_keys, status, y, row_tickets, split_tickets, splits, knorm));
  return SA_OK;
}

template <typename T, typename TY>
int decode_impl(const DecodeStep& d, cudaStream_t s) {
  const int rows = d.batch * d.heads, t = d.length + 1, D = d.head_dim;
  // With key norms most CTAs find nothing to stream and only the selecting heads stay dense: short key ranges (1024
  // keys; 512 and 2048 measured slower) then spread those heads over the whole GPU.
  const int split_keys = (d.key_norms != nullptr) ? kDecLiveSplit : decode_split_keys(t, rows);
  const int splits = (t + split_keys - 1) / split_keys;
  // Tickets first: where they are kept (`tickets_zero`), at a size that does not change from step to step, so that what the last CTAs leave at zero
  // is where the next step looks.
  const int ticket_splits = d.tickets_zero ? decode_splits_max(d.capacity, rows) : splits;
  unsigned int* row_tickets = reinterpret_cast<unsigned int*>(d.workspace);
  unsigned int* split_tickets = row_tickets + rows;
  const size_t n_tickets = (size_t)rows + (size_t)d.batch * d.groups * ticket_splits;
  float* partial = d.workspace + n_tickets;
  float* sel_new = partial + (size_t)rows * splits * (D + 2);
  tc::WaitCtx status;
  if (int st = tc::wait_ctx(&status)) return st;
  ProfileScope prof(SA_KERNEL_DECODE, s);
  if (d.tickets_zero != 1) SA_CUDA_CHECK(cudaMemsetAsync(row_tickets, 0, n_tickets * 4, s));
  // dead stages are left out when the norms are given and a CTA's range fits the stage list
  const bool live = d.key_norms != nullptr && split_keys / (kDecStageBytes / (D * (int)sizeof(T))) <= kDecMaxLive;
  auto attend = [&](auto dim, auto live_tag) {
    return launch_attend<T, TY, decltype(dim)::value, decltype(live_tag)::value>(
        (unsigned)rows * (unsigned)splits, s, static_cast<const T*>(d.q1), static_cast<const T*>(d.k1),
        static_cast<const T*>(d.v1), static_cast<T*>(d.k_cache), static_cast<T*>(d.v_cache), d.selected, partial, sel_new, d.heads, d.groups, t, d.capacity, d.exempt, split_keys,
        status, static_cast<TY*>(d.y), row_tickets, split_tickets, splits, d.key_norms);
  };
  auto by_live = [&](auto dim) { return live ? attend(dim, std::true_type{}) : attend(dim, std::false_type{}); };
  switch (D) {
    case 16: return by_live(std::integral_constant<int, 16>{});
    case 32: return by_live(std::integral_constant<int, 32>{});
    case 64: return by_live(std::integral_constant<int, 64>{});
    case 128: return by_live(std::integral_constant<int, 128>{});
  }
  return SA_ERR_UNSUPPORTED;
}

// ---- new rows of a decode cache ---------------------------------------------------------------------
// blockIdx.y is the (batch, head) row, blockIdx.z 0: keys, 1: values, 2: the history sums behind the prompt.  Units are 16
// bytes of a cache row.  Bound by memory: one read and one write of the new rows, one write of the zeros; the same in torch
// is two fills and two strided copies (1.0 ms for 131,072 tokens of 16 heads).
__global__ void __launch_bounds__(256) cache_store_kernel(const uint8_t* k, RowLayout k_rows, const uint8_t* v, RowLayout v_rows,
                                                          uint8_t* kc, uint8_t* vc, float* selected, int heads, int groups, int seq,
                                                          int capacity, int row_bytes, int elem_bytes, int at, bool begin, bool vec) {
  const int n = blockIdx.y, b = n / heads, h = n - b * heads;
  const int64_t first = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, step = (int64_t)gridDim.x * blockDim.x;
  if (blockIdx.z == 2) {
    if (h >= groups) return;
    float* sel = selected + ((int64_t)b * groups + h) * capacity;
    for (int64_t j = at + seq + first; j < capacity; j += step) sel[j] = 0.f;
    return;
  }
  const RowLayout& rows = blockIdx.z == 0 ? k_rows : v_rows;
  const uint8_t* src = (blockIdx.z == 0 ? k : v) + (rows.at(b, h, 0)) * elem_bytes;
  uint8_t* dst = (blockIdx.z == 0 ? kc : vc) + (int64_t)n * capacity * row_bytes;
  const int units = row_bytes / 16;
  const int64_t last = (int64_t)(begin ? capacity : at + seq) * units;
  for (int64_t u = (int64_t)at * units + first; u < last; u += step) {
    const int t = (int)(u / units), c = (int)(u - (int64_t)t * units);
    uint4 x = make_uint4(0u, 0u, 0u, 0u);
    if (t < at + seq) {
      const uint8_t* from = src + (int64_t)(t - at) * rows.st * elem_bytes + c * 16;
      if (vec) {
        x = *reinterpret_cast<const uint4*>(from);
      } else {                                       // rows at a multiple of the element size only
        uint32_t w[4];
#pragma unroll
        for (int e = 0; e < 4; ++e)
          w[e] = elem_bytes == 4 ? *reinterpret_cast<const uint32_t*>(from + 4 * e)
                                 : ((uint32_t)*reinterpret_cast<const uint16_t*>(from + 4 * e) |
                                    ((uint32_t)*reinterpret_cast<const uint16_t*>(from + 4 * e + 2) << 16));
        x = make_uint4(w[0], w[1], w[2], w[3]);
      }
    }
    *reinterpret_cast<uint4*>(dst + u * 16) = x;
  }
}

}  // namespace

int launch_dbar(const float* out, const void* d_out, int d_out_dtype, int64_t rows, int head_dim, float* dbar, float* d_out_f32,
                cudaStream_t s) {
  switch (d_out_dtype) {
    case SA_F32: return dbar_by_dim<float>(out, d_out, rows, head_dim, dbar, d_out_f32, s);
    case SA_BF16: return dbar_by_dim<__nv_bfloat16>(out, d_out, rows, head_dim, dbar, d_out_f32, s);
    case SA_F16: return dbar_by_dim<__half>(out, d_out, rows, head_dim, dbar, d_out_f32, s);
  }
  return SA_ERR_BAD_ARGUMENT;
}

namespace {
bool aligned_rows(const void* ptr, const RowLayout& r, int64_t elem_bytes, int64_t align) {
  return (reinterpret_cast<uintptr_t>(ptr) & (align - 1)) == 0 && (r.sb * elem_bytes) % align == 0 &&
         (r.sh * elem_bytes) % align == 0 && (r.st * elem_bytes) % align == 0;
}
template <typename TDO>
int row_stats_by_dim(const float* out, const void* d_out, const RowLayout& in_rows, bool vec, const float* lse2, float* stats,
                     void* d_out_bf16, float* dq_acc, float* zero_a, float* zero_b, int batch, int heads, int seq, int head_dim,
                     cudaStream_t s) {
  const int padded = (seq + 127) / 128 * 128;
  const int64_t rows = (int64_t)batch * heads * padded;          // a multiple of 128: a warp's rows exist or not together
  const unsigned blocks = (unsigned)((rows * (head_dim / 4) + 255) / 256);
  const TDO* g = static_cast<const TDO*>(d_out);
  __nv_bfloat16* low = static_cast<__nv_bfloat16*>(d_out_bf16);
  ProfileScope prof(SA_KERNEL_DBAR, s);
  count_launch();
  if (head_dim == 64)
    row_stats_kernel<TDO, 64><<<blocks, 256, 0, s>>>(out, g, in_rows, vec, lse2, stats, low, dq_acc, zero_a, zero_b, heads, seq, padded, rows);
  else if (head_dim == 128)
    row_stats_kernel<TDO, 128><<<blocks, 256, 0, s>>>(out, g, in_rows, vec, lse2, stats, low, dq_acc, zero_a, zero_b, heads, seq, padded, rows);
  else
    return SA_ERR_UNSUPPORTED;
  SA_CUDA_CHECK(cudaGetLastError());
  return SA_OK;
}
}  // namespace

int launch_row_stats(const float* out, const void* d_out, int d_out_dtype, const RowLayout& in_rows, const float* lse2,
                     float* stats, void* d_out_bf16, float* dq_acc, float* zero_a, float* zero_b, int batch, int heads, int seq,
                     int head_dim, cudaStream_t s) {
  const int64_t es = d_out_dtype == SA_F32 ? 4 : 2;
  const bool vec = aligned_rows(d_out, in_rows, es, 4 * es);
  switch (d_out_dtype) {
    case SA_F32: return row_stats_by_dim<float>(out, d_out, in_rows, vec, lse2, stats, d_out_bf16, dq_acc, zero_a, zero_b, batch, heads, seq, head_dim, s);
    case SA_BF16: return row_stats_by_dim<__nv_bfloat16>(out, d_out, in_rows, vec, lse2, stats, d_out_bf16, dq_acc, zero_a, zero_b, batch, heads, seq, head_dim, s);
    case SA_F16: return row_stats_by_dim<__half>(out, d_out, in_rows, vec, lse2, stats, d_out_bf16, dq_acc, zero_a, zero_b, batch, heads, seq, head_dim, s);
  }
  return SA_ERR_BAD_ARGUMENT;
}

int launch_fold_cast(const float* acc, const float* acc0, void* dst, int dtype, int batch, int heads, int seq, int head_dim,
                     const RowLayout* dst_rows, cudaStream_t s) {
  const RowLayout rl = dst_rows ? *dst_rows : contiguous_rows(heads, seq, head_dim);
  const int64_t per_head = (int64_t)seq * head_dim;
  const int64_t total8 = (int64_t)batch * heads * per_head / 8;
  const unsigned blocks = (unsigned)((total8 + 255) / 256);
  const bool vec = aligned_rows(dst, rl, dtype == SA_F32 ? 4 : 2, 16);
  switch (dtype) {
    case SA_F32:
      count_launch();
      fold_cast_kernel<float><<<blocks, 256, 0, s>>>(acc, acc0, static_cast<float*>(dst), heads, per_head, total8, vec, rl, head_dim);
      break;
    case SA_BF16:
      count_launch();
      fold_cast_kernel<__nv_bfloat16><<<blocks, 256, 0, s>>>(acc, acc0, static_cast<__nv_bfloat16*>(dst), heads, per_head, total8,
                                                             vec, rl, head_dim);
      break;
    case SA_F16:
      count_launch();
      fold_cast_kernel<__half><<<blocks, 256, 0, s>>>(acc, acc0, static_cast<__half*>(dst), heads, per_head, total8, vec, rl,
                                                      head_dim);
      break;
    default: return SA_ERR_BAD_ARGUMENT;
  }
  SA_CUDA_CHECK(cudaGetLastError());
  return SA_OK;
}

int cache_store(int dtype, int batch, int heads, int groups, int seq, int capacity, int head_dim, int at, bool begin, const void* k,
                const RowLayout& k_rows, const void* v, const RowLayout& v_rows, void* k_cache, void* v_cache, float* selected,
                cudaStream_t s) {
  if (((reinterpret_cast<uintptr_t>(k_cache) | reinterpret_cast<uintptr_t>(v_cache)) & 15) != 0) return SA_ERR_ALIGNMENT;
  if ((int64_t)batch * heads > 65535) return SA_ERR_UNSUPPORTED;
  const int es = dtype == SA_F32 ? 4 : 2;
  // A chunk whose rows are dense per head, heads at one pitch, is a plain 2-D copy: no kernel of ours.  The pitch has to be one
  // that the copy takes: not less than a row of it (keys broadcast over heads have a pitch of 0), and below 2^31.
  const size_t row = (size_t)head_dim * es, width = seq * row, dst_pitch = capacity * row, nrows = (size_t)batch * heads;
  auto pitch = [&](const RowLayout& r) -> size_t { return nrows == 1 ? width : (size_t)(r.sh * es); };
  auto pitched = [&](const RowLayout& r) {
    return r.st == head_dim && (batch == 1 || r.sb == heads * r.sh) && r.sh >= 0 && pitch(r) >= width && pitch(r) < (1u << 31);
  };
  if (!begin && dst_pitch < (1u << 31) && pitched(k_rows) && pitched(v_rows)) {
    SA_CUDA_CHECK(cudaMemcpy2DAsync(static_cast<char*>(k_cache) + at * row, dst_pitch, k, pitch(k_rows), width, nrows,
                                    cudaMemcpyDeviceToDevice, s));
    SA_CUDA_CHECK(cudaMemcpy2DAsync(static_cast<char*>(v_cache) + at * row, dst_pitch, v, pitch(v_rows), width, nrows,
                                    cudaMemcpyDeviceToDevice, s));
    return SA_OK;
  }
  const bool vec = aligned_rows(k, k_rows, es, 16) && aligned_rows(v, v_rows, es, 16);
  const int64_t units = (int64_t)((begin ? capacity : at + seq) - at) * head_dim * es / 16;
  const unsigned blocks = (unsigned)max((int64_t)1, min((int64_t)256, (units + 1023) / 1024));
  count_launch();
  cache_store_kernel<<<dim3(blocks, batch * heads, begin && selected != nullptr ? 3 : 2), 256, 0, s>>>(
      static_cast<const uint8_t*>(k), k_rows, static_cast<const uint8_t*>(v), v_rows, static_cast<uint8_t*>(k_cache),
      static_cast<uint8_t*>(v_cache), selected, heads, groups, seq, capacity, head_dim * es, es, at, begin, vec);
  SA_CUDA_CHECK(cudaGetLastError());
  return SA_OK;
}

size_t decode_workspace_floats(int batch, int heads, int groups, int length, int head_dim) {
  const int t = length + 1;
  const size_t splits = decode_splits_max(t, batch * heads);
  return (size_t)batch * heads * splits * (head_dim + 2) + (size_t)batch * groups * t   // partials, new selection
         + (size_t)batch * heads + (size_t)batch * groups * splits;                       // tickets
}

int decode_step(const DecodeStep& d, cudaStream_t s) {
  const bool y_low = d.y_dtype != SA_F32;             // y in the cache's own type
  switch (d.dtype) {
    case SA_F32: return decode_impl<float, float>(d, s);
    case SA_BF16: return y_low ? decode_impl<__nv_bfloat16, __nv_bfloat16>(d, s) : decode_impl<__nv_bfloat16, float>(d, s);
    case SA_F16: return y_low ? decode_impl<__half, __half>(d, s) : decode_impl<__half, float>(d, s);
  }
  return SA_ERR_BAD_ARGUMENT;
}

}  // namespace sa
