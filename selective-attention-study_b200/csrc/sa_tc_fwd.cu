// Tensor-core engine, forward side (sm_100a: TMA loads, tcgen05 MMAs, fp32 accumulators in TMEM).
//
//   colsum_kernel   selection pass: for one 128-key tile and a run of 128-query tiles, the product
//                   K0 Q0^T with KEYS on the TMEM lanes, so a thread owns one key and the column sum of
//                   relu'd, masked logits over the tile's queries is a register reduction.  Writes
//                   COLSUM[b][query tile][key].
//   scan_kernel     exclusive prefix of COLSUM across query tiles, in place (-> CARRY), plus one extra
//                   row holding the grand total.  One thread per key column; bandwidth-bound.
//   forward_wide_kernel  flash-style forward for one 128-query tile of one head over 128-key steps, taken from
//                   the diagonal back to key 0: S = Q K^T and L0 = Q0 K0^T by MMA (Q, Q0 in TMEM); relu(L0) under
//                   the selection mask is written to shared memory as bf16 and the in-tile exclusive running
//                   sum over queries is one more MMA, (-strictly-lower-triangular ones) x selection,
//                   accumulated into S; then online softmax in the log2 domain with the cross-tile carry
//                   subtracted per key, and O += P V in TMEM.  Four arithmetic warpgroups and a control warp
//                   that issues every load and MMA; steps software-pipelined so the tensor pipe works under
//                   the exponentials.  head_dim 128, and head_dim 64 where two heads a CTA would leave SMs idle; few rows
//                   after many cached keys: a piece of the walk each, merged by the CTA that finishes last.
//                   Bound by the chain of a step (L0, selection, running sum, maximum over four warpgroups, exponentials,
//                   P V): 3.1 k cycles at head_dim 64, 3.7 k at 128 (one head per selector, whose single K tile is waited
//                   for: 5.0 k), counted over T = 16384 with the split walk in the same
//                   kernel (it is 1 to 5 % shorter without); the tensor pipe is busy 57 % of them at 128.
//
// Reference for the arithmetic: src/selective_attention/kernels.py:100-194 (selection, carry, forward).
#include <float.h>

#include <type_traits>

#include "sa_tc_fwd.cuh"

namespace sa {
namespace tc {
namespace {

constexpr int kTile = 128;          // query rows per CTA; also the carry checkpoint spacing
constexpr int kRowTile = 16384;     // bytes of a [128][64] bf16 operand tile

// ---------------------------------------------------------------------------------------------------
// selection column sums
// ---------------------------------------------------------------------------------------------------
// 128 threads own a key each; a fifth warp's elected lane issues the loads and MMAs, one tile ahead.  Bound by latency and
// issue: 128 compares and 64 packed additions a thread and tile.  (One accumulator and a block-wide barrier a tile, with the
// issuing thread among the 128, took 2.1 k cycles a tile and CTA: the additions alone were a chain of 512.)
constexpr int kColsumThreads = 160;

template <int D>
__global__ void __launch_bounds__(kColsumThreads) colsum_kernel(const __grid_constant__ CUtensorMap map_q,
                                                                const __grid_constant__ CUtensorMap map_k,
                                                                float* __restrict__ carry, int seq, int ntiles, int exempt,
                                                                float scale, WaitCtx status, int q_offset, int mi_first,
                                                                int chunk) {
  constexpr int DK = D / 64;
  const int nj = blockIdx.x, b = blockIdx.z;
  // Query tiles from the key tile's own (the diagonal) on; in a prefill continuation from the first tile that holds a
  // new query on (rows before q_offset are not in the query tensor: TMA fills them with zeros, which select nothing).
  const int mi0 = max(nj, mi_first) + blockIdx.y * chunk;
  if (mi0 >= ntiles) return;
  const int count = min(chunk, ntiles - mi0);

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* k0s = smem;                               // DK tiles [128 keys][64]
  uint8_t* q0s = smem + DK * kRowTile;               // 2 stages x DK tiles [128 queries][64]
  __shared__ uint64_t bar_k, bar_q[2], bar_mma[2], bar_read[2];
  __shared__ uint32_t tmem_base_s;

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (tid == 0) {
    mbar_init(&bar_k, 1);
    for (int u = 0; u < 2; ++u) {
      mbar_init(&bar_q[u], 1);
      mbar_init(&bar_mma[u], 1);
      mbar_init(&bar_read[u], 4);
    }
    mbar_init_fence();
  }
  if (warp == 0) tmem_alloc(&tmem_base_s, 256);
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem = tmem_base_s;

  if (warp == 4) {
    if (lane == 0) {
      const uint32_t idesc = instr_desc_bf16(128, 128, false, false);
      const uint32_t k_low = desc_low(smem_u32(k0s), 16), q_low = desc_low(smem_u32(q0s), 16);
      auto load_q = [&](int it) {
        uint64_t* bar = &bar_q[it & 1];
        mbar_expect_tx(bar, DK * kRowTile);
        for (int s = 0; s < DK; ++s)
          tma_load_4d(q0s + ((it & 1) * DK + s) * kRowTile, &map_q, bar, s * 64, (mi0 + it) * kTile - q_offset, 0, b);
      };
      mbar_expect_tx(&bar_k, DK * kRowTile);
      for (int s = 0; s < DK; ++s) tma_load_4d(k0s + s * kRowTile, &map_k, &bar_k, s * 64, nj * kTile, 0, b);
      load_q(0);
      if (count > 1) load_q(1);
      mbar_wait(&bar_k, 0, status, 201);
#pragma unroll 1
      for (int it = 0; it < count; ++it) {
        const int st = it & 1;
        const uint32_t ph = (uint32_t)((it >> 1) & 1);
        if (it >= 2) mbar_wait(&bar_read[st], ph ^ 1u, status, 203);      // the columns' last tile has been read
        mbar_wait(&bar_q[st], ph, status, 200);
        tc_fence_after_sync();
        for (int ks = 0; ks < 4 * DK; ++ks) {
          const uint32_t off = (uint32_t)((ks >> 2) * kRowTile + (ks & 3) * 32) >> 4;
          const uint32_t ql = q_low + (uint32_t)(st * DK * kRowTile >> 4) + off;
          if (ks == 0) mma_ss_low<false>(tmem + st * 128, k_low + off, ql, idesc);
          else mma_ss_low<true>(tmem + st * 128, k_low + off, ql, idesc);
        }
        mma_commit(&bar_mma[st]);
        if (it >= 1 && it + 1 < count) {                                  // the other stage: its MMA has completed
          mbar_wait(&bar_mma[st ^ 1], (uint32_t)(((it - 1) >> 1) & 1), status, 204);
          load_q(it + 1);
        }
      }
    }
    __syncwarp();
  } else {
    const uint32_t lane_base = tmem + ((uint32_t)(warp * 32) << 16);
    const int j = nj * kTile + tid;
    float* dst = carry + ((int64_t)b * (ntiles + 1) + mi0) * seq + j;
#pragma unroll 1
    for (int it = 0; it < count; ++it, dst += seq) {
      mbar_wait(&bar_mma[it & 1], (uint32_t)((it >> 1) & 1), status, 202);
      tc_fence_after_sync();
      const bool diag = mi0 + it == nj;
      float2 acc[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) acc[u] = make_float2(0.f, 0.f);
#pragma unroll
      for (int c0 = 0; c0 < 128; c0 += 32) {
        uint32_t r[32];
        tmem_ld32(lane_base + (it & 1) * 128 + c0, r);
        tmem_ld_wait();
        if (diag) {                                                        // (key and query count from the same position)
#pragma unroll
          for (int e = 0; e < 32; ++e)
            if (tid >= c0 + e) r[e] = 0u;
        }
#pragma unroll
        for (int e = 0; e < 32; e += 2)
          acc[(e >> 1) & 3] = __fadd2_rn(acc[(e >> 1) & 3], make_float2(fmaxf(__uint_as_float(r[e]), 0.f),
                                                                        fmaxf(__uint_as_float(r[e + 1]), 0.f)));
      }
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(&bar_read[it & 1]);
      const float2 s2 = __fadd2_rn(__fadd2_rn(acc[0], acc[1]), __fadd2_rn(acc[2], acc[3]));
      if (j < seq) *dst = (j < exempt) ? 0.f : (s2.x + s2.y) * scale;
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tmem, 256);
}

// One thread per key column: CARRY[b][mi][j] = sum of COLSUM[b][m'][j] over m' < mi, in place; row `ntiles`
// and total[b][j] receive the sum over all query tiles.  Only rows mi >= j / 128 exist.
__global__ void __launch_bounds__(256) scan_kernel(float* __restrict__ carry, float* total, int64_t total_stride, int seq,
                                                   int ntiles, int mi_first, const float* init,
                                                   int64_t init_stride, bool keep_init, unsigned int* tickets, int n_tickets) {
  if (blockIdx.x == 0 && blockIdx.y == 0 && (int)threadIdx.x < n_tickets) tickets[threadIdx.x] = 0u;   // of a split forward
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  const int b = blockIdx.y;
  if (j >= seq) return;
  float* col = carry + (int64_t)b * (ntiles + 1) * seq + j;
  const float before = init ? init[(int64_t)b * init_stride + j] : 0.f;   // what the key received before the first query given
  float run = before;
  int mi = max(j / kTile, mi_first);
  for (; mi + 8 <= ntiles; mi += 8) {
    float x[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) x[u] = col[(int64_t)(mi + u) * seq];
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      col[(int64_t)(mi + u) * seq] = run;
      run += x[u];
    }
  }
  for (; mi < ntiles; ++mi) {
    float x = col[(int64_t)mi * seq];
    col[(int64_t)mi * seq] = run;
    run += x;
  }
  col[(int64_t)ntiles * seq] = keep_init ? before : run;
  total[(int64_t)b * total_stride + j] = run;                    // (a continued prefill: where `init` was)
}

// ---------------------------------------------------------------------------------------------------
// forward
// ---------------------------------------------------------------------------------------------------
template <int N>
__device__ __forceinline__ void tmem_ld_n(uint32_t taddr, uint32_t (&r)[N]) {
  if constexpr (N == 16) tmem_ld16(taddr, r);
  else tmem_ld32(taddr, r);
}
template <int N>
__device__ __forceinline__ void tmem_st_n(uint32_t taddr, const uint32_t (&r)[N]) {
  if constexpr (N == 8) tmem_st8(taddr, r);
  else if constexpr (N == 16) tmem_st16(taddr, r);
  else tmem_st32(taddr, r);
}

// ---------------------------------------------------------------------------------------------------
// forward: 128-query tile x 128-key steps, one CTA per SM
// ---------------------------------------------------------------------------------------------------
// One 128-query tile of one head.  Key steps of 128 run from the diagonal back to key 0: the keys nearest the query
// carry the least history, so the running maximum settles within the first steps and the output accumulator,
// which stays in TMEM for the whole loop, is rescaled only while the maximum still moves.  One CTA keeps the tensor
// pipe and four warpgroups busy without a second resident CTA: a step covers 128 keys (N = 128 MMAs run at the full tensor rate and the per-step barriers
// are paid half as often), a control warp issues every load and MMA, and the steps are software-pipelined: after
// the logits and the row maximum of step t the arithmetic warps write the selection tile of step t + 1 (its L0 was
// issued right behind the running sum of step t), and only then do the exponentials of step t, so S and the
// triangular running sum of step t + 1 run on the tensor pipe under the exponentials instead of being waited for.
// head_dim 64 keeps two stages of K, K0 and V in shared memory; head_dim 128 has room for one and refills a
// tile as soon as the MMA that read it has completed.
template <int D>
struct WideSmem {
  static constexpr int DK = D / 64;
  static constexpr int kStages = (D == 64) ? 2 : 1;
  static constexpr int kTileBytes = DK * kRowTile;     // one [128 keys][D] operand
  static constexpr int q = 0;                          // landing tiles of Q (and Q0 at head_dim 64), then the triangular ones
  static constexpr int sel = q + 2 * kRowTile;         // [128 queries][128 keys] bf16 as two key tiles (B of the running sum);
                                                       //   head_dim 128: first the landing tiles of Q0
  static constexpr int p = sel + 2 * kRowTile;         // the same shape: P (A of P V)
  static constexpr int k = p + 2 * kRowTile;
  static constexpr int k0 = k + kStages * kTileBytes;
  static constexpr int v = k0 + kStages * kTileBytes;
  static constexpr int total = v + kStages * kTileBytes;   // 192 KB for both head dims
  static constexpr int q0_landing = (D == 64) ? q + kRowTile : sel;
};
constexpr int kWideCompute = 512;                      // four warpgroups: 32 of a step's 128 key columns, D / 4 of the d each
constexpr int kWideThreads = kWideCompute + 32;        // + the control warp: one lane issues every TMA load and MMA
constexpr int kWideBarrier = 1;                        // hardware barrier id of the arithmetic warps

// With pieces > 1 a CTA walks one piece of its query tile's key tiles (nothing goes from key tile to key tile but the softmax
// state: the history at the query tile is given) and leaves its rows, normalised, and their lse2 in [piece][batch * heads].
struct SplitWalk {
  int pieces;
  unsigned int* tickets;       // one per (query tile, row), zero
  float *part, *lse;
};

// LIVE: a table of live key tiles is given and the dead ones are left out.  SPLIT: more than one piece; walks of one piece have
// a kernel without the other code, which took 5 % longer with it (15 heads of T = 16384, head_dim 64: 1.41 -> 1.37 ms).
template <int D, bool SELF, bool LIVE, bool SPLIT>
__global__ void __launch_bounds__(kWideThreads, 1)
    forward_wide_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                        const __grid_constant__ CUtensorMap map_v, const __grid_constant__ CUtensorMap map_q0,
                        const __grid_constant__ CUtensorMap map_k0, const float* __restrict__ carry,
                        float* __restrict__ out, float* __restrict__ lse2, int heads, int seq, int ntiles, int exempt,
                        float scale, WaitCtx status, __nv_bfloat16* __restrict__ out_lowp, RowLayout out_lowp_rows,
                        int q_offset, const uint8_t* __restrict__ alive, SplitWalk split) {
  using L = WideSmem<D>;
  constexpr int DK = D / 64, DH = D / 4, NC = 32, ST = L::kStages;
  // TMEM columns: S and L0 (fp32, 128 each), the output accumulator (D), Q and Q0 as bf16 pairs (D / 2 each)
  constexpr uint32_t kColS = 0, kColL = 128, kColO = 256, kColQ = kColO + D, kColQ0 = kColQ + D / 2;
  // head_dim 64 leaves 128 columns: the triangular matrix and P live there as bf16 pairs (64 columns each), so the
  // running-sum and P V MMAs fetch only their B operands from shared memory.  head_dim 128 keeps both in shared memory.
  constexpr bool kTmemAB = (D == 64);
  constexpr uint32_t kColTri = 384, kColP = 448;

  const int pieces = SPLIT ? split.pieces : 1;
  const int piece = SPLIT ? (int)blockIdx.x % pieces : 0, cta = SPLIT ? (int)blockIdx.x / pieces : (int)blockIdx.x;
  const int nrows = gridDim.x / pieces / (ntiles - q_offset / kTile);  // batch * heads (the grid covers the query tiles with rows to compute)
  const int mi = ntiles - 1 - cta / nrows;                    // heaviest query tiles first
  const int n = cta % nrows;
  const int b = n / heads, h = n - b * heads;
  const int i0 = mi * kTile;
  // this piece's key tiles: last, last - 1, .. lowest (the last pieces may have none)
  const int piece_tiles = SPLIT ? (mi + pieces) / pieces : mi + 1;
  const int last = mi - piece * piece_tiles, lowest = SPLIT ? max(0, last - piece_tiles + 1) : 0;

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  // Completion barriers (one MMA commit each): bar_l0 L0 of a step; bar_tri S and running sum of a step; bar_pv
  // P V of a step; bar_fin the last P V.  Arrival barriers (one arrival per arithmetic warp and step): bar_sel
  // selection tile written and the previous step's logits read; bar_p P written and O rescaled.
  __shared__ uint64_t bar_q, bar_k[2], bar_k0[2], bar_v[2], bar_l0, bar_tri, bar_pv, bar_fin, bar_sel, bar_p, bar_setup;
  __shared__ uint32_t tmem_base_s;
  __shared__ __align__(16) float carry_s[2][kTile];
  __shared__ float rmax_s[4][kTile];
  __shared__ uint16_t live_s[kMaxLiveTiles + 1];              // with a table of live tiles: this query tile's key tiles,
  __shared__ int live_count_s;                                //   nearest first
  __shared__ bool last_s;

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (LIVE && warp == 1) {
    const uint8_t* live_row = alive + ((int64_t)n * ntiles + mi) * ntiles;
    int cnt = 0;
    for (int base = last; base >= lowest; base -= 32) {
      const int nj = base - lane;
      const bool f = nj >= lowest && live_row[nj] != 0;
      const unsigned m = __ballot_sync(0xffffffffu, f);
      if (f) live_s[cnt + __popc(m & ((1u << lane) - 1u))] = (uint16_t)nj;
      cnt += __popc(m);
    }
    if (lane == 0) live_count_s = cnt;
  }
  if (tid == 0) {
    mbar_init(&bar_q, 1);
    for (int u = 0; u < 2; ++u) {
      mbar_init(&bar_k[u], 1);
      mbar_init(&bar_k0[u], 1);
      mbar_init(&bar_v[u], 1);
    }
    mbar_init(&bar_l0, 1);
    mbar_init(&bar_tri, 1);
    mbar_init(&bar_pv, 1);
    mbar_init(&bar_fin, 1);
    mbar_init(&bar_sel, kWideCompute / 32);
    mbar_init(&bar_p, kWideCompute / 32);
    mbar_init(&bar_setup, kWideCompute / 32);
    mbar_init_fence();
  }
  if (warp == 0) tmem_alloc(&tmem_base_s, 512);
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem = tmem_base_s;
  const uint32_t sa = smem_u32(smem);
  // 128-key steps: every key tile up to and including the diagonal one, or the live ones only.  Step index `it`
  // counts from the diagonal (it = 0) back towards key 0; key_tile(it) is the tile it covers.
  const int steps = LIVE ? live_count_s : last - lowest + 1;
  auto key_tile = [&](int it) { return LIVE ? (it < steps ? (int)live_s[it] : 0) : last - it; };
  const int q_rows = seq - q_offset;

  if (SPLIT && steps <= 0) {                                   // a piece without keys
    if (tid < kTile && i0 + tid < seq && i0 + tid >= q_offset)
      split.lse[((int64_t)piece * nrows + n) * q_rows + i0 + tid - q_offset] = -INFINITY;
  } else if (warp == kWideCompute / 32) {
    // =============================== control warp: TMA loads and MMA issue ===============================
    // The warp stays converged and one elected lane issues: inside a divergent branch an MMA took about 75 cycles to issue.  One
    // head per selector issues fewer MMAs and waits at as many places: a single lane that polls is the faster there (15 rows of
    // T = 16384 at head_dim 128 2.20 ms, converged 2.23; 5 rows of 1,000 at 64 22.7 us, converged 23.4).
    constexpr bool kOneLane = SELF;
    Waiter wait;
    if (!kOneLane) wait.begin(status);
    auto elected = [&] { return kOneLane || elect_one(); };
    auto converge = [&] { if (!kOneLane) __syncwarp(); };
    if (!kOneLane || lane == 0) {
    // A tile of step it lives in stage slot(it); the j-th fill of a stage completes its barrier's phase j.
    auto slot = [](int it) { return ST == 2 ? (it & 1) : 0; };
    auto fill = [](int it) { return (uint32_t)((ST == 2 ? (it >> 1) : it) & 1); };
    auto await = [&](uint64_t* bar, uint32_t parity, int site) {
      if (kOneLane) {
        mbar_wait(bar, parity, status, site);
        tc_fence_after_sync();
      } else {
        wait.left = wait_call(smem_u32(bar), parity, site, wait.left);
      }
    };
    auto load_tile = [&](int off, const CUtensorMap* map, uint64_t* bars, int it, int head) {
      const int j0 = key_tile(it) * kTile;
      if (elected()) {
        uint64_t* bar = &bars[slot(it)];
        mbar_expect_tx(bar, L::kTileBytes);
        for (int s2 = 0; s2 < DK; ++s2)
          tma_load_4d(smem + off + slot(it) * L::kTileBytes + s2 * kRowTile, map, bar, s2 * 64, j0, head, b);
      }
      converge();
    };
    auto load_k = [&](int it) { load_tile(L::k, &map_k, bar_k, it, h); };
    auto load_k0 = [&](int it) { if (!SELF) load_tile(L::k0, &map_k0, bar_k0, it, 0); };   // SELF: K0 is K
    auto load_v = [&](int it) { load_tile(L::v, &map_v, bar_v, it, h); };
    const uint32_t idesc_s = instr_desc_bf16(128, 128, false, false);
    const uint32_t idesc_tri = instr_desc_bf16(128, 128, false, true, /*negate_a=*/true);
    const uint32_t idesc_pv = instr_desc_bf16(128, D, false, true);
    const uint32_t kBase = desc_low(sa, 16);                   // K-major views (rows = M or N index)
    const uint32_t mBase = desc_low(sa, kRowTile);             // MN-major views (rows = K index)
    auto at = [](uint32_t low, uint32_t byte_off) { return low + (byte_off >> 4); };
    auto kstep = [](int ks) { return (uint32_t)((ks >> 2) * kRowTile + (ks & 3) * 32); };
    auto issue_l0 = [&](int it) {                              // L0 = Q0 K0^T
      await(SELF ? &bar_k[slot(it)] : &bar_k0[slot(it)], fill(it), 311);
      if (elected()) {
        const uint32_t tile = at(kBase, (SELF ? L::k : L::k0) + slot(it) * L::kTileBytes);
#pragma unroll
        for (int ks = 0; ks < 4 * DK; ++ks)
          mma_ts_low(tmem + kColL, tmem + (SELF ? kColQ : kColQ0) + ks * 8, at(tile, kstep(ks)), idesc_s, ks > 0);
        mma_commit(&bar_l0);
      }
      converge();
    };
    auto issue_s_tri = [&](int it) {                           // S = Q K^T, then S -= TRI x selection
      await(&bar_k[slot(it)], fill(it), 312);
      if (elected()) {
        const uint32_t tile = at(kBase, L::k + slot(it) * L::kTileBytes);
#pragma unroll
        for (int ks = 0; ks < 4 * DK; ++ks) mma_ts_low(tmem + kColS, tmem + kColQ + ks * 8, at(tile, kstep(ks)), idesc_s, ks > 0);
#pragma unroll
        for (int ks = 0; ks < 8; ++ks) {
          if (kTmemAB) mma_ts_low(tmem + kColS, tmem + kColTri + ks * 8, at(mBase, L::sel + ks * 2048), idesc_tri, 1u);
          else mma_ss_low<true>(tmem + kColS, at(kBase, L::q + kstep(ks)), at(mBase, L::sel + ks * 2048), idesc_tri);
        }
        mma_commit(&bar_tri);
      }
      converge();
    };
    auto issue_pv = [&](int it, uint64_t* bar) {               // O += P V
      await(&bar_v[slot(it)], fill(it), 315);
      if (elected()) {
        const uint32_t v = at(mBase, L::v + slot(it) * L::kTileBytes);
        const uint32_t more = it > 0 ? 1u : 0u;
#pragma unroll
        for (int ks = 0; ks < 8; ++ks) {
          if (kTmemAB) mma_ts_low(tmem + kColO, tmem + kColP + ks * 8, at(v, ks * 2048), idesc_pv, ks > 0 ? 1u : more);
          else if (ks > 0) mma_ss_low<true>(tmem + kColO, at(kBase, L::p + kstep(ks)), at(v, ks * 2048), idesc_pv);
          else if (it > 0) mma_ss_low<true>(tmem + kColO, at(kBase, L::p), v, idesc_pv);
          else mma_ss_low<false>(tmem + kColO, at(kBase, L::p), v, idesc_pv);
        }
        mma_commit(bar);
      }
      converge();
    };

    if (elected()) {
      mbar_expect_tx(&bar_q, (SELF ? 1 : 2) * DK * kRowTile);
      for (int s2 = 0; s2 < DK; ++s2) {
        tma_load_4d(smem + L::q + s2 * kRowTile, &map_q, &bar_q, s2 * 64, i0 - q_offset, h, b);
        if (!SELF) tma_load_4d(smem + L::q0_landing + s2 * kRowTile, &map_q0, &bar_q, s2 * 64, i0 - q_offset, 0, b);
      }
    }
    converge();
    load_k0(0);
    load_k(0);
    load_v(0);
    if (ST == 2 && steps > 1) {
      load_k0(1);
      load_k(1);
      load_v(1);
    }
    await(&bar_setup, 0, 317);                                 // Q, Q0 in TMEM and the triangular tile in place
    issue_l0(0);
#pragma unroll(D == 64 ? 2 : 1)   // head_dim 64: the stage and phase parities become constants
    for (int it = 0; it < steps; ++it) {
      await(&bar_sel, it & 1, 318);                            // selection of step it written; logits of it - 1 read;
      if (it + ST < steps) load_k0(it + ST);                   //   L0 of step it consumed: its K0 tile is free
      issue_s_tri(it);
      const bool l0_now = !(SELF && ST == 1);                  // one-stage SELF: K of the next step is not loaded yet
      if (l0_now && it + 1 < steps) issue_l0(it + 1);
      if (it > 0) {
        await(&bar_p, (it - 1) & 1, 320);                      // P of step it - 1 written, O rescaled
        if (ST == 2 && it >= 2) {                              // before this barrier's next commit: P V of it - 2 done,
          await(&bar_pv, it & 1, 321);                         //   so its V tile may be refilled
          load_v(it);
        }
        issue_pv(it - 1, &bar_pv);
      }
      await(&bar_tri, it & 1, 319);                            // S of step it done: its K tile is free
      if (it + ST < steps) load_k(it + ST);
      if (!l0_now && it + 1 < steps) issue_l0(it + 1);
      if (ST == 1 && it > 0) {                                 // the single V tile: refilled with V of step it (for the
        await(&bar_pv, (it - 1) & 1, 321);                     //   P V issued in the next iteration) once P V of step
        load_v(it);                                            //   it - 1 has completed
      }
    }
    await(&bar_p, (steps - 1) & 1, 322);
    issue_pv(steps - 1, &bar_fin);
    if (!kOneLane && lane == 0) wait.end(status);
    }
    __syncwarp();
  } else {
    // ======================================= arithmetic warps ============================================
    const int row = tid & 127, wg = tid >> 7;
    const uint32_t lane_base = tmem + ((uint32_t)((warp & 3) * 32) << 16);
    auto arrive = [&](uint64_t* bar) {                         // this warp's shared-memory and TMEM accesses are done
      fence_async_smem();
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar);
    };
    // Q and Q0 rows from the landing tiles into TMEM as bf16 pairs; warpgroup wg moves D / 4 of the D columns
    mbar_wait(&bar_q, 0, status, 310);
    {
      constexpr int kChunks = D / 32;                          // 16-byte chunks per thread and matrix
#pragma unroll
      for (int m = 0; m < (SELF ? 1 : 2); ++m) {
        const uint8_t* src = smem + (m == 0 ? L::q : L::q0_landing);
        uint32_t w[kChunks * 4];
#pragma unroll
        for (int c = 0; c < kChunks; ++c) {
          const int chunk = wg * kChunks + c;                  // chunk index along D (8 elements each)
          const uint4 v4 = *reinterpret_cast<const uint4*>(src + (chunk >> 3) * kRowTile + swz_off(row, chunk & 7));
          w[4 * c] = v4.x; w[4 * c + 1] = v4.y; w[4 * c + 2] = v4.z; w[4 * c + 3] = v4.w;
        }
        tmem_st_n<kChunks * 4>(lane_base + (m == 0 ? kColQ : kColQ0) + wg * (kChunks * 4), w);
      }
    }
    tmem_st_wait();
    named_barrier(kWideBarrier, kWideCompute);                 // the landing tiles have been read by everyone
    // strictly-lower-triangular ones TRI[i][r] = 1 for r < i over the landing area: a K-major A operand of two
    // [128][64] tiles; thread (row, wg) writes running-sum indices r = 32 wg .. 32 wg + 31 of its row
    if (kTmemAB) {                                             // 32 running-sum indices = 16 packed columns per thread
      uint32_t w[16];
#pragma unroll
      for (int e = 0; e < 16; ++e) {
        const int r = wg * 32 + 2 * e;
        w[e] = pack_bf16(r < row ? 1.f : 0.f, (r + 1) < row ? 1.f : 0.f);
      }
      tmem_st16(lane_base + kColTri + wg * 16, w);
      tmem_st_wait();
    } else {
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const int chunk = wg * 4 + c;
        uint32_t w[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int r = chunk * 8 + 2 * e;
          w[e] = pack_bf16(r < row ? 1.f : 0.f, (r + 1) < row ? 1.f : 0.f);
        }
        *reinterpret_cast<uint4*>(smem + L::q + (chunk >> 3) * kRowTile + swz_off(row, chunk & 7)) =
            make_uint4(w[0], w[1], w[2], w[3]);
      }
    }
    arrive(&bar_setup);

    const float c1 = scale * kLog2e;
    const float* carry_row = carry + ((int64_t)b * (ntiles + 1) + mi) * seq;
    const int i = i0 + row;
    const int cw = wg * NC;                                    // this warpgroup's key columns within a step

    // The carry of a step's keys is fetched from global memory a step before it is staged, so the load's latency
    // is spent under the exponentials of the step before.
    auto fetch_carry = [&](int it) {
      const int j = key_tile(it) * kTile + tid;
      return (tid < kTile && it < steps && j < seq) ? load_ahead(carry_row + j) : 0.f;
    };
    // selection relu(L0) under the mask of step `it` -> bf16 tile, in two halves of 16 columns; also stages the
    // step's carry (scaled) for the logits pass
    auto selection = [&](int it, float carry_value) {
      const int j0 = key_tile(it) * kTile;
      if (tid < kTile) carry_s[it & 1][tid] = -carry_value * kLog2e;   // negated: the logits pass adds it in an FMA
      mbar_wait(&bar_l0, it & 1, status, 313);
      tc_fence_after_sync();
      const bool masked = (j0 + kTile > i0) || (j0 < exempt);
      uint32_t r32[32];
      tmem_ld32(lane_base + kColL + cw, r32);                 // one load and one wait for the step's 32 columns
      tmem_ld_wait();
#pragma unroll
      for (int hc = 0; hc < 2; ++hc) {
        const uint32_t* r = r32 + hc * 16;
        float s[16];
        if (masked) {
#pragma unroll
          for (int e = 0; e < 16; ++e) {
            const int j = j0 + cw + hc * 16 + e;
            s[e] = (j < i && j >= exempt) ? __uint_as_float(r[e]) : 0.f;
          }
        } else {
#pragma unroll
          for (int e = 0; e < 16; ++e) s[e] = __uint_as_float(r[e]);
        }
#pragma unroll
        for (int c = 0; c < 2; ++c) {                          // the relu rides on the bf16 conversion
          uint4 w = make_uint4(pack_bf16_relu(s[c * 8 + 0], s[c * 8 + 1]), pack_bf16_relu(s[c * 8 + 2], s[c * 8 + 3]),
                               pack_bf16_relu(s[c * 8 + 4], s[c * 8 + 5]), pack_bf16_relu(s[c * 8 + 6], s[c * 8 + 7]));
          *reinterpret_cast<uint4*>(smem + L::sel + (wg >> 1) * kRowTile + swz_off(row, (wg & 1) * 4 + hc * 2 + c)) = w;
        }
      }
      arrive(&bar_sel);
    };

    // run_den: this warpgroup's share of the denominator.  The maximum starts at the lowest finite value: a later piece of a walk
    // can begin with key tiles whose history is infinite (keys taken out by their caller), and -inf - (-inf) is not a number.
    float run_max = -FLT_MAX, run_den = 0.f;
    selection(0, fetch_carry(0));
    float next_carry = fetch_carry(1);
    // One 128-key step.  The diagonal step (it = 0: causal mask inside the tile, nothing to wait for or rescale yet) is
    // peeled off the loop.
    auto step = [&](int it, auto first_tag) {
      constexpr bool kFirst = decltype(first_tag)::value;
      const int j0 = key_tile(it) * kTile;
      // ---- logits z = (S * scale - carry) * log2(e) after S -= TRI x selection, and the row maximum -----------
      mbar_wait(&bar_tri, it & 1, status, 314);
      tc_fence_after_sync();
      // Packed fp32x2 arithmetic (two results per issue slot) for the logits, the shift by the maximum and the row sum.
      float2 z[NC / 2];
      {
        uint32_t r[NC];
        tmem_ld32(lane_base + kColS + cw, r);
        tmem_ld_wait();
        const float4* ncs = reinterpret_cast<const float4*>(carry_s[it & 1] + cw);   // -carry * log2(e), broadcast loads
        const float2 cc = make_float2(c1, c1);
        float tile_max = -INFINITY;
#pragma unroll
        for (int e4 = 0; e4 < NC / 4; ++e4) {
          const float4 nc = ncs[e4];
          float2 a = __ffma2_rn(make_float2(__uint_as_float(r[4 * e4]), __uint_as_float(r[4 * e4 + 1])), cc,
                                make_float2(nc.x, nc.y));
          float2 b2 = __ffma2_rn(make_float2(__uint_as_float(r[4 * e4 + 2]), __uint_as_float(r[4 * e4 + 3])), cc,
                                 make_float2(nc.z, nc.w));
          if (kFirst) {                                        // the diagonal tile
            const int jj = j0 + cw + 4 * e4;
            if (jj > i) a.x = -INFINITY;
            if (jj + 1 > i) a.y = -INFINITY;
            if (jj + 2 > i) b2.x = -INFINITY;
            if (jj + 3 > i) b2.y = -INFINITY;
          }
          tile_max = fmaxf(fmaxf(tile_max, fmaxf(a.x, a.y)), fmaxf(b2.x, b2.y));
          z[2 * e4] = a;
          z[2 * e4 + 1] = b2;
        }
        rmax_s[wg][row] = tile_max;
      }
      named_barrier(kWideBarrier, kWideCompute);
      const float new_max =
          fmaxf(fmaxf(run_max, fmaxf(rmax_s[0][row], rmax_s[1][row])), fmaxf(rmax_s[2][row], rmax_s[3][row]));
      const float alpha = ex2(run_max - new_max);
      run_max = new_max;

      // ---- the next step's selection tile first: its S and running sum then run under the exponentials --------
      if (it + 1 < steps) selection(it + 1, next_carry);
      next_carry = fetch_carry(it + 2);

      // ---- exponentials, P, and the accumulator rescale ---------------------------------------------------------
      float2 rs = make_float2(0.f, 0.f);
      const float2 nm = make_float2(-new_max, -new_max);
#pragma unroll
      for (int e = 0; e < NC / 2; ++e) {
        const float2 x = __fadd2_rn(z[e], nm);
        z[e] = make_float2(ex2(x.x), ex2(x.y));
        rs = __fadd2_rn(rs, z[e]);
      }
      run_den = run_den * alpha + (rs.x + rs.y);
      if (!kFirst) {
        mbar_wait(&bar_pv, (it - 1) & 1, status, 323);         // P V of the previous step: P tile and O are free
        tc_fence_after_sync();
      }
      if (kTmemAB) {                                           // P as bf16 pairs: keys 32 wg .. at column 16 wg of P
        uint32_t w[16];
#pragma unroll
        for (int e = 0; e < 16; ++e) w[e] = pack_bf16(z[e].x, z[e].y);
        tmem_st16(lane_base + kColP + wg * 16, w);
      } else {
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          uint4 w = make_uint4(pack_bf16(z[c * 4].x, z[c * 4].y), pack_bf16(z[c * 4 + 1].x, z[c * 4 + 1].y),
                               pack_bf16(z[c * 4 + 2].x, z[c * 4 + 2].y), pack_bf16(z[c * 4 + 3].x, z[c * 4 + 3].y));
          *reinterpret_cast<uint4*>(smem + L::p + (wg >> 1) * kRowTile + swz_off(row, (wg & 1) * 4 + c)) = w;
        }
      }
      if (!kFirst && __any_sync(0xffffffffu, alpha != 1.f)) {  // the accumulator follows the maximum while it moves
        uint32_t r[DH];
        tmem_ld_n<DH>(lane_base + kColO + wg * DH, r);
        tmem_ld_wait();
#pragma unroll
        for (int e = 0; e < DH; ++e) r[e] = __float_as_uint(__uint_as_float(r[e]) * alpha);
        tmem_st_n<DH>(lane_base + kColO + wg * DH, r);
      }
      tmem_st_wait();                                          // P (head_dim 64) and the rescaled accumulator are in TMEM
      arrive(&bar_p);
    };
    step(0, std::true_type{});
    for (int it = 1; it < steps; ++it) step(it, std::false_type{});
    mbar_wait(&bar_fin, 0, status, 316);                       // the last P V
    tc_fence_after_sync();

    named_barrier(kWideBarrier, kWideCompute);                 // everyone has read the last row maxima
    rmax_s[wg][row] = run_den;                                 // the warpgroups hold disjoint shares of the denominator
    named_barrier(kWideBarrier, kWideCompute);
    const float den = (rmax_s[0][row] + rmax_s[1][row]) + (rmax_s[2][row] + rmax_s[3][row]);
    const float inv = 1.f / den;
    uint32_t r[DH];
    tmem_ld_n<DH>(lane_base + kColO + wg * DH, r);
    tmem_ld_wait();
    if (i < seq && i >= q_offset) {                            // rows before q_offset belong to an earlier call
      const int iq = i - q_offset;                             // row inside the query tensor
      constexpr bool whole = !SPLIT;
      const int64_t nr = ((int64_t)piece * nrows + n) * q_rows + iq;
      float* rows_to = whole ? out : split.part;
      if (rows_to != nullptr) {
        float4* orow = reinterpret_cast<float4*>(rows_to + nr * D + wg * DH);
#pragma unroll
        for (int d = 0; d < DH; d += 4)
          orow[d >> 2] = make_float4(__uint_as_float(r[d]) * inv, __uint_as_float(r[d + 1]) * inv,
                                     __uint_as_float(r[d + 2]) * inv, __uint_as_float(r[d + 3]) * inv);
      }
      if (wg == 0) (whole ? lse2 : split.lse)[nr] = run_max + log2f(den);
      if (whole && out_lowp != nullptr) {                               // the same rows in the operand dtype, in the caller's layout
        uint4* lrow = reinterpret_cast<uint4*>(out_lowp + out_lowp_rows.at(b, h, iq) + wg * DH);
#pragma unroll
        for (int d = 0; d < DH; d += 8)
          lrow[d >> 3] = make_uint4(pack_bf16(__uint_as_float(r[d]) * inv, __uint_as_float(r[d + 1]) * inv),
                                    pack_bf16(__uint_as_float(r[d + 2]) * inv, __uint_as_float(r[d + 3]) * inv),
                                    pack_bf16(__uint_as_float(r[d + 4]) * inv, __uint_as_float(r[d + 5]) * inv),
                                    pack_bf16(__uint_as_float(r[d + 6]) * inv, __uint_as_float(r[d + 7]) * inv));
      }
    }
  }
  if (SPLIT) __threadfence();
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tmem, 512);
  if constexpr (!SPLIT) return;
  // The CTA that finishes last merges the pieces of its 128 rows, D / 8 threads a row.
  if (tid == 0) last_s = atomicAdd(split.tickets + cta, 1u) == (unsigned)pieces - 1;
  __syncthreads();
  if (!last_s || tid >= kWideCompute) return;
  __threadfence();
  constexpr int kLanes = D / 8;
  const int64_t stride = (int64_t)nrows * q_rows;              // rows of a piece
  for (int r = tid / kLanes; r < kTile; r += kWideCompute / kLanes) {
    const int iq = i0 + r - q_offset, d = tid % kLanes * 8;
    if (iq < 0 || iq >= q_rows) continue;
    const int64_t at = (int64_t)n * q_rows + iq;
    float top = -INFINITY;
    for (int s2 = 0; s2 < pieces; ++s2) top = fmaxf(top, __ldcg(split.lse + s2 * stride + at));
    float acc[8] = {}, den = 0.f;
    for (int s2 = 0; s2 < pieces; ++s2) {
      const float l = __ldcg(split.lse + s2 * stride + at);
      if (l == -INFINITY) continue;                            // no keys, and no rows written
      const float w = ex2(l - top);
      const float4* src = reinterpret_cast<const float4*>(split.part + (s2 * stride + at) * D + d);
      const float4 x = __ldcg(src), y = __ldcg(src + 1);
      den += w;
      acc[0] = fmaf(w, x.x, acc[0]); acc[1] = fmaf(w, x.y, acc[1]); acc[2] = fmaf(w, x.z, acc[2]); acc[3] = fmaf(w, x.w, acc[3]);
      acc[4] = fmaf(w, y.x, acc[4]); acc[5] = fmaf(w, y.y, acc[5]); acc[6] = fmaf(w, y.z, acc[6]); acc[7] = fmaf(w, y.w, acc[7]);
    }
    const float inv = 1.f / den;
    if (d == 0) lse2[at] = top + log2f(den);
    if (out != nullptr) {
      float4* dst = reinterpret_cast<float4*>(out + at * D + d);
      dst[0] = make_float4(acc[0] * inv, acc[1] * inv, acc[2] * inv, acc[3] * inv);
      dst[1] = make_float4(acc[4] * inv, acc[5] * inv, acc[6] * inv, acc[7] * inv);
    }
    if (out_lowp != nullptr)
      *reinterpret_cast<uint4*>(out_lowp + out_lowp_rows.at(b, h, iq) + d) =
          make_uint4(pack_bf16(acc[0] * inv, acc[1] * inv), pack_bf16(acc[2] * inv, acc[3] * inv),
                     pack_bf16(acc[4] * inv, acc[5] * inv), pack_bf16(acc[6] * inv, acc[7] * inv));
  }
}

template <int D>
int forward_impl(const Problem& p, float* out, float* lse2, float* carry, float* total, cudaStream_t s) {
  const int ntiles = (p.seq + kTile - 1) / kTile;
  const int q_rows = p.seq - p.q_offset;                 // rows of the query tensor (all of them unless continuing a prefill)
  const int mi_first = p.q_offset / kTile;               // first query tile with a row to compute
  ForwardMaps m;
  int st = make_map_16bit(&m.q, p.q.ptr, D, q_rows, p.heads, p.batch, p.q.st, p.q.sh, p.q.sb, kTile);
  if (st != SA_OK) return st;
  st = make_map_16bit(&m.k, p.k.ptr, D, p.seq, p.heads, p.batch, p.k.st, p.k.sh, p.k.sb, kTile);
  if (st != SA_OK) return st;
  st = make_map_16bit(&m.v, p.v.ptr, D, p.seq, p.heads, p.batch, p.v.st, p.v.sh, p.v.sb, kTile);
  if (st != SA_OK) return st;
  // the selector's rows: (d, token, 1, batch)
  st = make_map_16bit(&m.q0, p.q0.ptr, D, q_rows, 1, p.batch, p.q0.st, 0, p.q0.sb, kTile);
  if (st != SA_OK) return st;
  st = make_map_16bit(&m.k0, p.k0.ptr, D, p.seq, 1, p.batch, p.k0.st, 0, p.k0.sb, kTile);
  if (st != SA_OK) return st;
  WaitCtx status;
  st = wait_ctx(&status);
  if (st != SA_OK) return st;

  constexpr int DK = D / 64;
  const int colsum_smem = 3 * DK * kRowTile + 1024;
  SA_CUDA_CHECK(allow_smem(colsum_kernel<D>, colsum_smem));
  // query tiles per CTA: 8, or 32 where that still gives every SM several CTAs (the key tile and the set-up are paid per CTA)
  const int64_t tiles = (int64_t)ntiles * (ntiles - mi_first) * p.batch;
  const int chunk = tiles >= 32 * 16 * kSms ? 32 : 8;
  dim3 gc(ntiles, (ntiles - mi_first + chunk - 1) / chunk, p.batch);
  {
    ProfileScope prof(SA_KERNEL_TC_COLSUM, s);
    count_launch();
    colsum_kernel<D><<<gc, kColsumThreads, colsum_smem, s>>>(m.q0, m.k0, carry, p.seq, ntiles, p.exempt, p.scale, status,
                                                             p.q_offset, mi_first, chunk);
  }
  SA_CUDA_CHECK(cudaGetLastError());
  const int pieces = p.split_scratch != nullptr ? prefill_split_pieces(p) : 1;
  const int64_t rows = (int64_t)p.batch * p.heads * q_rows;
  SplitWalk split{pieces, nullptr, nullptr, nullptr};
  if (pieces > 1) {
    split.tickets = reinterpret_cast<unsigned int*>(p.split_scratch);
    split.part = p.split_scratch + kSplitTickets;
    split.lse = split.part + pieces * rows * D;
  }
  dim3 gs((p.seq + 255) / 256, p.batch);
  {
    ProfileScope prof(SA_KERNEL_TC_SCAN, s);
    count_launch();
    scan_kernel<<<gs, 256, 0, s>>>(carry, total, p.total_stride, p.seq, ntiles, mi_first, p.carry_init, p.carry_init_stride,
                                    p.history_moved != nullptr, split.tickets, pieces > 1 ? kSplitTickets : 0);
  }
  SA_CUDA_CHECK(cudaGetLastError());
  if (p.history_moved != nullptr) *p.history_moved = true;

  const uint8_t* alive = nullptr;
  if (p.tile_table != nullptr && ntiles <= kMaxLiveTiles) {
    st = build_tile_table(p, carry, s);
    if (st != SA_OK) return st;
    alive = static_cast<const uint8_t*>(p.tile_table);
  }
  const bool self = self_selecting(p);
  // Heads that share a selector go two to a CTA: its selection is made once and the two overlap (1.3x a head-tile).  While
  // one head a CTA still fits the GPU in one wave, that is faster: a step of it takes 3.1 k cycles, of a pair 4.4 k.
  const int64_t ctas = (int64_t)(ntiles - mi_first) * p.batch * p.heads;
  if (D == 64 && !self && p.heads % 2 == 0 && ctas > kSms) return forward_pair(p, m, carry, out, lse2, status, alive, s);
  if (D == 64 && self && p.batch % 2 == 0 && ctas > kSms) return forward_self(p, m, carry, out, lse2, status, alive, s);
  const unsigned grid = (unsigned)(ntiles - mi_first) * p.batch * p.heads * pieces;
  const int wide_smem = WideSmem<D>::total + 1024;
  auto launch = [&](auto kernel) -> int {
    SA_CUDA_CHECK(allow_smem(kernel, wide_smem));
    ProfileScope prof(SA_KERNEL_TC_FORWARD, s);
    count_launch();
    kernel<<<grid, kWideThreads, wide_smem, s>>>(m.q, m.k, m.v, m.q0, m.k0, carry, out, lse2, p.heads, p.seq,
                                                 ntiles, p.exempt, p.scale, status,
                                                 static_cast<__nv_bfloat16*>(p.out_lowp), p.out_lowp_rows,
                                                 p.q_offset, alive, split);
    return SA_OK;
  };
  auto by_split = [&](auto self_tag, auto live_tag) {
    constexpr bool kSelf = decltype(self_tag)::value, kLive = decltype(live_tag)::value;
    return pieces > 1 ? launch(forward_wide_kernel<D, kSelf, kLive, true>) : launch(forward_wide_kernel<D, kSelf, kLive, false>);
  };
  const std::true_type yes;
  const std::false_type no;
  if (alive != nullptr) st = self ? by_split(yes, yes) : by_split(no, yes);
  else st = self ? by_split(yes, no) : by_split(no, no);
  if (st != SA_OK) return st;
  SA_CUDA_CHECK(cudaGetLastError());
  return SA_OK;
}

}  // namespace

// A short chunk after a long cache has few (query tile, head) pairs, each with a long walk: where half of the SMs or more would
// have nothing to do, a walk is cut into as many pieces as give each its SM, of at least 4 steps of 128 keys (a piece pays a
// set-up of about two, and the last one reads all of them).  A prompt is not cut: its rows do not depend on what follows them.
int prefill_split_pieces(const Problem& p) {
  if (p.q_offset == 0) return 1;
  const int ntiles = (p.seq + kTile - 1) / kTile;
  const int64_t ctas = (int64_t)(ntiles - p.q_offset / kTile) * p.batch * p.heads;
  const int64_t pieces = ctas > 0 ? kSms / ctas : 1;
  return (int)(pieces < ntiles / 4 ? (pieces > 1 ? pieces : 1) : (ntiles / 4 > 1 ? ntiles / 4 : 1));
}

int forward(const Problem& p, float* out, float* lse2, float* carry, float* total, cudaStream_t s) {
  if (p.head_dim == 64) return forward_impl<64>(p, out, lse2, carry, total, s);
  if (p.head_dim == 128) return forward_impl<128>(p, out, lse2, carry, total, s);
  return SA_ERR_UNSUPPORTED;
}

}  // namespace tc
}  // namespace sa
