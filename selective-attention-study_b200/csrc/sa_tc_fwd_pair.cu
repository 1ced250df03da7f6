// Tensor-core engine, forward for two heads that share a selector (head_dim 64; sm_100a: TMA loads, tcgen05 MMAs, fp32
// accumulators in TMEM).
//
// One CTA owns one 128-query tile of two neighbouring heads and takes 128-key steps from the diagonal back to key 0.  The
// selection of a step -- the logits L0 = Q0 K0^T, relu and mask to bf16, and the exclusive running sum over the tile's
// queries as an MMA with a strictly-lower-triangular ones matrix, F = -TRI x selection -- does not depend on the head, so it
// is made once for both, by a warpgroup of its own, one step ahead of the softmax.  The two heads are two chains (scores ->
// softmax -> P V) that take turns on the exponential unit: one computes while the products of the other run.
//
// Roles.  Warps 0-3 and 4-7: the softmax of the two heads; a thread owns a query row and its 128 logits of the step.  Warps
// 8-11: the selection (and the carry of the step's keys).  Warp 12: MMAs of the heads (P V of a step, then S of the next).
// Warp 13: TMA loads.  Warp 14: MMAs of the selection (L0, then F over the same columns).
//
// TMEM, 512 columns: S of the two heads (128 each; P as bf16 pairs over its first 64) | L0, then F (128) | O of the two
// heads (64 each).  Shared memory, 224 KB: Q, Q of the two heads and Q0 48 KB, TRI 32, selection 32, K and V rings of three
// tiles 48 each (the heads alternate), K0 16.
//
// What bounds it: latency around F.  The step of both heads takes 4.4 k cycles: F read by both -> L0 -> selection -> running
// sum -> F read by both is a chain of hand-overs, and a head's own chain is as long (S after P V of the step before 1.2 k, read
// 0.8 k, 128 exponentials a thread 1.5 k).  The exponential unit (16 ex2 a clock and SM) needs 2.0 k of them and is busy 48 % of
// the time, the tensor pipe 41 %, the issue slots 42 %.  TMEM is full, so neither S nor F can have a second buffer; S in two halves
// of 64 keys around P V (N = 64 products read shared memory 1.5 times as much), four softmax warpgroups and two for the
// selection were slower.
// Measured at B = 4, H = 16, T = 16384: 4.25 ms (forward_wide_kernel, which makes the selection and its running sum for each
// head and keeps its sixteen warps in step: 6.06 ms); B = 1, H = 16, T = 131072: 95.1 -> 66.2 ms.
//
// Reference for the arithmetic: src/selective_attention/kernels.py:140-194 (one head), :366-424 (heads sharing S and F).
#include <type_traits>

#include "sa_tc_fwd.cuh"

namespace sa {
namespace tc {
namespace {

constexpr int kTile = 128;          // query rows per CTA; also the carry checkpoint spacing
constexpr int kRowTile = 16384;     // bytes of a [128][64] bf16 operand tile
constexpr int kThreads = 512;       // two softmax warpgroups, the selection, four single warps (one idle)
constexpr int kRing = 3;
// Registers: 512 x 128 at launch; the softmax keeps 128 logits: 256 x 176 + 256 x 80.
constexpr int kSoftmaxRegs = 176, kOtherRegs = 80;

struct PairSmem {
  static constexpr int q = 0;                              // Q of the two heads, Q0
  static constexpr int tri = q + 3 * kRowTile;             // [128][128] ones below the diagonal: two K-major tiles
  static constexpr int sel = tri + 2 * kRowTile;           // [128 queries][128 keys] bf16 as two key tiles
  static constexpr int k = sel + 2 * kRowTile;
  static constexpr int v = k + kRing * kRowTile;
  static constexpr int k0 = v + kRing * kRowTile;
  static constexpr int total = k0 + kRowTile;              // 224 KB
};
constexpr uint32_t kS = 0, kF = 256, kO = 384;             // TMEM columns: S of head x at 128 x, O at kO + 64 x

template <bool LIVE>
__global__ void __launch_bounds__(kThreads, 1) forward_pair_kernel(
    const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
    const __grid_constant__ CUtensorMap map_v, const __grid_constant__ CUtensorMap map_q0,
    const __grid_constant__ CUtensorMap map_k0, const float* __restrict__ carry, float* __restrict__ out,
    float* __restrict__ lse2, int heads, int seq, int ntiles, int exempt, float scale, const __grid_constant__ WaitCtx status,
    __nv_bfloat16* __restrict__ out_lowp, RowLayout out_lowp_rows, int q_offset, const uint8_t* __restrict__ alive) {
  using L = PairSmem;
  constexpr int D = 64;
  const int npairs = gridDim.x / (ntiles - q_offset / kTile);  // batch * heads / 2 (the grid covers the query tiles with rows to compute)
  const int mi = ntiles - 1 - (int)(blockIdx.x / npairs);      // heaviest query tiles first
  const int n0 = 2 * (int)(blockIdx.x % npairs);               // the pair's first (batch, head) row
  const int b = n0 / heads, h0 = n0 - b * heads;
  const int i0 = mi * kTile;

  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = smem_raw;                                    // 1024-byte aligned: the static part is rounded up to it
  // Completion barriers: QF the query tiles; LDK, LDV, LDK0 loads; FREEK, FREEV the MMA that read a slot; SF S of a head's
  // step (and P V of the step before); L0F, FF the selection's products; OF the last P V of a head.  Arrival barriers (one
  // arrival per warp): SELW selection and carry written; FREAD F read (both heads); PW P written and O rescaled.
  enum : int { QF = 0, LDK0 = 1, L0F = 2, FF = 3, SELW = 4, FREAD = 5, SF = 6, PW = 8, OF = 10, LDK = 12, FREEK = 15, LDV = 18,
               FREEV = 21, kBars = 24 };
  __shared__ uint64_t bars[kBars];
  __shared__ uint32_t tmem_base_s;
  __shared__ __align__(16) float carry_s[kTile];
  __shared__ unsigned live_s[LIVE ? kMaxLiveTiles / 32 : 1];   // with a table of live tiles: bit nj of this query tile's row
  __shared__ int live_count_s;

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (LIVE && warp == 1) {                                     // live in either head (in the other one the step adds zeros)
    const uint8_t* row_a = alive + ((int64_t)n0 * ntiles + mi) * ntiles;
    const uint8_t* row_b = row_a + (int64_t)ntiles * ntiles;
    int cnt = 0;
    for (int base = 0; base <= mi; base += 32) {
      const int nj = base + lane;
      const unsigned m = __ballot_sync(0xffffffffu, nj <= mi && (row_a[nj] != 0 || row_b[nj] != 0));
      if (lane == 0) live_s[base >> 5] = m;
      cnt += __popc(m);
    }
    if (lane == 0) live_count_s = cnt;
  }
  if (tid == 0) {
    for (int u = 0; u < kBars; ++u) mbar_init(&bars[u], u == FREAD ? 8 : (u == SELW || u == PW || u == PW + 1) ? 4 : 1);
    mbar_init_fence();
  }
  if (warp == 0) tmem_alloc(&tmem_base_s, 512);
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t sa = smem_u32(smem), bar0 = smem_u32(bars);
  auto bar = [&](int id) { return bar0 + 8u * (uint32_t)id; };
  Waiter wait;
  wait.begin(status);
  const int steps = LIVE ? live_count_s : mi + 1;              // step 0 is the diagonal tile
  auto step_back = [&](int nj) {                               // the key tile of the step after the one of tile nj
    if (!LIVE) return nj - 1;
    int w = nj >> 5;
    unsigned m = live_s[w] & ((1u << (nj & 31)) - 1u);
    while (m == 0u && w > 0) m = live_s[--w];
    return m != 0u ? 32 * w + 31 - __clz(m) : 0;
  };
  auto arrive = [&](int id) {
    __syncwarp();
    if (lane == 0) mbar_arrive(bar(id));
  };

  if (warp >= 8) {
    regs_shrink<kOtherRegs>();
    auto at = [](uint32_t low, uint32_t byte_off) { return low + (byte_off >> 4); };
    auto await = [&](int id, uint32_t parity, int site) { wait.left = wait_call(bar(id), parity, site, wait.left); };
    const uint32_t kBase = desc_low(sa, 16);                   // K-major views (rows = M or N index)
    const uint32_t mBase = desc_low(sa, kRowTile);             // MN-major views (rows = K index)
    struct Ring { uint32_t slot, par; };
    auto next = [](Ring& x) {
      if (++x.slot == kRing) { x.slot = 0; x.par ^= 1u; }
    };
    if (warp == 13) {
      // ============================================ TMA loads =============================================
      if (lane == 0) {
        auto load = [&](int off, const CUtensorMap* map, int id, int row, int head) {
          mbar_expect_tx(&bars[id], kRowTile);
          tma_load_4d(smem + off, map, &bars[id], 0, row, head, b);
        };
        mbar_expect_tx(&bars[QF], 3 * kRowTile);
        tma_load_4d(smem + L::q + 2 * kRowTile, &map_q0, &bars[QF], 0, i0 - q_offset, 0, b);
        tma_load_4d(smem + L::q, &map_q, &bars[QF], 0, i0 - q_offset, h0, b);
        tma_load_4d(smem + L::q + kRowTile, &map_q, &bars[QF], 0, i0 - q_offset, h0 + 1, b);
        load(L::k0, &map_k0, LDK0, i0, 0);
        // Tile n of the K and V rings: step n / 2 of head n & 1.  K runs one tile ahead of V.
        const int tiles = 2 * steps;
        int nj_k = mi, nj_v = mi, nj_k0 = mi;
        Ring rk{0, 1}, rv{0, 1};                               // par: of the freeing before the fill (the first three wait for none)
#pragma unroll 1
        for (int n = 0; n <= tiles; ++n) {
          if (n < tiles) {
            if (n >= kRing) wait(bar(FREEK + (int)rk.slot), rk.par, 501);
            load(L::k + rk.slot * kRowTile, &map_k, LDK + (int)rk.slot, nj_k * kTile, h0 + (n & 1));
            next(rk);
            if (n & 1) nj_k = step_back(nj_k);
          }
          if (n > 0) {
            if (n - 1 >= kRing) wait(bar(FREEV + (int)rv.slot), rv.par, 502);
            load(L::v + rv.slot * kRowTile, &map_v, LDV + (int)rv.slot, nj_v * kTile, h0 + ((n - 1) & 1));
            next(rv);
            if (!(n & 1)) nj_v = step_back(nj_v);
          }
          if ((n & 1) && (n >> 1) + 1 < steps) {               // K0 of the next step, once this step's L0 is done
            wait(bar(L0F), (uint32_t)((n >> 1) & 1), 503);
            nj_k0 = step_back(nj_k0);
            load(L::k0, &map_k0, LDK0, nj_k0 * kTile, 0);
          }
        }
      }
      __syncwarp();
    } else if (warp == 12) {
      // ============================ MMAs of the heads: S, and O += P V ====================================
      const uint32_t idesc_s = instr_desc_bf16(128, 128, false, false), idesc_pv = instr_desc_bf16(128, D, false, true);
      Ring rk{0, 0}, rv{0, 0};
      auto issue_s = [&](uint32_t x) {
        await(LDK + (int)rk.slot, rk.par, 511);
        if (elect_one()) {
          const uint32_t ql = at(kBase, L::q + x * kRowTile), kl = at(kBase, L::k + rk.slot * kRowTile);
          mma_ss_low<false>(kS + 128 * x, ql, kl, idesc_s);
#pragma unroll
          for (int ks = 1; ks < 4; ++ks) mma_ss_low<true>(kS + 128 * x, at(ql, ks * 32), at(kl, ks * 32), idesc_s);
          mma_commit(bar(SF + (int)x));
          mma_commit(bar(FREEK + (int)rk.slot));
        }
        __syncwarp();
        next(rk);
      };
      await(QF, 0, 510);
#pragma unroll 1
      for (uint32_t x = 0; x < 2; ++x) issue_s(x);
#pragma unroll 1
      for (int n = 0; n < 2 * steps; ++n) {
        const uint32_t x = (uint32_t)(n & 1);
        const int t = n >> 1;
        await(LDV + (int)rv.slot, rv.par, 512);
        await(PW + (int)x, (uint32_t)(t & 1), 513);            // P written, O rescaled
        if (elect_one()) {
          const uint32_t vl = at(mBase, L::v + rv.slot * kRowTile);
#pragma unroll
          for (int ks = 0; ks < 8; ++ks)
            mma_ts_low(kO + 64 * x, kS + 128 * x + ks * 8, at(vl, ks * 2048), idesc_pv, (t > 0 || ks > 0) ? 1u : 0u);
          mma_commit(bar(FREEV + (int)rv.slot));
          if (t + 1 == steps) mma_commit(bar(OF + (int)x));
        }
        __syncwarp();
        next(rv);
        if (t + 1 < steps) issue_s(x);                         // over P, which the MMAs before it read
      }
    } else if (warp == 14) {
      // ============================ MMAs of the selection: L0, and F = -TRI x selection ====================
      const uint32_t idesc_s = instr_desc_bf16(128, 128, false, false);
      const uint32_t idesc_tri = instr_desc_bf16(128, 128, false, true, /*negate_a=*/true);
      await(QF, 0, 520);
#pragma unroll 1
      for (int t = 0; t < steps; ++t) {
        if (t > 0) await(FREAD, (uint32_t)((t - 1) & 1), 521); // both heads have read F of the step before
        await(LDK0, (uint32_t)(t & 1), 522);
        if (elect_one()) {
          const uint32_t ql = at(kBase, L::q + 2 * kRowTile), kl = at(kBase, L::k0);
          mma_ss_low<false>(kF, ql, kl, idesc_s);
#pragma unroll
          for (int ks = 1; ks < 4; ++ks) mma_ss_low<true>(kF, at(ql, ks * 32), at(kl, ks * 32), idesc_s);
          mma_commit(bar(L0F));
        }
        __syncwarp();
        await(SELW, (uint32_t)(t & 1), 523);                   // L0 read, the selection in shared memory
        if (elect_one()) {
          mma_ss_low<false>(kF, at(kBase, L::tri), at(mBase, L::sel), idesc_tri);
#pragma unroll
          for (int ks = 1; ks < 8; ++ks)
            mma_ss_low<true>(kF, at(kBase, L::tri + (ks >> 2) * kRowTile + (ks & 3) * 32), at(mBase, L::sel + ks * 2048), idesc_tri);
          mma_commit(bar(FF));
        }
        __syncwarp();
      }
    } else if (warp < 12) {
      // ================================= selection: relu(L0) under the mask, the carry ========================
      const int row = tid & 127;                               // query row; also the key whose carry this thread fetches
      const uint32_t lane_base = (uint32_t)((warp & 3) * 32) << 16;
      const uint32_t row_off = (uint32_t)(row * 128 + ((row & 7) << 4));   // 16-byte chunk x of this row is at ^ 16 x
#pragma unroll 1
      for (int chunk = 0; chunk < 16; ++chunk) {               // strictly-lower-triangular ones TRI[i][r] = 1 for r < i
        uint32_t w[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int r = chunk * 8 + 2 * e;
          w[e] = pack_bf16(r < row ? 1.f : 0.f, (r + 1) < row ? 1.f : 0.f);
        }
        st_shared16(sa + L::tri + (chunk >> 3) * kRowTile + (row_off ^ (uint32_t)((chunk & 7) << 4)), w[0], w[1], w[2], w[3]);
      }
      const float* carry_row = carry + ((int64_t)b * (ntiles + 1) + mi) * seq;
      auto fetch_carry = [&](int nj) {
        const int j = nj * kTile + row;
        return j < seq ? load_ahead(carry_row + j) : 0.f;
      };
      int nj = mi;
      float next_carry = fetch_carry(nj);
      const int i = i0 + row;
#pragma unroll 1
      for (int t = 0; t < steps; ++t) {
        const int j0 = nj * kTile;
        const bool masked = t == 0 || j0 < exempt;
        wait(bar(L0F), (uint32_t)(t & 1), 530);
        tc_fence_after_sync();
        uint32_t r[2][16];                                     // 16 columns are converted while the next 16 arrive
        tmem_ld16(lane_base + kF, r[0]);
        carry_s[row] = -next_carry * kLog2e;                   // negated: the softmax adds it in an FMA (both heads have read the
                                                               //   last one, with F: L0 came after that)
#pragma unroll
        for (int c = 0; c < 8; ++c) {
          uint32_t* cur = r[c & 1];
          tmem_ld_wait();
          if (c + 1 < 8) tmem_ld16(lane_base + kF + 16 * (c + 1), r[(c + 1) & 1]);
          if (masked) {
#pragma unroll
            for (int e = 0; e < 16; ++e) {
              const int j = j0 + 16 * c + e;
              if (!(j < i && j >= exempt)) cur[e] = 0u;
            }
          }
#pragma unroll
          for (int u = 0; u < 2; ++u) {                        // the relu rides on the bf16 conversion
            uint32_t w[4];
#pragma unroll
            for (int e = 0; e < 4; ++e)
              w[e] = pack_bf16_relu(__uint_as_float(cur[8 * u + 2 * e]), __uint_as_float(cur[8 * u + 2 * e + 1]));
            const uint32_t chunk = (uint32_t)(((c & 3) * 2 + u) << 4);
            st_shared16(sa + L::sel + (c >> 2) * kRowTile + (row_off ^ chunk), w[0], w[1], w[2], w[3]);
          }
        }
        fence_async_smem();
        tc_fence_before_sync();
        arrive(SELW);
        if (t + 1 < steps) {                                   // the next step's carry arrives while its L0 is awaited
          nj = step_back(nj);
          next_carry = fetch_carry(nj);
        }
      }
    }
  } else {
    regs_grow<kSoftmaxRegs>();
    // ========================================= softmax of one head =============================================
    const int x = warp >> 2, row = tid & 127;
    const uint32_t lane_base = (uint32_t)((warp & 3) * 32) << 16;
    const uint32_t s_cols = lane_base + kS + 128 * x, o_cols = lane_base + kO + 64 * x;
    const uint32_t carry_base = smem_u32(carry_s);
    const float c1 = scale * kLog2e;
    const float2 cc = make_float2(c1, c1);
    const int i = i0 + row;
    float run_max = -INFINITY, run_den = 0.f;
    auto step = [&](int t, auto first_tag) {
      constexpr bool kFirst = decltype(first_tag)::value;      // the diagonal tile: causal mask inside it, nothing to rescale yet
      const uint32_t ph = (uint32_t)(t & 1);
      // ---- the history part of the logits, F * scale - carry in log2 units, as soon as F is there and not when S is: the next
      // step's selection starts when both heads have it (packed fp32x2 arithmetic throughout)
      float2 z[64];
      wait(bar(SELW), ph, 540);                                // (complete: F came after it) the carry of the step's keys
      wait(bar(FF), ph, 542);
      tc_fence_after_sync();
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        uint32_t f[32];
        tmem_ld32(lane_base + kF + 32 * c, f);
        tmem_ld_wait();
#pragma unroll
        for (int e4 = 0; e4 < 32; e4 += 4) {
          const float4 nc = ld_shared_f4(carry_base + 4 * (32 * c + e4));
          float2* zz = &z[16 * c + (e4 >> 1)];
          zz[0] = __ffma2_rn(make_float2(__uint_as_float(f[e4]), __uint_as_float(f[e4 + 1])), cc, make_float2(nc.x, nc.y));
          zz[1] = __ffma2_rn(make_float2(__uint_as_float(f[e4 + 2]), __uint_as_float(f[e4 + 3])), cc, make_float2(nc.z, nc.w));
        }
      }
      tc_fence_before_sync();
      arrive(FREAD);                                           // F may take the next step's L0, carry_s its carry
      // ---- logits and the row maximum -------------------------------------------------------------------------------
      wait(bar(SF + x), ph, 541);
      tc_fence_after_sync();
      float tile_max = -INFINITY;
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        uint32_t s[32];
        tmem_ld32(s_cols + 32 * c, s);
        tmem_ld_wait();
#pragma unroll
        for (int e = 0; e < 16; ++e) {
          float2 a = __ffma2_rn(make_float2(__uint_as_float(s[2 * e]), __uint_as_float(s[2 * e + 1])), cc, z[16 * c + e]);
          if (kFirst) {
            const int j = 32 * c + 2 * e;                      // key and query count from the same position
            if (j > row) a.x = -INFINITY;
            if (j + 1 > row) a.y = -INFINITY;
          }
          tile_max = fmaxf(tile_max, fmaxf(a.x, a.y));
          z[16 * c + e] = a;
        }
      }
      // every row has its own key in the diagonal tile, so the maximum is finite from the first step on
      const float new_max = fmaxf(run_max, tile_max);
      const float alpha = ex2(run_max - new_max);
      run_max = new_max;
      // ---- exponentials, P as bf16 pairs over the S columns that have been read ----------------------------------------
      // Four sums: with one, its additions and the exponentials form a chain (31 cycles a pair instead of 18 when the warp has
      // the scheduler to itself).
      float2 sum[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) sum[e] = make_float2(0.f, 0.f);
      const float2 nm = make_float2(-new_max, -new_max);
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        uint32_t w[32];
#pragma unroll
        for (int e = 0; e < 32; ++e) {
          const float2 y = __fadd2_rn(z[32 * c + e], nm);
          const float2 p = make_float2(ex2(y.x), ex2(y.y));
          sum[e & 3] = __fadd2_rn(sum[e & 3], p);
          w[e] = pack_bf16(p.x, p.y);
        }
        tmem_st32(s_cols + 32 * c, w);
      }
      const float2 s2 = __fadd2_rn(__fadd2_rn(sum[0], sum[1]), __fadd2_rn(sum[2], sum[3]));
      run_den = run_den * alpha + (s2.x + s2.y);
      // the accumulator follows the maximum while it moves (P V of the step before is done: this step's S came after it)
      if (!kFirst && __any_sync(0xffffffffu, alpha != 1.f)) {
#pragma unroll 1
        for (int c = 0; c < 4; ++c) {
          uint32_t r[16];
          tmem_ld16(o_cols + 16 * c, r);
          tmem_ld_wait();
#pragma unroll
          for (int e = 0; e < 16; ++e) r[e] = __float_as_uint(__uint_as_float(r[e]) * alpha);
          tmem_st16(o_cols + 16 * c, r);
        }
      }
      tmem_st_wait();
      tc_fence_before_sync();
      arrive(PW + x);
    };
    step(0, std::true_type{});
#pragma unroll 1
    for (int t = 1; t < steps; ++t) step(t, std::false_type{});

    wait(bar(OF + x), 0, 543);                                 // the last P V
    tc_fence_after_sync();
    const float inv = 1.f / run_den;
    const int iq = i - q_offset, q_rows = seq - q_offset;      // row inside the query tensor
    const bool mine = i < seq && i >= q_offset;                // rows before q_offset belong to an earlier call
    const int64_t n = n0 + x;
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      uint32_t r[32];
      tmem_ld32(o_cols + 32 * c, r);
      tmem_ld_wait();
      float o[32];
#pragma unroll
      for (int e = 0; e < 32; ++e) o[e] = __uint_as_float(r[e]) * inv;
      if (mine) {
        float* orow = out + (n * q_rows + iq) * D + 32 * c;
#pragma unroll
        for (int e = 0; e < 32 && out != nullptr; e += 4) *reinterpret_cast<float4*>(orow + e) = make_float4(o[e], o[e + 1], o[e + 2], o[e + 3]);
        if (out_lowp != nullptr) {                             // the same rows in the operand dtype, in the caller's layout
          uint4* lrow = reinterpret_cast<uint4*>(out_lowp + out_lowp_rows.at(b, h0 + x, iq) + 32 * c);
#pragma unroll
          for (int e = 0; e < 32; e += 8)
            lrow[e >> 3] = make_uint4(pack_bf16(o[e], o[e + 1]), pack_bf16(o[e + 2], o[e + 3]), pack_bf16(o[e + 4], o[e + 5]),
                                      pack_bf16(o[e + 6], o[e + 7]));
        }
      }
    }
    if (mine) lse2[n * q_rows + iq] = run_max + log2f(run_den);
  }
  wait.end(status);
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tmem_base_s, 512);
}

}  // namespace

int forward_pair(const Problem& p, const ForwardMaps& m, const float* carry, float* out, float* lse2, const WaitCtx& status,
                 const uint8_t* alive, cudaStream_t s) {
  const int ntiles = (p.seq + kTile - 1) / kTile;
  const unsigned grid = (unsigned)(ntiles - p.q_offset / kTile) * p.batch * (p.heads / 2);
  const int smem = PairSmem::total;
  auto launch = [&](auto kernel) -> int {
    SA_CUDA_CHECK(allow_smem(kernel, smem));
    ProfileScope prof(SA_KERNEL_TC_FORWARD, s);
    count_launch();
    kernel<<<grid, kThreads, smem, s>>>(m.q, m.k, m.v, m.q0, m.k0, carry, out, lse2, p.heads, p.seq, ntiles, p.exempt, p.scale,
                                        status, static_cast<__nv_bfloat16*>(p.out_lowp), p.out_lowp_rows, p.q_offset, alive);
    SA_CUDA_CHECK(cudaGetLastError());
    return SA_OK;
  };
  return alive != nullptr ? launch(forward_pair_kernel<true>) : launch(forward_pair_kernel<false>);
}

}  // namespace tc
}  // namespace sa
