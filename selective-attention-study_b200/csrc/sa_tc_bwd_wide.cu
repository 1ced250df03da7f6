// Tensor-core engine, backward at head_dim 128 (sm_100a: TMA loads, tcgen05 MMAs, fp32 accumulators in TMEM).
//
// The scheme is the one of sa_tc_bwd.cu: one 128-key tile of one head, query tiles walked last to first, the upper and the
// lower 64-query halves as two chains of a warpgroup each, score-shaped tiles transposed with KEYS on the TMEM lanes, P^T /
// dz^T / g^T consumed from TMEM.  At head_dim 128 the three per-key accumulators alone (dV, dK, dK0: 128 fp32 columns each)
// and the score tiles of two chains would need 640 of the 512 TMEM columns, so TWO CTAs share a (head, key tile), one per
// 64-wide half `dh` of the head dimension:
//   * both compute the full-depth score products (8 MMAs of K = 16 each: S^T, dP^T, L0^T) and the whole arithmetic,
//   * each accumulates only its own 64 columns of dV, dK, dK0 (B operand: the `dh` box of dO, Q, Q0),
//   * the query-side gradients are computed TRANSPOSED per half, d on the lanes: dQ^T = K^T dz^T (CTA dh = 0) and
//     dQ0^T = K0^T g^T (CTA dh = 1), M = 128 = the full head dimension, N = 64 queries, K = 128 keys, so the two CTAs
//     split that work instead of repeating it, each keeps only ONE of the dz / g tiles in shared memory, and the result is
//     staged over that half tile on its way to the TMA reduce-add.  One head per selector: dQ^T = K^T (dz + g)^T, the CTAs take one chain's halves each.
// TMEM, 512 columns: dV | dK | dQ^T | W1, W2 of the two chains | dK0 (64 each; one head per selector: V as bf16 pairs, A of
// dP^T).  Shared memory: K, V, K0 32 KB each, dz-or-g 32 KB, two slots of (Q, dO, Q0) half tiles, 48 KB each: all 227 KB with
// the statistics (one head per selector: no K0 and Q0, three slots of (Q, dO)).  What a half frees at its dz takes what the
// chain's next half needs first (Q0, Q), what it frees at g the rest (dO): no load is waited for.
//
// What bounds it: shared memory, 688 KB a CTA and 128 x 128 tile = 5.5 k cycles (score operands 288, dQ^T staged and reduced 128,
// its operands 96, loads 96, B operands of the accumulators 48, dz or g written 32); a tile takes 6.4 k (one head per
// selector 4.9 k).  Measured at B = 2, H = 8, T = 4097: 817 us
// with sixteen warps in lock step and reductions from registers, 553 us.
//
// Reference for the arithmetic: src/selective_attention/kernels.py:196-268 (one head), :271-364 (the shared
// selection-gradient products); head_dim 128 in the reference's tests: tests/test_selective_kernels.py:159-172.
#include "sa_tc_bwd_chain.cuh"

namespace sa {
namespace tc {
namespace {

using namespace bwd;

constexpr int kOpTile = 2 * kHalfTile;   // a [64 queries][128] bf16 operand half tile: two 64-column boxes

template <bool SELF>
struct Layout {
  static constexpr int kRing = SELF ? 3 : 2;                // half tiles of Q, dO (and Q0) in flight
  static constexpr int kSlot = (SELF ? 2 : 3) * kOpTile;
  static constexpr int k = 0;                               // [128 keys][128] as two 64-column boxes, stationary
  static constexpr int v = k + 2 * kRowTile;
  static constexpr int k0 = v + 2 * kRowTile;
  static constexpr int t = SELF ? k0 : k0 + 2 * kRowTile;   // dz or g (one head per selector: dz + g): [128 keys][2 x 64 queries]
  static constexpr int ring = t + 2 * kRowTile;
  static constexpr int stat = ring + kRing * kSlot;
  static constexpr int total = stat + kRing * kStatBytes;
  // One head per selector: slot `x` holds Q, then dO.  Otherwise chain c owns three tiles whose roles rotate from tile to
  // tile (`turn` = tile mod 3): the two that dz frees take the next Q0 and Q, the one that g frees the next dO.
  static __device__ __forceinline__ uint32_t q0(uint32_t c, uint32_t turn) { return ring + c * kSlot + turn * kOpTile; }
  static __device__ __forceinline__ uint32_t q(uint32_t x, uint32_t turn) {
    return ring + x * kSlot + (SELF ? 0u : (turn == 2 ? 0u : turn + 1) * kOpTile);
  }
  static __device__ __forceinline__ uint32_t d_out(uint32_t x, uint32_t turn) {
    return ring + x * kSlot + (SELF ? 1u : (turn == 0 ? 2u : turn - 1)) * kOpTile;
  }
};

// TMEM columns (W1, W2: sa_tc_bwd_chain.cuh)
constexpr uint32_t kDV = 0, kDK = 64, kDQT = 128, kDK0 = 448, kVA = 448;

// LIVE: a table of live tiles is given (sa_tc_skip.cu).  ANY: rows of dk, dv that are not 16-byte aligned.
template <bool SELF, bool LIVE, bool ANY>
__global__ void __launch_bounds__(kThreads, 1) backward_wide_kernel(
    const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
    const __grid_constant__ CUtensorMap map_v, const __grid_constant__ CUtensorMap map_do,
    const __grid_constant__ CUtensorMap map_q0, const __grid_constant__ CUtensorMap map_k0,
    const __grid_constant__ CUtensorMap map_dq, const __grid_constant__ CUtensorMap map_dq0,
    const float* __restrict__ stats, const float* __restrict__ carry, int dq0_rows,
    __nv_bfloat16* __restrict__ dk, float* __restrict__ dk0, __nv_bfloat16* __restrict__ dv, int heads, int seq, int ntiles,
    int exempt, float scale, const __grid_constant__ WaitCtx status, RowLayout dk_rows, RowLayout dv_rows,
    const uint8_t* __restrict__ alive) {
  using L = Layout<SELF>;
  constexpr int D = 128, R = L::kRing;
  // Consecutive CTAs: the two halves of the head dimension of one (row, key tile), then the row's next key tile, so
  // the CTAs resident at one time walk the same query tiles and share them through L2.
  const int dh = (int)(blockIdx.x & 1);
  int n, nj;
  tile_of_block(blockIdx.x >> 1, ntiles, (gridDim.x >> 1) / ntiles, LIVE, n, nj);
  const int b = n / heads, h = n - b * heads;

  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = smem_raw;                       // 1024-byte aligned: the static part is rounded up to it
  __shared__ uint64_t bars[kBars];                // (per chain here: DQ + chain)
  __shared__ uint32_t tmem_base_s;
  __shared__ float run_s[kTile], sel_s[2 * kTile];
  __shared__ int top_s;

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (LIVE && warp == 1) find_top_tile(alive, n, nj, ntiles, lane, &top_s);
  if (tid == 0) init_bars(bars);
  if (tid < kTile) run_s[tid] = 0.f;
  if (warp == 0) tmem_alloc(&tmem_base_s, 512);
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t sa = smem_u32(smem), bar0 = smem_u32(bars);
  auto bar = [&](int id) { return bar0 + 8u * (uint32_t)id; };
  Waiter wait;
  wait.begin(status);
  const int mi_top = LIVE ? top_s : ntiles - 1;   // the walk starts at the last query tile, or at the last live one
  const int n_iter = mi_top - nj + 1;
  const int n_half = 2 * n_iter;                  // half hn: tile mi_top - hn / 2, chain hn & 1 (chain 0: the upper half)

  if (warp >= 8) {
    regs_shrink<kOtherRegs>();
    if (warp == kLoadWarp) {
      // ========================================== TMA loads ================================================
      if (lane == 0) {
        auto row_of = [&](int hn) { return (mi_top - (hn >> 1)) * kTile + (1 - (hn & 1)) * 64; };
        auto load = [&](uint32_t off, const CUtensorMap* map, int id, int row0, int head) {
          for (int x = 0; x < 2; ++x) tma_load_4d(smem + off + x * kHalfTile, map, &bars[id], 64 * x, row0, head, b);
        };
        auto load_stat = [&](int slot, int row0) {
          bulk_load(smem + L::stat + slot * kStatBytes, stats + ((int64_t)n * 2 * ntiles + (row0 >> 6)) * (kStatBytes / 4), kStatBytes,
                    &bars[LD + slot]);
        };
        mbar_expect_tx(&bars[KV], (SELF ? 4 : 6) * kRowTile);
        for (int x = 0; x < 2; ++x) {
          if (!SELF) tma_load_4d(smem + L::k0 + x * kRowTile, &map_k0, &bars[KV], 64 * x, nj * kTile, 0, b);
          tma_load_4d(smem + L::k + x * kRowTile, &map_k, &bars[KV], 64 * x, nj * kTile, h, b);
          tma_load_4d(smem + L::v + x * kRowTile, &map_v, &bars[KV], 64 * x, nj * kTile, h, b);
        }
        if constexpr (SELF) {
          int slot = 0;
          uint32_t par = 1;                                        // of the freeing before this fill (the first fills wait for none)
#pragma unroll 1
          for (int hn = 0; hn < n_half; ++hn) {
            if (hn >= R) wait(bar(FREE + slot), par, 442);
            const int row0 = row_of(hn);
            mbar_expect_tx(&bars[LD + slot], 2 * kOpTile + kStatBytes);
            load(L::q(slot, 0), &map_q, LD + slot, row0, h);
            load(L::d_out(slot, 0), &map_do, LD + slot, row0, h);
            load_stat(slot, row0);
            if (++slot == R) { slot = 0; par ^= 1u; }
          }
        } else {
          // Tiles come free in the order dz, g of one half, then of the next.
          uint32_t turn = 0;
#pragma unroll 1
          for (int hn = 0; hn < n_half; ++hn) {
            const int c = hn & 1, row0 = row_of(hn);
            const uint32_t par = (uint32_t)((hn >> 1) & 1) ^ 1u;   // of the freeing before this fill (at first it passes)
            wait(bar(FREE + c), par, 442);
            mbar_expect_tx(&bars[LD0 + c], kOpTile);
            load(L::q0(c, turn), &map_q0, LD0 + c, row0, 0);
            mbar_expect_tx(&bars[LD + c], kOpTile + kStatBytes);
            load(L::q(c, turn), &map_q, LD + c, row0, h);
            load_stat(c, row0);
            wait(bar(FREE0 + c), par, 443);
            mbar_expect_tx(&bars[LD + 2 + c], kOpTile);
            load(L::d_out(c, turn), &map_do, LD + 2 + c, row0, h);
            if (c == 1 && ++turn == 3) turn = 0;
          }
        }
      }
      __syncwarp();
    } else if (warp >= 12) {
      // ========================================== MMA issue ================================================
      // A whole warp walks this code and one elected lane issues; the warps as in sa_tc_bwd.cu.
      const uint32_t idesc_t = instr_desc_bf16(128, 64, false, false);     // keys x 64 queries, K = D
      const uint32_t idesc_acc = instr_desc_bf16(128, 64, false, true);    // A K-major (keys x queries), B MN-major
      const uint32_t idesc_dq = instr_desc_bf16(128, 64, true, true);      // A MN-major (d x keys), B MN-major (keys x queries)
      const uint32_t kBase = desc_low(sa, 16);                             // K-major views (rows = M or N index)
      const uint32_t mBase = desc_low(sa, kRowTile);                       // MN-major views (rows = K index)
      auto at = [](uint32_t low, uint32_t byte_off) { return low + (byte_off >> 4); };
      const int halves = 2 * (LIVE ? __shfl_sync(0xffffffffu, n_iter, 0) : n_iter);
      auto await = [&](int id, uint32_t parity, int site) { wait.left = wait_call(bar(id), parity, site, wait.left); };
      // d (64 columns) = A x B over eight K steps of 16: operands of two 64-column boxes, A from shared memory or from TMEM
      auto product = [&](uint32_t d, bool from_tmem, uint32_t a_at, uint32_t b_off, int done) {
        if (elect_one()) {
          const uint32_t bl = at(kBase, b_off);
          auto kstep = [](int ks, int box) { return (uint32_t)((ks >> 2) * box + (ks & 3) * 32); };
          if (from_tmem) {
#pragma unroll
            for (int ks = 0; ks < 8; ++ks) mma_ts_low(d, a_at + ks * 8, at(bl, kstep(ks, kHalfTile)), idesc_t, ks > 0 ? 1u : 0u);
          } else {
            mma_ss_low<false>(d, at(kBase, a_at), bl, idesc_t);
#pragma unroll
            for (int ks = 1; ks < 8; ++ks)
              mma_ss_low<true>(d, at(kBase, a_at + kstep(ks, kRowTile)), at(bl, kstep(ks, kHalfTile)), idesc_t);
          }
          mma_commit(bar(done));
        }
        __syncwarp();
      };
      auto issue_s = [&](uint32_t c, uint32_t q_off) { product(w2_of(c), false, L::k, q_off, S + (int)c); };
      auto issue_dp = [&](uint32_t c, uint32_t do_off) {
        product(w1_of(c), SELF, SELF ? kVA : (uint32_t)L::v, do_off, DP + (int)c);
      };
      // acc (64 columns) += A (TMEM, 16 queries are 8 packed columns) x this CTA's box of the half tile at `off`
      auto accumulate = [&](uint32_t acc, uint32_t a_col, uint32_t off, uint32_t keep) {
        const uint32_t rows = at(mBase, off + dh * kHalfTile);
#pragma unroll
        for (int ks = 0; ks < 4; ++ks) mma_ts_low(acc, a_col + ks * 8, at(rows, ks * 2048), idesc_acc, ks > 0 ? 1u : keep);
      };
      struct Ring { uint32_t slot, par; };
      auto next = [](Ring& x) {
        if (++x.slot == R) { x.slot = 0; x.par ^= 1u; }
      };
      auto next_turn = [](uint32_t& turn, uint32_t c) {
        if (c == 1 && ++turn == 3) turn = 0;
      };
      await(SELF ? SETUP : KV, 0, 440);                                    // K, V (and K0) in place
      if (warp == kMmaWarp) {
        // -- the per-key accumulators, and the products whose columns they free: L0^T (SELF: S^T and dP^T) of the half after next
        Ring use{0, 0}, ahead{0, 0};                                       // SELF: slots
        uint32_t turn = 0, l0_turn = 0;
        int l0_half = 0;
        auto ask_l0 = [&](uint32_t c) {
          await(LD0 + (int)c, (uint32_t)((l0_half >> 1) & 1), 444);
          product(w1_of(c), false, L::k0, L::q0(c, l0_turn), L0 + (int)c);
          next_turn(l0_turn, c);
          ++l0_half;
        };
        auto ask_s = [&](uint32_t c) {
          await(LD + (int)ahead.slot, ahead.par, 445);
          issue_s(c, L::q(ahead.slot, 0));
        };
        auto ask_dp = [&](uint32_t c) {
          issue_dp(c, L::d_out(ahead.slot, 0));
          next(ahead);
        };
#pragma unroll 1
        for (uint32_t c = 0; c < 2; ++c) {
          if (SELF) ask_s(c), ask_dp(c);
          else ask_l0(c);
        }
#pragma unroll 1
        for (int hn = 0; hn < halves; ++hn) {
          const uint32_t c = (uint32_t)(hn & 1), ph = (uint32_t)((hn >> 1) & 1), keep = hn > 0 ? 1u : 0u;
          const uint32_t x = SELF ? use.slot : c;
          await(DZ + (int)c, ph, 446);                                     // P^T (and dz^T) written: dV, dK
          if (elect_one()) {
            accumulate(kDV, w2_of(c) + 32, L::d_out(x, turn), keep);
            if (!SELF) {
              accumulate(kDK, w2_of(c), L::q(x, turn), keep);
              mma_commit(bar(FREE + (int)c));
            }
          }
          __syncwarp();
          if (SELF && hn + 2 < halves) ask_s(c);
          await(G + (int)c, ph, 447);                                      // g^T written: dK0
          if (elect_one()) {
            if (SELF) {
              accumulate(kDK, w1_of(c), L::q(x, turn), keep);
              mma_commit(bar(FREE + (int)x));
            } else {
              accumulate(kDK0, w1_of(c), L::q0(c, turn), keep);
              mma_commit(bar(FREE0 + (int)c));
            }
          }
          __syncwarp();
          if (hn + 2 < halves) {
            if (SELF) ask_dp(c);
            else ask_l0(c);
          }
          next(use);
          next_turn(turn, c);
        }
        if (elect_one()) mma_commit(bar(FIN));
        __syncwarp();
      } else if (warp == kDqWarp) {
        // -- dQ^T = K^T dz^T, or dQ0^T = K0^T g^T, of a half: A = the stationary key-side tile seen transposed
        uint32_t acc_par = 1;                                              // of the read-out before (the first passes)
#pragma unroll 1
        for (int hn = SELF ? dh : 0; hn < halves; hn += SELF ? 2 : 1) {
          const uint32_t c = (uint32_t)(hn & 1);
          await((!SELF && dh == 0 ? DZ : G) + (int)c, (uint32_t)((hn >> 1) & 1), 448);
          await(ACC, acc_par, 449);
          acc_par ^= 1u;
          if (elect_one()) {
            const uint32_t a_off = (SELF || dh == 0) ? L::k : L::k0, b_off = L::t + (1 - c) * kRowTile;
            mma_ss_low<false>(kDQT, at(mBase, a_off), at(mBase, b_off), idesc_dq);
#pragma unroll
            for (int ks = 1; ks < 8; ++ks) mma_ss_low<true>(kDQT, at(mBase, a_off + ks * 2048), at(mBase, b_off + ks * 2048), idesc_dq);
            mma_commit(bar(DQ + (int)c));
          }
          __syncwarp();
        }
      } else if (!SELF && warp == kScoreWarp) {
        // -- dP^T of half hn when its L0^T has been read, S^T of half hn + 1 when dV, dK of half hn - 1 are done
        uint32_t s_turn = 0, dp_turn = 0;
        auto ask_s = [&](int hn) {
          const uint32_t c = (uint32_t)(hn & 1);
          await(LD + (int)c, (uint32_t)((hn >> 1) & 1), 445);
          issue_s(c, L::q(c, s_turn));
          next_turn(s_turn, c);
        };
        ask_s(0);
        ask_s(1);
#pragma unroll 1
        for (int hn = 0; hn < halves; ++hn) {
          const uint32_t c = (uint32_t)(hn & 1), ph = (uint32_t)((hn >> 1) & 1);
          await(SEL + (int)c, ph, 450);
          await(LD + 2 + (int)c, ph, 456);
          issue_dp(c, L::d_out(c, dp_turn));
          next_turn(dp_turn, c);
          if (hn > 0 && hn + 1 < halves) {
            await(FREE + (int)(c ^ 1u), (uint32_t)(((hn - 1) >> 1) & 1), 451);
            ask_s(hn + 1);
          }
        }
      }
    } else {
      // ============ read-out: the lane is d, a query column of a warp is 32 consecutive floats of its row ==========
      // Staged over the dz (or g) half tile that the product has just consumed, 32 queries at a time, a [32 queries][32 d]
      // box a warp, and reduce-added from there by TMA.  (Reductions from registers, 128 bytes a warp, took 25 cycles each:
      // 6.5 k a half, which is what bounded both this kernel and the form before it.)
      const uint32_t lane_base = (uint32_t)((warp & 3) * 32) << 16;
      const bool zero_path = !SELF && dh == 1;
      const CUtensorMap* map = zero_path ? &map_dq0 : &map_dq;
      const int grad_row = zero_path ? b * dq0_rows : n;
#pragma unroll 1
      for (int hn = SELF ? dh : 0; hn < n_half; hn += SELF ? 2 : 1) {
        const int c = hn & 1;
        const int i_first = (mi_top - (hn >> 1)) * kTile + (1 - c) * 64;
        uint8_t* stage = smem + L::t + (1 - c) * kRowTile + (warp - 8) * 4096;
        wait(bar(DQ + c), (uint32_t)((hn >> 1) & 1), 452);
        tc_fence_after_sync();
#pragma unroll 1
        for (int x = 0; x < 2; ++x) {
          uint32_t r[32];
          tmem_ld32(lane_base + kDQT + 32 * x, r);
          tmem_ld_wait();
          if (x == 1) {
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) {
              mbar_arrive(bar(ACC));                               // the accumulator may be overwritten
              bulk_wait_read();                                    // the first 32 queries have left
            }
            __syncwarp();
          }
          const uint32_t at = smem_u32(stage) + lane * 4;
#pragma unroll
          for (int e = 0; e < 32; ++e)
            asm volatile("st.shared.f32 [%0], %1;" ::"r"(at + e * 128), "f"(__uint_as_float(r[e]) * scale) : "memory");
          fence_async_smem();
          __syncwarp();
          if (lane == 0 && i_first + 32 * x < seq) {
            tma_reduce_add_4d(map, stage, (warp - 8) * 32, i_first + 32 * x, grad_row, 0);
            bulk_commit();
          }
        }
        if (lane == 0) {
          bulk_wait_read();
          mbar_arrive(bar(TFREE + c));                             // the half tile may be written again
        }
        __syncwarp();
      }
      if (lane == 0) bulk_wait_all();                              // the last reduce-adds must land before the CTA exits
      __syncwarp();
      if (!SELF) {                                                 // this head's share of dK0
        wait(bar(FIN), 0, 453);
        tc_fence_after_sync();
        const int j = nj * kTile + (warp - 8) * 32 + lane;
        float* row = dk0 + ((int64_t)b * seq + j) * D + dh * 64;
#pragma unroll 1
        for (int x = 0; x < 4; ++x) {
          uint32_t r0[16];
          tmem_ld16(lane_base + kDK0 + 16 * x, r0);
          tmem_ld_wait();
          if (j < seq) store_key_grads<false, 16, ANY>(nullptr, nullptr, r0, scale, nullptr, nullptr, row + 16 * x, false);
        }
      }
    }
  } else {
    regs_grow<kChainRegs>();
    // ============================================ the two chains ============================================
    const int c = warp >> 2, row = tid & 127;
    const uint32_t lane_base = (uint32_t)((warp & 3) * 32) << 16;      // a warp reaches lanes 32 (warp % 4) ..
    const int j = nj * kTile + row;
    Chain ch;
    ch.c = c; ch.row = row; ch.lane = lane; ch.j = j; ch.n_iter = n_iter;
    ch.w1 = lane_base + w1_of(c);
    ch.w2 = lane_base + w2_of(c);
    ch.bar0 = bar0;
    ch.stat0 = sa + L::stat;
    ch.dz_row = ch.g_row = sa + L::t + (1 - c) * kRowTile + row * 128 + ((row & 7) << 4);
    ch.keep_dz = dh == 0;                                          // one of the two goes to shared memory (SELF: dz + g, if
    ch.keep_g = SELF ? c == dh : dh == 1;                          //   this CTA computes the chain's dQ^T)
    ch.free_bar = (SELF && c != dh) ? G + c : TFREE + c;             // (nothing to wait for: the chain's own last half)
    ch.c1 = scale * kLog2e;
    ch.inv_scale = 1.f / scale;
    ch.shut = (j >= exempt) ? 0.f : -INFINITY;                     // an exempt key is never selected
    ch.carry = (j < seq) ? carry + ((int64_t)b * (ntiles + 1) + mi_top + 1) * seq + j : nullptr;
    ch.carry_step = seq;
    ch.run_s = run_s;
    ch.sel_s = sel_s;
    ch.slot = c;
    ch.ld_par = 0;
    ch.wait = wait;
    ch.fetch_carry();

    if (SELF) {                                                    // V rows into TMEM as bf16 pairs, a 64-column box each
      ch.wait(bar(KV), 0, 454);
      const uint8_t* src = smem + L::v + c * kRowTile;
      uint32_t w32[32];
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const uint4 v4 = *reinterpret_cast<const uint4*>(src + swz_off(row, u));
        w32[4 * u] = v4.x; w32[4 * u + 1] = v4.y; w32[4 * u + 2] = v4.z; w32[4 * u + 3] = v4.w;
      }
      tmem_st32(lane_base + kVA + 32 * c, w32);
      tmem_st_wait();
      tc_fence_before_sync();
      ch.arrive(SETUP);
    }
    for (int it = 0; it + 1 < n_iter; ++it) half_pass<SELF, false, R>(ch, it);
    half_pass<SELF, true, R>(ch, n_iter - 1);
    wait = ch.wait;

    // ---- epilogue: this CTA's 64 columns of dV (chain 0) and dK (chain 1) of the key tile ----------------------------
    wait(bar(FIN), 0, 455);
    tc_fence_after_sync();
#pragma unroll
    for (int x = 0; x < 2; ++x) {
      uint32_t r[32];
      tmem_ld32(lane_base + (c == 0 ? kDV : kDK) + 32 * x, r);
      tmem_ld_wait();
      if (j < seq) {
        const int col = dh * 64 + 32 * x;
        if (c == 0)
          store_key_grads<SELF, 32, ANY>(r, nullptr, nullptr, scale, dv + dv_rows.at(b, h, j) + col, nullptr, nullptr, false);
        else
          store_key_grads<SELF, 32, ANY>(nullptr, r, nullptr, scale, nullptr, dk + dk_rows.at(b, h, j) + col,
                                    dk0 + ((int64_t)b * seq + j) * D + col, SELF || (h == 0 && dq0_rows != 1));
      }
    }
  }
  wait.end(status);
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tmem_base_s, 512);
}

}  // namespace

int backward_wide(const Problem& p, const float* stats, const float* carry, const void* d_out, const RowLayout& d_out_rows,
                  float* dq_acc, float* dq0, float* dk0, void* dk, void* dv, cudaStream_t s) {
  if (p.head_dim != 128) return SA_ERR_UNSUPPORTED;
  const int ntiles = (p.seq + kTile - 1) / kTile;
  const int nrows = p.batch * p.heads;
  CUtensorMap map_q, map_k, map_v, map_do, map_q0, map_k0, map_dq, map_dq0;
  int st = make_map_16bit(&map_q, p.q.ptr, 128, p.seq, p.heads, p.batch, p.q.st, p.q.sh, p.q.sb, 64);
  if (st != SA_OK) return st;
  st = make_map_16bit(&map_k, p.k.ptr, 128, p.seq, p.heads, p.batch, p.k.st, p.k.sh, p.k.sb, kTile);
  if (st != SA_OK) return st;
  st = make_map_16bit(&map_v, p.v.ptr, 128, p.seq, p.heads, p.batch, p.v.st, p.v.sh, p.v.sb, kTile);
  if (st != SA_OK) return st;
  st = make_map_16bit(&map_do, d_out, 128, p.seq, p.heads, p.batch, d_out_rows.st, d_out_rows.sh, d_out_rows.sb, 64);
  if (st != SA_OK) return st;
  st = make_map_16bit(&map_q0, p.q0.ptr, 128, p.seq, 1, p.batch, p.q0.st, 0, p.q0.sb, 64);
  if (st != SA_OK) return st;
  st = make_map_16bit(&map_k0, p.k0.ptr, 128, p.seq, 1, p.batch, p.k0.st, 0, p.k0.sb, kTile);
  if (st != SA_OK) return st;
  st = make_map_f32_rows(&map_dq, dq_acc, p.seq, nrows, 128, false);
  if (st != SA_OK) return st;
  st = dq0 != nullptr ? make_map_f32_rows(&map_dq0, dq0, p.seq, p.batch, 128, false)
                      : make_map_f32_rows(&map_dq0, dq_acc, p.seq, nrows, 128, false);
  if (st != SA_OK) return st;
  WaitCtx status;
  st = wait_ctx(&status);
  if (st != SA_OK) return st;
  const bool self = self_selecting(p);
  const int smem = self ? Layout<true>::total : Layout<false>::total;
  const uint8_t* alive = static_cast<const uint8_t*>(p.tile_table);
  const unsigned grid = 2u * (unsigned)ntiles * (unsigned)nrows;
  auto launch = [&](auto kernel) -> int {
    SA_CUDA_CHECK(allow_smem(kernel, smem));
    ProfileScope prof(SA_KERNEL_TC_BACKWARD, s);
    count_launch();
    kernel<<<grid, kThreads, smem, s>>>(map_q, map_k, map_v, map_do, map_q0, map_k0, map_dq, map_dq0, stats, carry, dq0 != nullptr ? 1 : p.heads,
                                        static_cast<__nv_bfloat16*>(dk), dk0, static_cast<__nv_bfloat16*>(dv), p.heads, p.seq,
                                        ntiles, p.exempt, p.scale, status, p.dk_rows, p.dv_rows, alive);
    return SA_OK;
  };
  // (the live-tile entry points, like all that take the caller's layout, ask for 16-byte aligned rows)
  if (alive != nullptr) st = self ? launch(backward_wide_kernel<true, true, false>) : launch(backward_wide_kernel<false, true, false>);
  else if (((reinterpret_cast<uintptr_t>(dk) | reinterpret_cast<uintptr_t>(dv)) & 15) != 0)
    st = self ? launch(backward_wide_kernel<true, false, true>) : launch(backward_wide_kernel<false, false, true>);
  else st = self ? launch(backward_wide_kernel<true, false, false>) : launch(backward_wide_kernel<false, false, false>);
  if (st != SA_OK) return st;
  SA_CUDA_CHECK(cudaGetLastError());
  return SA_OK;
}

}  // namespace tc
}  // namespace sa
