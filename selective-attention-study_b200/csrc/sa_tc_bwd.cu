// Tensor-core engine, backward at head_dim 64 (sm_100a: TMA loads and reduce-adds, tcgen05 MMAs, fp32 accumulators in TMEM).
//
// One CTA owns one 128-key tile of one head and walks the query tiles LAST TO FIRST in 64-query halves.  All
// score-shaped tiles are computed transposed, KEYS on the TMEM lanes (S^T = K Q^T, dP^T = V dO^T, L0^T = K0 Q0^T), so
// one thread owns one key and sees all 64 queries of a half along its registers, the last one first.  The two running sums down the query
// axis are then thread-local fp32 recurrences walked from the last query to the first:
//     F[i]  = carry_after_tile - sum_{r >= i} sel[r]          (history term rebuilt per key)
//     U[i]  = suffix + sum_{i' > i} dz[i']                      (logit gradient of later queries)
// with  P = exp2(z - lse),  dz = P (dP - dbar),  g = gate ? -U : 0.
//
// TWO CHAINS.  A half is a serial chain (scores -> selection -> probabilities -> dz -> g -> the products that consume
// them) whose links are hand-overs between the arithmetic warps and the tensor pipe.  With all warps on one half at a time
// the SM idles at each of them: 10.4 k cycles per 128 x 128 tile of which ~3.8 k were issue slots.  Here the upper halves
// (chain 0) and the lower halves (chain 1) of the tiles belong to one warpgroup each, with their own two score tiles in TMEM,
// so that one chain computes while the other waits.  What couples them is little: the per key, the upper half
// hands the sum of its selection to the lower half of the same tile (`sel_s`), and the running sum of dz goes from half to
// half (`run_s`).
//
// Roles.  Warps 0-3 and 4-7: the two chains.  Warps 8-11: read dQ and dQ0 out of TMEM, scale, stage and TMA-reduce-add them
// into fp32 global rows.  Warps 12, 14, 15: MMA issue (per-key accumulators and L0^T; dQ and dQ0; S^T and dP^T).  Warp 13, one
// lane: TMA loads.
//
// TMEM, 512 columns: dV | dK | one accumulator shared by dQ and dQ0 | per chain W1 and W2 | dK0 (64 each).
//     W1: L0^T of half n -> (read) -> dP^T of half n -> (read) -> g^T as bf16 pairs -> dK0 -> L0^T of half n + 2
//     W2: S^T of half n -> (read) -> P^T and dz^T as bf16 pairs -> dV, dK -> S^T of half n + 2
// so each product is issued as soon as the columns that it goes to are free, a pass or more before it is needed; only L0^T
// is waited for, and the other chain covers that.  P^T, dz^T, g^T are A operands from TMEM; dz and g also go to shared
// memory, from where dQ = dz K and dQ0 = g K0 are computed per 128-query tile.
//
// What bounds it.  Shared memory (128 B/clk) moves 528 KB per 128 x 128 tile: score operands 144, B operands of dV, dK, dK0
// 48, dQ, dQ0 operands 96, dz and g written 64, dQ, dQ0 staged and reduced 128, loads 48 = 4.2 k cycles; the tensor pipe needs
// 2.7 k, the issue slots ~3 k.  And the INSTRUCTION CACHE: everything that runs at one time has to fit 32 KB (measured: what
// does not fit is fetched at 2.7 cycles an instruction, for each chain separately since they are half a tile apart).  The
// first form of this kernel, with 45 KB of loops, ran at 15.5 k cycles a tile; hence the compact waits (Waiter), rolled MMA
// loops over halves (the order is the same for both chains), low words of descriptors, 32-bit shared addresses.
// Measured at B = 4, H = 16, T = 16384: 16.6 ms with sixteen warps in lock step, 12.1 ms with two chains and one MMA warp,
// 10.3 ms (5.4 k cycles a tile) with three (SELF: 12.3, 8.7, 8.0).
//
// SELF variant (one head per selector, i.e. the per-head form reshaped to (B H, 1, T, D)): the selection logits are the
// head's own logits, so S^T serves as L0^T (read twice), and since Q0 = Q and K0 = K the two gradient paths add before the
// MMAs: dK += (dz + g)^T Q and dQ = (dz + g) K, with (dz + g)^T in W1.  40 MMAs per query tile instead of 64, no Q0 / K0
// tiles, and the columns of dK0 hold K and V as bf16 pairs (A of the score products, 64 KB less shared-memory traffic).
// It moves 240 KB a tile (score operands 32, dV, dK 32, dQ 48, dz + g 32, staged and reduced 64, loads 32), 1.9 k of its 4.2 k
// cycles; the tensor pipe is busy 32 % of them, the issue slots 60 %.  What bounds it has not been found.
//
// The diagonal tile, the only one that needs the causal mask inside the tile, is the LAST tile of a CTA's walk: the loop
// holds the unmasked form only and the masked form runs once after it.  LIVE: with a table of live tiles (sa_tc_skip.cu)
// the walk starts at the key tile's last live query tile.
//
// Reference for the arithmetic: src/selective_attention/kernels.py:196-268 (one head), :271-364 (the shared
// selection-gradient products).
#include <type_traits>

#include "sa_tc_bwd_chain.cuh"

namespace sa {
namespace tc {
namespace {

using namespace bwd;

template <bool SELF>
struct PairSmem {
  static constexpr int kRing = SELF ? 5 : 3;                                 // half tiles of Q, dO in flight
  static constexpr int kRing0 = SELF ? 0 : 3;                                // half tiles of Q0
  static constexpr int kSlot = 2 * kHalfTile;                                // Q, dO
  static constexpr int k = 0;                                                // [128 keys][64], stationary
  static constexpr int v = k + kRowTile;
  static constexpr int k0 = v + kRowTile;
  static constexpr int ring = SELF ? k0 : k0 + kRowTile;
  static constexpr int ring0 = ring + kRing * kSlot;
  static constexpr int dz = ring0 + kRing0 * kHalfTile;                      // [128 keys][128 queries] bf16 as two query-half tiles
  static constexpr int g = dz + 2 * kRowTile;
  static constexpr int out = SELF ? g : g + 2 * kRowTile;                    // fp32 [128 queries][64]: per warp two [32][32] boxes
  static constexpr int stat = out + 2 * kRowTile;                            // kRing x (-lse2, -dbar)
  static constexpr int total = stat + kRing * kStatBytes;
};

// TMEM columns (W1, W2: sa_tc_bwd_chain.cuh)
constexpr uint32_t kDV = 0, kDK = 64, kDQ = 128, kDK0 = 448, kKA = 448, kVA = 480;
constexpr int DQ0 = DQ + 1;           // completes per tile like DQ

// LIVE: a table of live tiles is given (sa_tc_skip.cu).  ANY: rows of dk, dv that are not 16-byte aligned.
template <bool SELF, bool LIVE, bool ANY>
__global__ void __launch_bounds__(kThreads, 1) backward_kernel(
    const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
    const __grid_constant__ CUtensorMap map_v, const __grid_constant__ CUtensorMap map_do,
    const __grid_constant__ CUtensorMap map_dq, const __grid_constant__ CUtensorMap map_dq0,
    const __grid_constant__ CUtensorMap map_q0, const __grid_constant__ CUtensorMap map_k0,
    const float* __restrict__ stats, const float* __restrict__ carry, __nv_bfloat16* __restrict__ dk,
    float* __restrict__ dk0, __nv_bfloat16* __restrict__ dv, int heads, int dq0_rows, int seq, int ntiles, int exempt, float scale,
    const __grid_constant__ WaitCtx status, RowLayout dk_rows, RowLayout dv_rows, const uint8_t* __restrict__ alive) {
  using L = PairSmem<SELF>;
  constexpr int D = 64, R = L::kRing;
  // One (batch, head) row after the other, and within a row the key tiles with the most query tiles first: the CTAs
  // resident at one time belong to one or two rows and walk the same query tiles from the last one down, so every
  // Q, Q0, dO tile is fetched from DRAM once and then served from L2 to the row's other CTAs.
  int n, nj;
  tile_of_block(blockIdx.x, ntiles, gridDim.x / ntiles, LIVE, n, nj);
  const int b = n / heads, h = n - b * heads;

  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  __shared__ uint64_t bars[kBars];
  __shared__ uint32_t tmem_base_s;
  __shared__ float run_s[kTile], sel_s[2 * kTile];
  __shared__ int top_s;

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (LIVE && warp == 1) find_top_tile(alive, n, nj, ntiles, lane, &top_s);
  if (tid == 0) {
    init_bars(bars);
  }
  if (tid < kTile) run_s[tid] = 0.f;
  if (warp == 0) tmem_alloc(&tmem_base_s, 512);
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem = tmem_base_s;
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
    // ========================================== TMA loads ==================================================
    if (lane == 0) {
      auto row_of = [&](int hn) { return (mi_top - (hn >> 1)) * kTile + (1 - (hn & 1)) * 64; };
      auto load_qdo = [&](int hn, int slot) {
        const int row0 = row_of(hn);
        uint8_t* st = smem + L::ring + slot * L::kSlot;
        mbar_expect_tx(&bars[LD + slot], 2 * kHalfTile + kStatBytes);
        tma_load_4d(st, &map_q, &bars[LD + slot], 0, row0, h, b);
        tma_load_4d(st + kHalfTile, &map_do, &bars[LD + slot], 0, row0, h, b);
        bulk_load(smem + L::stat + slot * kStatBytes, stats + ((int64_t)n * 2 * ntiles + (row0 >> 6)) * (kStatBytes / 4), kStatBytes,
                  &bars[LD + slot]);
      };
      auto load_q0 = [&](int hn, int slot) {
        mbar_expect_tx(&bars[LD0 + slot], kHalfTile);
        tma_load_4d(smem + L::ring0 + slot * kHalfTile, &map_q0, &bars[LD0 + slot], 0, row_of(hn), 0, b);
      };
      mbar_expect_tx(&bars[KV], (SELF ? 2 : 3) * kRowTile);
      if (!SELF) tma_load_4d(smem + L::k0, &map_k0, &bars[KV], 0, nj * kTile, 0, b);
      tma_load_4d(smem + L::k, &map_k, &bars[KV], 0, nj * kTile, h, b);
      tma_load_4d(smem + L::v, &map_v, &bars[KV], 0, nj * kTile, h, b);
      // The slots of a half come free in the order dz, g of one half, then of the next: (Q, dO) first, then Q0.
      int slot = 0, slot0 = 0;
      uint32_t par = 1, par0 = 1;                                  // of the freeing before this fill (the first fills wait for none)
#pragma unroll 1
      for (int hn = 0; hn < n_half; ++hn) {
        if (hn >= R) wait(bar(FREE + slot), par, 402);
        load_qdo(hn, slot);
        if (++slot == R) { slot = 0; par ^= 1u; }
        if (!SELF) {
          if (hn >= 3) wait(bar(FREE0 + slot0), par0, 403);
          load_q0(hn, slot0);
          if (++slot0 == 3) { slot0 = 0; par0 ^= 1u; }
        }
      }
    }
    __syncwarp();
  } else if (warp >= 12) {
    // ========================================== MMA issue ==================================================
    // A whole warp walks this code and one elected lane issues.  Issuing is slow enough (an await that finds its phase
    // complete ~120 cycles, four MMAs ~300) that one warp for the 64 MMAs of a tile was the bottleneck at 6.2 k cycles a tile.
    // Products that must follow one another in the pipe (what reads a column range, then what overwrites it) are issued by
    // the same warp, or wait for the commit of the first.
    const uint32_t idesc_t = instr_desc_bf16(128, 64, false, false);     // keys x 64 queries, K = D
    const uint32_t idesc_acc = instr_desc_bf16(128, 64, false, true);    // A K-major (keys x queries), B MN-major
    const uint32_t idesc_dq = instr_desc_bf16(128, 64, true, true);      // A MN-major (queries x keys), B MN-major
    const uint32_t kBase = desc_low(sa, 16);                             // K-major views (rows = M or N index)
    const uint32_t mBase = desc_low(sa, kRowTile);                       // MN-major views (rows = K index)
    auto at = [](uint32_t low, uint32_t byte_off) { return low + (byte_off >> 4); };
    const int tiles = LIVE ? __shfl_sync(0xffffffffu, n_iter, 0) : n_iter;
    auto await = [&](int id, uint32_t parity, int site) {
      wait.left = wait_call(bar(id), parity, site, wait.left);
    };
    // TMEM addresses: the CTA owns all 512 columns, so they start at column 0.
    // d (64 columns) = A x B over four K steps of 16: A from shared memory, or from TMEM (8 packed columns a step)
    auto product_ss = [&](uint32_t d, uint32_t a_off, uint32_t b_off, int done) {
      if (elect_one()) {
        const uint32_t bl = at(kBase, b_off);
        mma_ss_low<false>(d, at(kBase, a_off), bl, idesc_t);
#pragma unroll
        for (int ks = 1; ks < 4; ++ks) mma_ss_low<true>(d, at(kBase, a_off + ks * 32), at(bl, ks * 32), idesc_t);
        mma_commit(bar(done));
      }
      __syncwarp();
    };
    auto product_ts = [&](uint32_t d, uint32_t a_col, uint32_t b_off, int done) {
      if (elect_one()) {
        const uint32_t bl = at(kBase, b_off);
#pragma unroll
        for (int ks = 0; ks < 4; ++ks) mma_ts_low(d, a_col + ks * 8, at(bl, ks * 32), idesc_t, ks > 0 ? 1u : 0u);
        mma_commit(bar(done));
      }
      __syncwarp();
    };
    auto issue_l0 = [&](uint32_t c, uint32_t slot) {                     // L0^T -> W1
      product_ss(w1_of(c), L::k0, L::ring0 + slot * kHalfTile, L0 + (int)c);
    };
    auto issue_s = [&](uint32_t c, uint32_t slot) {                      // S^T -> W2
      if (SELF) product_ts(w2_of(c), kKA, L::ring + slot * L::kSlot, S + (int)c);
      else product_ss(w2_of(c), L::k, L::ring + slot * L::kSlot, S + (int)c);
    };
    auto issue_dp = [&](uint32_t c, uint32_t slot) {                     // dP^T -> W1
      if (SELF) product_ts(w1_of(c), kVA, L::ring + slot * L::kSlot + kHalfTile, DP + (int)c);
      else product_ss(w1_of(c), L::v, L::ring + slot * L::kSlot + kHalfTile, DP + (int)c);
    };
    // acc (64 columns) += A (TMEM, 16 queries are 8 packed columns) x the half tile at `off`
    auto accumulate = [&](uint32_t acc, uint32_t a_col, uint32_t off, uint32_t keep) {
      const uint32_t rows = at(mBase, off);
#pragma unroll
      for (int ks = 0; ks < 4; ++ks) mma_ts_low(acc, a_col + ks * 8, at(rows, ks * 2048), idesc_acc, ks > 0 ? 1u : keep);
    };
    auto issue_dq = [&](uint32_t a_off, uint32_t b_off, int done) {  // dQ = dz K, dQ0 = g K0 over the tile's 128 keys
      if (elect_one()) {
        mma_ss_low<false>(kDQ, at(mBase, a_off), at(mBase, b_off), idesc_dq);
#pragma unroll
        for (int ks = 1; ks < 8; ++ks) mma_ss_low<true>(kDQ, at(mBase, a_off + ks * 2048), at(mBase, b_off + ks * 2048), idesc_dq);
        mma_commit(bar(done));
      }
      __syncwarp();
    };
    // Half hn of chain hn & 1 uses slot hn mod ring; `Ring` walks the halves in order.
    struct Ring { uint32_t slot, par; };
    auto next = [](Ring& x, uint32_t ring) {
      if (++x.slot == ring) { x.slot = 0; x.par ^= 1u; }
    };
    const int halves = 2 * tiles;
    await(SELF ? SETUP : KV, 0, 400);                                    // K, V (and K0) in place
    if (warp == kMmaWarp) {
      // -- the per-key accumulators, and the products whose columns they free: L0^T (SELF: S^T and dP^T) of the half after next
      Ring use{0, 0}, use0{0, 0}, ahead{0, 0};
      auto ask_l0 = [&](uint32_t c) {
        await(LD0 + (int)ahead.slot, ahead.par, 404);
        issue_l0(c, ahead.slot);
        next(ahead, 3);
      };
      auto ask_s = [&](uint32_t c) {
        await(LD + (int)ahead.slot, ahead.par, 403);
        issue_s(c, ahead.slot);
      };
      auto ask_dp = [&](uint32_t c) {
        issue_dp(c, ahead.slot);
        next(ahead, R);
      };
#pragma unroll 1
      for (uint32_t c = 0; c < 2; ++c) {
        if (SELF) ask_s(c), ask_dp(c);
        else ask_l0(c);
      }
#pragma unroll 1
      for (int hn = 0; hn < halves; ++hn) {
        const uint32_t c = (uint32_t)(hn & 1), ph = (uint32_t)((hn >> 1) & 1), keep = hn > 0 ? 1u : 0u;
        await(DZ + (int)c, ph, 406);                                     // P^T (and dz^T) written: dV, dK
        if (elect_one()) {
          accumulate(kDV, w2_of(c) + 32, L::ring + use.slot * L::kSlot + kHalfTile, keep);
          if (!SELF) {
            accumulate(kDK, w2_of(c), L::ring + use.slot * L::kSlot, keep);
            mma_commit(bar(FREE + (int)use.slot));
          }
        }
        __syncwarp();
        if (SELF && hn + 2 < halves) ask_s(c);
        await(G + (int)c, ph, 407);                                      // g^T written: dK0
        if (elect_one()) {
          if (SELF) {
            accumulate(kDK, w1_of(c), L::ring + use.slot * L::kSlot, keep);
            mma_commit(bar(FREE + (int)use.slot));
          } else {
            accumulate(kDK0, w1_of(c), L::ring0 + use0.slot * kHalfTile, keep);
            mma_commit(bar(FREE0 + (int)use0.slot));
          }
        }
        __syncwarp();
        if (hn + 2 < halves) {
          if (SELF) ask_dp(c);
          else ask_l0(c);
        }
        next(use, R);
        next(use0, 3);
      }
      if (elect_one()) mma_commit(bar(FIN));
      __syncwarp();
    } else if (warp == kDqWarp) {
      // -- the query-side products of a tile, once both halves are there and the accumulator has been read
#pragma unroll 1
      for (int t = 0; t < tiles; ++t) {
        const uint32_t ph = (uint32_t)(t & 1);
        if (!SELF) {
          await(DZ, ph, 408);
          await(DZ + 1, ph, 408);
          await(ACC, 1u, 409);                                           // (the first passes) dQ0 of the tile before
          issue_dq(L::dz, L::k, DQ);
        }
        await(G, ph, 410);
        await(G + 1, ph, 410);
        await(ACC, SELF ? ph ^ 1u : 0u, 411);                            // dQ of this tile; SELF: of the tile before
        issue_dq(SELF ? L::dz : L::g, SELF ? L::k : L::k0, SELF ? DQ : DQ0);
      }
    } else if (!SELF && warp == kScoreWarp) {
      // -- dP^T of half hn when its L0^T has been read, S^T of half hn + 1 when dV, dK of half hn - 1 are done
      Ring ahead{0, 0}, freed{0, 0}, sel{0, 0};
      auto ask_s = [&](uint32_t c) {
        await(LD + (int)ahead.slot, ahead.par, 403);
        issue_s(c, ahead.slot);
        next(ahead, R);
      };
      ask_s(0);
      ask_s(1);
#pragma unroll 1
      for (int hn = 0; hn < halves; ++hn) {
        const uint32_t c = (uint32_t)(hn & 1);
        await(SEL + (int)c, (uint32_t)((hn >> 1) & 1), 405);
        issue_dp(c, sel.slot);
        next(sel, R);
        if (hn > 0 && hn + 1 < halves) {
          await(FREE + (int)freed.slot, freed.par, 412);
          next(freed, R);
          ask_s(c ^ 1u);
        }
      }
    }
  } else {
    // ==================== read-out of dQ, dQ0: lanes are queries, a warp's 32 rows at a time ====================
    const uint32_t lane_base = tmem + ((uint32_t)((warp & 3) * 32) << 16);
    uint8_t* stage = smem + L::out + (warp - 8) * 8192;           // two [32 queries][32 floats] boxes, 128-byte swizzle
    const int n_reads = SELF ? n_iter : n_half;
    for (int r = 0; r < n_reads; ++r) {
      const int t = SELF ? r : r >> 1;
      const bool second = !SELF && (r & 1);
      wait(bar(second ? DQ0 : DQ), (uint32_t)(t & 1), 413);
      tc_fence_after_sync();
      if (lane == 0) bulk_wait_read();                            // the last reduce-add has read the staging boxes
#pragma unroll 1
      for (int x = 0; x < 2; ++x) {
        uint32_t a[32];
        tmem_ld32(lane_base + kDQ + 32 * x, a);
        tmem_ld_wait();
        if (x == 1) {
          tc_fence_before_sync();
          __syncwarp();
          if (lane == 0) mbar_arrive(bar(ACC));                   // the accumulator may be overwritten
        }
#pragma unroll
        for (int c = 0; c < 8; ++c)
          *reinterpret_cast<float4*>(stage + x * 4096 + swz_off(lane, c)) =
              make_float4(__uint_as_float(a[4 * c]) * scale, __uint_as_float(a[4 * c + 1]) * scale,
                          __uint_as_float(a[4 * c + 2]) * scale, __uint_as_float(a[4 * c + 3]) * scale);
      }
      fence_async_smem();
      __syncwarp();
      if (lane == 0) {
        const CUtensorMap* map = second ? &map_dq0 : &map_dq;
        const int row = second ? b * dq0_rows : n, q0 = (mi_top - t) * kTile + (warp - 8) * 32;
        if (q0 < seq) {
          tma_reduce_add_4d(map, stage, 0, q0, row, 0);
          tma_reduce_add_4d(map, stage + 4096, 32, q0, row, 0);
          bulk_commit();
        }
      }
    }
    if (!SELF) {                                                  // this head's share of dK0
      wait(bar(FIN), 0, 415);
      tc_fence_after_sync();
      const int j = nj * kTile + (warp - 8) * 32 + lane;
      float* row = dk0 + ((int64_t)b * seq + j) * D;
#pragma unroll
      for (int x = 0; x < 2; ++x) {
        uint32_t r0[32];
        tmem_ld32(lane_base + kDK0 + 32 * x, r0);
        tmem_ld_wait();
        if (j < seq) store_key_grads<false, 32, ANY>(nullptr, nullptr, r0, scale, nullptr, nullptr, row + 32 * x, false);
      }
    }
    if (lane == 0) bulk_wait_all();                               // the last reduce-adds must land before the CTA exits
    __syncwarp();
  }
  } else {
    regs_grow<kChainRegs>();
    // ============================================ the two chains ============================================
    const int c = warp >> 2, row = tid & 127;
    const uint32_t lane_base = tmem + ((uint32_t)((warp & 3) * 32) << 16);   // a warp reaches lanes 32 (warp % 4) ..
    const int j = nj * kTile + row;
    Chain ch;
    ch.c = c; ch.row = row; ch.lane = lane; ch.j = j; ch.n_iter = n_iter;
    ch.w1 = lane_base + w1_of(c);
    ch.w2 = lane_base + w2_of(c);
    ch.bar0 = bar0;
    ch.stat0 = sa + L::stat;
    ch.dz_row = sa + L::dz + (1 - c) * kRowTile + row * 128 + ((row & 7) << 4);
    ch.g_row = ch.dz_row + (SELF ? 0 : L::g - L::dz);              // (SELF: dz + g go to the dz tile, in the g pass)
    ch.keep_dz = ch.keep_g = true;
    ch.free_bar = SELF ? DQ : DQ0;                                 // of the tile before: has read dz and, later, g
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

    if (SELF) {                                                    // K (chain 0) and V (chain 1) rows into TMEM as bf16 pairs
      ch.wait(bar(KV), 0, 409);
      const uint8_t* src = smem + (c == 0 ? L::k : L::v);
      uint32_t w32[32];
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const uint4 v4 = *reinterpret_cast<const uint4*>(src + swz_off(row, u));
        w32[4 * u] = v4.x; w32[4 * u + 1] = v4.y; w32[4 * u + 2] = v4.z; w32[4 * u + 3] = v4.w;
      }
      tmem_st32(lane_base + (c == 0 ? kKA : kVA), w32);
      tmem_st_wait();
      tc_fence_before_sync();
      ch.arrive(SETUP);
    }
    for (int it = 0; it + 1 < n_iter; ++it) half_pass<SELF, false, R>(ch, it);
    half_pass<SELF, true, R>(ch, n_iter - 1);
    wait = ch.wait;

    // ---- epilogue: dV (chain 0) and dK (chain 1) of this key tile -------------------------------------------------
    wait(bar(FIN), 0, 415);
    tc_fence_after_sync();
#pragma unroll
    for (int x = 0; x < 2; ++x) {
      uint32_t r[32];
      tmem_ld32(lane_base + (c == 0 ? kDV : kDK) + 32 * x, r);
      tmem_ld_wait();
      if (j < seq) {
        if (c == 0)
          store_key_grads<SELF, 32, ANY>(r, nullptr, nullptr, scale, dv + dv_rows.at(b, h, j) + 32 * x, nullptr, nullptr, false);
        else
          store_key_grads<SELF, 32, ANY>(nullptr, r, nullptr, scale, nullptr, dk + dk_rows.at(b, h, j) + 32 * x,
                                    dk0 + ((int64_t)b * seq + j) * D + 32 * x, SELF || (h == 0 && dq0_rows != 1));
      }
    }
  }
  wait.end(status);
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tmem, 512);
}

}  // namespace

int backward(const Problem& p, const float* stats, const float* carry, const void* d_out, const RowLayout& d_out_rows,
             float* dq_acc, float* dq0, float* dk0, void* dk, void* dv, cudaStream_t s) {
  if (p.head_dim != 64) return SA_ERR_UNSUPPORTED;
  const int ntiles = (p.seq + kTile - 1) / kTile;
  const int nrows = p.batch * p.heads;
  CUtensorMap map_q, map_k, map_v, map_do, map_dq, map_dq0, map_q0, map_k0;
  int st = make_map_16bit(&map_q, p.q.ptr, 64, p.seq, p.heads, p.batch, p.q.st, p.q.sh, p.q.sb, 64);
  if (st != SA_OK) return st;
  st = make_map_16bit(&map_k, p.k.ptr, 64, p.seq, p.heads, p.batch, p.k.st, p.k.sh, p.k.sb, kTile);
  if (st != SA_OK) return st;
  st = make_map_16bit(&map_v, p.v.ptr, 64, p.seq, p.heads, p.batch, p.v.st, p.v.sh, p.v.sb, kTile);
  if (st != SA_OK) return st;
  st = make_map_16bit(&map_do, d_out, 64, p.seq, p.heads, p.batch, d_out_rows.st, d_out_rows.sh, d_out_rows.sb, 64);
  if (st != SA_OK) return st;
  st = make_map_f32_rows(&map_dq, dq_acc, p.seq, nrows, 64, true);
  if (st != SA_OK) return st;
  st = dq0 != nullptr ? make_map_f32_rows(&map_dq0, dq0, p.seq, p.batch, 64, true)
                      : make_map_f32_rows(&map_dq0, dq_acc, p.seq, nrows, 64, true);
  if (st != SA_OK) return st;
  st = make_map_16bit(&map_q0, p.q0.ptr, 64, p.seq, 1, p.batch, p.q0.st, 0, p.q0.sb, 64);
  if (st != SA_OK) return st;
  st = make_map_16bit(&map_k0, p.k0.ptr, 64, p.seq, 1, p.batch, p.k0.st, 0, p.k0.sb, kTile);
  if (st != SA_OK) return st;
  WaitCtx status;
  st = wait_ctx(&status);
  if (st != SA_OK) return st;
  const bool self = self_selecting(p);
  const int smem = (self ? PairSmem<true>::total : PairSmem<false>::total) + 1024;
  const uint8_t* alive = static_cast<const uint8_t*>(p.tile_table);
  auto launch = [&](auto kernel) -> int {
    SA_CUDA_CHECK(allow_smem(kernel, smem));
    ProfileScope prof(SA_KERNEL_TC_BACKWARD, s);
    count_launch();
    kernel<<<(unsigned)ntiles * nrows, kThreads, smem, s>>>(
        map_q, map_k, map_v, map_do, map_dq, map_dq0, map_q0, map_k0, stats, carry, static_cast<__nv_bfloat16*>(dk), dk0,
        static_cast<__nv_bfloat16*>(dv), p.heads, dq0 != nullptr ? 1 : p.heads, p.seq, ntiles, p.exempt, p.scale, status,
        p.dk_rows, p.dv_rows, alive);
    return SA_OK;
  };
  // (the live-tile entry points, like all that take the caller's layout, ask for 16-byte aligned rows)
  if (alive != nullptr) st = self ? launch(backward_kernel<true, true, false>) : launch(backward_kernel<false, true, false>);
  else if (((reinterpret_cast<uintptr_t>(dk) | reinterpret_cast<uintptr_t>(dv)) & 15) != 0)
    st = self ? launch(backward_kernel<true, false, true>) : launch(backward_kernel<false, false, true>);
  else st = self ? launch(backward_kernel<true, false, false>) : launch(backward_kernel<false, false, false>);
  if (st != SA_OK) return st;
  SA_CUDA_CHECK(cudaGetLastError());
  return SA_OK;
}

}  // namespace tc
}  // namespace sa
