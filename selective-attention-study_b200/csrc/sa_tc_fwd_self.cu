// Tensor-core engine, forward for heads that each select for themselves (head_dim 64; sm_100a: TMA loads, tcgen05 MMAs, fp32
// accumulators in TMEM).
//
// One CTA owns one 128-query tile of two neighbouring rows (batch x head) and takes 128-key steps from the diagonal back to
// key 0.  The selection logits are the head's own, S = Q K^T, so S is read twice: by a warpgroup that writes relu(S) under
// the mask to shared memory as bf16, and, after S -= TRI x selection (the exclusive running sum over the tile's queries as
// an MMA with a strictly-lower-triangular ones matrix), by the softmax.  Tile n is step n / 2 of row n & 1; three tiles are in
// flight, each in its own 128 TMEM columns (n mod 3): while the two softmax warpgroups work on two of them, the third goes
// through its product, selection and running sum.
//
// Roles.  Warps 0-3 and 4-7: the softmax of the two rows; a thread owns a query row and its 128 logits of the step.  Warps
// 8-11: the selection of both, and the carry of the step's keys.  Warp 12: S and P V.  Warp 13: TMA loads.  Warp 14: the
// running sums.
//
// TMEM, 512 columns: S x 3 (P as bf16 pairs over the first 64 of each) | O of the two rows (64 each).  Shared memory, 224 KB: Q
// 32, TRI 32, selection 2 x 32, K and V rings of three tiles 48 each.
//
// What bounds it: the latency of a tile over three tiles in flight (S 0.4 k cycles, selection 1.0, running sum 0.7, softmax 2.6,
// P V 0.5, and the waits between them: a tile takes 2.2 k of the CTA's time, so its columns are in use for 6.5 k); the
// exponential unit needs 1.0 k a tile, the tensor pipe 1.0 k, neither is busy half of the time.  Measured at 64 rows of T = 16384: 4.21 ms
// (forward_wide_kernel, one row a CTA in lock step: 5.77 ms).
//
// Reference for the arithmetic: src/selective_attention/kernels.py:140-194; per-head form: mixers.py:76-98.
#include <type_traits>

#include "sa_tc_fwd.cuh"

namespace sa {
namespace tc {
namespace {

constexpr int kTile = 128;          // query rows per CTA; also the carry checkpoint spacing
constexpr int kRowTile = 16384;     // bytes of a [128][64] bf16 operand tile
constexpr int kThreads = 512;       // two softmax warpgroups, the selection, four single warps (one idle)
constexpr int kRing = 3;            // tiles in flight
// Registers: 512 x 128 at launch; the softmax keeps 128 logits: 256 x 168 + 256 x 88.
constexpr int kSoftmaxRegs = 168, kOtherRegs = 88;
constexpr int kMmaWarp = 12, kLoadWarp = 13, kSumWarp = 14;

struct SelfSmem {
  static constexpr int q = 0;                              // Q of the two rows
  static constexpr int tri = q + 2 * kRowTile;             // [128][128] ones below the diagonal: two K-major tiles
  static constexpr int sel = tri + 2 * kRowTile;           // 2 x [128 queries][128 keys] bf16 as two key tiles
  static constexpr int k = sel + 4 * kRowTile;
  static constexpr int v = k + kRing * kRowTile;
  static constexpr int total = v + kRing * kRowTile;       // 224 KB
};
constexpr uint32_t kO = 384;                               // TMEM columns: S of slot i at 128 i, O of row x at kO + 64 x

// Tiles in order; slot n mod 3 and the parity of its use.
struct Turn {
  uint32_t slot = 0, par = 0;
  __device__ __forceinline__ void next(uint32_t by = 1) {
    slot += by;
    if (slot >= kRing) { slot -= kRing; par ^= 1u; }
  }
};

template <bool LIVE>
__global__ void __launch_bounds__(kThreads, 1) forward_self_kernel(
    const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
    const __grid_constant__ CUtensorMap map_v, const float* __restrict__ carry, float* __restrict__ out, float* __restrict__ lse2,
    int seq, int ntiles, int exempt, float scale, const __grid_constant__ WaitCtx status, __nv_bfloat16* __restrict__ out_lowp,
    RowLayout out_lowp_rows, int q_offset, const uint8_t* __restrict__ alive) {
  using L = SelfSmem;
  constexpr int D = 64;
  const int npairs = gridDim.x / (ntiles - q_offset / kTile);  // rows / 2 (the grid covers the query tiles with rows to compute)
  const int mi = ntiles - 1 - (int)(blockIdx.x / npairs);      // heaviest query tiles first
  const int n0 = 2 * (int)(blockIdx.x % npairs);               // the pair's first row
  const int i0 = mi * kTile;

  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = smem_raw;                                    // 1024-byte aligned: the static part is rounded up to it
  // Completion barriers: QF the query tiles; LDK, LDV loads; FREEK, FREEV the MMAs that read a slot (FREEV: P V of its tile);
  // SF S of a tile; FF its running sum; OF the last P V of a row.  Arrival barriers (one arrival per warp): SELW selection and
  // carry written; PW P written and O rescaled.
  enum : int { QF = 0, OF = 1, SF = 3, SELW = 6, FF = 9, PW = 12, LDK = 15, FREEK = 18, LDV = 21, FREEV = 24, kBars = 27 };
  __shared__ uint64_t bars[kBars];
  __shared__ uint32_t tmem_base_s;
  __shared__ __align__(16) float carry_s[kRing][kTile];
  __shared__ unsigned live_s[LIVE ? kMaxLiveTiles / 32 : 1];   // with a table of live tiles: bit nj of this query tile's row
  __shared__ int live_count_s;

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (LIVE && warp == 1) {                                     // live in either row (in the other one the step adds zeros)
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
    for (int u = 0; u < kBars; ++u) mbar_init(&bars[u], ((u >= SELW && u < FF) || (u >= PW && u < LDK)) ? 4 : 1);
    mbar_init_fence();
  }
  if (warp == 0) tmem_alloc(&tmem_base_s, 512);
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t sa = smem_u32(smem), bar0 = smem_u32(bars);
  auto bar = [&](uint32_t id) { return bar0 + 8u * id; };
  Waiter wait;
  wait.begin(status);
  const int steps = LIVE ? live_count_s : mi + 1;              // step 0 is the diagonal tile
  const int tiles = 2 * steps;
  auto step_back = [&](int nj) {                               // the key tile of the step after the one of tile nj
    if (!LIVE) return nj - 1;
    int w = nj >> 5;
    unsigned m = live_s[w] & ((1u << (nj & 31)) - 1u);
    while (m == 0u && w > 0) m = live_s[--w];
    return m != 0u ? 32 * w + 31 - __clz(m) : 0;
  };
  auto arrive = [&](uint32_t id) {
    __syncwarp();
    if (lane == 0) mbar_arrive(bar(id));
  };

  if (warp >= 8) {
    regs_shrink<kOtherRegs>();
    auto at = [](uint32_t low, uint32_t byte_off) { return low + (byte_off >> 4); };
    auto await = [&](uint32_t id, uint32_t parity, int site) { wait.left = wait_call(bar(id), parity, site, wait.left); };
    const uint32_t kBase = desc_low(sa, 16);                   // K-major views (rows = M or N index)
    const uint32_t mBase = desc_low(sa, kRowTile);             // MN-major views (rows = K index)
    if (warp == kLoadWarp) {
      // ============================================ TMA loads =============================================
      if (lane == 0) {
        auto load = [&](int off, const CUtensorMap* map, int id, int row, int x) {
          mbar_expect_tx(&bars[id], kRowTile);
          tma_load_4d(smem + off, map, &bars[id], 0, row, 0, n0 + x);
        };
        mbar_expect_tx(&bars[QF], 2 * kRowTile);
        for (int x = 0; x < 2; ++x) tma_load_4d(smem + L::q + x * kRowTile, &map_q, &bars[QF], 0, i0 - q_offset, 0, n0 + x);
        // K runs one tile ahead of V: that is the order in which their slots come free (S of n + 3 follows P V of n)
        int nj_k = mi, nj_v = mi;
        Turn rk, rv;
#pragma unroll 1
        for (int n = 0; n <= tiles; ++n) {
          if (n < tiles) {
            if (n >= kRing) wait(bar(FREEK + rk.slot), rk.par ^ 1u, 601);
            load(L::k + rk.slot * kRowTile, &map_k, LDK + (int)rk.slot, nj_k * kTile, n & 1);
            rk.next();
            if (n & 1) nj_k = step_back(nj_k);
          }
          if (n > 0) {
            if (n - 1 >= kRing) wait(bar(FREEV + rv.slot), rv.par ^ 1u, 602);
            load(L::v + rv.slot * kRowTile, &map_v, LDV + (int)rv.slot, nj_v * kTile, (n - 1) & 1);
            rv.next();
            if (!(n & 1)) nj_v = step_back(nj_v);
          }
        }
      }
      __syncwarp();
    } else if (warp == kMmaWarp) {
      // ======================================= S, and O += P V ============================================
      const uint32_t idesc_s = instr_desc_bf16(128, 128, false, false), idesc_pv = instr_desc_bf16(128, D, false, true);
      Turn rs, rp;
      auto issue_s = [&](uint32_t x) {
        await(LDK + rs.slot, rs.par, 611);
        if (elect_one()) {
          const uint32_t ql = at(kBase, L::q + x * kRowTile), kl = at(kBase, L::k + rs.slot * kRowTile);
          mma_ss_low<false>(128 * rs.slot, ql, kl, idesc_s);
#pragma unroll
          for (int ks = 1; ks < 4; ++ks) mma_ss_low<true>(128 * rs.slot, at(ql, ks * 32), at(kl, ks * 32), idesc_s);
          mma_commit(bar(SF + rs.slot));
          mma_commit(bar(FREEK + rs.slot));
        }
        __syncwarp();
        rs.next();
      };
      await(QF, 0, 610);
#pragma unroll 1
      for (int n = 0; n < kRing && n < tiles; ++n) issue_s((uint32_t)(n & 1));
#pragma unroll 1
      for (int n = 0; n < tiles; ++n) {
        const uint32_t x = (uint32_t)(n & 1);
        await(LDV + rp.slot, rp.par, 612);
        await(PW + rp.slot, rp.par, 613);                      // P written, O rescaled
        if (elect_one()) {
          const uint32_t vl = at(mBase, L::v + rp.slot * kRowTile);
#pragma unroll
          for (int ks = 0; ks < 8; ++ks)
            mma_ts_low(kO + 64 * x, 128 * rp.slot + ks * 8, at(vl, ks * 2048), idesc_pv, (n > 1 || ks > 0) ? 1u : 0u);
          mma_commit(bar(FREEV + rp.slot));
          if (n + 2 >= tiles) mma_commit(bar(OF + x));
        }
        __syncwarp();
        rp.next();
        if (n + kRing < tiles) issue_s((uint32_t)((n + kRing) & 1));   // over P, which the MMAs before it read
      }
    } else if (warp == kSumWarp) {
      // ======================================= S -= TRI x selection =======================================
      const uint32_t idesc_tri = instr_desc_bf16(128, 128, false, true, /*negate_a=*/true);
      Turn r;
#pragma unroll 1
      for (int n = 0; n < tiles; ++n) {
        await(SELW + r.slot, r.par, 620);                      // S read, its selection in shared memory
        if (elect_one()) {
          const uint32_t sl = at(mBase, L::sel + (n & 1) * 2 * kRowTile);
#pragma unroll
          for (int ks = 0; ks < 8; ++ks)
            mma_ss_low<true>(128 * r.slot, at(kBase, L::tri + (ks >> 2) * kRowTile + (ks & 3) * 32), at(sl, ks * 2048), idesc_tri);
          mma_commit(bar(FF + r.slot));
        }
        __syncwarp();
        r.next();
      }
    } else if (warp < kMmaWarp) {
      // ================================= selection: relu(S) under the mask, the carry =========================
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
      const float* carry_row = carry + ((int64_t)n0 * (ntiles + 1) + mi) * seq;
      auto fetch_carry = [&](int x, int nj) {
        const int j = nj * kTile + row;
        return j < seq ? load_ahead(carry_row + (int64_t)x * (ntiles + 1) * seq + j) : 0.f;
      };
      int nj = mi, nj_next = mi;
      float next_carry = fetch_carry(0, mi);
      const int i = i0 + row;
      Turn r;
#pragma unroll 1
      for (int n = 0; n < tiles; ++n) {
        const int j0 = nj * kTile;
        const bool masked = n < 2 || j0 < exempt;
        if (n >= 2) wait(bar(FF + (r.slot == 2 ? 0 : r.slot + 1)), r.slot == 2 ? r.par : r.par ^ 1u, 631);   // tile n - 2: its selection has been read
        wait(bar(SF + r.slot), r.par, 630);
        tc_fence_after_sync();
        const uint32_t sel = sa + L::sel + (n & 1) * 2 * kRowTile;
        const uint32_t cols = lane_base + 128 * r.slot;
        uint32_t q[2][32];                                     // 32 columns are converted while the next 32 arrive
        tmem_ld32(cols, q[0]);
        carry_s[r.slot][row] = -next_carry * kLog2e;           // negated: the softmax adds it in an FMA (the slot's last carry has
                                                               //   been read: S came after P V of its last tile)
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          uint32_t* cur = q[c & 1];
          tmem_ld_wait();
          if (c + 1 < 4) tmem_ld32(cols + 32 * (c + 1), q[(c + 1) & 1]);
          if (masked) {
#pragma unroll
            for (int e = 0; e < 32; ++e) {
              const int j = j0 + 32 * c + e;
              if (!(j < i && j >= exempt)) cur[e] = 0u;
            }
          }
#pragma unroll
          for (int u = 0; u < 4; ++u) {                        // the relu rides on the bf16 conversion
            uint32_t w[4];
#pragma unroll
            for (int e = 0; e < 4; ++e)
              w[e] = pack_bf16_relu(__uint_as_float(cur[8 * u + 2 * e]), __uint_as_float(cur[8 * u + 2 * e + 1]));
            const uint32_t chunk = (uint32_t)(((c & 1) * 4 + u) << 4);
            st_shared16(sel + (c >> 1) * kRowTile + (row_off ^ chunk), w[0], w[1], w[2], w[3]);
          }
        }
        fence_async_smem();
        tc_fence_before_sync();
        arrive(SELW + r.slot);
        if (n + 1 < tiles) {                                   // the next tile's carry arrives while its S is awaited
          if (n & 1) nj = nj_next;
          else if (n + 2 < tiles) nj_next = step_back(nj);
          next_carry = fetch_carry((n + 1) & 1, nj);
        }
        r.next();
      }
    }
  } else {
    regs_grow<kSoftmaxRegs>();
    // ========================================== softmax of one row ==============================================
    const int x = warp >> 2, row = tid & 127;
    const uint32_t lane_base = (uint32_t)((warp & 3) * 32) << 16;
    const uint32_t o_cols = lane_base + kO + 64 * x;
    const uint32_t carry_base = smem_u32(carry_s);
    const float c1 = scale * kLog2e;
    const float2 cc = make_float2(c1, c1);
    const int i = i0 + row;
    float run_max = -INFINITY, run_den = 0.f;
    Turn r, last;                                              // this tile, and the row's tile before it
    r.slot = (uint32_t)x;
    auto step = [&](auto first_tag) {
      constexpr bool kFirst = decltype(first_tag)::value;      // the diagonal tile: causal mask inside it, nothing to rescale yet
      const uint32_t s_cols = lane_base + 128 * r.slot, nc_at = carry_base + r.slot * (kTile * 4);
      wait(bar(SELW + r.slot), r.par, 640);                    // (complete: the running sum came after it) the carry
      wait(bar(FF + r.slot), r.par, 641);
      tc_fence_after_sync();
      // ---- logits z = S * scale - carry in log2 units, and the row maximum (packed fp32x2 arithmetic) ------------------
      float2 z[64];
      float tile_max = -INFINITY;
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        uint32_t s[32];
        tmem_ld32(s_cols + 32 * c, s);
        tmem_ld_wait();
#pragma unroll
        for (int e4 = 0; e4 < 32; e4 += 4) {
          const float4 nc = ld_shared_f4(nc_at + 4 * (32 * c + e4));
#pragma unroll
          for (int k = 0; k < 2; ++k) {
            const int e = e4 + 2 * k;
            float2 a = __ffma2_rn(make_float2(__uint_as_float(s[e]), __uint_as_float(s[e + 1])), cc,
                                  k ? make_float2(nc.z, nc.w) : make_float2(nc.x, nc.y));
            if (kFirst) {
              const int j = 32 * c + e;                        // key and query count from the same position
              if (j > row) a.x = -INFINITY;
              if (j + 1 > row) a.y = -INFINITY;
            }
            tile_max = fmaxf(tile_max, fmaxf(a.x, a.y));
            z[16 * c + (e >> 1)] = a;
          }
        }
      }
      // every row has its own key in the diagonal tile, so the maximum is finite from the first step on
      const float new_max = fmaxf(run_max, tile_max);
      const float alpha = ex2(run_max - new_max);
      run_max = new_max;
      // ---- exponentials, P as bf16 pairs over the S columns that have been read (four sums: one would chain them) -------
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
      if (!kFirst) {
        wait(bar(FREEV + last.slot), last.par, 642);           // P V of the row's step before is done
        tc_fence_after_sync();
        if (__any_sync(0xffffffffu, alpha != 1.f)) {           // the accumulator follows the maximum while it moves
#pragma unroll 1
          for (int c = 0; c < 4; ++c) {
            uint32_t a[16];
            tmem_ld16(o_cols + 16 * c, a);
            tmem_ld_wait();
#pragma unroll
            for (int e = 0; e < 16; ++e) a[e] = __float_as_uint(__uint_as_float(a[e]) * alpha);
            tmem_st16(o_cols + 16 * c, a);
          }
        }
      }
      tmem_st_wait();
      tc_fence_before_sync();
      arrive(PW + r.slot);
      last = r;
      r.next(2);
    };
    step(std::true_type{});
#pragma unroll 1
    for (int t = 1; t < steps; ++t) step(std::false_type{});

    wait(bar(OF + x), 0, 643);                                 // the last P V
    tc_fence_after_sync();
    const float inv = 1.f / run_den;
    const int iq = i - q_offset, q_rows = seq - q_offset;      // row inside the query tensor
    const bool mine = i < seq && i >= q_offset;                // rows before q_offset belong to an earlier call
    const int64_t n = n0 + x;
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      uint32_t a[32];
      tmem_ld32(o_cols + 32 * c, a);
      tmem_ld_wait();
      float o[32];
#pragma unroll
      for (int e = 0; e < 32; ++e) o[e] = __uint_as_float(a[e]) * inv;
      if (mine) {
        if (out != nullptr) {
          float* orow = out + (n * q_rows + iq) * D + 32 * c;
#pragma unroll
          for (int e = 0; e < 32; e += 4) *reinterpret_cast<float4*>(orow + e) = make_float4(o[e], o[e + 1], o[e + 2], o[e + 3]);
        }
        if (out_lowp != nullptr) {                             // the same rows in the operand dtype, in the caller's layout
          uint4* lrow = reinterpret_cast<uint4*>(out_lowp + out_lowp_rows.at((int)n, 0, iq) + 32 * c);
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

int forward_self(const Problem& p, const ForwardMaps& m, const float* carry, float* out, float* lse2, const WaitCtx& status,
                 const uint8_t* alive, cudaStream_t s) {
  const int ntiles = (p.seq + kTile - 1) / kTile;
  const unsigned grid = (unsigned)(ntiles - p.q_offset / kTile) * (p.batch / 2);
  const int smem = SelfSmem::total;
  auto launch = [&](auto kernel) -> int {
    SA_CUDA_CHECK(allow_smem(kernel, smem));
    ProfileScope prof(SA_KERNEL_TC_FORWARD, s);
    count_launch();
    kernel<<<grid, kThreads, smem, s>>>(m.q, m.k, m.v, carry, out, lse2, p.seq, ntiles, p.exempt, p.scale, status,
                                        static_cast<__nv_bfloat16*>(p.out_lowp), p.out_lowp_rows, p.q_offset, alive);
    SA_CUDA_CHECK(cudaGetLastError());
    return SA_OK;
  };
  return alive != nullptr ? launch(forward_self_kernel<true>) : launch(forward_self_kernel<false>);
}

}  // namespace tc
}  // namespace sa
