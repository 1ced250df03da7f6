// Tensor-core engine, backward: what its two kernels share -- which CTA takes which key tile, the arithmetic of a chain's
// half tile (one thread owns one key row and sees all 64 queries of the half along its registers) and the key-side
// epilogue.  The scheme is described in sa_tc_bwd.cu.
#pragma once

#include "sa_tc_host.cuh"
#include "sa_tc_ptx.cuh"

namespace sa {
namespace tc {
namespace bwd {

constexpr int kTile = 128;
constexpr int kRowTile = 16384;      // bytes of a [128][64] bf16 operand tile
constexpr int kHalfTile = 8192;      // bytes of a [64][64] bf16 operand tile
constexpr int kThreads = 512;        // two chains, the read-out warpgroup, three MMA warps and a load warp
constexpr int kMmaWarp = 12, kLoadWarp = 13, kDqWarp = 14, kScoreWarp = 15;
constexpr int kStatBytes = 512;      // -lse2 and -dbar of 64 queries
// Registers: 512 x 128 at launch; the chains keep 64 values and their gates, the rest needs little: 256 x 168 + 256 x 88.
constexpr int kChainRegs = 168, kOtherRegs = 88;

// Barriers.  Completion: LD, LD0 TMA loads; L0, S, DP score products of a chain's half; FREE, FREE0 the last MMA that reads
// a slot; DQ query-side products.  Arrival, one arrival per warp: SEL L0^T read; DZ P^T and dz^T written, S^T and dP^T read;
// G g^T written; TOK the running sum of dz handed on; SUM the upper half's selection handed to the lower (even and odd
// tiles); ACC the shared accumulator read; TFREE (head_dim 128) a
// half tile of dz or g free again.
enum Bar : int { KV = 0, SETUP = 1, FIN = 2, DQ = 3, ACC = 5, L0 = 6, S = 8, DP = 10, SEL = 12, DZ = 14, G = 16, TOK = 18,
                 SUM = 20, LD = 22, FREE = 27, LD0 = 32, FREE0 = 35, TFREE = 38, kBars = 40 };
__device__ __forceinline__ void init_bars(uint64_t* bars) {
  for (int u = 0; u < kBars; ++u) mbar_init(&bars[u], u == SETUP ? 8 : (u == ACC || (u >= SEL && u < LD) || u >= TFREE) ? 4 : 1);
  mbar_init_fence();
}

// Which (row n = batch x head, key tile nj) a CTA takes.  Dense: one row after the other, key tile 0 (the longest
// walk) first.  With a table of live tiles most walks are a few tiles long, except those of the key tiles that hold an
// exempt key, which stay live for every query tile: all rows' key tile 0 go first so that the long walks start together.
__device__ __forceinline__ void tile_of_block(unsigned block, int ntiles, int nrows, bool sparse, int& n, int& nj) {
  if (!sparse) {
    n = (int)(block / ntiles);
    nj = (int)(block % ntiles);
  } else if ((int)block < nrows) {
    n = (int)block;
    nj = 0;
  } else {
    const unsigned r = block - nrows;
    n = (int)(r / (ntiles - 1));
    nj = 1 + (int)(r % (ntiles - 1));
  }
}

// The last query tile from which key tile nj of row n gets anything: ntiles - 1, or with a table of live tiles
// (alive[n][mi][nj], sa_tc_skip.cu) the largest live mi; the diagonal tile is always live.  One warp.
__device__ __forceinline__ void find_top_tile(const uint8_t* alive, int n, int nj, int ntiles, int lane, int* top) {
  int found = ntiles - 1;
  if (alive != nullptr) {
    const uint8_t* col = alive + (int64_t)n * ntiles * ntiles + nj;
    found = nj;
    for (int base = ntiles - 1; base >= nj; base -= 32) {
      const int mi = base - lane;
      const bool f = mi >= nj && col[(int64_t)mi * ntiles] != 0;
      const unsigned m = __ballot_sync(0xffffffffu, f);
      if (m != 0) {
        found = base - (__ffs(m) - 1);
        break;
      }
    }
  }
  if (lane == 0) *top = found;
}

// Eight bf16 of a gradient row.  ANY: the row is at any address of an element (what the plain entry points take).
template <bool ANY>
__device__ __forceinline__ void store8(__nv_bfloat16* to, uint4 w) {
  if constexpr (!ANY) {
    *reinterpret_cast<uint4*>(to) = w;
  } else {
    const uint32_t x[4] = {w.x, w.y, w.z, w.w};
    uint16_t* out = reinterpret_cast<uint16_t*>(to);
#pragma unroll
    for (int u = 0; u < 8; ++u) out[u] = (uint16_t)(x[u >> 1] >> (16 * (u & 1)));
  }
}

// N columns of one key row's gradients from the accumulators: dV in bf16, dK and dK0 scaled.  dK0 is added to the selecting
// head's fp32 rows (every head of the sequence adds its share); `own` says that dK belongs there too (head 0, whose dk is
// that sum), otherwise dK goes out in bf16.  SELF: dK holds both gradient paths and no one else adds to the row.
template <bool SELF, int N, bool ANY>
__device__ __forceinline__ void store_key_grads(const uint32_t* rv, const uint32_t* rk, const uint32_t* r0, float scale,
                                                __nv_bfloat16* dv_row, __nv_bfloat16* dk_row, float* dk0_row, bool own) {
#pragma unroll
  for (int e = 0; e < N; e += 8) {
    auto f = [&](const uint32_t* r, int u) { return __uint_as_float(r[e + u]); };
    if (rv != nullptr)
      store8<ANY>(dv_row + e, make_uint4(pack_bf16(f(rv, 0), f(rv, 1)), pack_bf16(f(rv, 2), f(rv, 3)),
                                         pack_bf16(f(rv, 4), f(rv, 5)), pack_bf16(f(rv, 6), f(rv, 7))));
    if (rk != nullptr && !own)
      store8<ANY>(dk_row + e,
                  make_uint4(pack_bf16(f(rk, 0) * scale, f(rk, 1) * scale), pack_bf16(f(rk, 2) * scale, f(rk, 3) * scale),
                             pack_bf16(f(rk, 4) * scale, f(rk, 5) * scale), pack_bf16(f(rk, 6) * scale, f(rk, 7) * scale)));
#pragma unroll
    for (int q = 0; q < 8; q += 4) {
      if (SELF) {
        if (rk != nullptr)
          *reinterpret_cast<float4*>(dk0_row + e + q) =
              make_float4(f(rk, q) * scale, f(rk, q + 1) * scale, f(rk, q + 2) * scale, f(rk, q + 3) * scale);
        continue;
      }
      float a[4] = {0.f, 0.f, 0.f, 0.f};
      if (rk == nullptr && r0 == nullptr) continue;
      if (r0 == nullptr && !own) continue;
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        if (r0 != nullptr) a[u] += f(r0, q + u) * scale;
        if (rk != nullptr && own) a[u] += f(rk, q + u) * scale;
      }
      asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(dk0_row + e + q), "f"(a[0]), "f"(a[1]), "f"(a[2]),
                   "f"(a[3])
                   : "memory");
    }
  }
}

// The gate of two selection logits, l > 0, as a bf16 pair: masks of 16 bits, or 1 and 0.  The comparison is made on the bf16
// roundings: they have the sign of the logit, and are zero only below 2^-134.
template <bool MASK>
__device__ __forceinline__ uint32_t gate_pair(float lo, float hi) {
  const __nv_bfloat162 x = __floats2bfloat162_rn(lo, hi), zero = __floats2bfloat162_rn(0.f, 0.f);
  if (MASK) return __hgt2_mask(x, zero);
  const __nv_bfloat162 g = __hgt2(x, zero);
  return *reinterpret_cast<const uint32_t*>(&g);
}

// TMEM: the score tiles of a chain, W1 and W2 (64 columns each).
constexpr uint32_t kW = 192;
__device__ __forceinline__ constexpr uint32_t w1_of(uint32_t chain) { return kW + 128 * chain; }
__device__ __forceinline__ constexpr uint32_t w2_of(uint32_t chain) { return kW + 128 * chain + 64; }

// One thread of a chain: chain 0 takes the upper halves of the query tiles, chain 1 the lower ones.
struct Chain {
  int c, row, lane, j, n_iter;
  uint32_t w1, w2;             // this thread's lane of the chain's columns
  uint32_t bar0, stat0;        // shared addresses: the barriers, the ring of query statistics
  uint32_t dz_row, g_row;      // this key's row of the dz and g half tiles (16-byte chunk x of it is at ^ 16 x)
  bool keep_dz, keep_g;        // whether an MMA of this CTA reads the half tile from there (otherwise TMEM alone has it)
  int free_bar;                // completes when the half tiles of the tile before may be overwritten
  float c1, inv_scale, shut;
  const float* carry;          // this key's column of the checkpoints at the tile after the one in hand
  int64_t carry_step;
  float* run_s;                // [128] the running sum of dz
  float* sel_s;                // [2][128] the upper half's selection
  int slot;
  uint32_t ld_par;
  float next_carry;
  Waiter wait;

  __device__ __forceinline__ uint32_t bar(int id) const { return bar0 + 8u * (uint32_t)id; }
  __device__ __forceinline__ void arrive(int id) const {
    __syncwarp();
    if (lane == 0) mbar_arrive(bar(id));
  }
  __device__ __forceinline__ void fetch_carry() {
    next_carry = carry != nullptr ? load_ahead(carry) : 0.f;
    carry -= carry != nullptr ? carry_step : 0;
  }
};
__device__ __forceinline__ void put8(uint32_t at, int chunk, const uint32_t* w) {             // eight queries of a key
  st_shared16(at ^ (uint32_t)(chunk << 4), w[0], w[1], w[2], w[3]);
}

// Half `it` of a chain.  DIAG: the diagonal tile, with the causal mask inside it.  RING: slots of (Q, dO) in flight.
template <bool SELF, bool DIAG, int RING>
__device__ __forceinline__ void half_pass(Chain& ch, int it) {
  const uint32_t ph = (uint32_t)(it & 1);
  const int c = ch.c, row = ch.row, other = c ^ 1;
  const int diag = row - (1 - c) * 64;                         // DIAG: query e of the half is this key itself
  const uint32_t stat = ch.stat0 + ch.slot * kStatBytes;
  const uint32_t w1 = ch.w1, w2 = ch.w2;
  float run = ch.next_carry;
  asm volatile("" : "+f"(run));                                // (the scaling stays here: next to the load it would wait for it)
  run *= -ch.inv_scale;                                        // minus the history after the tile, in units of q . k
  if (it + 1 < ch.n_iter) ch.fetch_carry();

  // ---- selection: relu(L0^T) and the gate ---------------------------------------------------------
  float v[64];
  uint32_t gate[32];                                           // bf16 pairs
  ch.wait(ch.bar((SELF ? S : L0) + c), ph, 410);
  tc_fence_after_sync();
  {
    uint32_t r[2][32];
    tmem_ld32((SELF ? w2 : w1), r[0]);
    tmem_ld32((SELF ? w2 : w1) + 32, r[1]);
    tmem_ld_wait();
    tc_fence_before_sync();
    if (!SELF) ch.arrive(SEL + c);                                // W1 may take dP^T
#pragma unroll
    for (int e = 0; e < 64; e += 2) {
      float l0 = __uint_as_float(r[e >> 5][e & 31]), l1 = __uint_as_float(r[e >> 5][(e & 31) + 1]);
      if (DIAG) {                                             // key strictly before the query
        if (e <= diag) l0 = -1.f;
        if (e + 1 <= diag) l1 = -1.f;
      }
      const float2 t = __fadd2_rn(make_float2(l0, l1), make_float2(ch.shut, ch.shut));
      gate[e >> 1] = gate_pair<!SELF>(t.x, t.y);
      v[e] = fmaxf(t.x, 0.f);
      v[e + 1] = fmaxf(t.y, 0.f);
    }
  }

  // ---- probabilities, last query first: P = exp2(c1 (S + run) - lse), run growing by the selection ---------------
  if (!SELF) {
    ch.wait(ch.bar(S + c), ph, 416);
    tc_fence_after_sync();
  }
  mbar_try_wait(ch.bar(LD + ch.slot), ch.ld_par);                    // (complete: S^T was made from the slot) its statistics are visible
  if (c == 1) {                                                // the upper half's selection comes first
    ch.wait(ch.bar(SUM + (int)ph), (uint32_t)((it >> 1) & 1), 421);
    run += ch.sel_s[ph * kTile + row];
  }
  const float2 cc = make_float2(ch.c1, ch.c1);
  const float run_in = run;
#pragma unroll
  for (int q = 1; q >= 0; --q) {
    uint32_t r[32], w[16];
    tmem_ld32(w2 + 32 * q, r);
    tmem_ld_wait();
#pragma unroll
    for (int e4 = 28; e4 >= 0; e4 -= 4) {
      const float4 nl = ld_shared_f4(stat + 4 * (32 * q + e4));
#pragma unroll
      for (int k = 1; k >= 0; --k) {
        const int e = 32 * q + e4 + 2 * k;
        const float hi = run + v[e + 1];
        run = hi + v[e];
        const float2 s = __fadd2_rn(make_float2(__uint_as_float(r[e4 + 2 * k]), __uint_as_float(r[e4 + 2 * k + 1])),
                                    make_float2(run, hi));
        const float2 x = __ffma2_rn(s, cc, k ? make_float2(nl.z, nl.w) : make_float2(nl.x, nl.y));
        v[e] = ex2(x.x);
        v[e + 1] = ex2(x.y);
        if (DIAG) {                                           // key after the query
          if (e < diag) v[e] = 0.f;
          if (e + 1 < diag) v[e + 1] = 0.f;
        }
        w[(e4 >> 1) + k] = pack_bf16(v[e], v[e + 1]);
      }
    }
    tmem_st16(w2 + 32 + 16 * q, w);                            // over S^T columns that have been read
  }
  if (c == 0) {
    ch.sel_s[ph * kTile + row] = run - run_in;
    ch.arrive(SUM + (int)ph);
  }

  // ---- dz = P (dP - dbar) ------------------------------------------------------------------------------------
  ch.wait(ch.bar(DP + c), ph, 411);
  tc_fence_after_sync();
  if (!SELF) ch.wait(ch.bar(ch.free_bar), ph ^ 1u, 418);                // the tile before has been read
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    uint32_t r[32], w[16];
    tmem_ld32(w1 + 32 * q, r);
    tmem_ld_wait();
#pragma unroll
    for (int e4 = 0; e4 < 32; e4 += 4) {
      const float4 nd = ld_shared_f4(stat + 4 * (64 + 32 * q + e4));
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        const int e = 32 * q + e4 + 2 * k;
        const float2 d = __fmul2_rn(make_float2(v[e], v[e + 1]),
                                    __fadd2_rn(make_float2(__uint_as_float(r[e4 + 2 * k]), __uint_as_float(r[e4 + 2 * k + 1])),
                                               k ? make_float2(nd.z, nd.w) : make_float2(nd.x, nd.y)));
        v[e] = d.x;
        v[e + 1] = d.y;
        if (!SELF) w[(e4 >> 1) + k] = pack_bf16(d.x, d.y);
      }
    }
    if (!SELF) {                                               // dz: to TMEM (A of dK) and shared memory (A of dQ)
      tmem_st16(w2 + 16 * q, w);
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (ch.keep_dz) put8(ch.dz_row, 4 * q + u, w + 4 * u);
    }
  }
  if (!SELF) fence_async_smem();                               // dz half tile -> visible to the MMAs
  tmem_st_wait();
  tc_fence_before_sync();
  ch.arrive(DZ + c);

  // ---- g = gate ? -(sum of dz over later queries) : 0; SELF: dz + g.  The sum goes from half to half --------------
  ch.wait(ch.bar(TOK + other), ph ^ (uint32_t)other, 419);
  float later = ch.run_s[row];                                    // minus the sum of dz over later queries
  if (SELF) ch.wait(ch.bar(ch.free_bar), ph ^ 1u, 420);
#pragma unroll
  for (int q = 1; q >= 0; --q) {
    uint32_t w[16];
#pragma unroll
    for (int e = 32 * q + 30; e >= 32 * q; e -= 2) {
      const float hi = later, lo = later - v[e + 1];
      later = lo - v[e];
      const uint32_t m = gate[e >> 1];
      if constexpr (SELF)
        w[(e >> 1) & 15] = pack_bf16(fmaf(__uint_as_float(m << 16), lo, v[e]), fmaf(__uint_as_float(m & 0xffff0000u), hi, v[e + 1]));
      else
        w[(e >> 1) & 15] = pack_bf16(lo, hi) & m;
    }
    tmem_st16(w1 + 16 * q, w);                                 // over dP^T columns that have been read
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (ch.keep_g) put8(ch.g_row, 4 * q + u, w + 4 * u);
  }
  ch.run_s[row] = later;
  fence_async_smem();
  tmem_st_wait();
  tc_fence_before_sync();
  __syncwarp();
  if (ch.lane == 0) {
    mbar_arrive(ch.bar(G + c));
    mbar_arrive(ch.bar(TOK + c));
  }
  ch.slot += 2;
  if (ch.slot >= RING) { ch.slot -= RING; ch.ld_par ^= 1u; }
}

}  // namespace bwd
}  // namespace tc
}  // namespace sa
