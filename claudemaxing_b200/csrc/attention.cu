// Causal attention inside the segments of one packed row (the batch rows of a packed training
// batch), forward and backward, for head_dim 128 and fp16 q/k/v with grouped-query heads.
//
// Forward. A CTA owns 128 consecutive query tokens of one segment for NT query heads (one, or two
// that share their key/value head) and walks the key tiles of 128 tokens these may see. Per tile
// and head: S = Q K^T into 128 columns of tensor memory; the head's softmax warpgroup (thread =
// query row) reads its row into registers, takes P = exp2(scale S - m) and writes it back as fp16
// over S's columns; O += P V with P as the tensor-memory operand. m is the row's maximum so far: O and
// the sum are rescaled when it grows. (Letting it lag by up to 2^8 saved those round trips, 101 against
// 117 us for 9215 tokens in 4 segments, but the largest P is then no longer 1, which fp16 holds exactly,
// and the output's error against float64 rises by up to a tenth on peaked rows.) The score product of
// the next tile is issued right behind O += P V of this one; the commit that announces it also says that
// O may be rescaled, which happens behind the exponentials, when the scores' registers are free to hold the
// whole row of O (ahead of them it went 16 columns at a time: 127.5 against 121.2 us).
//
// What bounds it: on long walks the exponentials (16 a clock and SM: 1024 clocks a tile) and the
// two products (1024 clocks a tile) alternate, so two tiles must be in flight on an SM. NT = 2 does
// that inside a CTA and loads every key and value tile once for both heads; NT = 1 fits twice on an
// SM (96 KB of shared memory, 256 columns) and does it with two CTAs: half the work per CTA and no
// second wave where the row has few tiles. forward_heads_per_cta() draws the line.
//
// CTAs take the tiles with the longest walks first, over all heads. Every wait is bounded
// (umma::mbar_wait).
//
// The reference calls torch SDPA here (solution/attention.py:332-343) on a [1, 1, N, N] mask
// built by its packing (solution/lm_head_loss.py:300-337); this kernel takes the segment offsets.
#include <cfloat>
#include <cmath>
#include <cuda.h>

#include "common.cuh"
#include "rowpipe.cuh"
#include "umma.cuh"

namespace soup {
namespace {

using namespace umma;

constexpr int kD = 128;                        // head dimension
constexpr int kBQ = 128;                       // query rows per tile
constexpr int kBKV = 128;                      // key/value rows per tile
constexpr int kTileBytes = 128 * kD * 2;       // 32 KB: a [128 x 128] fp16 tile, two swizzled boxes
constexpr int kBox = kTileBytes / 2;           // one [128 rows x 64 cols] box
constexpr float kLog2e = 1.4426950408889634f;
constexpr float kLn2 = 0.6931471805599453f;

// Which tile a slot is. Slots go through the 128-row tiles of all segments in the order of their
// depth inside the segment, deepest first (`depth` = tiles before it in its segment): the longest
// walks of the forward, and, read from the other end, of the backward. More than 64 segments: plain
// order. Called by whole warps; false for a slot past the last tile.
struct Tile {
  int seg_begin, seg_end, depth, tiles;   // tiles: of the whole segment
};
__device__ __forceinline__ bool locate_tile(const int32_t* cu, int segments, int slot, Tile& t) {
  const int lane = threadIdx.x & 31;
  if (segments <= 64) {
    int b0 = 0, e0 = 0, b1 = 0, e1 = 0;
    if (lane < segments) { b0 = cu[lane]; e0 = cu[lane + 1]; }
    if (lane + 32 < segments) { b1 = cu[lane + 32]; e1 = cu[lane + 33]; }
    const int n0 = (e0 - b0 + kBQ - 1) / kBQ, n1 = (e1 - b1 + kBQ - 1) / kBQ;
    int left = slot;
    for (int level = __reduce_max_sync(0xffffffffu, max(n0, n1)) - 1; level >= 0; --level) {
      const uint32_t m0 = __ballot_sync(0xffffffffu, n0 > level), m1 = __ballot_sync(0xffffffffu, n1 > level);
      const int c0 = __popc(m0), c = c0 + __popc(m1);
      if (left < c) {
        const bool low = left < c0;
        const int src = __fns(low ? m0 : m1, 0, (low ? left : left - c0) + 1);
        t.seg_begin = __shfl_sync(0xffffffffu, low ? b0 : b1, src);
        t.seg_end = __shfl_sync(0xffffffffu, low ? e0 : e1, src);
        t.tiles = __shfl_sync(0xffffffffu, low ? n0 : n1, src);
        t.depth = level;
        return true;
      }
      left -= c;
    }
    return false;
  }
  int base = 0;
  for (int s0 = 0; s0 < segments; s0 += 32) {
    int b = 0, e = 0;
    if (s0 + lane < segments) { b = cu[s0 + lane]; e = cu[s0 + lane + 1]; }
    const int n = (e - b + kBQ - 1) / kBQ;
    int upto = n;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, upto, o);
      if (lane >= o) upto += y;
    }
    const uint32_t past = __ballot_sync(0xffffffffu, slot < base + upto);
    if (past) {
      const int src = __ffs(past) - 1;
      t.seg_begin = __shfl_sync(0xffffffffu, b, src);
      t.seg_end = __shfl_sync(0xffffffffu, e, src);
      t.tiles = __shfl_sync(0xffffffffu, n, src);
      t.depth = slot - base - (__shfl_sync(0xffffffffu, upto, src) - t.tiles);
      return true;
    }
    base += __shfl_sync(0xffffffffu, upto, 31);
  }
  return false;
}

__device__ __forceinline__ uint32_t kstep(int k8) {   // K-major step of 16 columns, in descriptor units
  return (uint32_t)(k8 >> 2) * (uint32_t)(kBox >> 4) + (uint32_t)(k8 & 3) * 2u;
}

struct AttnArgs {
  const int32_t* cu;     // [segments + 1]
  __half* out;           // [n, hq, 128]
  float* lse;            // [hq, n]
  int n, segments, hq, group;
  float scale_log2;      // softmax scale * log2(e), above zero (attn_fwd_kernel's NEG has the sign)
  float scale_far;       // the power of two at or above it (softmax_tile)
  int* status;
};

template <int NT>
struct __align__(1024) FwdSmem {
  static constexpr int kRing = 2 * NT;         // key and value tiles alternate: K0 V0 K1 V1 ...
  uint8_t q[NT][kTileBytes];
  uint8_t kv[kRing][kTileBytes];
  uint64_t q_full, kv_full[kRing], kv_empty[kRing], s_full[NT], p_full[NT], o_full[NT];
  uint32_t tmem_base;
  int abort_flag;
};

template <int NT>
constexpr int kFwdThreads = NT * 128 + 64;     // softmax warpgroups, then the TMA warp and the MMA warp

// What a row's exponentials are taken against: exp2(x * sl - msl), msl being the row's maximum so far
// times sl, rounded once and used everywhere, so that its rounding cancels between P, the sum and the
// log-sum-exp. sl is the softmax scale (times log2 e), except that from kFarScore on that rounding is more
// than 2^3, for which P's fp16 range has no room, and scores that differ at all differ by 2^4: there a power
// of two takes its place, whose products are exact, and only the largest score has weight either way.
// (It costs 119.3 against 116.5 us for 9215 tokens in 4 segments with two heads per CTA, 130.8 against 126.3
// with one, 11.4 against 11.3 for 1280 in 5; subtracting the maximum from every score 118.1, 135.4 and 11.6.)
// A row whose scores so far are all -inf has the finite maximum kLowest: they weigh nothing.
constexpr float kFarScore = 268435456.f;   // 2^28
constexpr float kLowest = -1e30f;          // below any product of 128 finite fp16 pairs
struct RowRef {
  float sl, msl;
  __device__ __forceinline__ void set(float top, float scale, float scale_far) {
    sl = scale;
    msl = __fmul_rn(top, scale);
    if (fabsf(msl) >= kFarScore) {
      sl = scale_far;
      msl = top * scale_far;
    }
  }
};

// One row of a score tile: its exponentials, as fp16 over the score columns, against the (possibly moved)
// reference, and the row's sum l. NEG: of the negated scores (a softmax scale below zero).
template <bool DIAG, bool NEG>
__device__ __forceinline__ void softmax_tile(uint32_t s_addr, uint32_t o_addr, int limit, bool first,
                                             float scale, float scale_far, RowRef& ref, float& l) {
  uint32_t x[4][32];
#pragma unroll
  for (int c = 0; c < 4; ++c) tmem_ld_32x32(s_addr + c * 32, x[c]);
#pragma unroll
  for (int c = 0; c < 4; ++c) tmem_ld_wait_on(x[c]);
  float mx[4] = {kLowest, kLowest, kLowest, kLowest};
#pragma unroll
  for (int c = 0; c < 4; ++c)
#pragma unroll
    for (int j = 0; j < 32; ++j) {
      if (NEG) x[c][j] ^= 0x80000000u;
      if (DIAG && c * 32 + j > limit) x[c][j] = 0xff800000u;   // -inf: no weight
      mx[j & 3] = fmaxf(mx[j & 3], __uint_as_float(x[c][j]));
    }
  const float top = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3]));
  float f = 1.f;
  bool rescale = false;   // of the whole warp
  if (first) {
    ref.set(top, scale, scale_far);
  } else {
    const bool grow = __fmul_rn(top, ref.sl) > ref.msl;
    rescale = __any_sync(0xffffffffu, grow);
    if (rescale) {
      if (grow) {   // from one reference, as it was used, to the next; a far one is left behind by 2^4 at least
        const float old = fabsf(ref.msl) < kFarScore ? ref.msl : -INFINITY;
        ref.set(top, scale, scale_far);
        f = exp2f(fabsf(ref.msl) < kFarScore ? old - ref.msl : -fmaf(top, scale, -old));
      }
      l *= f;
    }
  }
  float s[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    uint32_t packed[16];
#pragma unroll
    for (int j = 0; j < 32; j += 2) {
      const float p0 = exp2f(fmaf(__uint_as_float(x[c][j]), ref.sl, -ref.msl));
      const float p1 = exp2f(fmaf(__uint_as_float(x[c][j + 1]), ref.sl, -ref.msl));
      s[j & 2] += p0;                      // the sum of exponentials, from the values before rounding
      s[(j & 2) + 1] += p1;
      __half2 hh = __floats2half2_rn(p0, p1);
      packed[j >> 1] = *reinterpret_cast<uint32_t*>(&hh);
    }
    tmem_st_32x16(s_addr + c * 16, packed);
  }
  l += (s[0] + s[1]) + (s[2] + s[3]);
  if (rescale) {   // the scores' registers are free now: all of O's row is on its way at once
    uint32_t o[4][32];
#pragma unroll
    for (int c = 0; c < 4; ++c) tmem_ld_32x32(o_addr + c * 32, o[c]);
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      tmem_ld_wait_on(o[c]);
#pragma unroll
      for (int j = 0; j < 32; ++j) o[c][j] = __float_as_uint(__uint_as_float(o[c][j]) * f);
      tmem_st_32x32(o_addr + c * 32, o[c]);
    }
  }
  tmem_st_wait();
}

template <int NT, bool NEG>
__global__ void __launch_bounds__(kFwdThreads<NT>, NT == 1 ? 2 : 1)
attn_fwd_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                const __grid_constant__ CUtensorMap map_v, const AttnArgs a) {
  extern __shared__ uint8_t raw[];
  using Smem = FwdSmem<NT>;
  constexpr int kRing = Smem::kRing;
  const int head_groups = a.hq / NT;
  Tile tile;
  // the whole CTA leaves when the slot is past the last tile
  if (!locate_tile(a.cu, a.segments, blockIdx.x / head_groups, tile)) return;
  Smem& s = *reinterpret_cast<Smem*>((reinterpret_cast<uintptr_t>(raw) + 1023) & ~uintptr_t(1023));
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int h0 = (blockIdx.x % head_groups) * NT, hk = h0 / a.group;
  const int q0 = tile.seg_begin + tile.depth * kBQ;
  const int n_kv = tile.depth + 1;                               // key tiles it may see
  constexpr int kLoadWarp = NT * 4, kMmaWarp = NT * 4 + 1;
  if (threadIdx.x == 0) {
    mbar_init(&s.q_full, 1);
    for (int i = 0; i < kRing; ++i) {
      mbar_init(&s.kv_full[i], 1);
      mbar_init(&s.kv_empty[i], 1);
    }
    for (int t = 0; t < NT; ++t) {
      mbar_init(&s.s_full[t], 1);
      mbar_init(&s.p_full[t], 4);
      mbar_init(&s.o_full[t], 1);
    }
    s.abort_flag = 0;
    fence_barrier_init();
  }
  if (warp == kMmaWarp) {
    tmem_alloc(&s.tmem_base, NT * 256);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem = s.tmem_base;   // score columns of head t from t * 128, its O behind all scores
  volatile int* abort_flag = &s.abort_flag;

  if (warp == kLoadWarp) {
    if (lane == 0) {
      prefetch_tensormap(&map_v);
      mbar_expect_tx(&s.q_full, NT * kTileBytes);
#pragma unroll
      for (int t = 0; t < NT; ++t) {
        tma_load_2d(s.q[t], &map_q, (h0 + t) * kD, q0, &s.q_full);
        tma_load_2d(s.q[t] + kBox, &map_q, (h0 + t) * kD + 64, q0, &s.q_full);
      }
      for (int g = 0; g < 2 * n_kv; ++g) {
        const int st = g % kRing;
        if (g >= kRing && !mbar_wait(&s.kv_empty[st], ((g / kRing) & 1) ^ 1, abort_flag, a.status, 41)) break;
        const CUtensorMap* map = (g & 1) ? &map_v : &map_k;
        const int row = tile.seg_begin + (g >> 1) * kBKV;
        mbar_expect_tx(&s.kv_full[st], kTileBytes);
        tma_load_2d(s.kv[st], map, hk * kD, row, &s.kv_full[st]);
        tma_load_2d(s.kv[st] + kBox, map, hk * kD + 64, row, &s.kv_full[st]);
      }
    }
  } else if (warp == kMmaWarp) {
    if (lane == 0) {
      constexpr uint32_t idesc_s = make_idesc_f16(kBQ, kBKV, kFmtF16, kFmtF16, false, false);
      constexpr uint32_t idesc_o = make_idesc_f16(kBQ, kD, kFmtF16, kFmtF16, false, true);
      auto full = [&](int g) {
        return mbar_wait(&s.kv_full[g % kRing], (g / kRing) & 1, abort_flag, a.status, 44);
      };
      auto mma_s = [&](int t, int g) {   // S = Q K^T: 8 steps of 16 along the head dimension
        const uint64_t dq = make_smem_desc(smem_u32(s.q[t]), 16, 1024);
        const uint64_t dk = make_smem_desc(smem_u32(s.kv[g % kRing]), 16, 1024);
#pragma unroll
        for (int k8 = 0; k8 < kD / 16; ++k8)
          mma_f16_ss(tmem + t * 128, dq + kstep(k8), dk + kstep(k8), idesc_s, k8 != 0);
        tc_commit(&s.s_full[t]);
      };
      bool ok = mbar_wait(&s.q_full, 0, abort_flag, a.status, 43) && full(0);
      if (ok) {
        tc_fence_after_sync();
#pragma unroll
        for (int t = 0; t < NT; ++t) mma_s(t, 0);
        tc_commit(&s.kv_empty[0]);
      }
      for (int i = 0; i < n_kv && ok; ++i) {
        const int gv = 2 * i + 1, gk = 2 * i + 2;
        const bool more = i + 1 < n_kv;
        ok = full(gv);
#pragma unroll
        for (int t = 0; t < NT; ++t) {
          ok = ok && mbar_wait(&s.p_full[t], i & 1, abort_flag, a.status, 47);
          if (!ok) break;
          tc_fence_after_sync();
          // O (+)= P V along the key rows of the tile: P from tensor memory, V MN-major
          const uint64_t dv = make_smem_desc(smem_u32(s.kv[gv % kRing]), kBox, 1024);
#pragma unroll
          for (int k8 = 0; k8 < kBKV / 16; ++k8)
            mma_f16_ts(tmem + (NT + t) * 128, tmem + t * 128 + k8 * 8, dv + k8 * (2048 >> 4), idesc_o, (i | k8) != 0);
          if (t == NT - 1) tc_commit(&s.kv_empty[gv % kRing]);
          if (more) {
            if (t == 0) {
              ok = full(gk);
              if (!ok) break;
              tc_fence_after_sync();
            }
            // over the columns of P, which the products above, in order before these, have read
            mma_s(t, gk);
            if (t == NT - 1) tc_commit(&s.kv_empty[gk % kRing]);
          } else {
            tc_commit(&s.o_full[t]);
          }
        }
      }
    }
  } else {
    // ---------------------------------------------------------------- softmax: thread = query row
    const int t = warp >> 2;
    const int r = threadIdx.x & 127;
    const int q_idx = q0 + r;
    const uint32_t lane_base = tmem + ((uint32_t)((warp & 3) * 32) << 16);
    const uint32_t s_addr = lane_base + t * 128, o_addr = lane_base + (NT + t) * 128;
    RowRef ref = {};
    float l = 0.f;
    bool ok = true;
    for (int i = 0; i < n_kv; ++i) {
      ok = __all_sync(0xffffffffu, mbar_wait(&s.s_full[t], i & 1, abort_flag, a.status, 48));
      if (!ok) break;
      tc_fence_after_sync();
      // only the last tile of the walk, the one on the diagonal, hides columns from a row
      if (i + 1 < n_kv) softmax_tile<false, NEG>(s_addr, o_addr, 0, i == 0, a.scale_log2, a.scale_far, ref, l);
      else softmax_tile<true, NEG>(s_addr, o_addr, r, i == 0, a.scale_log2, a.scale_far, ref, l);
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(&s.p_full[t]);
    }
    if (ok) ok = __all_sync(0xffffffffu, mbar_wait(&s.o_full[t], 0, abort_flag, a.status, 50));
    if (ok) {
      tc_fence_after_sync();
      const float inv = 1.f / l;
      const bool valid = q_idx < tile.seg_end;
      const int h = h0 + t;
      __half* dst = a.out + ((size_t)q_idx * a.hq + h) * kD;
#pragma unroll
      for (int c0 = 0; c0 < kD; c0 += 32) {
        uint32_t o[32];
        tmem_ld_32x32(o_addr + c0, o);
        tmem_ld_wait_on(o);
        if (valid) {
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            uint32_t w[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              __half2 hh = __floats2half2_rn(__uint_as_float(o[8 * j + 2 * e]) * inv,
                                             __uint_as_float(o[8 * j + 2 * e + 1]) * inv);
              w[e] = *reinterpret_cast<uint32_t*>(&hh);
            }
            *reinterpret_cast<uint4*>(dst + c0 + 8 * j) = make_uint4(w[0], w[1], w[2], w[3]);
          }
        }
      }
      if (valid) a.lse[(size_t)h * a.n + q_idx] = (ref.msl * (ref.sl == a.scale_log2 ? 1.f : a.scale_log2 / ref.sl) + log2f(l)) * kLn2;
      tc_fence_before_sync();
    }
  }
  __syncthreads();
  if (s.abort_flag) {   // copies that may still be in flight land before the shared memory is released
    for (int i = 0; i < 64; ++i) __nanosleep(2000);
    __syncthreads();
  }
  if (warp == kMmaWarp) {
    tc_fence_after_sync();
    tmem_dealloc(tmem, NT * 256);
  }
}

// ------------------------------------------------------------------------------------------
// Backward. A CTA owns one 128-token key/value tile of a segment and one query head, or a few that share their
// key/value head, keeps K, V and the accumulators dV and dK (tensor memory) and walks the query tiles from the
// diagonal to the segment's end, head after head. Per query tile, everything transposed (lanes = key rows):
//   S^T = K Q^T, dP^T = V dO^T               tensor-memory columns 0-127 / 128-255
//   P^T = exp2(scale S^T - lse)              two compute warpgroups (64 query columns each), fp16 over S^T
//   dV += P^T dO                             A from tensor memory, columns 256-383
//   dS^T = P^T (dP^T - D)                    fp16 to shared memory
//   dQ  = dS K                               A from shared memory, over dP^T's columns; a third
//                                            warpgroup adds it to fp32 global memory (bulk reductions)
//   dK += dS^T Q                             A from shared memory, columns 384-511, while dQ is read out
// The score product of the next tile is issued as soon as dV has consumed P^T, so the exponentials of
// tile i + 1 run under the dQ / dK products of tile i. dK and dV leave once per CTA.
//
// What bounds it: shared memory, at 128 B a clock. A tile's products read 288 KB of operands (S^T, dP^T, dQ and dK
// both of theirs, dV one), loads, dS^T and the staging of dQ move 224 KB more and the rows' statistics 32: 4250
// clocks by count, about 5200 measured between tiles (9215 tokens in 4 segments: 236 us), and the thread that
// issues the products waits on none of the warps for long. The tensor core needs 2560. With dS^T in tensor memory as
// dK's operand 32 KB fewer are read, but dQ, over the same columns, has to wait for dK and the next dP^T for both:
// 5600 clocks, 290 us. (A query-stationary walk reads and moves 700 KB per tile: it stages and adds dK and dV, 128
// KB, where this one adds dQ, 64 KB. It took 35.8 us for 1280 tokens in 5 segments, 12 / 2 heads, and 790 us for
// 9215 tokens in 4; this one 20 and 236 us.)
// ------------------------------------------------------------------------------------------
constexpr int kBwdThreads = 448;   // warps 0-7 compute, 8-11 dQ, 12 loads, 13 products
constexpr int kDqWarp = 8, kBwdLoadWarp = 12, kBwdMmaWarp = 13;
constexpr uint32_t kColS = 0, kColP = 128, kColDv = 256, kColDk = 384;

struct KvSmem {
  uint8_t k[kTileBytes];
  uint8_t v[kTileBytes];
  uint8_t q[2][kTileBytes];    // k, v and q stage dV and dK (fp32) when the walk is over
  uint8_t d_o[kTileBytes];
  uint8_t ds[kTileBytes];      // dS^T [key rows x query columns]
  uint8_t stage[4][8192];      // per dQ warp two 32 x 32 fp32 boxes
  float lse[2][kBQ], d[2][kBQ];   // lse * log2 e and D of the query tile's rows
  uint64_t k_full, v_full, q_full[2], q_empty[2], do_full, do_empty, s_full, p_full, dp_full, ds_full,
      dq_full, dq_free, stats_full[2], done;
  uint32_t tmem_base;
  int abort_flag;
};
static_assert(sizeof(KvSmem) <= 232448, "shared memory of one CTA");

struct AttnKvArgs {
  const int32_t* cu;
  const float2* stats;   // [hq, n]
  int n, segments, hq, group;
  int heads;             // query heads of a CTA, one after another: a divisor of group
  float scale_log2, scale;
  int* status;
};

// D = rowsum(dO o O) and lse in powers of two per (token, head), and the cleared accumulators. 16
// lanes per row of 128; bound by memory (512 B read, 512 B + cleared per row).
constexpr int kPrepThreads = 256;
__global__ void __launch_bounds__(kPrepThreads)
attn_bwd_prep_kernel(const __half* __restrict__ out, const __half* __restrict__ d_out,
                     const float* __restrict__ lse, float2* __restrict__ stats, float4* __restrict__ dq,
                     float4* __restrict__ dk, float4* __restrict__ dv, int64_t rows_q, int64_t rows_k,
                     int n, int hq) {
  const int64_t row = (int64_t)blockIdx.x * (kPrepThreads / 16) + (threadIdx.x >> 4);
  const int lane = threadIdx.x & 15;
  const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
  if (row < rows_k) {
    dk[row * 32 + lane] = dk[row * 32 + 16 + lane] = zero;
    dv[row * 32 + lane] = dv[row * 32 + 16 + lane] = zero;
  }
  float d = 0.f;
  if (row < rows_q) {
    const uint4 x = reinterpret_cast<const uint4*>(out)[row * 16 + lane];
    const uint4 y = reinterpret_cast<const uint4*>(d_out)[row * 16 + lane];
    const __half2* xh = reinterpret_cast<const __half2*>(&x);
    const __half2* yh = reinterpret_cast<const __half2*>(&y);
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float2 xf = __half22float2(xh[e]), yf = __half22float2(yh[e]);
      d = fmaf(xf.x, yf.x, fmaf(xf.y, yf.y, d));
    }
    dq[row * 32 + lane] = dq[row * 32 + 16 + lane] = zero;
  }
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) d += __shfl_xor_sync(0xffffffffu, d, o);
  if (row < rows_q && lane == 0) {
    const int64_t token = row / hq;
    const int64_t at = (row - token * hq) * n + token;
    stats[at] = make_float2(lse[at] * kLog2e, d);
  }
}

// 32 fp32 columns of row `lane` of a 32 x 32 fp32 box with the 128-byte swizzle (8 pieces of 16 B).
__device__ __forceinline__ void write_box_row(uint8_t* box, int lane, const uint32_t (&x)[32], float f, bool keep) {
  uint8_t* mine = box + lane * 128;
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    float4 v = make_float4(__uint_as_float(x[4 * j]) * f, __uint_as_float(x[4 * j + 1]) * f,
                           __uint_as_float(x[4 * j + 2]) * f, __uint_as_float(x[4 * j + 3]) * f);
    if (!keep) v = make_float4(0.f, 0.f, 0.f, 0.f);
    *reinterpret_cast<float4*>(mine + ((j ^ (lane & 7)) << 4)) = v;
  }
}

// One query tile for one compute thread: key row r, query columns [64 * wg, 64 * wg + 64).
struct ComputeTile {
  uint32_t s_addr, dp_addr;   // this thread's lane, columns of its warpgroup
  const float *lse, *d;       // of its 64 columns
  uint8_t* ds_box;            // its 64-column box of dS^T
  int r;
};

template <bool DIAG>
__device__ __forceinline__ void probabilities(const ComputeTile& t, int first_col, float sl, float (&p)[64]) {
  uint32_t x[2][32];
  tmem_ld_32x32(t.s_addr, x[0]);
  tmem_ld_32x32(t.s_addr + 32, x[1]);
  tmem_ld_wait_on(x[0]);
  tmem_ld_wait_on(x[1]);
#pragma unroll
  for (int c = 0; c < 2; ++c) {
    uint32_t packed[16];
#pragma unroll
    for (int j = 0; j < 32; j += 4) {
      // four columns' lse at a time; every thread of the warpgroup reads the same ones
      const float4 l = *reinterpret_cast<const float4*>(t.lse + c * 32 + j);
      const float neg[4] = {-l.x, -l.y, -l.z, -l.w};
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        float v = exp2f(fmaf(__uint_as_float(x[c][j + k]), sl, neg[k]));
        if (DIAG && first_col + c * 32 + j + k < t.r) v = 0.f;   // a query sees the keys up to its own row
        p[c * 32 + j + k] = v;
      }
#pragma unroll
      for (int k = 0; k < 4; k += 2) {
        __half2 hh = __floats2half2_rn(p[c * 32 + j + k], p[c * 32 + j + k + 1]);
        packed[(j + k) >> 1] = *reinterpret_cast<uint32_t*>(&hh);
      }
    }
    tmem_st_32x16(t.s_addr + c * 16, packed);
  }
  tmem_st_wait();
}

__device__ __forceinline__ void score_gradients(const ComputeTile& t, const float (&p)[64]) {
  uint8_t* row = t.ds_box + t.r * 128;
#pragma unroll
  for (int c = 0; c < 2; ++c) {
    uint32_t y[32], packed[16];
    tmem_ld_32x32(t.dp_addr + c * 32, y);
    tmem_ld_wait_on(y);
#pragma unroll
    for (int j = 0; j < 32; j += 4) {
      const float4 d = *reinterpret_cast<const float4*>(t.d + c * 32 + j);
      const int at = c * 32 + j;
      __half2 lo = __floats2half2_rn(p[at] * (__uint_as_float(y[j]) - d.x), p[at + 1] * (__uint_as_float(y[j + 1]) - d.y));
      __half2 hi = __floats2half2_rn(p[at + 2] * (__uint_as_float(y[j + 2]) - d.z), p[at + 3] * (__uint_as_float(y[j + 3]) - d.w));
      packed[j >> 1] = *reinterpret_cast<uint32_t*>(&lo);
      packed[(j >> 1) + 1] = *reinterpret_cast<uint32_t*>(&hi);
    }
#pragma unroll
    for (int j = 0; j < 4; ++j)
      *reinterpret_cast<uint4*>(row + (((c * 4 + j) ^ (t.r & 7)) << 4)) =
          make_uint4(packed[4 * j], packed[4 * j + 1], packed[4 * j + 2], packed[4 * j + 3]);
  }
}

__global__ void __launch_bounds__(kBwdThreads, 1)
attn_bwd_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_do,
                   const __grid_constant__ CUtensorMap map_k, const __grid_constant__ CUtensorMap map_v,
                   const __grid_constant__ CUtensorMap map_dq, const __grid_constant__ CUtensorMap map_dk,
                   const __grid_constant__ CUtensorMap map_dv, const AttnKvArgs a) {
  extern __shared__ __align__(1024) uint8_t raw_kv[];
  Tile tile;
  const int head_groups = a.hq / a.heads;
  if (!locate_tile(a.cu, a.segments, blockIdx.x / head_groups, tile)) return;   // the whole CTA leaves
  KvSmem& s = *reinterpret_cast<KvSmem*>(raw_kv);
  if (smem_u32(raw_kv) & 1023) {   // the swizzled tiles and their descriptors want it; no room to align by hand
    if (threadIdx.x == 0) atomicCAS(a.status, 0, 60);
    return;
  }
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int h0 = (blockIdx.x % head_groups) * a.heads, hk = h0 / a.group;
  // depth counts from the walk's end: the tile with the longest walk is the segment's first
  const int n_q = tile.depth + 1;                                   // query tiles of a head's walk
  const int n_it = n_q * a.heads;
  const int kv0 = tile.seg_begin + (tile.tiles - 1 - tile.depth) * kBKV;
  if (threadIdx.x == 0) {
    mbar_init(&s.k_full, 1);
    mbar_init(&s.v_full, 1);
    for (int i = 0; i < 2; ++i) {
      mbar_init(&s.q_full[i], 1);
      mbar_init(&s.q_empty[i], 1);
      mbar_init(&s.stats_full[i], 4);
    }
    mbar_init(&s.do_full, 1);
    mbar_init(&s.do_empty, 1);
    mbar_init(&s.s_full, 1);
    mbar_init(&s.p_full, 8);
    mbar_init(&s.dp_full, 1);
    mbar_init(&s.ds_full, 8);
    mbar_init(&s.dq_full, 1);
    mbar_init(&s.dq_free, 4);
    mbar_init(&s.done, 1);
    s.abort_flag = 0;
    fence_barrier_init();
  }
  if (warp == kBwdMmaWarp) {
    tmem_alloc(&s.tmem_base, 512);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem = s.tmem_base;
  volatile int* abort_flag = &s.abort_flag;
  const uint32_t lane_base = tmem + ((uint32_t)((warp & 3) * 32) << 16);

  if (warp == kBwdLoadWarp) {
    if (lane == 0) {
      auto tile_in = [&](uint8_t* dst, const CUtensorMap* map, int col, int row, uint64_t* bar) {
        mbar_expect_tx(bar, kTileBytes);
        tma_load_2d(dst, map, col, row, bar);
        tma_load_2d(dst + kBox, map, col + 64, row, bar);
      };
      tile_in(s.k, &map_k, hk * kD, kv0, &s.k_full);
      tile_in(s.q[0], &map_q, h0 * kD, kv0, &s.q_full[0]);
      tile_in(s.v, &map_v, hk * kD, kv0, &s.v_full);
      tile_in(s.d_o, &map_do, h0 * kD, kv0, &s.do_full);
      int step = 0, h = h0;
      for (int i = 1; i < n_it; ++i) {
        if (++step == n_q) { step = 0; ++h; }
        const int row = kv0 + step * kBQ;
        if (i >= 2 && !mbar_wait(&s.q_empty[i & 1], ((i >> 1) & 1) ^ 1, abort_flag, a.status, 61)) break;
        tile_in(s.q[i & 1], &map_q, h * kD, row, &s.q_full[i & 1]);
        if (!mbar_wait(&s.do_empty, (i - 1) & 1, abort_flag, a.status, 62)) break;
        tile_in(s.d_o, &map_do, h * kD, row, &s.do_full);
      }
    }
  } else if (warp == kBwdMmaWarp) {
    if (lane == 0) {
      constexpr uint32_t idesc_nn = make_idesc_f16(128, 128, kFmtF16, kFmtF16, false, false);
      constexpr uint32_t idesc_nt = make_idesc_f16(128, 128, kFmtF16, kFmtF16, false, true);
      constexpr uint32_t idesc_tt = make_idesc_f16(128, 128, kFmtF16, kFmtF16, true, true);
      const uint64_t k_k = make_smem_desc(smem_u32(s.k), 16, 1024), k_mn = make_smem_desc(smem_u32(s.k), kBox, 1024);
      const uint64_t v_k = make_smem_desc(smem_u32(s.v), 16, 1024);
      const uint64_t do_k = make_smem_desc(smem_u32(s.d_o), 16, 1024);
      const uint64_t do_mn = make_smem_desc(smem_u32(s.d_o), kBox, 1024);
      const uint64_t ds_mn = make_smem_desc(smem_u32(s.ds), kBox, 1024), ds_k = make_smem_desc(smem_u32(s.ds), 16, 1024);
      auto wait = [&](uint64_t* bar, int turn, int code) {
        const bool got = mbar_wait(bar, turn & 1, abort_flag, a.status, code);
        tc_fence_after_sync();
        return got;
      };
      auto scores = [&](int i) {
        const uint64_t q_k = make_smem_desc(smem_u32(s.q[i & 1]), 16, 1024);
#pragma unroll
        for (int k8 = 0; k8 < 8; ++k8)
          mma_f16_ss(tmem + kColS, k_k + kstep(k8), q_k + kstep(k8), idesc_nn, k8 != 0);
        tc_commit(&s.s_full);
      };
      auto d_prob = [&]() {
#pragma unroll
        for (int k8 = 0; k8 < 8; ++k8)
          mma_f16_ss(tmem + kColP, v_k + kstep(k8), do_k + kstep(k8), idesc_nn, k8 != 0);
        tc_commit(&s.dp_full);
      };
      // columns of the 16 query tokens of step k8 in an fp16 operand that two warpgroups wrote over
      // their own halves of 128 fp32 columns
      auto packed_col = [](int k8) { return (uint32_t)((k8 >> 2) * 64 + (k8 & 3) * 8); };
      bool ok = wait(&s.k_full, 0, 63) && wait(&s.q_full[0], 0, 64);
      if (ok) scores(0);
      ok = ok && wait(&s.v_full, 0, 65) && wait(&s.do_full, 0, 66);
      if (ok) d_prob();
      for (int i = 0; i < n_it && ok; ++i) {
        const bool more = i + 1 < n_it;
        ok = wait(&s.p_full, i, 67);
        if (!ok) break;
#pragma unroll
        for (int k8 = 0; k8 < 8; ++k8)
          mma_f16_ts(tmem + kColDv, tmem + kColS + packed_col(k8), do_mn + k8 * (2048 >> 4), idesc_nt, (i | k8) != 0);
        tc_commit(&s.do_empty);
        if (more) {   // over the columns of P^T, which the products above, in order before these, have read
          ok = wait(&s.q_full[(i + 1) & 1], (i + 1) >> 1, 68);
          if (!ok) break;
          scores(i + 1);
        }
        ok = wait(&s.ds_full, i, 69);
        if (!ok) break;
        const uint64_t q_mn = make_smem_desc(smem_u32(s.q[i & 1]), kBox, 1024);
#pragma unroll
        for (int k8 = 0; k8 < 8; ++k8)   // over the columns of dP^T, which the compute warps have read
          mma_f16_ss(tmem + kColP, ds_mn + k8 * (2048 >> 4), k_mn + k8 * (2048 >> 4), idesc_tt, k8 != 0);
        tc_commit(&s.dq_full);
#pragma unroll
        for (int k8 = 0; k8 < 8; ++k8)   // while dQ is read out
          mma_f16_ss(tmem + kColDk, ds_k + kstep(k8), q_mn + k8 * (2048 >> 4), idesc_nt, (i | k8) != 0);
        tc_commit(&s.q_empty[i & 1]);
        if (more) {
          ok = wait(&s.do_full, i + 1, 70) && wait(&s.dq_free, i, 71);
          if (ok) d_prob();
        }
      }
      if (ok) tc_commit(&s.done);
    }
  } else if (warp >= kDqWarp) {
    // ---------------------------------------------------------------- dQ, and the rows' statistics
    const int r = threadIdx.x - kDqWarp * 32;
    uint8_t* stage = s.stage[warp - kDqWarp];
    struct At {   // a step of the walk: query tile and head
      int step, head;
    };
    auto after = [&](At at) { return at.step + 1 == n_q ? At{0, at.head + 1} : At{at.step + 1, at.head}; };
    auto fetch = [&](At at) {   // a query past the segment gets weight exp2(-inf) = 0
      const int token = kv0 + at.step * kBQ + r;
      return at.head < h0 + a.heads && token < tile.seg_end ? a.stats[(size_t)at.head * a.n + token]
                                                            : make_float2(INFINITY, 0.f);
    };
    auto put = [&](int i, float2 v) {
      s.lse[i & 1][r] = v.x;
      s.d[i & 1][r] = v.y;
      __syncwarp();
      if (lane == 0) mbar_arrive(&s.stats_full[i & 1]);
    };
    At now = {0, h0}, next = after(now);
    put(0, fetch(now));
    put(1, fetch(next));
    next = after(next);
    bool ok = true;
    for (int i = 0; i < n_it; ++i, now = after(now), next = after(next)) {
      const float2 ahead = fetch(next);
      ok = __all_sync(0xffffffffu, mbar_wait(&s.dq_full, i & 1, abort_flag, a.status, 72));
      if (!ok) break;
      tc_fence_after_sync();
      put(i + 2, ahead);   // dq_full(i): nobody reads the statistics of tile i any more
      const bool keep = kv0 + now.step * kBQ + r < tile.seg_end;   // the tile's other rows belong to other segments
      const int row0 = kv0 + now.step * kBQ + (warp - kDqWarp) * 32;
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        uint32_t x[32], y[32];
        tmem_ld_32x32(lane_base + kColP + half * 64, x);
        tmem_ld_32x32(lane_base + kColP + half * 64 + 32, y);
        tmem_ld_wait_on(x);
        tmem_ld_wait_on(y);
        if (half == 1) {
          tc_fence_before_sync();
          __syncwarp();
          if (lane == 0) mbar_arrive(&s.dq_free);
        }
        if (lane == 0) tma_store_wait_read<0>();   // both boxes have been read
        __syncwarp();
        write_box_row(stage, lane, x, a.scale, keep);
        write_box_row(stage + 4096, lane, y, a.scale, keep);
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0 && row0 < tile.seg_end) {
          tma_reduce_add_2d(&map_dq, stage, now.head * kD + half * 64, row0);
          tma_reduce_add_2d(&map_dq, stage + 4096, now.head * kD + half * 64 + 32, row0);
          tma_store_commit();
        }
      }
    }
    if (lane == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");   // the sums have landed
  } else {
    // ---------------------------------------------------------------- P^T and dS^T: thread = key row
    const int wg = warp >> 2;
    ComputeTile t;
    t.r = threadIdx.x & 127;
    t.s_addr = lane_base + kColS + wg * 64;
    t.dp_addr = lane_base + kColP + wg * 64;
    t.ds_box = s.ds + wg * kBox;
    const float sl = a.scale_log2;
    bool ok = true;
    int step = 0;
    for (int i = 0; i < n_it; ++i) {
      t.lse = s.lse[i & 1] + wg * 64;
      t.d = s.d[i & 1] + wg * 64;
      ok = mbar_wait(&s.stats_full[i & 1], (i >> 1) & 1, abort_flag, a.status, 73) &&
           mbar_wait(&s.s_full, i & 1, abort_flag, a.status, 74);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      tc_fence_after_sync();
      float p[64];
      if (step == 0) probabilities<true>(t, wg * 64, sl, p);   // the tile on the diagonal
      else probabilities<false>(t, wg * 64, sl, p);
      if (++step == n_q) step = 0;
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(&s.p_full);
      ok = __all_sync(0xffffffffu, mbar_wait(&s.dp_full, i & 1, abort_flag, a.status, 75));
      if (!ok) break;
      tc_fence_after_sync();
      score_gradients(t, p);
      tc_fence_before_sync();
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(&s.ds_full);
    }
    if (ok) ok = __all_sync(0xffffffffu, mbar_wait(&s.done, 0, abort_flag, a.status, 76));
    if (ok) {   // the first warpgroup adds dV, the second dK, through the tiles nobody reads any more
      tc_fence_after_sync();
      uint8_t* stage = s.k + warp * 16384;
      const uint32_t src = lane_base + (wg == 0 ? kColDv : kColDk);
      const float f = wg == 0 ? 1.f : a.scale;
      const bool keep = kv0 + t.r < tile.seg_end;
      const int row0 = kv0 + (warp & 3) * 32;
#pragma unroll 1
      for (int c = 0; c < 4; ++c) {
        uint32_t x[32];
        tmem_ld_32x32(src + c * 32, x);
        tmem_ld_wait_on(x);
        write_box_row(stage + c * 4096, lane, x, f, keep);
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0 && row0 < tile.seg_end) {
          tma_reduce_add_2d(wg == 0 ? &map_dv : &map_dk, stage + c * 4096, hk * kD + c * 32, row0);
          tma_store_commit();
        }
      }
      if (lane == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
      tc_fence_before_sync();
    }
  }
  __syncthreads();
  if (s.abort_flag) {   // copies that may still be in flight land before the shared memory is released
    for (int i = 0; i < 64; ++i) __nanosleep(2000);
    __syncthreads();
  }
  if (warp == kBwdMmaWarp) {
    tc_fence_after_sync();
    tmem_dealloc(tmem, 512);
  }
}
}  // namespace
}  // namespace soup

namespace soup {
namespace {

// every segment adds at most one partial tile to the tiles of the packed row
inline int64_t tile_slots(int64_t n_tokens, int64_t n_segments) { return (n_tokens + kBQ - 1) / kBQ + n_segments; }

// Heads of a forward CTA. Two per CTA (both heads use every key and value tile) pay once an SM has
// more than about fourteen (tile, key tile) steps to walk, estimated from the mean segment; below, twice
// as many CTAs of half the work finish earlier. One and two heads, in us, by steps per SM: 12 query and 2
// key heads 1: 11.4 and 13.8 (1280 tokens in 5 segments), 5: 24.1 and 25.2 (4607 in 16), 8: 28.7 and 28.0
// (4604 in 8), 11: 42.2 and 46.7 (2048 in 1), 15: 46.5 and 47.2 (4607 in 4), 29: 72.9 and 69.9 (9212 in 8),
// 55: 130.6 and 119.4 (9215 in 4); 32 and 8 heads 13: 51.7 and 54.8 (4607 in 16), 16: 36.3 and 33.3 (2048 in
// 2), 39: 98.2 and 92.3 (4607 in 4). The two heads share one key/value head.
inline int forward_heads_per_cta(int64_t n_tokens, int64_t n_segments, int64_t hq, int64_t hk) {
  if ((hq / hk) % 2) return 1;
  const double tiles = (double)n_tokens / kBQ, walk = (tiles / (double)n_segments + 1.0) / 2.0;
  return tiles * walk * (double)hq > 14.0 * sm_count() ? 2 : 1;
}

// Query heads of a backward CTA, one after another on the same key/value tile: K, V, the prologue and the sums
// of dK and dV are paid once for all of them. More heads make fewer and longer units, so the choice is the one
// with the smallest estimate of the last SM's end, in steps of a walk (`cost` of a number of heads). One, two and three
// heads, in us (both launches, 12 query and 2 key heads; "even": equal lengths, else falling to an eighth of the longest):
// 1280 tokens in 5 24.6, 34.4, 44.6; 4607 in 16 62.8, 51.3, 54.2; 4607 in 4 93.2, 105, 146; 8192 in 16 118, 98.5, 94.8
// and even 106, 84.9, 81.0; 8192 in 1 537, 556, 544; 9212 in 8 171, 150, 157; 9215 in 4 276, 257, 284; 13496 in 8 326,
// 296, 286; 1200 in 30 even 30.7, 27.4, 22.6; one of 512 and 15 of 64 24.9, 35.2, 45.4; one of 2000 and 20 of 20 65.9, 101, 141;
// one of 1024 and 30 of 100 55.1, 61.5, 81.8; one of 4096 and 100 of 20 220, 245, 280, and 16 of 512 257, 227, 289.
template <class Cost>
inline int cheapest_heads(int64_t hq, int64_t hk, Cost cost) {
  int best = 1;
  double best_cost = cost(1.0);
  for (int heads = 2; heads <= 4 && heads <= hq / hk; ++heads) {
    if ((hq / hk) % heads) continue;
    const double c = cost((double)heads);
    if (c < best_cost) { best = heads; best_cost = c; }
  }
  return best;
}

// For segments of similar lengths (the lengths are on the device), the longest taken as 1.5 times the mean: the SMs'
// share of all units (whole waves of the mean one where they are few) or the longest unit, an end of 1.5 steps each.
inline int heads_for_similar_segments(int64_t n_tokens, int64_t n_segments, int64_t hq, int64_t hk) {
  const double depth = (double)((n_tokens + n_segments * kBQ - 1) / (n_segments * kBQ)), end = 1.5;
  const double walk = (depth + 1.0) / 2.0, all = depth * (double)n_segments * (double)hq / sm_count();
  return cheapest_heads(hq, hk, [&](double heads) {
    const double units = all / heads, share = (units < 3.0 ? ceil(units) : units) * (heads * walk + end);
    return fmax(share, 1.5 * heads * depth + end);
  });
}

// With a bound on the longest segment (the others taken as equal): the SMs' share of all units or the unit on its
// first tile, three steps each for what a unit pays besides its walk; both where the tiles are in plain order (more
// than 64 segments), which starts the longest walks anywhere. A bound that is too large leaves heads apart that
// could have gone together; one that is too small costs time, nothing else. Of 27 rows of 64 to 13496 tokens, 12 / 2 and 32 /
// 8 heads, this takes the fastest number of heads or one at most 4 % slower; the rule above is up to 50 % slower on
// rows of which one segment is long (2000 and 20 of 20: 99 us, this one 65).
inline int heads_for_bounded_segments(int64_t n_tokens, int64_t n_segments, int64_t longest, int64_t hq, int64_t hk) {
  auto tiles_of = [](double tokens) { return ceil(tokens / kBQ); };
  if (longest > n_tokens) longest = n_tokens;
  const double others = (double)(n_segments - 1), deep = tiles_of((double)longest), end = 3.0;
  const double rest = others > 0.0 ? tiles_of((double)(n_tokens - longest) / others) : 0.0;
  const double tiles = deep + others * rest, steps = (deep * (deep + 1.0) + others * rest * (rest + 1.0)) / 2.0;
  return cheapest_heads(hq, hk, [&](double heads) {
    const double share = (steps * heads + tiles * end) * ((double)hq / heads) / sm_count(), unit = heads * deep + end;
    return n_segments > 64 ? share + unit : fmax(share, unit);
  });
}

// longest 0: no bound is known.
inline int backward_heads_per_cta(int64_t n_tokens, int64_t n_segments, int64_t longest, int64_t hq, int64_t hk) {
  return longest > 0 ? heads_for_bounded_segments(n_tokens, n_segments, longest, hq, hk)
                     : heads_for_similar_segments(n_tokens, n_segments, hq, hk);
}

}  // namespace
}  // namespace soup

extern "C" int soup_attn_fwd(const void* q, const void* k, const void* v, const int32_t* cu_rows,
                             void* out, float* lse, int64_t n_tokens, int64_t n_segments,
                             int64_t hq, int64_t hk, int64_t head_dim, int64_t q_pitch,
                             int64_t k_pitch, int64_t v_pitch, float scale, void* stream) {
  using namespace soup;
  if (n_tokens == 0 || n_segments == 0) return SOUP_OK;
  if (!q || !k || !v || !cu_rows || !out || !lse) SOUP_FAIL(SOUP_ERR_ARG, "attn_fwd: null pointer");
  if (head_dim != kD) SOUP_FAIL(SOUP_ERR_ARG, "attn_fwd: head_dim must be 128");
  if (n_tokens < 0 || n_segments < 0 || hq <= 0 || hk <= 0 || hq % hk)
    SOUP_FAIL(SOUP_ERR_ARG, "attn_fwd: bad sizes (query heads must be a multiple of key heads)");
  if (n_tokens > (1 << 30) || n_segments > 65535 || hq > 65535)
    SOUP_FAIL(SOUP_ERR_ARG, "attn_fwd: too many tokens, segments or heads");
  if (q_pitch < hq * kD || k_pitch < hk * kD || v_pitch < hk * kD || (q_pitch | k_pitch | v_pitch) & 7)
    SOUP_FAIL(SOUP_ERR_ARG, "attn_fwd: row pitches must cover the heads and be multiples of 8 elements");
  if (!aligned16(q) || !aligned16(k) || !aligned16(v) || !aligned16(out))
    SOUP_FAIL(SOUP_ERR_ARG, "attn_fwd: pointers must be 16-byte aligned");
  // a runtime call first: it makes the device's context current on this thread (autograd runs
  // backward on threads of its own), which the driver's tensor-map encoder needs
  const bool negative = scale < 0.f;
  const int heads = negative ? 1 : forward_heads_per_cta(n_tokens, n_segments, hq, hk);
  const auto kernel = negative ? attn_fwd_kernel<1, true> : heads == 1 ? attn_fwd_kernel<1, false> : attn_fwd_kernel<2, false>;
  const size_t smem = (heads == 1 ? sizeof(FwdSmem<1>) : sizeof(FwdSmem<2>)) + 1024;
  if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)
    SOUP_FAIL(SOUP_ERR_LAUNCH, "attn_fwd: shared memory attribute");
  CUtensorMap mq, mk, mv;
  if (umma::encode_map_2d_16bit(&mq, q, (uint64_t)n_tokens, (uint64_t)(hq * kD), (uint64_t)q_pitch, kBQ, 64, false) ||
      umma::encode_map_2d_16bit(&mk, k, (uint64_t)n_tokens, (uint64_t)(hk * kD), (uint64_t)k_pitch, kBKV, 64, false) ||
      umma::encode_map_2d_16bit(&mv, v, (uint64_t)n_tokens, (uint64_t)(hk * kD), (uint64_t)v_pitch, kBKV, 64, false))
    SOUP_FAIL(SOUP_ERR_LAUNCH, "attn_fwd: cuTensorMapEncodeTiled failed");
  AttnArgs a;
  a.cu = cu_rows;
  a.out = reinterpret_cast<__half*>(out);
  a.lse = lse;
  a.n = (int)n_tokens;
  a.segments = (int)n_segments;
  a.hq = (int)hq;
  a.group = (int)(hq / hk);
  // a scale of zero as the smallest above it: x * scale is as good as zero, and a hidden key's -inf stays -inf
  a.scale_log2 = fmaxf(fabsf(scale) * kLog2e, FLT_MIN);
  a.scale_far = exp2f(ceilf(log2f(a.scale_log2)));
  a.status = rowpipe::status_word();
  const int64_t ctas = tile_slots(n_tokens, n_segments) * (hq / heads);
  if (ctas > INT32_MAX) SOUP_FAIL(SOUP_ERR_ARG, "attn_fwd: too many tokens, segments or heads");
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  kernel<<<(unsigned)ctas, heads == 1 ? kFwdThreads<1> : kFwdThreads<2>, smem, st>>>(mq, mk, mv, a);
  SOUP_CHECK_LAUNCH("attn_fwd");
  return SOUP_OK;
}

extern "C" int soup_attn_bwd_bounded(const void* q, const void* k, const void* v, const void* out,
                                     const void* d_out, const float* lse, const int32_t* cu_rows, float* dq,
                                     float* dk, float* dv, void* workspace, int64_t workspace_bytes,
                                     int64_t n_tokens, int64_t n_segments, int64_t longest, int64_t hq, int64_t hk,
                                     int64_t head_dim, int64_t q_pitch, int64_t k_pitch, int64_t v_pitch,
                                     float scale, void* stream) {
  using namespace soup;
  if (n_tokens == 0) return SOUP_OK;
  if (!q || !k || !v || !out || !d_out || !lse || !cu_rows || !dq || !dk || !dv || !workspace)
    SOUP_FAIL(SOUP_ERR_ARG, "attn_bwd: null pointer");
  if (head_dim != kD) SOUP_FAIL(SOUP_ERR_ARG, "attn_bwd: head_dim must be 128");
  if (n_tokens < 0 || n_segments < 0 || hq <= 0 || hk <= 0 || hq % hk)
    SOUP_FAIL(SOUP_ERR_ARG, "attn_bwd: bad sizes (query heads must be a multiple of key heads)");
  if (longest < 0) SOUP_FAIL(SOUP_ERR_ARG, "attn_bwd: the longest segment's bound is negative");
  const int heads = n_segments > 0 ? backward_heads_per_cta(n_tokens, n_segments, longest, hq, hk) : 1;
  const int64_t ctas = tile_slots(n_tokens, n_segments) * (hq / heads);
  if (n_tokens > (1 << 30) || n_segments > 65535 || hq > 65535 || ctas > INT32_MAX)
    SOUP_FAIL(SOUP_ERR_ARG, "attn_bwd: too many tokens, segments or heads");
  if (q_pitch < hq * kD || k_pitch < hk * kD || v_pitch < hk * kD || (q_pitch | k_pitch | v_pitch) & 7)
    SOUP_FAIL(SOUP_ERR_ARG, "attn_bwd: row pitches must cover the heads and be multiples of 8 elements");
  if (!aligned16(q) || !aligned16(k) || !aligned16(v) || !aligned16(out) || !aligned16(d_out) ||
      !aligned16(dq) || !aligned16(dk) || !aligned16(dv) || !aligned16(workspace))
    SOUP_FAIL(SOUP_ERR_ARG, "attn_bwd: pointers must be 16-byte aligned");
  if (workspace_bytes < n_tokens * hq * (int64_t)sizeof(float2))
    SOUP_FAIL(SOUP_ERR_ARG, "attn_bwd: workspace too small (%lld < %lld)", (long long)workspace_bytes,
              (long long)(n_tokens * hq * (int64_t)sizeof(float2)));
  // a runtime call first (see soup_attn_fwd): backward usually runs on an autograd thread
  if (cudaFuncSetAttribute(attn_bwd_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           (int)sizeof(KvSmem)) != cudaSuccess)
    SOUP_FAIL(SOUP_ERR_LAUNCH, "attn_bwd: shared memory attribute");
  CUtensorMap mq, mdo, mk, mv, mdq, mdk, mdv;
  const uint64_t n = (uint64_t)n_tokens, wq = (uint64_t)(hq * kD), wk = (uint64_t)(hk * kD);
  if (umma::encode_map_2d_16bit(&mq, q, n, wq, (uint64_t)q_pitch, kBQ, 64, false) ||
      umma::encode_map_2d_16bit(&mdo, d_out, n, wq, wq, kBQ, 64, false) ||
      umma::encode_map_2d_16bit(&mk, k, n, wk, (uint64_t)k_pitch, kBKV, 64, false) ||
      umma::encode_map_2d_16bit(&mv, v, n, wk, (uint64_t)v_pitch, kBKV, 64, false) ||
      umma::encode_map_2d_f32(&mdq, dq, n, wq, wq, 32, 32) || umma::encode_map_2d_f32(&mdk, dk, n, wk, wk, 32, 32) ||
      umma::encode_map_2d_f32(&mdv, dv, n, wk, wk, 32, 32))
    SOUP_FAIL(SOUP_ERR_LAUNCH, "attn_bwd: cuTensorMapEncodeTiled failed");
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  const int64_t rows = n_tokens * hq;
  attn_bwd_prep_kernel<<<(unsigned)((rows + kPrepThreads / 16 - 1) / (kPrepThreads / 16)), kPrepThreads, 0, st>>>(
      reinterpret_cast<const __half*>(out), reinterpret_cast<const __half*>(d_out), lse,
      reinterpret_cast<float2*>(workspace), reinterpret_cast<float4*>(dq), reinterpret_cast<float4*>(dk),
      reinterpret_cast<float4*>(dv), rows, n_tokens * hk, (int)n_tokens, (int)hq);
  SOUP_CHECK_LAUNCH("attn_bwd_prep");
  if (n_segments == 0) return SOUP_OK;
  AttnKvArgs a;
  a.cu = cu_rows;
  a.stats = reinterpret_cast<const float2*>(workspace);
  a.n = (int)n_tokens;
  a.segments = (int)n_segments;
  a.hq = (int)hq;
  a.group = (int)(hq / hk);
  a.heads = heads;
  a.scale = scale;
  a.scale_log2 = scale * kLog2e;
  a.status = rowpipe::status_word();
  attn_bwd_kernel<<<(unsigned)ctas, kBwdThreads, sizeof(KvSmem), st>>>(mq, mdo, mk, mv, mdq, mdk, mdv, a);
  SOUP_CHECK_LAUNCH("attn_bwd");
  return SOUP_OK;
}

extern "C" int soup_attn_bwd(const void* q, const void* k, const void* v, const void* out, const void* d_out,
                             const float* lse, const int32_t* cu_rows, float* dq, float* dk, float* dv,
                             void* workspace, int64_t workspace_bytes, int64_t n_tokens, int64_t n_segments,
                             int64_t hq, int64_t hk, int64_t head_dim, int64_t q_pitch, int64_t k_pitch,
                             int64_t v_pitch, float scale, void* stream) {
  return soup_attn_bwd_bounded(q, k, v, out, d_out, lse, cu_rows, dq, dk, dv, workspace, workspace_bytes, n_tokens,
                               n_segments, 0, hq, hk, head_dim, q_pitch, k_pitch, v_pitch, scale, stream);
}

extern "C" int soup_attn_plan_bounded(int64_t n_tokens, int64_t n_segments, int64_t longest, int64_t hq, int64_t hk,
                                      int* forward_heads, int* backward_heads) {
  using namespace soup;
  if (n_tokens <= 0 || n_segments <= 0 || longest < 0 || hq <= 0 || hk <= 0 || hq % hk)
    SOUP_FAIL(SOUP_ERR_ARG, "attn_plan: bad sizes");
  if (forward_heads) *forward_heads = forward_heads_per_cta(n_tokens, n_segments, hq, hk);
  if (backward_heads) *backward_heads = backward_heads_per_cta(n_tokens, n_segments, longest, hq, hk);
  return SOUP_OK;
}

extern "C" int soup_attn_plan(int64_t n_tokens, int64_t n_segments, int64_t hq, int64_t hk, int* forward_heads,
                              int* backward_heads) {
  return soup_attn_plan_bounded(n_tokens, n_segments, 0, hq, hk, forward_heads, backward_heads);
}

extern "C" int soup_attn_bound_matters(int64_t n_tokens, int64_t n_segments, int64_t longest, int64_t hq, int64_t hk) {
  using namespace soup;
  if (n_tokens <= 0 || n_segments <= 0 || longest <= 0 || hq <= 0 || hk <= 0 || hq % hk) return 0;
  return backward_heads_per_cta(n_tokens, n_segments, longest, hq, hk) !=
         backward_heads_per_cta(n_tokens, n_segments, 0, hq, hk);
}
