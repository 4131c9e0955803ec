// The four products of a gated MLP with frozen weights, y = residual + down(silu(gate(x)) * up(x)), forward and
// input gradient, on CTA pairs (tcgen05.mma.cta_group::2, 256 x 256 tiles), each with the elementwise pass
// next to it in its epilogue:
//
//   kUp    gate and up of 128 columns are the two halves of one tile (each CTA of the pair loads one weight's
//          rows); a thread then holds both for its row and writes gate, up and silu(gate) * up
//   kDown  residual + act Wd^T, fp32
//   kDact  d_act = dy Wd stays in tensor memory; gate and up of the tile come in by TMA and leave as their gradients
//   kDx    d_gate Wg + d_up Wu as one product over both, fp32
//
// As library products with elementwise kernels between them a block of the 1.5B model (hidden 1536,
// intermediate 8960) takes 202 us forward and backward at 1280 tokens and 656 at 4608, ten launches that write and
// read d_act, gate, up and the residual once more than needed; here four and 193 and 617 us. What bounds it: at 4608
// tokens, 1.2 PFLOP/s, the power cap: at the 1.55 GHz it leaves the tensor pipe is active 68 (kUp), 71 (kDown) and 51 % (kDact, whose
// tiles are only 24 K blocks long) of the cycles, L2 moves 12 to 14 TB/s, 38 to 43 % of its peak, and the ports into the SMs are
// busy 30 to 37 %. At 1280 tokens, 1.1 PFLOP/s, the last wave of tiles as well: the busiest pair walks 402 K blocks where 341 are
// its share. soup_mlp_pays has the sizes at which the library's products, in other tile shapes, are faster.
//
// Tiles are 256 columns wide because shared memory serves the tensor core 128 bytes a clock: a 256 x 128
// tile wants 96 for operands and 96 for the loads that replace them, a 256 x 256 tile 64 and 64. The two products
// that end in [rows, hidden] have few such tiles, so K may be split in two (`splits`); the halves are added to
// zeros, which the launch before has written with an idle warp, so the result has one value whichever comes first.
//
// Roles per CTA: warp 0 loads the operands (a ring of five 32 KB stages), warp 1 of the leader issues the
// products, warp 3 clears, warps 4-11 are the epilogue (two per quarter of the lanes) on one of two
// accumulators while the products fill the other. Every wait is bounded (umma::mbar_wait), codes 111-115.
#include <cuda.h>

#include "common.cuh"
#include "rowpipe.cuh"
#include "silu.cuh"
#include "umma.cuh"

namespace soup {
namespace {

using namespace umma;

constexpr int kBM = 128;             // rows per CTA; a pair owns 256
constexpr int kBN = 256;             // columns per tile
constexpr int kBK = 64;              // one 128-byte swizzle row
constexpr int kABytes = kBM * kBK * 2;
constexpr int kStageBytes = kABytes + (kBN / 2) * kBK * 2;
constexpr int kStages = 5;
constexpr int kEpiWarps = 8, kFirstEpi = 4, kClearWarp = 3;
constexpr int kThreads = (kFirstEpi + kEpiWarps) * 32;
constexpr int kBoxBytes = 4096;      // 32 rows x 128 bytes: 64 fp16 or 32 fp32 columns, swizzled
constexpr int kSmem = kStages * kStageBytes + kEpiWarps * 2 * kBoxBytes + 1024 + 256;

enum Mode { kUp, kDown, kDact, kDx };

struct Smem {
  uint8_t* tiles;
  uint8_t* boxes;         // [kEpiWarps][2]
  uint64_t *full, *empty, *acc_full, *acc_empty, *in_full;   // in_full: [kEpiWarps]
  uint32_t* tmem_base;
  int* abort_flag;
};
__device__ __forceinline__ Smem carve(uint8_t* raw) {
  Smem s;
  s.tiles = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(raw) + 1023u) & ~uintptr_t(1023u));
  s.boxes = s.tiles + kStages * kStageBytes;
  s.full = reinterpret_cast<uint64_t*>(s.boxes + kEpiWarps * 2 * kBoxBytes);
  s.empty = s.full + kStages;
  s.acc_full = s.empty + kStages;
  s.acc_empty = s.acc_full + 2;
  s.in_full = s.acc_empty + 2;
  s.tmem_base = reinterpret_cast<uint32_t*>(s.in_full + kEpiWarps);
  s.abort_flag = reinterpret_cast<int*>(s.tmem_base + 1);
  return s;
}

struct MlpArgs {
  int rows, cols;          // of the output; kUp: columns of gate and of up
  int n_kb;                // 64-wide K blocks of a source
  int sources, splits;     // kDx has two operand pairs; K splits of a tile (with two sources: one each)
  const float* residual;   // kDown
  float4* clear;           // nullable: zeros for the next launch
  int64_t clear_vecs;
  int keep_act;            // kUp: the activation is wanted too
  int* status;
};

// Row `lane` of a 32-row swizzled box: eight 16-byte pieces.
__device__ __forceinline__ uint4* piece_of(uint8_t* box, int lane, int j) {
  return reinterpret_cast<uint4*>(box + lane * 128 + ((j ^ (lane & 7)) << 4));
}
__device__ __forceinline__ uint32_t pack_half2(float a, float b) {
  const __half2 h = __floats2half2_rn(a, b);
  return *reinterpret_cast<const uint32_t*>(&h);
}
__device__ __forceinline__ float2 unpack_half2(uint32_t v) {
  return __half22float2(*reinterpret_cast<const __half2*>(&v));
}

template <int MODE>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kThreads, 1)
mlp_gemm_kernel(const __grid_constant__ CUtensorMap map_a0, const __grid_constant__ CUtensorMap map_a1,
                const __grid_constant__ CUtensorMap map_b0, const __grid_constant__ CUtensorMap map_b1,
                const __grid_constant__ CUtensorMap map_in0, const __grid_constant__ CUtensorMap map_in1,
                const __grid_constant__ CUtensorMap map_o0, const __grid_constant__ CUtensorMap map_o1,
                const __grid_constant__ CUtensorMap map_o2, const MlpArgs a) {
  constexpr bool kBMN = MODE == kDact || MODE == kDx;             // the weight's columns are the tile's
  constexpr int kTileCols = MODE == kUp ? kBN / 2 : kBN;          // output columns of a tile
  extern __shared__ uint8_t raw[];
  const Smem s = carve(raw);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();
  pdl_trigger();
  if (threadIdx.x == 0) {
    for (int i = 0; i < kStages; ++i) { mbar_init(&s.full[i], 1); mbar_init(&s.empty[i], 1); }
    for (int i = 0; i < 2; ++i) { mbar_init(&s.acc_full[i], 1); mbar_init(&s.acc_empty[i], 2 * kEpiWarps); }
    for (int i = 0; i < kEpiWarps; ++i) mbar_init(&s.in_full[i], 1);
    *s.abort_flag = 0;
    fence_barrier_init();
    prefetch_tensormap(&map_a0);
    prefetch_tensormap(&map_b0);
  }
  __syncthreads();
  cluster_sync_all();   // the peer's barriers are there before anything signals them
  if (warp == 1) {
    tmem_alloc_pair(s.tmem_base, 512);
    tmem_relinquish_pair();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem = *s.tmem_base;
  pdl_wait();
  volatile int* abort_flag = s.abort_flag;

  // Units: row tile fastest, so that the row tiles that share weight columns run together; then columns, then splits.
  const int pair = blockIdx.x >> 1, n_pairs = gridDim.x >> 1;
  const int rt = (a.rows + 2 * kBM - 1) / (2 * kBM);
  const int n_tiles = rt * ((a.cols + kTileCols - 1) / kTileCols);
  const int n_units = n_tiles * a.splits, kb_total = a.n_kb * a.sources;

  if (warp == 0) {
    if (lane == 0) {
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int unit = pair; unit < n_units && ok; unit += n_pairs) {
        const int tile = unit % n_tiles, ks = unit / n_tiles;
        const int row0 = (tile % rt) * 2 * kBM + (int)rank * kBM;
        const int col0 = (tile / rt) * kTileCols;
        const int kb_end = kb_total * (ks + 1) / a.splits;
        for (int kb = kb_total * ks / a.splits; kb < kb_end; ++kb) {
          ok = mbar_wait(&s.empty[stage], phase ^ 1u, abort_flag, a.status, 111);
          if (!ok) break;
          uint8_t* st = s.tiles + stage * kStageBytes;
          const uint32_t full = mapa_u32(smem_u32(&s.full[stage]), 0);   // both CTAs' bytes, on the leader's barrier
          if (rank == 0) mbar_expect_tx(&s.full[stage], 2 * kStageBytes);
          const bool second = MODE == kDx && kb >= a.n_kb;
          const int k0 = (second ? kb - a.n_kb : kb) * kBK;
          tma_load_2d_pair(st, second ? &map_a1 : &map_a0, k0, row0, full);
          if (kBMN) {
            const CUtensorMap* mb = second ? &map_b1 : &map_b0;
#pragma unroll
            for (int j = 0; j < 2; ++j)
              tma_load_2d_pair(st + kABytes + j * kBK * 128, mb, col0 + (int)rank * (kBN / 2) + j * 64, k0, full);
          } else if (MODE == kUp) {
            tma_load_2d_pair(st + kABytes, rank ? &map_b1 : &map_b0, k0, col0, full);
          } else {
            tma_load_2d_pair(st + kABytes, &map_b0, k0, col0 + (int)rank * (kBN / 2), full);
          }
          if (++stage == kStages) { stage = 0; phase ^= 1u; }
        }
      }
    }
  } else if (warp == 1) {
    if (lane == 0 && rank == 0) {
      constexpr uint32_t idesc = make_idesc_f16(2 * kBM, kBN, kFmtF16, kFmtF16, false, kBMN);
      int stage = 0, it = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int unit = pair; unit < n_units && ok; unit += n_pairs, ++it) {
        const int ks = unit / n_tiles, ab = it & 1;
        ok = mbar_wait(&s.acc_empty[ab], ((it >> 1) & 1) ^ 1, abort_flag, a.status, 112);
        if (!ok) break;
        tc_fence_after_sync();
        const uint32_t d = tmem + ab * kBN;
        const int kb0 = kb_total * ks / a.splits, kb_end = kb_total * (ks + 1) / a.splits;
        for (int kb = kb0; kb < kb_end; ++kb) {
          ok = mbar_wait(&s.full[stage], phase, abort_flag, a.status, 113);
          if (!ok) break;
          tc_fence_after_sync();
          const uint32_t at = smem_u32(s.tiles + stage * kStageBytes);
          const uint64_t da = make_smem_desc(at, 16, 1024);
          // MN-major: the two 64-column boxes are 8 KB apart (leading offset), a step of 16 k is 2 KB
          const uint64_t db = make_smem_desc(at + kABytes, kBMN ? kBK * 128 : 16, 1024);
#pragma unroll
          for (int k4 = 0; k4 < kBK / 16; ++k4)
            mma_f16_ss_pair(d, da + k4 * 2, db + k4 * (kBMN ? 2048 >> 4 : 2), idesc, kb != kb0 || k4 != 0);
          tc_commit_pair(&s.empty[stage], 3);
          if (++stage == kStages) { stage = 0; phase ^= 1u; }
        }
        if (ok) tc_commit_pair(&s.acc_full[ab], 3);
      }
    }
  } else if (warp == kClearWarp) {
    if (a.clear)
      for (int64_t i = (int64_t)blockIdx.x * 32 + lane; i < a.clear_vecs; i += (int64_t)gridDim.x * 32)
        a.clear[i] = make_float4(0.f, 0.f, 0.f, 0.f);
  } else if (warp >= kFirstEpi) {
    const int q = warp & 3, e = (warp - kFirstEpi) >> 2;   // lanes [32 q, 32 q + 32), column half or block e
    uint8_t* box = s.boxes + (warp - kFirstEpi) * 2 * kBoxBytes;
    const uint32_t lanes = tmem + ((uint32_t)(q * 32) << 16);
    auto release = [&](int ab) {
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) {
        if (rank == 0) mbar_arrive(&s.acc_empty[ab]);
        else mbar_arrive_remote(mapa_u32(smem_u32(&s.acc_empty[ab]), 0));
      }
    };
    auto row_of = [&](int unit) { return ((unit % n_tiles) % rt) * 2 * kBM + (int)rank * kBM + q * 32; };
    auto col_of = [&](int unit) { return ((unit % n_tiles) / rt) * kTileCols; };
    int it = 0, turn = 0;
    uint32_t in_phase = 0;
    bool ok = true;
    // kDact: this warp's 32 x 64 boxes of gate and up, for the next block of columns it works on
    auto request = [&](int row, int col) {
      if (lane == 0) {
        tma_store_wait_read<0>();   // the gradients stored from the same boxes
        mbar_expect_tx(&s.in_full[warp - kFirstEpi], 2 * kBoxBytes);
        tma_load_2d(box, &map_in0, col, row, &s.in_full[warp - kFirstEpi]);
        tma_load_2d(box + kBoxBytes, &map_in1, col, row, &s.in_full[warp - kFirstEpi]);
      }
    };
    if (MODE == kDact && pair < n_units) request(row_of(pair), col_of(pair) + e * 64);
    for (int unit = pair; unit < n_units; unit += n_pairs, ++it) {
      const int ab = it & 1;
      const int row0 = row_of(unit), col0 = col_of(unit);
      float4 res[8];
      auto residual = [&](int col) {   // 32 columns of this thread's row
        const int row = row0 + lane;
#pragma unroll
        for (int j = 0; j < 8; ++j)
          res[j] = row < a.rows && col + 4 * j < a.cols
                       ? *reinterpret_cast<const float4*>(a.residual + (int64_t)row * a.cols + col + 4 * j)
                       : make_float4(0.f, 0.f, 0.f, 0.f);
      };
      const bool add = MODE == kDown && unit < n_tiles;   // the first split brings the residual
      if (MODE == kDown && add) residual(col0 + e * 128);
      ok = __all_sync(0xffffffffu, mbar_wait(&s.acc_full[ab], (it >> 1) & 1, abort_flag, a.status, 114));
      if (!ok) break;
      tc_fence_after_sync();
      const uint32_t acc = lanes + ab * kBN;
      if (MODE == kUp) {
        uint32_t gp[32], up[32], ap[32];
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          uint32_t x[32], y[32];
          tmem_ld_32x32(acc + e * 64 + c * 32, x);
          tmem_ld_32x32(acc + 128 + e * 64 + c * 32, y);
          tmem_ld_wait_on(x);
          tmem_ld_wait_on(y);
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            const uint32_t g = pack_half2(__uint_as_float(x[2 * j]), __uint_as_float(x[2 * j + 1]));
            const uint32_t u = pack_half2(__uint_as_float(y[2 * j]), __uint_as_float(y[2 * j + 1]));
            const float2 gf = unpack_half2(g), uf = unpack_half2(u);
            gp[c * 16 + j] = g;
            up[c * 16 + j] = u;
            ap[c * 16 + j] = pack_half2(silu_of(gf.x) * uf.x, silu_of(gf.y) * uf.y);
          }
        }
        release(ab);
        const int col = col0 + e * 64;
        if (row0 < a.rows && col < a.cols) {
          auto leave = [&](const uint32_t (&v)[32], const CUtensorMap* map) {
            uint8_t* b = box + turn * kBoxBytes;
            turn ^= 1;
            if (lane == 0) tma_store_wait_read<1>();   // the store two boxes ago has read this one
            __syncwarp();
#pragma unroll
            for (int j = 0; j < 8; ++j) *piece_of(b, lane, j) = make_uint4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
            fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) {
              tma_store_2d(map, b, col, row0);
              tma_store_commit();
            }
          };
          leave(gp, &map_o0);
          leave(up, &map_o1);
          if (a.keep_act) leave(ap, &map_o2);
        }
      } else if (MODE == kDact) {
#pragma unroll 1
        for (int h = 0; h < 2; ++h) {
          const int block = e + 2 * h, col = col0 + block * 64;
          ok = __all_sync(0xffffffffu, mbar_wait(&s.in_full[warp - kFirstEpi], in_phase, abort_flag, a.status, 115));
          if (!ok) break;
          in_phase ^= 1u;
#pragma unroll
          for (int c = 0; c < 2; ++c) {
            uint32_t y[32];
            tmem_ld_32x32(acc + block * 64 + c * 32, y);
            tmem_ld_wait_on(y);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              uint4* pg = piece_of(box, lane, c * 4 + j);
              uint4* pu = piece_of(box + kBoxBytes, lane, c * 4 + j);
              const uint4 gv = *pg, uv = *pu;
              const uint32_t g[4] = {gv.x, gv.y, gv.z, gv.w}, u[4] = {uv.x, uv.y, uv.z, uv.w};
              uint32_t dg[4], du[4];
#pragma unroll
              for (int k = 0; k < 4; ++k) {
                // the gradient of the activation rounded to fp16, as a tensor of its own would be
                const float2 d = unpack_half2(pack_half2(__uint_as_float(y[8 * j + 2 * k]), __uint_as_float(y[8 * j + 2 * k + 1])));
                const float2 gf = unpack_half2(g[k]), uf = unpack_half2(u[k]);
                const float s0 = __fdividef(1.0f, silu_denom(gf.x)), s1 = __fdividef(1.0f, silu_denom(gf.y));
                dg[k] = pack_half2(d.x * uf.x * silu_slope(gf.x, s0), d.y * uf.y * silu_slope(gf.y, s1));
                du[k] = pack_half2(d.x * (gf.x * s0), d.y * (gf.y * s1));
              }
              *pg = make_uint4(dg[0], dg[1], dg[2], dg[3]);
              *pu = make_uint4(du[0], du[1], du[2], du[3]);
            }
          }
          if (h == 1) release(ab);
          fence_proxy_async_smem();
          __syncwarp();
          if (lane == 0 && row0 < a.rows && col < a.cols) {
            tma_store_2d(&map_o0, box, col, row0);
            tma_store_2d(&map_o1, box + kBoxBytes, col, row0);
            tma_store_commit();
          }
          if (h == 0) request(row0, col + 128);
          else if (unit + n_pairs < n_units) request(row_of(unit + n_pairs), col_of(unit + n_pairs) + e * 64);
        }
        if (!ok) break;
      } else {
        const CUtensorMap* map = &map_o0;
        const int left = a.cols - (col0 + e * 128);
        const int n_boxes = row0 < a.rows ? min(4, (left + 31) / 32) : 0;
#pragma unroll 1
        for (int c = 0; c < n_boxes; ++c) {
          const int col = col0 + e * 128 + c * 32;
          uint32_t x[32];
          tmem_ld_32x32(acc + e * 128 + c * 32, x);
          uint8_t* b = box + turn * kBoxBytes;
          turn ^= 1;
          if (lane == 0) tma_store_wait_read<1>();
          __syncwarp();
          tmem_ld_wait_on(x);
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            float4 v = make_float4(__uint_as_float(x[4 * j]), __uint_as_float(x[4 * j + 1]),
                                   __uint_as_float(x[4 * j + 2]), __uint_as_float(x[4 * j + 3]));
            if (MODE == kDown && add) { v.x += res[j].x; v.y += res[j].y; v.z += res[j].z; v.w += res[j].w; }
            *reinterpret_cast<float4*>(piece_of(b, lane, j)) = v;
          }
          if (MODE == kDown && add && c + 1 < n_boxes) residual(col + 32);
          fence_proxy_async_smem();
          __syncwarp();
          if (lane == 0) {
            if (a.splits > 1) tma_reduce_add_2d(map, b, col, row0);
            else tma_store_2d(map, b, col, row0);
            tma_store_commit();
          }
        }
        release(ab);
      }
    }
    if (!ok && MODE == kDact) {   // a requested box may still be on its way
      for (int i = 0; i < 64; ++i) __nanosleep(2000);
    }
    if (lane == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");   // everything has left
  }
  tc_fence_before_sync();
  __syncthreads();
  if (*abort_flag) {   // copies that may still be in flight land before the shared memory is released
    for (int i = 0; i < 64; ++i) __nanosleep(2000);
    __syncthreads();
  }
  // the leader's products read the peer's shared memory and both signal each other's barriers
  cluster_sync_all();
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc_pair(tmem, 512);
  }
}

// A runtime call before the tensor maps: it makes the device's context current on this thread (autograd runs
// backward on threads of its own), which the driver's encoder needs.
template <int MODE>
bool allow_smem() {
  return cudaFuncSetAttribute(mlp_gemm_kernel<MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem) == cudaSuccess;
}

template <int MODE>
int launch(const char* name, const CUtensorMap (&m)[9], const MlpArgs& a, cudaStream_t st) {
  const int64_t tile_cols = MODE == kUp ? kBN / 2 : kBN;
  const int64_t units = (int64_t)((a.rows + 2 * kBM - 1) / (2 * kBM)) * ((a.cols + tile_cols - 1) / tile_cols) * a.splits;
  const int64_t pairs = sm_count() / 2;
  const unsigned grid = 2u * (unsigned)(units < pairs ? units : pairs);
  launch_dependent(mlp_gemm_kernel<MODE>, grid, kThreads, kSmem, st, m[0], m[1], m[2], m[3], m[4], m[5], m[6], m[7], m[8], a);
  SOUP_CHECK_LAUNCH(name);
  return SOUP_OK;
}

// K blocks on the busiest pair of a product with `tiles` tiles of `kb` blocks in `splits` K ranges, and eight for
// what a launch's end does not hide.
inline int64_t span(int64_t tiles, int64_t kb, int splits) {
  const int64_t pairs = sm_count() / 2;
  return (tiles * splits + pairs - 1) / pairs * ((kb + splits - 1) / splits) + 8;
}
inline int64_t tiles_of(int64_t rows, int64_t cols, int64_t tile_cols) {
  return (rows + 2 * kBM - 1) / (2 * kBM) * ((cols + tile_cols - 1) / tile_cols);
}
// K splits (one or two) of the products that end in [rows, hidden].
inline int pick_splits(int64_t rows, int64_t hidden, int64_t kb_total) {
  const int64_t tiles = tiles_of(rows, hidden, kBN);
  return span(tiles, kb_total, 2) < span(tiles, kb_total, 1) ? 2 : 1;
}

// Sizes whose tile counts and coordinates stay far inside 32 bits.
inline bool fits(int64_t rows, int64_t hidden, int64_t inter) {
  return rows <= (1 << 22) && hidden <= (1 << 20) && inter <= (1 << 20);
}

int check(const char* name, int64_t rows, int64_t hidden, int64_t inter) {
  if (rows < 0 || hidden <= 0 || inter <= 0 || hidden % 8 || inter % 8)
    SOUP_FAIL(SOUP_ERR_ARG, "%s: the widths must be multiples of 8", name);
  if (!fits(rows, hidden, inter)) SOUP_FAIL(SOUP_ERR_ARG, "%s: too large", name);
  return SOUP_OK;
}

}  // namespace
}  // namespace soup

// Whether the two launches of a direction take these sizes and are faster than the library's products with the
// elementwise kernel between them: a question of how full the last wave of 256 x 256 tiles is. The share of the busiest
// pair's K blocks that the rows need (in per cent), and the library's time over this file's, forward; backward, by rows
// (each the median of 9 to 15 replays in turn):
//   896 / 4864     1280 56 0.90; 45 0.83, 2816 63 1.00; 56 1.04, 4096 83 1.12; 73 1.14, 8192 83 1.14; 78 1.15, 24576 1.05; 1.12
//   1536 / 8960    512 51 0.83; 38 0.81, 1152 74 0.96; 67 0.97, 1280 83 1.06; 75 1.04, 2048 78 1.02; 70 1.02, 3072 92 1.13;
//                  93 1.18, 4608 93 1.07; 94 1.06, 8192 92 1.11; 88 1.09, 16384 1.01; 1.10, 49152 1.03; 1.34
//   2048 / 11008   512 56 0.93; 44 0.84, 1024 85 1.11; 79 1.05, 1280 73 0.94; 61 0.86, 1536 82 1.04; 69 0.97, 3072 93 1.15; 89 1.06
//   2560 / 9728    2048 79 1.01; 73 0.95, 3072 92 1.17; 85 1.11
//   3584 / 18944   512 87 0.99; 80 1.01, 768 78 0.93; 65 0.89, 896 77 0.96; 71 0.92, 1280 1.09; 1.08, 2048 1.06; 1.07, 8192 1.06; 1.19
//   4096 / 14336   1152 76 0.91; 69 0.86, 1280 84 0.99; 77 0.98, 2048 1.08; 1.03, 8192 1.20; 1.21
//   5120 / 27648   896 75 0.88; 68 0.82, 1024 86 0.98; 78 0.86, 1152 84 1.03; 81 0.95, 1280 1.08; 1.05, 4096 1.06; 1.07
//   8192 / 28672   512 85 0.98; 82 0.96, 1152 82 0.93; 80 0.90, 1280 1.04; 1.02, 4096 1.21; 1.22
// Up to a width of 2048 a share of 76, backward 69, per cent draws the line. Wider weights have tiles enough at any
// number of rows, and the library's smaller tiles win where the rows are not: the line is five row tiles there.
extern "C" int soup_mlp_pays(int64_t rows, int64_t hidden, int64_t inter, int backward) {
  using namespace soup;
  if (rows <= 0 || hidden <= 0 || inter <= 0 || !fits(rows, hidden, inter)) return 0;
  const int64_t kb_in = (hidden + kBK - 1) / kBK, kb_mid = (inter + kBK - 1) / kBK;
  const int64_t kb_out = backward ? 2 * kb_mid : kb_mid, outer = tiles_of(rows, hidden, kBN);
  const int64_t wide = tiles_of(rows, inter, backward ? kBN : kBN / 2);
  const int64_t busy = span(wide, kb_in, 1) + span(outer, kb_out, pick_splits(rows, hidden, kb_out));
  const double needed = 3.0 * (double)rows * (double)hidden * (double)inter /
                        ((double)(2 * kBM) * kBN * kBK * (double)(sm_count() / 2));
  const bool narrow = hidden <= 2048;
  if (!narrow && rows < 5 * 2 * kBM) return 0;
  return needed >= (backward && narrow ? 0.69 : 0.76) * (double)busy;
}

extern "C" int soup_mlp_fwd(const void* x16, const float* residual, const void* w_gate, const void* w_up,
                            const void* w_down, void* gate, void* up, void* act, float* out, int64_t rows,
                            int64_t hidden, int64_t inter, void* stream) {
  using namespace soup;
  const int rc = check("mlp_fwd", rows, hidden, inter);
  if (rc != SOUP_OK || rows == 0) return rc;
  const void* all[] = {x16, w_gate, w_up, gate, up, w_down, residual, act, out};
  for (int i = 0; i < (out ? 9 : 5); ++i)
    if (!all[i] || !aligned16(all[i])) SOUP_FAIL(SOUP_ERR_ARG, "mlp_fwd: pointers must be set and 16-byte aligned");
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  const int64_t kb_in = (hidden + kBK - 1) / kBK, kb_mid = (inter + kBK - 1) / kBK;
  const int splits = pick_splits(rows, hidden, kb_mid);
  if (!allow_smem<kUp>() || !allow_smem<kDown>()) SOUP_FAIL(SOUP_ERR_LAUNCH, "mlp_fwd: shared memory attribute");
  int* status = rowpipe::status_word();
  using umma::encode_map_2d_16bit;
  CUtensorMap x, g, u, og, ou, oa, ain, wd, o;
  if (encode_map_2d_16bit(&x, x16, rows, hidden, hidden, kBM, kBK, false) ||
      encode_map_2d_16bit(&g, w_gate, inter, hidden, hidden, kBN / 2, kBK, false) ||
      encode_map_2d_16bit(&u, w_up, inter, hidden, hidden, kBN / 2, kBK, false) ||
      encode_map_2d_16bit(&og, gate, rows, inter, inter, 32, 64, false) ||
      encode_map_2d_16bit(&ou, up, rows, inter, inter, 32, 64, false) ||
      (out && (encode_map_2d_16bit(&oa, act, rows, inter, inter, 32, 64, false) ||
               encode_map_2d_16bit(&ain, act, rows, inter, inter, kBM, kBK, false) ||
               encode_map_2d_16bit(&wd, w_down, hidden, inter, inter, kBN / 2, kBK, false) ||
               umma::encode_map_2d_f32(&o, out, rows, hidden, hidden, 32, 32))))
    SOUP_FAIL(SOUP_ERR_LAUNCH, "mlp_fwd: cuTensorMapEncodeTiled failed");
  MlpArgs a = {};
  a.status = status;
  a.rows = (int)rows;
  a.cols = (int)inter;
  a.n_kb = (int)kb_in;
  a.sources = a.splits = 1;
  if (!out) {
    const CUtensorMap m_pair[9] = {x, x, g, u, x, x, og, ou, ou};
    return launch<kUp>("mlp_up", m_pair, a, st);
  }
  a.keep_act = 1;
  if (splits > 1) {
    a.clear = reinterpret_cast<float4*>(out);
    a.clear_vecs = rows * hidden / 4;
  }
  const CUtensorMap m_up[9] = {x, x, g, u, x, x, og, ou, oa};
  const int r1 = launch<kUp>("mlp_up", m_up, a, st);
  if (r1 != SOUP_OK) return r1;
  a.clear = nullptr;
  a.cols = (int)hidden;
  a.n_kb = (int)kb_mid;
  a.splits = splits;
  a.residual = residual;
  const CUtensorMap m_down[9] = {ain, ain, wd, wd, ain, ain, o, o, o};
  return launch<kDown>("mlp_down", m_down, a, st);
}

extern "C" int soup_mlp_bwd(const void* dy16, const void* gate, const void* up, const void* w_gate,
                            const void* w_up, const void* w_down, void* d_gate, void* d_up, float* dx,
                            int64_t rows, int64_t hidden, int64_t inter, void* stream) {
  using namespace soup;
  const int rc = check("mlp_bwd", rows, hidden, inter);
  if (rc != SOUP_OK || rows == 0) return rc;
  const void* all[] = {dy16, gate, up, w_gate, w_up, w_down, d_gate, d_up, dx};
  for (const void* p : all)
    if (!p || !aligned16(p)) SOUP_FAIL(SOUP_ERR_ARG, "mlp_bwd: pointers must be set and 16-byte aligned");
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  const int64_t kb_in = (hidden + kBK - 1) / kBK, kb_mid = (inter + kBK - 1) / kBK;
  const int splits = pick_splits(rows, hidden, 2 * kb_mid);
  if (!allow_smem<kDact>() || !allow_smem<kDx>()) SOUP_FAIL(SOUP_ERR_LAUNCH, "mlp_bwd: shared memory attribute");
  int* status = rowpipe::status_word();
  using umma::encode_map_2d_16bit;
  CUtensorMap y, wd, gi, ui, og, ou, ga, ua, wg, wu, o;
  if (encode_map_2d_16bit(&y, dy16, rows, hidden, hidden, kBM, kBK, false) ||
      encode_map_2d_16bit(&wd, w_down, hidden, inter, inter, kBK, 64, false) ||
      encode_map_2d_16bit(&gi, gate, rows, inter, inter, 32, 64, false) ||
      encode_map_2d_16bit(&ui, up, rows, inter, inter, 32, 64, false) ||
      encode_map_2d_16bit(&og, d_gate, rows, inter, inter, 32, 64, false) ||
      encode_map_2d_16bit(&ou, d_up, rows, inter, inter, 32, 64, false) ||
      encode_map_2d_16bit(&ga, d_gate, rows, inter, inter, kBM, kBK, false) ||
      encode_map_2d_16bit(&ua, d_up, rows, inter, inter, kBM, kBK, false) ||
      encode_map_2d_16bit(&wg, w_gate, inter, hidden, hidden, kBK, 64, false) ||
      encode_map_2d_16bit(&wu, w_up, inter, hidden, hidden, kBK, 64, false) ||
      umma::encode_map_2d_f32(&o, dx, rows, hidden, hidden, 32, 32))
    SOUP_FAIL(SOUP_ERR_LAUNCH, "mlp_bwd: cuTensorMapEncodeTiled failed");
  MlpArgs a = {};
  a.status = status;
  a.rows = (int)rows;
  a.cols = (int)inter;
  a.n_kb = (int)kb_in;
  a.sources = a.splits = 1;
  if (splits > 1) {
    a.clear = reinterpret_cast<float4*>(dx);
    a.clear_vecs = rows * hidden / 4;
  }
  const CUtensorMap m_act[9] = {y, y, wd, wd, gi, ui, og, ou, ou};
  const int r1 = launch<kDact>("mlp_dact", m_act, a, st);
  if (r1 != SOUP_OK) return r1;
  a.clear = nullptr;
  a.cols = (int)hidden;
  a.n_kb = (int)kb_mid;
  a.sources = 2;
  a.splits = splits;
  const CUtensorMap m_dx[9] = {ga, ua, wg, wu, ga, ga, o, o, o};
  return launch<kDx>("mlp_dx", m_dx, a, st);
}
