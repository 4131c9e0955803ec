// The rank-16 LoRA branch B(A(dropout(x))) * scaling: the product with B of one adapter, or of two, with its
// scaling, and the backward of one.
//
// As torch products the branch's backward is a scaling pass over [rows, out], four products with an extent of
// 16 and a mask kernel between them, and its forward ends in another scaling pass: 151 us for 16384 x 1536
// behind the product with A. Here backward reads the output gradient twice (the second time largely from L2) and
// the fp16 input once and writes the input gradient; the dropped input exists in registers only. 84 us. With dropout,
// packing and the product with A, the branch forward and backward took, as torch products and now, in us: 1536 -> 1536 columns
// 28.6 and 19.0 at 16 rows, 46.8 and 32.1 at 1024, 238 and 172 at 16384; 896 -> 128 28.9 and 18.6 at 128 rows; 4096 -> 4096
// 303 and 233 at 8192; 1536 -> 8960 154 and 119 at 4096; 8960 -> 1536 263 and 212 at 4096: the faster one at each of 76 sizes.
// (The product with A stays the library's: summed in another order its fp16 results, and with them the
// branch's, are no longer those of the plain formula bit for bit.)
//
// Roundings are those of the products: fp32 accumulators; the product with B rounded to fp16, then its scaling;
// in backward the scaled gradient, the rank-16 gradient and the product back to the input's width. Weight
// gradients are summed from partial sums in a fixed order.
#include "common.cuh"
#include "rank16.cuh"

namespace soup {
namespace {

using namespace rank16;

constexpr int kRows = 16;        // rows of an m tile
constexpr int kWarps = 16;       // gain: warps that share 16 rows' columns
constexpr int kChunk = 32;       // columns a warp takes at a time

__device__ __forceinline__ uint32_t half2_bits(float x, float y) {
  const __half2 h = __floats2half2_rn(x, y);
  return *reinterpret_cast<const uint32_t*>(&h);
}
// Two fp16 values times a scale, rounded to fp16 again.
__device__ __forceinline__ uint32_t scale2(uint32_t v, float scale) {
  const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&v));
  return half2_bits(f.x * scale, f.y * scale);
}

// ------------------------------------------------------------------------------------------
// out = fp16(fp16(low B^T) * scale). A warp keeps the fragments of 32 columns of B and walks its CTA's share of the
// 16-row tiles. Bound by the writes: 11.6 us for 16384 x 1536 (a library product and a scaling pass 29.4).
// ------------------------------------------------------------------------------------------
constexpr int kUpWarps = 8;
struct UpArgs {
  const __half* low;        // [adapters, rows, 16]
  const __half* b[2];       // [out, 16]
  __half* out[2];           // [rows, out]
  int width[2];             // a multiple of 8
  int first_ctas;           // CTAs along x that work on the first adapter
  int tiles_per_cta;
  float scale;
  int64_t rows;
};

__global__ void __launch_bounds__(kUpWarps * 32) lora_up_kernel(const __grid_constant__ UpArgs p) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int g = lane >> 2, t = lane & 3;
  const bool second = (int)blockIdx.x >= p.first_ctas;
  const int block = second ? blockIdx.x - p.first_ctas : blockIdx.x;
  const int width = second ? p.width[1] : p.width[0];
  const __half* b = second ? p.b[1] : p.b[0];
  __half* out = second ? p.out[1] : p.out[0];
  const __half* low = p.low + (second ? p.rows * kRank : 0);
  const int col0 = (block * kUpWarps + warp) * kChunk;
  if (col0 >= width) return;
  uint2 bv[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const int col = col0 + column_of(j, g);
    bv[j] = col < width ? __ldg(reinterpret_cast<const uint2*>(b + (int64_t)col * kRank + 4 * t)) : make_uint2(0u, 0u);
  }
  const bool mine = col0 + 8 * t < width;
  const int64_t n_tiles = (p.rows + kRows - 1) / kRows;
  const int64_t begin = (int64_t)blockIdx.y * p.tiles_per_cta;
  const int64_t end = begin + p.tiles_per_cta < n_tiles ? begin + p.tiles_per_cta : n_tiles;
#pragma unroll 2
  for (int64_t tile = begin; tile < end; ++tile) {
    uint32_t af[4], o[2][4];
    load_rank_fragment(low, tile * kRows, p.rows, lane, af);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      float c[4] = {0.f, 0.f, 0.f, 0.f};
      mma16816(c, af, bv[j].x, bv[j].y);
      o[0][j] = half2_bits(c[0], c[1]);
      o[1][j] = half2_bits(c[2], c[3]);
      if (p.scale != 1.f) {
        o[0][j] = scale2(o[0][j], p.scale);
        o[1][j] = scale2(o[1][j], p.scale);
      }
    }
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      const int64_t row = tile * kRows + g + half * 8;
      if (mine && row < p.rows)
        *reinterpret_cast<uint4*>(out + row * width + col0 + 8 * t) = make_uint4(o[half][0], o[half][1], o[half][2], o[half][3]);
    }
  }
}

// fp16 copies of the two weights (50 KB each).
__global__ void __launch_bounds__(256) lora_cast_kernel(const void* __restrict__ a, const void* __restrict__ b,
                                                        __half* __restrict__ a16, __half* __restrict__ b16,
                                                        int64_t n_a, int64_t n_b, int adt, int bdt) {
  const int64_t i = ((int64_t)blockIdx.x * 256 + threadIdx.x) * 8;
  if (i >= n_a + n_b) return;
  float v[8];
  if (i < n_a) {
    load8(a, i, adt, v);
    store8(a16, i, SOUP_F16, v);
  } else {
    load8(b, i - n_a, bdt, v);
    store8(b16, i - n_a, SOUP_F16, v);
  }
}

// ------------------------------------------------------------------------------------------
// Backward, first launch: gain = fp16(fp16(g * scale) B), [rows, 16]. A CTA owns RB blocks of 16 rows; its
// warps take 32-column chunks of the gradient in turn and add up in shared memory in a fixed order. Two blocks
// share the fragments of B, as many bytes as a block's gradient, once there are CTAs enough for every SM.
// ------------------------------------------------------------------------------------------
struct GainArgs {
  const __half* g;
  int64_t pitch;
  const __half* b;    // [out, 16]
  __half* gain;       // [rows, 16]
  float scale;
  int64_t rows;
  int out;            // a multiple of 8
};

template <int RB>
__global__ void __launch_bounds__(kWarps * 32, 2) lora_branch_gain_kernel(const __grid_constant__ GainArgs p) {
  __shared__ __align__(16) float s_part[kWarps][RB * kRows * kRank];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int g = lane >> 2, t = lane & 3;
  const int64_t row0 = (int64_t)blockIdx.x * RB * kRows;
  float acc[RB][2][4] = {};
#pragma unroll 1
  for (int col0 = warp * kChunk; col0 < p.out; col0 += kWarps * kChunk) {
    uint32_t gf[RB][2][4], bf[4][2];
#pragma unroll
    for (int rb = 0; rb < RB; ++rb)
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        const int64_t row = row0 + rb * kRows + g + half * 8;
        const uint4 v = row < p.rows && col0 + 8 * t < p.out
                            ? __ldg(reinterpret_cast<const uint4*>(p.g + row * p.pitch + col0 + 8 * t))
                            : make_uint4(0u, 0u, 0u, 0u);
        gf[rb][half][0] = v.x; gf[rb][half][1] = v.y; gf[rb][half][2] = v.z; gf[rb][half][3] = v.w;
      }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int col = col0 + column_of(j, g);
      const uint2 v = col < p.out ? __ldg(reinterpret_cast<const uint2*>(p.b + (int64_t)col * kRank + 4 * t))
                                  : make_uint2(0u, 0u);
      bf[j][0] = transpose8x8(v.x);
      bf[j][1] = transpose8x8(v.y);
    }
#pragma unroll
    for (int rb = 0; rb < RB; ++rb) {
      if (p.scale != 1.f) {
#pragma unroll
        for (int half = 0; half < 2; ++half)
#pragma unroll
          for (int j = 0; j < 4; ++j) gf[rb][half][j] = scale2(gf[rb][half][j], p.scale);
      }
#pragma unroll
      for (int s = 0; s < 2; ++s) {
        const uint32_t ga[4] = {gf[rb][0][2 * s], gf[rb][1][2 * s], gf[rb][0][2 * s + 1], gf[rb][1][2 * s + 1]};
        mma16816(acc[rb][0], ga, bf[2 * s][0], bf[2 * s + 1][0]);
        mma16816(acc[rb][1], ga, bf[2 * s][1], bf[2 * s + 1][1]);
      }
    }
  }
#pragma unroll
  for (int rb = 0; rb < RB; ++rb)
#pragma unroll
    for (int half = 0; half < 2; ++half)   // ranks 4 t .. 4 t + 3: rank_of(block, 2 t), + 1
      *reinterpret_cast<float4*>(&s_part[warp][(rb * kRows + g + 8 * half) * kRank + 4 * t]) =
          make_float4(acc[rb][0][2 * half], acc[rb][0][2 * half + 1], acc[rb][1][2 * half], acc[rb][1][2 * half + 1]);
  __syncthreads();
  const int e = threadIdx.x;
  if (e < RB * kRows * kRank && row0 + e / kRank < p.rows) {
    float sum = 0.f;
#pragma unroll
    for (int k = 0; k < kWarps; ++k) sum += s_part[k][e];
    p.gain[row0 * kRank + e] = __float2half_rn(sum);
  }
}

// ------------------------------------------------------------------------------------------
// Second launch: sums over the rows. Strips of 32 columns of the input form dx = keep * scale * fp16(gain A)
// and dA = gain^T (keep * scale * x); strips of the output form dB^T = a^T fp16(g * scale). A warp owns a
// strip and every fourth 16-row block of its CTA's share of the rows; the four warps on a strip add up in
// shared memory, and each share leaves its sums as a partial [16, width].
// ------------------------------------------------------------------------------------------
constexpr int kStrips = 2, kGroups = 4;   // per CTA: 32-column strips, warps on each

struct StripArgs {
  const __half* x;        // [rows, in]
  const uint8_t* bits;
  const __half* gain;     // [rows, 16]
  const __half* a;        // [16, in]
  float* dx;              // [rows, in]
  const __half* g;        // [rows, out]
  int64_t pitch;
  const __half* low;      // [rows, 16]
  float* part;            // [shares, 16, in + out]
  float keep_scale, g_scale;
  int64_t rows;
  int in, out, in_ctas, blocks_per_cta;   // CTAs along x that work on the input; 16-row blocks of a share
  int add_dx;             // dx holds the gradient of another adapter already
};

template <bool INPUT>
__device__ __forceinline__ void strip_sums(const StripArgs& p, float4 (*s_sum)[kGroups][4][32]) {
  const int lane = threadIdx.x & 31, group = (threadIdx.x >> 5) % kGroups, local = (threadIdx.x >> 5) / kGroups;
  const int g = lane >> 2, t = lane & 3;
  const int width = INPUT ? p.in : p.out;
  const int strip = (INPUT ? blockIdx.x : blockIdx.x - p.in_ctas) * kStrips + local;
  const int col = strip * 32 + t * 8;
  const bool mine = col < width;
  uint32_t af[4][2];
  if (INPUT) {
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      const uint4 v = mine ? __ldg(reinterpret_cast<const uint4*>(p.a + (int64_t)rank_of(half, g) * p.in + col))
                           : make_uint4(0u, 0u, 0u, 0u);
      af[0][half] = transpose8x8(v.x);
      af[1][half] = transpose8x8(v.y);
      af[2][half] = transpose8x8(v.z);
      af[3][half] = transpose8x8(v.w);
    }
  }
  float sum[4][4] = {};
  const int64_t n_blocks = (p.rows + 15) / 16;
  const int64_t begin = (int64_t)blockIdx.y * p.blocks_per_cta;
  const int64_t end = begin + p.blocks_per_cta < n_blocks ? begin + p.blocks_per_cta : n_blocks;
  const __half* factor = INPUT ? p.gain : p.low;
  const __half* values = INPUT ? p.x : p.g;
  const int64_t pitch = INPUT ? p.in : p.pitch;
  struct Block {
    uint4 v[2];
    uint32_t bits[2], f[4];
  };
  auto fetch = [&](int64_t rb, Block& k) {
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      const int64_t row = rb * 16 + g + half * 8;
      const bool ok = row < p.rows && mine;
      k.v[half] = ok ? *reinterpret_cast<const uint4*>(values + row * pitch + col) : make_uint4(0u, 0u, 0u, 0u);
      if (INPUT) k.bits[half] = ok ? *reinterpret_cast<const uint32_t*>(p.bits + ((row * p.in + strip * 32) >> 3)) : 0u;
    }
    load_rank_fragment(factor, rb * 16, p.rows, lane, k.f);
  };
  Block now, next;
  if (begin + group < end) fetch(begin + group, now);
#pragma unroll 1
  for (int64_t rb = begin + group; rb < end; rb += kGroups) {
    if (rb + kGroups < end) fetch(rb + kGroups, next);
    const uint32_t ft[4] = {transpose8x8(now.f[0]), transpose8x8(now.f[2]), transpose8x8(now.f[1]),
                            transpose8x8(now.f[3])};
    float d[2][8];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      float c[4] = {0.f, 0.f, 0.f, 0.f};
      if (INPUT) mma16816(c, now.f, af[j][0], af[j][1]);
      uint32_t vf[2];
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        uint32_t v = j == 0 ? now.v[half].x : j == 1 ? now.v[half].y : j == 2 ? now.v[half].z : now.v[half].w;
        if (INPUT) {
          const uint32_t keep = now.bits[half] >> (t * 8 + 2 * j);
          const bool k0 = keep & 1u, k1 = keep & 2u;
          const float2 xv = __half22float2(*reinterpret_cast<const __half2*>(&v));
          v = half2_bits(k0 ? __fmul_rn(xv.x, p.keep_scale) : 0.f, k1 ? __fmul_rn(xv.y, p.keep_scale) : 0.f);
          // the product rounded to fp16, as a tensor of its own would be
          const float g0 = __half2float(__float2half_rn(c[2 * half])), g1 = __half2float(__float2half_rn(c[2 * half + 1]));
          d[half][2 * j] = k0 ? __fmul_rn(g0, p.keep_scale) : 0.f;
          d[half][2 * j + 1] = k1 ? __fmul_rn(g1, p.keep_scale) : 0.f;
        } else if (p.g_scale != 1.f) {
          v = scale2(v, p.g_scale);
        }
        vf[half] = transpose8x8(v);
      }
      mma16816(sum[j], ft, vf[0], vf[1]);
    }
    if (INPUT && mine) {
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        const int64_t row = rb * 16 + g + half * 8;
        if (row < p.rows) {
          if (p.add_dx) {
            const float4* dst = reinterpret_cast<const float4*>(p.dx + row * p.in + col);
            const float4 u = dst[0], v = dst[1];
            d[half][0] = __fadd_rn(u.x, d[half][0]); d[half][1] = __fadd_rn(u.y, d[half][1]);
            d[half][2] = __fadd_rn(u.z, d[half][2]); d[half][3] = __fadd_rn(u.w, d[half][3]);
            d[half][4] = __fadd_rn(v.x, d[half][4]); d[half][5] = __fadd_rn(v.y, d[half][5]);
            d[half][6] = __fadd_rn(v.z, d[half][6]); d[half][7] = __fadd_rn(v.w, d[half][7]);
          }
          store_sector(p.dx + row * p.in + col, d[half]);
        }
      }
    }
    now = next;
  }
#pragma unroll
  for (int half = 0; half < 2; ++half)
#pragma unroll
    for (int q = 0; q < 2; ++q)
      s_sum[local][group][half * 2 + q][lane] = make_float4(sum[2 * q][2 * half], sum[2 * q][2 * half + 1],
                                                            sum[2 * q + 1][2 * half], sum[2 * q + 1][2 * half + 1]);
  __syncthreads();
  // the strip's four warps finish one of its four pieces each
  float4 total = s_sum[local][0][group][lane];
#pragma unroll
  for (int k = 1; k < kGroups; ++k) {
    const float4 v = s_sum[local][k][group][lane];
    total.x += v.x; total.y += v.y; total.z += v.z; total.w += v.w;
  }
  if (mine)
    *reinterpret_cast<float4*>(p.part + ((int64_t)blockIdx.y * kRank + rank_of(group >> 1, g)) * (p.in + p.out) +
                               (INPUT ? 0 : p.in) + col + (group & 1) * 4) = total;
}

__global__ void __launch_bounds__(kStrips * kGroups * 32, 2)
lora_branch_strip_kernel(const __grid_constant__ StripArgs p) {
  __shared__ float4 s_sum[kStrips][kGroups][4][32];   // [..][row half, column half][lane]
  if ((int)blockIdx.x < p.in_ctas) strip_sums<true>(p, s_sum);
  else strip_sums<false>(p, s_sum);
}

// Third launch: dA [16, in] and dB [out, 16] from the shares' partial sums, in the shares' order.
struct TotalArgs {
  const float* part;
  float *da, *db;
  int shares, in, out, add_a, add_b;   // add: to what da / db hold
  float alpha;                         // of dB
};

__global__ void __launch_bounds__(256) lora_branch_total_kernel(const __grid_constant__ TotalArgs p) {
  const int width = p.in + p.out;
  const int i = blockIdx.x * 256 + threadIdx.x;
  if (i >= kRank * width) return;
  const int rank = i / width, col = i - rank * width;
  float sum = 0.f;
#pragma unroll 8
  for (int s = 0; s < p.shares; ++s) sum += p.part[(int64_t)s * kRank * width + i];
  if (col < p.in) {
    float* dst = p.da + (int64_t)rank * p.in + col;
    *dst = p.add_a ? *dst + sum : sum;
  } else {
    float* dst = p.db + (int64_t)(col - p.in) * kRank + rank;
    *dst = p.add_b ? *dst + sum * p.alpha : sum * p.alpha;
  }
}

// Row blocks of a share: whole rounds of a CTA's four warps, so that the two CTAs an SM holds have one each.
inline int64_t share_blocks(int64_t rows, int64_t in, int64_t out) {
  const int64_t ctas = (in / 32 + kStrips - 1) / kStrips + ((out + 31) / 32 + kStrips - 1) / kStrips;
  const int64_t n_blocks = (rows + 15) / 16;
  int64_t per = (ctas * n_blocks + 2ll * sm_count() - 1) / (2ll * sm_count());
  if (per < (n_blocks + 65534) / 65535) per = (n_blocks + 65534) / 65535;
  return (per + kGroups - 1) / kGroups * kGroups;
}
inline int64_t shares_of(int64_t rows, int64_t in, int64_t out) {
  const int64_t per = share_blocks(rows, in, out);
  return ((rows + 15) / 16 + per - 1) / per;
}

inline int check_widths(const char* name, int64_t rows, int64_t in, int64_t out, int64_t rank) {
  if (rows < 0 || rank != kRank) SOUP_FAIL(SOUP_ERR_ARG, "%s: the rank must be 16", name);
  if (in <= 0 || in % 32 || in > (1 << 24) || out <= 0 || out % 8 || out > (1 << 24))
    SOUP_FAIL(SOUP_ERR_ARG, "%s: the input width must be a multiple of 32, the output's of 8", name);
  if (rows > (1ll << 34)) SOUP_FAIL(SOUP_ERR_ARG, "%s: too many rows", name);
  return SOUP_OK;
}

}  // namespace
}  // namespace soup

extern "C" int soup_lora_cast(const void* a, const void* b, void* a16, void* b16, int64_t n_a, int64_t n_b,
                              int a_dtype, int b_dtype, void* stream) {
  using namespace soup;
  if (n_a < 0 || n_b < 0 || n_a % 8 || n_b % 8 || n_a + n_b > (1ll << 38))
    SOUP_FAIL(SOUP_ERR_ARG, "lora_cast: sizes must be multiples of 8");
  if (n_a + n_b == 0) return SOUP_OK;
  if ((n_a && (!a || !a16)) || (n_b && (!b || !b16))) SOUP_FAIL(SOUP_ERR_ARG, "lora_cast: null pointer");
  if (!is_float_dtype(a_dtype) || !is_float_dtype(b_dtype)) SOUP_FAIL(SOUP_ERR_ARG, "lora_cast: unsupported dtype");
  if (!aligned16(a) || !aligned16(b) || !aligned16(a16) || !aligned16(b16))
    SOUP_FAIL(SOUP_ERR_ARG, "lora_cast: pointers must be 16-byte aligned");
  lora_cast_kernel<<<(unsigned)((n_a + n_b + 2047) / 2048), 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(
      a, b, reinterpret_cast<__half*>(a16), reinterpret_cast<__half*>(b16), n_a, n_b, a_dtype, b_dtype);
  SOUP_CHECK_LAUNCH("lora_cast");
  return SOUP_OK;
}

extern "C" int soup_lora_up(const void* low, const void* b16_first, const void* b16_second, void* out_first,
                            void* out_second, float scale, int64_t rows, int64_t width_first, int64_t width_second,
                            int64_t rank, void* stream) {
  using namespace soup;
  const bool two = b16_second != nullptr;
  int rc = check_widths("lora_up", rows, 32, width_first, rank);
  if (rc == SOUP_OK && two) rc = check_widths("lora_up", rows, 32, width_second, rank);
  if (rc != SOUP_OK || rows == 0) return rc;
  if (!low || !b16_first || !out_first || (two && !out_second)) SOUP_FAIL(SOUP_ERR_ARG, "lora_up: null pointer");
  if (!aligned16(low) || !aligned16(b16_first) || !aligned16(b16_second) || !aligned16(out_first) || !aligned16(out_second))
    SOUP_FAIL(SOUP_ERR_ARG, "lora_up: pointers must be 16-byte aligned");
  UpArgs p;
  p.low = reinterpret_cast<const __half*>(low);
  p.b[0] = reinterpret_cast<const __half*>(b16_first);
  p.b[1] = reinterpret_cast<const __half*>(b16_second);
  p.out[0] = reinterpret_cast<__half*>(out_first);
  p.out[1] = reinterpret_cast<__half*>(out_second);
  p.width[0] = (int)width_first;
  p.width[1] = two ? (int)width_second : 0;
  p.scale = scale;
  p.rows = rows;
  auto ctas = [](int64_t width) { return (width + kUpWarps * kChunk - 1) / (kUpWarps * kChunk); };
  p.first_ctas = (int)ctas(width_first);
  const int64_t columns = ctas(width_first) + (two ? ctas(width_second) : 0), n_tiles = (rows + kRows - 1) / kRows;
  // row tiles per CTA that leave eight CTAs an SM, all resident at once
  int64_t per = (columns * n_tiles + 8ll * sm_count() - 1) / (8ll * sm_count());
  if (per < (n_tiles + 65534) / 65535) per = (n_tiles + 65534) / 65535;
  p.tiles_per_cta = (int)per;
  lora_up_kernel<<<dim3((unsigned)columns, (unsigned)((n_tiles + per - 1) / per)), kUpWarps * 32, 0,
                   reinterpret_cast<cudaStream_t>(stream)>>>(p);
  SOUP_CHECK_LAUNCH("lora_up");
  return SOUP_OK;
}

extern "C" int64_t soup_lora_branch_workspace_bytes(int64_t rows, int64_t in, int64_t out) {
  using namespace soup;
  if (rows <= 0 || in <= 0 || out <= 0) return 0;
  return rows * kRank * 2 + 16 + shares_of(rows, in, out) * kRank * (in + out) * 4;
}

extern "C" int soup_lora_branch_bwd(const void* g, int64_t g_pitch, const void* x16, const uint8_t* bits,
                                    const void* low, const void* a16, const void* b16, float* dx, float* da,
                                    float* db, int add_dx, int add_da, int add_db, float keep_scale, float g_scale,
                                    float db_alpha, void* workspace, int64_t workspace_bytes, int64_t rows,
                                    int64_t in, int64_t out, int64_t rank, void* stream) {
  using namespace soup;
  const int rc = check_widths("lora_branch_bwd", rows, in, out, rank);
  if (rc != SOUP_OK) return rc;
  if (g_pitch < out || g_pitch % 8)
    SOUP_FAIL(SOUP_ERR_ARG, "lora_branch_bwd: the row pitch must cover the output and be a multiple of 8");
  if (!da || !db) SOUP_FAIL(SOUP_ERR_ARG, "lora_branch_bwd: null pointer");
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  if (rows == 0) {
    if (!add_da) cudaMemsetAsync(da, 0, (size_t)(kRank * in) * sizeof(float), st);
    if (!add_db) cudaMemsetAsync(db, 0, (size_t)(kRank * out) * sizeof(float), st);
    return SOUP_OK;
  }
  if (!g || !x16 || !bits || !low || !a16 || !b16 || !dx || !workspace)
    SOUP_FAIL(SOUP_ERR_ARG, "lora_branch_bwd: null pointer");
  if (!aligned16(g) || !aligned16(x16) || (reinterpret_cast<uintptr_t>(bits) & 3u) || !aligned16(low) ||
      !aligned16(a16) || !aligned16(b16) || !aligned32(dx) || !aligned16(workspace))
    SOUP_FAIL(SOUP_ERR_ARG, "lora_branch_bwd: pointers must be 16-byte aligned, dx 32-byte aligned");
  if (workspace_bytes < soup_lora_branch_workspace_bytes(rows, in, out))
    SOUP_FAIL(SOUP_ERR_ARG, "lora_branch_bwd: workspace too small");
  const int64_t shares = shares_of(rows, in, out);
  GainArgs ga;
  ga.g = reinterpret_cast<const __half*>(g);
  ga.pitch = g_pitch;
  ga.b = reinterpret_cast<const __half*>(b16);
  ga.gain = reinterpret_cast<__half*>(workspace);
  ga.scale = g_scale;
  ga.rows = rows;
  ga.out = (int)out;
  const int64_t blocks = (rows + kRows - 1) / kRows;
  if (blocks >= 4ll * sm_count()) lora_branch_gain_kernel<2><<<(unsigned)((blocks + 1) / 2), kWarps * 32, 0, st>>>(ga);
  else lora_branch_gain_kernel<1><<<(unsigned)blocks, kWarps * 32, 0, st>>>(ga);
  SOUP_CHECK_LAUNCH("lora_branch_gain");
  StripArgs sa;
  sa.x = reinterpret_cast<const __half*>(x16);
  sa.bits = bits;
  sa.gain = ga.gain;
  sa.a = reinterpret_cast<const __half*>(a16);
  sa.dx = dx;
  sa.g = ga.g;
  sa.pitch = g_pitch;
  sa.low = reinterpret_cast<const __half*>(low);
  sa.part = reinterpret_cast<float*>(reinterpret_cast<uint8_t*>(workspace) + (rows * kRank * 2 + 15) / 16 * 16);
  sa.keep_scale = keep_scale;
  sa.g_scale = g_scale;
  sa.rows = rows;
  sa.in = (int)in;
  sa.out = (int)out;
  sa.in_ctas = (int)((in / 32 + kStrips - 1) / kStrips);
  sa.blocks_per_cta = (int)share_blocks(rows, in, out);
  sa.add_dx = add_dx;
  const dim3 grid((unsigned)(sa.in_ctas + ((out + 31) / 32 + kStrips - 1) / kStrips), (unsigned)shares);
  lora_branch_strip_kernel<<<grid, kStrips * kGroups * 32, 0, st>>>(sa);
  SOUP_CHECK_LAUNCH("lora_branch_strip");
  TotalArgs ta;
  ta.part = sa.part;
  ta.da = da;
  ta.db = db;
  ta.shares = (int)shares;
  ta.in = (int)in;
  ta.out = (int)out;
  ta.add_a = add_da;
  ta.add_b = add_db;
  ta.alpha = db_alpha;
  lora_branch_total_kernel<<<(unsigned)((kRank * (in + out) + 255) / 256), 256, 0, st>>>(ta);
  SOUP_CHECK_LAUNCH("lora_branch_total");
  return SOUP_OK;
}
