// Backward of a block's two rank-16 adapters (q_proj's and v_proj's, sharing their input) in two
// launches: everything that reads the output gradients, and everything that reads the shared input.
//
// As torch products the pair takes eight launches at a few thousand tokens (two per weight gradient,
// two for the rank-16 gradients, a batched product back to the input's width and the mask kernel),
// 37 us a block at 1280 tokens, most of it launches of GEMMs with an extent of 16, and writes and
// reads four [tokens, hidden] fp16 tensors in between. Here a rank of 16 is one k step (or one m tile)
// of mma.sync.m16n8k16, operands go from global memory to fragments without shared memory, and a
// fragment's transpose is a movmatrix away, so that each [tokens, width] tensor is read once and the
// only one written is the input gradient. (A tcgen05 tile would be 128 wide where these are 16.)
// Bound by latency at the step's token counts: 5.4 + 8.7 us at 1280 tokens (hidden 1536, outputs 1536
// and 256; buffers larger than L2 in turn) where the eight launches take 37.2 us, 10.6 + 22.9 and 70.0 us at 4608.
//
// Roundings are those of the products they replace: fp32 accumulators, the rank-16 gradient and the
// product back to the input's width rounded to fp16 once, weight gradients added in fp32 (by
// reductions, in any order).
#include "common.cuh"
#include "rank16.cuh"

namespace soup {
namespace {

using namespace rank16;

__device__ __forceinline__ void red_add4(float* p, float x, float y, float z, float w) {
  asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(p), "f"(x), "f"(y), "f"(z), "f"(w));
}

// ------------------------------------------------------------------------------------------
// gain = g B (fp16 [rows, 16], B already scaled) and dB += alpha g^T a, for both adapters, by CTAs of two kinds that
// do not wait for one another. One kind takes four strips of 32 output columns and a share of the rows, four
// warps on each strip, whose sums meet in shared memory and leave as reductions. The other owns one or two
// blocks of 16 rows; its 16 warps take 32-column chunks of the gradients in turn and their partial products meet
// in shared memory, summed in a fixed order. Both read the gradients (one of them from L2), so that neither's
// chain of loads waits for the other's. With both products in the CTAs that own the rows, and now: 128 rows 7.9 and
// 3.5 us, 1280 8.4 and 5.4, 4608 12.1 and 10.6, 16384 38.4 and 28.3 (the first kind last in the grid: 8192 rows 22.0, now 16.6).
// ------------------------------------------------------------------------------------------
constexpr int kGainWarps = 16, kChunk = 32;
constexpr int kGainValues = 16 * kRank;          // of one adapter and 16 rows
constexpr int kDbStrips = 4, kDbGroups = 4;      // strips of a CTA, warps on each
constexpr int kStripValues = kChunk * kRank;

struct GainArgs {
  const __half* g[2];
  int64_t pitch[2];
  int out[2];             // columns of each gradient, a multiple of 16
  const __half* a;        // [2, rows, 16]
  const __half* b[2];     // [out, 16]
  float* db[2];           // [out, 16]
  float alpha[2];
  __half* gain;           // [2, rows, 16]
  int64_t rows;
  int db_ctas, db_columns, blocks_per_share;   // CTAs of the first kind, along the strips; 16-row blocks of a share
};

// 16 rows x 32 columns of a gradient: [row half][column block], rows past the end and columns past `left` zero.
__device__ __forceinline__ void load_chunk(const __half* g, int64_t pitch, int64_t row0, int64_t rows, int left, int lane,
                                           uint32_t (&f)[2][4]) {
#pragma unroll
  for (int half = 0; half < 2; ++half) {
    const int64_t row = row0 + (lane >> 2) + half * 8;
    const uint4 v = row < rows && 8 * (lane & 3) < left ? __ldg(reinterpret_cast<const uint4*>(g + row * pitch + 8 * (lane & 3)))
                                                        : make_uint4(0u, 0u, 0u, 0u);
    f[half][0] = v.x; f[half][1] = v.y; f[half][2] = v.z; f[half][3] = v.w;
  }
}

// RB: 16-row blocks of a CTA of the second kind. Two share the fragments of B, as many bytes as a block's gradient,
// once there are blocks enough for every SM.
template <int RB>
constexpr int kGainSmem = RB * 2 * kGainWarps * kGainValues * (int)sizeof(float);
template <int RB>
__global__ void __launch_bounds__(kGainWarps * 32, 2) lora_gain_kernel(const __grid_constant__ GainArgs p) {
  extern __shared__ __align__(16) float s_sum[];   // either kind's partial sums
  static_assert(2 * kGainWarps * kGainValues == kDbStrips * kDbGroups * kStripValues, "the first kind's fit");
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int g = lane >> 2, t = lane & 3;
  if ((int)blockIdx.x >= p.db_ctas) {   // the shorter chains start last
    const int64_t row0 = (int64_t)(blockIdx.x - p.db_ctas) * (16 * RB);
#pragma unroll
    for (int w = 0; w < 2; ++w) {
      float gain[RB][2][4] = {};   // [row block][rank block]
#pragma unroll 1
      for (int col0 = warp * kChunk; col0 < p.out[w]; col0 += kGainWarps * kChunk) {
        const int left = p.out[w] - col0;   // 16 in the last chunk of an odd number of sixteens
        uint32_t gf[RB][2][4], bf[4][2];
#pragma unroll
        for (int rb = 0; rb < RB; ++rb) load_chunk(p.g[w] + col0, p.pitch[w], row0 + rb * 16, p.rows, left, lane, gf[rb]);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int col = column_of(j, g);
          const uint2 v = col < left ? __ldg(reinterpret_cast<const uint2*>(p.b[w] + (int64_t)(col0 + col) * kRank + 4 * t))
                                     : make_uint2(0u, 0u);
          bf[j][0] = transpose8x8(v.x);
          bf[j][1] = transpose8x8(v.y);
        }
#pragma unroll
        for (int rb = 0; rb < RB; ++rb)
#pragma unroll
          for (int s = 0; s < 2; ++s) {
            const uint32_t ga[4] = {gf[rb][0][2 * s], gf[rb][1][2 * s], gf[rb][0][2 * s + 1], gf[rb][1][2 * s + 1]};
            mma16816(gain[rb][0], ga, bf[2 * s][0], bf[2 * s + 1][0]);
            mma16816(gain[rb][1], ga, bf[2 * s][1], bf[2 * s + 1][1]);
          }
      }
#pragma unroll
      for (int rb = 0; rb < RB; ++rb)
#pragma unroll
        for (int half = 0; half < 2; ++half)
          *reinterpret_cast<float4*>(s_sum + ((warp * 2 + w) * RB + rb) * kGainValues + (g + half * 8) * kRank + 4 * t) =
              make_float4(gain[rb][0][2 * half], gain[rb][0][2 * half + 1], gain[rb][1][2 * half],
                          gain[rb][1][2 * half + 1]);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < 2 * RB * kGainValues; i += kGainWarps * 32) {
      const int w = i / (RB * kGainValues), e = i % (RB * kGainValues);
      float sum = 0.f;   // in the warps' order: the same bits every time
#pragma unroll
      for (int k = 0; k < kGainWarps; ++k) sum += s_sum[(k * 2 + w) * RB * kGainValues + e];
      if (row0 + e / kRank < p.rows) p.gain[((int64_t)w * p.rows + row0) * kRank + e] = __float2half_rn(sum);
    }
    return;
  }
  const int share = blockIdx.x / p.db_columns;
  const int strips_first = (p.out[0] + kChunk - 1) / kChunk, strips = strips_first + (p.out[1] + kChunk - 1) / kChunk;
  const int local = warp / kDbGroups, group = warp % kDbGroups;
  const int strip = ((int)blockIdx.x - share * p.db_columns) * kDbStrips + local;
  const int w = strip >= strips_first;
  const int col0 = (w ? strip - strips_first : strip) * kChunk;
  const int left = strip < strips ? p.out[w] - col0 : 0;
  float db[2][2][4] = {};   // [16-column half][rank block]
  const int64_t n_blocks = (p.rows + 15) / 16, begin = (int64_t)share * p.blocks_per_share;
  const int64_t end = begin + p.blocks_per_share < n_blocks ? begin + p.blocks_per_share : n_blocks;
#pragma unroll 2
  for (int64_t rb = begin + group; rb < end; rb += kDbGroups) {
    uint32_t gf[2][4], f[4];
    load_chunk(p.g[w] + col0, p.pitch[w], rb * 16, p.rows, left, lane, gf);
    load_rank_fragment(p.a + (int64_t)w * p.rows * kRank, rb * 16, p.rows, lane, f);
    // a, rows along the contraction: B fragments [16 rows x 8 ranks]
    const uint32_t ab[2][2] = {{transpose8x8(f[0]), transpose8x8(f[1])}, {transpose8x8(f[2]), transpose8x8(f[3])}};
#pragma unroll
    for (int s = 0; s < 2; ++s) {
      const uint32_t gt[4] = {transpose8x8(gf[0][2 * s]), transpose8x8(gf[0][2 * s + 1]), transpose8x8(gf[1][2 * s]),
                              transpose8x8(gf[1][2 * s + 1])};
      mma16816(db[s][0], gt, ab[0][0], ab[0][1]);
      mma16816(db[s][1], gt, ab[1][0], ab[1][1]);
    }
  }
#pragma unroll
  for (int s = 0; s < 2; ++s)
#pragma unroll
    for (int half = 0; half < 2; ++half)
      *reinterpret_cast<float4*>(s_sum + warp * kStripValues + column_of(2 * s + half, g) * kRank + 4 * t) =
          make_float4(db[s][0][2 * half], db[s][0][2 * half + 1], db[s][1][2 * half], db[s][1][2 * half + 1]);
  __syncthreads();
  // the strip's four warps finish eight of its columns each: a lane four ranks of one
  const int value = group * (kStripValues / kDbGroups) + lane * 4;
  const float* sums = s_sum + local * kDbGroups * kStripValues + value;
  float4 v = *reinterpret_cast<const float4*>(sums);
#pragma unroll
  for (int k = 1; k < kDbGroups; ++k) {
    const float4 o = *reinterpret_cast<const float4*>(sums + k * kStripValues);
    v.x += o.x; v.y += o.y; v.z += o.z; v.w += o.w;
  }
  const float al = p.alpha[w];
  if (value / kRank < left) red_add4(p.db[w] + (int64_t)col0 * kRank + value, v.x * al, v.y * al, v.z * al, v.w * al);
}

// ------------------------------------------------------------------------------------------
// From the shared input x (fp16) and the two masks: dx = sum over the adapters of
// keep * scale * fp16(gain A), and dA += gain^T (keep * scale * x). A warp owns 32 columns and walks
// every fourth 16-row block of its CTA; the CTA's four warps on the same columns add up their dA in
// shared memory first, because the reductions into dA, the same [16, hidden] for every block of rows,
// are what bounds it (8.4 us at 1280 rows and 22.0 at 4608 with a reduction per warp, now 6.3 and 19.1).
// ------------------------------------------------------------------------------------------
constexpr int kInputStrips = 2, kInputGroups = 4;   // per CTA: 32-column strips, warps on each

struct InputArgs {
  const __half* x;
  const uint8_t* bits[2];
  const __half* gain;     // [2, rows, 16]
  const __half* a;        // [2, 16, hidden]
  float* dx;
  float* da[2];           // [16, hidden]
  float scale[2];
  int64_t rows;
  int hidden, strips, blocks_per_cta;   // strips: hidden / 32
  int wide_dx;            // dx is 32-byte aligned
};

__global__ void __launch_bounds__(kInputStrips * kInputGroups * 32)
lora_input_kernel(const __grid_constant__ InputArgs p) {
  __shared__ float4 s_da[kInputStrips][kInputGroups][8][32];   // [..][adapter, row half, column half][lane]
  const int lane = threadIdx.x & 31, group = (threadIdx.x >> 5) % kInputGroups;
  const int local = (threadIdx.x >> 5) / kInputGroups;
  const int strip = min((int)blockIdx.x * kInputStrips + local, p.strips - 1);   // the odd last one twice
  const bool mine = blockIdx.x * kInputStrips + local < p.strips;
  const int g = lane >> 2, t = lane & 3;
  const int col = strip * 32 + t * 8;
  // A of both adapters: B fragments [16 x 8] of the four tiles
  uint32_t af[2][4][2];
#pragma unroll
  for (int w = 0; w < 2; ++w)
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      const uint4 v = *reinterpret_cast<const uint4*>(p.a + ((int64_t)w * kRank + rank_of(half, g)) * p.hidden + col);
      const uint32_t r[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
      for (int j = 0; j < 4; ++j) af[w][j][half] = transpose8x8(r[j]);
    }
  float da[2][4][4] = {};
  const int64_t n_blocks = (p.rows + 15) / 16;
  const int64_t begin = (int64_t)blockIdx.y * p.blocks_per_cta;
  const int64_t end = begin + p.blocks_per_cta < n_blocks ? begin + p.blocks_per_cta : n_blocks;
  const int64_t first = begin + group, last = mine ? end : 0;
  const int bit_shift = t * 8;
  auto fetch = [&](int64_t rb, uint4 (&x)[2], uint32_t (&bits)[2][2], uint32_t (&gf)[2][4]) {
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      const int64_t row = rb * 16 + g + half * 8;
      const bool ok = row < p.rows;
      const int64_t at = row * p.hidden + col;
      x[half] = ok ? *reinterpret_cast<const uint4*>(p.x + at) : make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
      for (int w = 0; w < 2; ++w)
        bits[w][half] = ok ? *reinterpret_cast<const uint32_t*>(p.bits[w] + ((at - t * 8) >> 3)) : 0u;
    }
#pragma unroll
    for (int w = 0; w < 2; ++w)
      load_rank_fragment(p.gain + (int64_t)w * p.rows * kRank, rb * 16, p.rows, lane, gf[w]);
  };
  uint4 x[2];
  uint32_t bits[2][2], gf[2][4];
  if (first < last) fetch(first, x, bits, gf);
#pragma unroll 1
  for (int64_t rb = first; rb < last; rb += kInputGroups) {
    uint4 nx[2];
    uint32_t nbits[2][2], ngf[2][4];
    if (rb + kInputGroups < last) fetch(rb + kInputGroups, nx, nbits, ngf);
    float sum[2][8];   // dx of rows g and g + 8
#pragma unroll
    for (int w = 0; w < 2; ++w) {
      const float scale = p.scale[w];
      const uint32_t gt[4] = {transpose8x8(gf[w][0]), transpose8x8(gf[w][2]), transpose8x8(gf[w][1]),
                              transpose8x8(gf[w][3])};
      const uint32_t keep[2] = {bits[w][0] >> bit_shift, bits[w][1] >> bit_shift};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        float c[4] = {0.f, 0.f, 0.f, 0.f};
        mma16816(c, gf[w], af[w][j][0], af[w][j][1]);
        uint32_t xf[2];
#pragma unroll
        for (int half = 0; half < 2; ++half) {
          const uint32_t raw = j == 0 ? x[half].x : j == 1 ? x[half].y : j == 2 ? x[half].z : x[half].w;
          const float2 xv = __half22float2(*reinterpret_cast<const __half2*>(&raw));
          const bool k0 = (keep[half] >> (2 * j)) & 1u, k1 = (keep[half] >> (2 * j + 1)) & 1u;
          __half2 dropped = __floats2half2_rn(k0 ? __fmul_rn(xv.x, scale) : 0.f, k1 ? __fmul_rn(xv.y, scale) : 0.f);
          xf[half] = transpose8x8(*reinterpret_cast<uint32_t*>(&dropped));
          // the product rounded to fp16, as a tensor of its own would be
          const float g0 = __half2float(__float2half_rn(c[2 * half])), g1 = __half2float(__float2half_rn(c[2 * half + 1]));
          const float d0 = k0 ? __fmul_rn(g0, scale) : 0.f, d1 = k1 ? __fmul_rn(g1, scale) : 0.f;
          sum[half][2 * j] = w ? __fadd_rn(sum[half][2 * j], d0) : d0;
          sum[half][2 * j + 1] = w ? __fadd_rn(sum[half][2 * j + 1], d1) : d1;
        }
        mma16816(da[w][j], gt, xf[0], xf[1]);
      }
    }
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      const int64_t row = rb * 16 + g + half * 8;
      if (row < p.rows) {
        float* dst = p.dx + row * p.hidden + col;
        if (p.wide_dx) {
          store_sector(dst, sum[half]);
        } else {
          reinterpret_cast<float4*>(dst)[0] = make_float4(sum[half][0], sum[half][1], sum[half][2], sum[half][3]);
          reinterpret_cast<float4*>(dst)[1] = make_float4(sum[half][4], sum[half][5], sum[half][6], sum[half][7]);
        }
      }
    }
    if (rb + kInputGroups < last) {
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        x[half] = nx[half];
        bits[0][half] = nbits[0][half];
        bits[1][half] = nbits[1][half];
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) { gf[0][i] = ngf[0][i]; gf[1][i] = ngf[1][i]; }
    }
  }
#pragma unroll
  for (int w = 0; w < 2; ++w)
#pragma unroll
    for (int half = 0; half < 2; ++half)
#pragma unroll
      for (int q = 0; q < 2; ++q)
        s_da[local][group][w * 4 + half * 2 + q][lane] =
            make_float4(da[w][2 * q][2 * half], da[w][2 * q][2 * half + 1], da[w][2 * q + 1][2 * half],
                        da[w][2 * q + 1][2 * half + 1]);
  __syncthreads();
  // the strip's four warps finish two of its eight pieces each
#pragma unroll
  for (int e = 0; e < 8 / kInputGroups; ++e) {
    const int piece = group * (8 / kInputGroups) + e, w = piece >> 2, half = (piece >> 1) & 1, q = piece & 1;
    float4 sum = s_da[local][0][piece][lane];
#pragma unroll
    for (int k = 1; k < kInputGroups; ++k) {
      const float4 v = s_da[local][k][piece][lane];
      sum.x += v.x; sum.y += v.y; sum.z += v.z; sum.w += v.w;
    }
    if (mine) red_add4(p.da[w] + (int64_t)rank_of(half, g) * p.hidden + col + q * 4, sum.x, sum.y, sum.z, sum.w);
  }
}

inline bool aligned4(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 3u) == 0; }

}  // namespace
}  // namespace soup

extern "C" int soup_lora_pair_gain(const void* g_first, int64_t pitch_first, int64_t out_first, const void* g_second,
                                   int64_t pitch_second, int64_t out_second, const void* a, const void* b_first,
                                   const void* b_second, void* gain, float* db_first, float* db_second,
                                   float alpha_first, float alpha_second, int64_t rows, int64_t rank, void* stream) {
  using namespace soup;
  if (rows < 0 || rank != kRank) SOUP_FAIL(SOUP_ERR_ARG, "lora_pair_gain: the rank must be 16");
  if (out_first <= 0 || out_second <= 0 || out_first % 16 || out_second % 16 || out_first > (1 << 24) ||
      out_second > (1 << 24))
    SOUP_FAIL(SOUP_ERR_ARG, "lora_pair_gain: output widths must be multiples of 16");
  if (pitch_first < out_first || pitch_second < out_second || (pitch_first | pitch_second) & 7)
    SOUP_FAIL(SOUP_ERR_ARG, "lora_pair_gain: row pitches must cover the outputs and be multiples of 8");
  if (rows == 0) return SOUP_OK;
  if (!g_first || !g_second || !a || !b_first || !b_second || !gain || !db_first || !db_second)
    SOUP_FAIL(SOUP_ERR_ARG, "lora_pair_gain: null pointer");
  if (!aligned16(g_first) || !aligned16(g_second) || !aligned16(a) || !aligned16(b_first) || !aligned16(b_second) ||
      !aligned16(db_first) || !aligned16(db_second))
    SOUP_FAIL(SOUP_ERR_ARG, "lora_pair_gain: unaligned pointer");
  GainArgs p;
  p.g[0] = reinterpret_cast<const __half*>(g_first);
  p.g[1] = reinterpret_cast<const __half*>(g_second);
  p.pitch[0] = pitch_first;
  p.pitch[1] = pitch_second;
  p.out[0] = (int)out_first;
  p.out[1] = (int)out_second;
  p.a = reinterpret_cast<const __half*>(a);
  p.b[0] = reinterpret_cast<const __half*>(b_first);
  p.b[1] = reinterpret_cast<const __half*>(b_second);
  p.db[0] = db_first;
  p.db[1] = db_second;
  p.alpha[0] = alpha_first;
  p.alpha[1] = alpha_second;
  p.gain = reinterpret_cast<__half*>(gain);
  p.rows = rows;
  const int64_t n_blocks = (rows + 15) / 16;
  const int64_t strips = (out_first + kChunk - 1) / kChunk + (out_second + kChunk - 1) / kChunk;
  const int64_t columns = (strips + kDbStrips - 1) / kDbStrips;
  // row blocks of a share, whole rounds of a strip's four warps, that leave about one CTA per SM
  int64_t per = (columns * n_blocks + sm_count() - 1) / sm_count();
  per = (per + kDbGroups - 1) / kDbGroups * kDbGroups;
  const int rb = n_blocks >= sm_count() ? 2 : 1;
  const int64_t db_ctas = columns * ((n_blocks + per - 1) / per), ctas = db_ctas + (n_blocks + rb - 1) / rb;
  if (ctas > INT32_MAX || per > (1 << 30)) SOUP_FAIL(SOUP_ERR_ARG, "lora_pair_gain: too many rows");
  p.db_ctas = (int)db_ctas;
  p.db_columns = (int)columns;
  p.blocks_per_share = (int)per;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  if (rb == 1) {
    lora_gain_kernel<1><<<(unsigned)ctas, kGainWarps * 32, kGainSmem<1>, st>>>(p);
  } else {
    if (cudaFuncSetAttribute(lora_gain_kernel<2>, cudaFuncAttributeMaxDynamicSharedMemorySize, kGainSmem<2>) != cudaSuccess)
      SOUP_FAIL(SOUP_ERR_LAUNCH, "lora_pair_gain: shared memory attribute");
    lora_gain_kernel<2><<<(unsigned)ctas, kGainWarps * 32, kGainSmem<2>, st>>>(p);
  }
  SOUP_CHECK_LAUNCH("lora_pair_gain");
  return SOUP_OK;
}

extern "C" int soup_lora_pair_input(const void* x16, const uint8_t* bits_first, const uint8_t* bits_second,
                                    const void* gain, const void* a_pair, float* dx, float* da_first,
                                    float* da_second, float scale_first, float scale_second, int64_t rows,
                                    int64_t hidden, int64_t rank, void* stream) {
  using namespace soup;
  if (rows < 0 || rank != kRank) SOUP_FAIL(SOUP_ERR_ARG, "lora_pair_input: the rank must be 16");
  if (hidden <= 0 || hidden % 32 || hidden > (1 << 24))
    SOUP_FAIL(SOUP_ERR_ARG, "lora_pair_input: the input width must be a multiple of 32");
  if (rows == 0) return SOUP_OK;
  if (!x16 || !bits_first || !bits_second || !gain || !a_pair || !dx || !da_first || !da_second)
    SOUP_FAIL(SOUP_ERR_ARG, "lora_pair_input: null pointer");
  if (!aligned16(x16) || !aligned4(bits_first) || !aligned4(bits_second) || !aligned16(gain) || !aligned16(a_pair) ||
      !aligned16(dx) || !aligned16(da_first) || !aligned16(da_second))
    SOUP_FAIL(SOUP_ERR_ARG, "lora_pair_input: unaligned pointer");
  InputArgs p;
  p.x = reinterpret_cast<const __half*>(x16);
  p.bits[0] = bits_first;
  p.bits[1] = bits_second;
  p.gain = reinterpret_cast<const __half*>(gain);
  p.a = reinterpret_cast<const __half*>(a_pair);
  p.dx = dx;
  p.da[0] = da_first;
  p.da[1] = da_second;
  p.scale[0] = scale_first;
  p.scale[1] = scale_second;
  p.rows = rows;
  p.hidden = (int)hidden;
  p.wide_dx = aligned32(dx);
  p.strips = (int)(hidden / 32);
  // row blocks per CTA, whole rounds of its four warps, that leave about one CTA per SM
  const int64_t columns = (p.strips + kInputStrips - 1) / kInputStrips, n_blocks = (rows + 15) / 16;
  int64_t per = (columns * n_blocks + sm_count() - 1) / sm_count();
  if (per < (n_blocks + 65534) / 65535) per = (n_blocks + 65534) / 65535;
  per = (per + kInputGroups - 1) / kInputGroups * kInputGroups;
  if (per > (1 << 20)) SOUP_FAIL(SOUP_ERR_ARG, "lora_pair_input: too many rows");
  p.blocks_per_cta = (int)per;
  const dim3 grid((unsigned)columns, (unsigned)((n_blocks + per - 1) / per));
  lora_input_kernel<<<grid, kInputStrips * kInputGroups * 32, 0, reinterpret_cast<cudaStream_t>(stream)>>>(p);
  SOUP_CHECK_LAUNCH("lora_pair_input");
  return SOUP_OK;
}
