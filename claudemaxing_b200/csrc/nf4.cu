// NF4 dequantisation with the nested 8-bit absmax fused in: an HBM-streaming kernel.
//
// A thread turns kGroups groups of 8 packed bytes (one 64-bit load each) into 16 outputs each: fp16 in
// one 256-bit store, fp32 in two, so that a lane fills whole 32-byte sectors and a warp 1 KB in a row.
// (Groups of 16 bytes stored as four 128-bit pieces wrote every sector in two halves, from different
// instructions: the 46.8 M weights of a Qwen2.5-1.5B block took 27.8 us to fp16 and 86.0 us to fp32, now
// 20.8 and 34.8 us, 5.7 and 6.1 TB/s.) The 16 outputs of a group share one absmax block because every supported
// blocksize is a multiple of 32. All loads a thread needs are issued before the first is used; the
// 256-entry table is read through L1, eight or fewer entries a warp. The arithmetic is the reference's,
// operation for operation, with explicitly unfused fp32 intrinsics:
//   scale = code2[absmax8[b]] * absmax2[b / blocksize2]   (__fmul_rn)
//   scale = scale + offset                                 (__fadd_rn)
//   out   = round(code[nibble] * scale)                    (__fmul_rn, then RN to the out dtype)
// which is what makes the result bit-identical (solution/nf4.py:31-46 of the reference).
#include "common.cuh"

namespace soup {
namespace {

constexpr int kThreads = 256;
constexpr int kGroups = 4;        // independent 64-bit loads in flight per thread

template <bool NESTED>
__device__ __forceinline__ float block_scale(const void* absmax, const float* code2, const float* absmax2,
                                             float offset, int64_t blk, int shift2) {
  if (NESTED) {
    const uint32_t q8 = reinterpret_cast<const uint8_t*>(absmax)[blk];
    return __fadd_rn(__fmul_rn(__ldg(code2 + q8), __ldg(absmax2 + (blk >> shift2))), offset);
  }
  return __ldg(reinterpret_cast<const float*>(absmax) + blk);
}

// 32 bytes to a 32-byte aligned address in one store.
__device__ __forceinline__ void store32(void* p, const uint32_t (&w)[8]) {
  asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
               ::"l"(p), "r"(w[0]), "r"(w[1]), "r"(w[2]), "r"(w[3]), "r"(w[4]), "r"(w[5]), "r"(w[6]), "r"(w[7])
               : "memory");
}

// One CTA's share of one tensor: blocks [0, n_blocks) of the tensor, this CTA being `block`.
template <bool NESTED, bool OUT_F16>
__device__ __forceinline__ void
nf4_dequant_body(const uint8_t* __restrict__ packed, const void* __restrict__ absmax,
                 const float* __restrict__ code, const float* __restrict__ code2,
                 const float* __restrict__ absmax2, const float* __restrict__ offset_ptr,
                 void* __restrict__ out, int64_t n_bytes, int shift, int shift2, int64_t block,
                 int64_t n_blocks) {
  __shared__ float s_code[16];
  const bool wide = (reinterpret_cast<uintptr_t>(out) & 31u) == 0;   // else 16-byte aligned
  const int64_t n_groups = n_bytes >> 3;
  const int64_t g_base = block * (kThreads * kGroups) + threadIdx.x;
  uint2 raw[kGroups];
  uint32_t q8[kGroups];
  float top[kGroups];   // absmax2 of the group's block (nested), or its absmax
#pragma unroll
  for (int u = 0; u < kGroups; ++u) {
    const int64_t g = g_base + (int64_t)u * kThreads;
    if (g < n_groups) {
      raw[u] = __ldcs(reinterpret_cast<const uint2*>(packed) + g);
      const int64_t blk = (g << 4) >> shift;
      if (NESTED) {
        q8[u] = __ldg(reinterpret_cast<const uint8_t*>(absmax) + blk);
        top[u] = __ldg(absmax2 + (blk >> shift2));
      } else {
        top[u] = __ldg(reinterpret_cast<const float*>(absmax) + blk);
      }
    }
  }
  const float offset = NESTED ? __ldg(offset_ptr) : 0.f;
  if (threadIdx.x < 16) s_code[threadIdx.x] = code[threadIdx.x];
  __syncthreads();
#pragma unroll
  for (int u = 0; u < kGroups; ++u) {
    const int64_t g = g_base + (int64_t)u * kThreads;
    if (g >= n_groups) continue;
    const int64_t e0 = g << 4;  // first output element of this group
    const float scale = NESTED ? __fadd_rn(__fmul_rn(__ldg(code2 + q8[u]), top[u]), offset) : top[u];
    const uint32_t w[2] = {raw[u].x, raw[u].y};
    if (OUT_F16) {
      uint32_t h[8];
#pragma unroll
      for (int b = 0; b < 8; ++b) {
        const uint32_t byte = (w[b >> 2] >> (8 * (b & 3))) & 0xffu;
        const float hi = __fmul_rn(s_code[byte >> 4], scale);
        const float lo = __fmul_rn(s_code[byte & 15u], scale);
        __half2 p = __floats2half2_rn(hi, lo);
        h[b] = *reinterpret_cast<uint32_t*>(&p);
      }
      __half* o = reinterpret_cast<__half*>(out) + e0;
      if (wide) {
        store32(o, h);
      } else {
        reinterpret_cast<uint4*>(o)[0] = make_uint4(h[0], h[1], h[2], h[3]);
        reinterpret_cast<uint4*>(o)[1] = make_uint4(h[4], h[5], h[6], h[7]);
      }
    } else {
      float* o = reinterpret_cast<float*>(out) + e0;
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        uint32_t f[8];
#pragma unroll
        for (int b = 0; b < 4; ++b) {
          const uint32_t byte = (w[half] >> (8 * b)) & 0xffu;
          f[2 * b] = __float_as_uint(__fmul_rn(s_code[byte >> 4], scale));
          f[2 * b + 1] = __float_as_uint(__fmul_rn(s_code[byte & 15u], scale));
        }
        if (wide) {
          store32(o + 8 * half, f);
        } else {
          reinterpret_cast<uint4*>(o)[2 * half] = make_uint4(f[0], f[1], f[2], f[3]);
          reinterpret_cast<uint4*>(o)[2 * half + 1] = make_uint4(f[4], f[5], f[6], f[7]);
        }
      }
    }
  }

  // Ragged tail (n_bytes not a multiple of 8): the last block's first threads go byte by byte.
  if (block == n_blocks - 1) {
    const int64_t tail0 = n_groups << 3;
    for (int64_t i = tail0 + threadIdx.x; i < n_bytes; i += kThreads) {
      const uint32_t byte = packed[i];
      const int64_t e = i << 1;
      const float scale = block_scale<NESTED>(absmax, code2, absmax2, offset, e >> shift, shift2);
      const float hi = __fmul_rn(s_code[byte >> 4], scale);
      const float lo = __fmul_rn(s_code[byte & 15u], scale);
      if (OUT_F16) {
        reinterpret_cast<__half*>(out)[e] = __float2half_rn(hi);
        reinterpret_cast<__half*>(out)[e + 1] = __float2half_rn(lo);
      } else {
        reinterpret_cast<float*>(out)[e] = hi;
        reinterpret_cast<float*>(out)[e + 1] = lo;
      }
    }
  }
}

inline int64_t blocks_of(int64_t n_bytes) {
  const int64_t blocks = ((n_bytes >> 3) + kThreads * kGroups - 1) / (kThreads * kGroups);
  return blocks < 1 ? 1 : blocks;
}

template <bool NESTED, bool OUT_F16>
__global__ void __launch_bounds__(kThreads)
nf4_dequant_kernel(const uint8_t* __restrict__ packed, const void* __restrict__ absmax,
                   const float* __restrict__ code, const float* __restrict__ code2,
                   const float* __restrict__ absmax2, const float* __restrict__ offset_ptr,
                   void* __restrict__ out, int64_t n_bytes, int shift, int shift2) {
  nf4_dequant_body<NESTED, OUT_F16>(packed, absmax, code, code2, absmax2, offset_ptr, out, n_bytes,
                                    shift, shift2, blockIdx.x, gridDim.x);
}

// Several tensors in one launch: removes the per-launch latency that dominates the small projection
// weights (k/v of Qwen2.5-1.5B are 0.4 M elements each). Their blocks follow one another in the grid.
constexpr int kMaxBatch = 8;
struct Nf4Batch {
  soup_nf4_item item[kMaxBatch];
  int64_t first_block[kMaxBatch + 1];
  int count;
};

template <bool NESTED, bool OUT_F16>
__global__ void __launch_bounds__(kThreads)
nf4_dequant_batch_kernel(const __grid_constant__ Nf4Batch b, const float* __restrict__ code, int shift, int shift2) {
  int i = 0;
  while (i + 1 < b.count && (int64_t)blockIdx.x >= b.first_block[i + 1]) ++i;
  const soup_nf4_item& it = b.item[i];
  nf4_dequant_body<NESTED, OUT_F16>(reinterpret_cast<const uint8_t*>(it.packed), it.absmax, code,
                                    it.code2, it.absmax2, it.offset, it.out, it.n_elems >> 1, shift,
                                    shift2, blockIdx.x - b.first_block[i], b.first_block[i + 1] - b.first_block[i]);
}

inline int log2_exact(int v) {
  int s = 0;
  while ((1 << s) < v) ++s;
  return (1 << s) == v ? s : -1;
}

}  // namespace
}  // namespace soup

extern "C" int soup_nf4_dequant(const void* packed, const void* absmax, const float* code,
                                const float* code2, const float* absmax2, const float* offset,
                                void* out, int64_t n_elems, int blocksize, int blocksize2,
                                int nested, int out_dtype, void* stream) {
  using namespace soup;
  if (n_elems == 0) return SOUP_OK;
  if (!packed || !absmax || !code || !out) SOUP_FAIL(SOUP_ERR_ARG, "nf4_dequant: null pointer");
  if (n_elems < 0 || (n_elems & 1)) SOUP_FAIL(SOUP_ERR_ARG, "nf4_dequant: n_elems must be even");
  const int shift = log2_exact(blocksize);
  if (shift < 5 || shift > 12)
    SOUP_FAIL(SOUP_ERR_ARG, "nf4_dequant: blocksize %d not a power of two in [32,4096]", blocksize);
  int shift2 = 0;
  if (nested) {
    if (!code2 || !absmax2 || !offset) SOUP_FAIL(SOUP_ERR_ARG, "nf4_dequant: nested tables missing");
    shift2 = log2_exact(blocksize2);
    if (shift2 < 0) SOUP_FAIL(SOUP_ERR_ARG, "nf4_dequant: blocksize2 %d not a power of two", blocksize2);
  }
  if (out_dtype != SOUP_F16 && out_dtype != SOUP_F32)
    SOUP_FAIL(SOUP_ERR_ARG, "nf4_dequant: out dtype must be fp16 or fp32");
  if (!aligned16(packed) || !aligned16(out))
    SOUP_FAIL(SOUP_ERR_ARG, "nf4_dequant: packed and out must be 16-byte aligned");
  const int64_t n_bytes = n_elems >> 1;
  const int64_t blocks = blocks_of(n_bytes);
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
#define SOUP_NF4_LAUNCH(N_, F_)                                                              \
  nf4_dequant_kernel<N_, F_><<<(unsigned)blocks, kThreads, 0, s>>>(                          \
      reinterpret_cast<const uint8_t*>(packed), absmax, code, code2, absmax2, offset, out,   \
      n_bytes, shift, shift2)
  if (nested) {
    if (out_dtype == SOUP_F16) SOUP_NF4_LAUNCH(true, true); else SOUP_NF4_LAUNCH(true, false);
  } else {
    if (out_dtype == SOUP_F16) SOUP_NF4_LAUNCH(false, true); else SOUP_NF4_LAUNCH(false, false);
  }
#undef SOUP_NF4_LAUNCH
  SOUP_CHECK_LAUNCH("nf4_dequant");
  return SOUP_OK;
}


extern "C" int soup_nf4_dequant_batch(const soup_nf4_item* items, int count, const float* code,
                                      int blocksize, int blocksize2, int nested, int out_dtype,
                                      void* stream) {
  using namespace soup;
  if (count == 0) return SOUP_OK;
  if (count < 0 || !items || !code) SOUP_FAIL(SOUP_ERR_ARG, "nf4_dequant_batch: bad argument");
  const int shift = log2_exact(blocksize);
  if (shift < 5 || shift > 12)
    SOUP_FAIL(SOUP_ERR_ARG, "nf4_dequant_batch: blocksize %d not a power of two in [32,4096]", blocksize);
  int shift2 = 0;
  if (nested) {
    shift2 = log2_exact(blocksize2);
    if (shift2 < 0) SOUP_FAIL(SOUP_ERR_ARG, "nf4_dequant_batch: blocksize2 %d not a power of two", blocksize2);
  }
  if (out_dtype != SOUP_F16 && out_dtype != SOUP_F32)
    SOUP_FAIL(SOUP_ERR_ARG, "nf4_dequant_batch: out dtype must be fp16 or fp32");
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  for (int i0 = 0; i0 < count; i0 += kMaxBatch) {
    Nf4Batch b;
    int m = 0;
    b.first_block[0] = 0;
    for (int i = i0; i < count && m < kMaxBatch; ++i) {
      const soup_nf4_item& it = items[i];
      if (it.n_elems == 0) continue;
      if (!it.packed || !it.absmax || !it.out || it.n_elems < 0 || (it.n_elems & 1) ||
          (nested && (!it.code2 || !it.absmax2 || !it.offset)) || !aligned16(it.packed) ||
          !aligned16(it.out))
        SOUP_FAIL(SOUP_ERR_ARG, "nf4_dequant_batch: item %d is malformed", i);
      b.item[m] = it;
      b.first_block[m + 1] = b.first_block[m] + blocks_of(it.n_elems >> 1);
      ++m;
    }
    if (m == 0) continue;
    b.count = m;
    const unsigned grid = (unsigned)b.first_block[m];
    if (nested) {
      if (out_dtype == SOUP_F16) nf4_dequant_batch_kernel<true, true><<<grid, kThreads, 0, s>>>(b, code, shift, shift2);
      else nf4_dequant_batch_kernel<true, false><<<grid, kThreads, 0, s>>>(b, code, shift, shift2);
    } else {
      if (out_dtype == SOUP_F16) nf4_dequant_batch_kernel<false, true><<<grid, kThreads, 0, s>>>(b, code, shift, shift2);
      else nf4_dequant_batch_kernel<false, false><<<grid, kThreads, 0, s>>>(b, code, shift, shift2);
    }
    SOUP_CHECK_LAUNCH("nf4_dequant_batch");
  }
  return SOUP_OK;
}
