// Fragments of the rank-16 adapter products (lora_pair.cu, lora_branch.cu) on mma.sync.m16n8k16: a rank of
// 16 is one k step or one m tile, operands go from global memory to fragments without shared memory, and a
// fragment's transpose is a movmatrix away. (A tcgen05 tile would be 128 wide where these are 16.)
#pragma once

#include "common.cuh"

namespace soup {
namespace rank16 {

constexpr int kRank = 16;

__device__ __forceinline__ uint32_t transpose8x8(uint32_t x) {
  uint32_t y;
  asm("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(y) : "r"(x));
  return y;
}

// c += a b: A [16 x 16] row, B [16 x 8] column fragments.
__device__ __forceinline__ void mma16816(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// The order of indices inside a product is free as long as both operands agree, so that a lane can move
// contiguous bytes: of 16 ranks, "index 2t, 2t + 1 of 8-block i" is rank 4t + 2i, 4t + 2i + 1, and of 32
// columns, "index 2t, 2t + 1 of 8-block j" is column 8t + 2j, 8t + 2j + 1 (t = lane % 4). With the plain
// order a fragment is four 4-byte loads a lane, 16 bytes of each of 8 rows, and the load unit is what
// bounds the kernel.
__device__ __forceinline__ int rank_of(int block, int index) { return 4 * (index >> 1) + 2 * block + (index & 1); }
__device__ __forceinline__ int column_of(int block, int index) { return 8 * (index >> 1) + 2 * block + (index & 1); }

// The A fragment of rows row0 .. row0 + 15 of a row-major fp16 [n_rows, 16] matrix; rows past n_rows read
// as zero.
__device__ __forceinline__ void load_rank_fragment(const __half* m, int64_t row0, int64_t n_rows, int lane,
                                                   uint32_t (&f)[4]) {
  const int g = lane >> 2, t = lane & 3;
#pragma unroll
  for (int half = 0; half < 2; ++half) {   // f[0], f[1]: rows g, g + 8 of block 0; f[2], f[3]: of block 1
    const int64_t row = row0 + g + half * 8;
    const uint2 v = row < n_rows ? __ldg(reinterpret_cast<const uint2*>(m + row * kRank + 4 * t)) : make_uint2(0u, 0u);
    f[half] = v.x;
    f[2 + half] = v.y;
  }
}

// Eight floats as one 32-byte store (p 32-byte aligned): two of 16 bytes would each leave half of a sector.
__device__ __forceinline__ void store_sector(float* p, const float (&v)[8]) {
  asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "f"(v[0]), "f"(v[1]), "f"(v[2]),
               "f"(v[3]), "f"(v[4]), "f"(v[5]), "f"(v[6]), "f"(v[7]) : "memory");
}
inline bool aligned32(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 31u) == 0; }

}  // namespace rank16
}  // namespace soup
