// RMSNorm forward and backward for Qwen2 (fp32 statistics, the reference's rounding points).
//
// Layout of the work: a thread owns VPT column vectors of 8 elements and keeps them in registers;
// a CTA of TPR threads covers one row (TPR * VPT * 8 >= n_cols) and processes R rows per step so
// that two rows' worth of 128-bit loads are in flight before the first reduction. The row sums are
// reduced with warp shuffles and one shared-memory exchange. Backward reads each row twice (the
// second time from L1/L2) instead of holding it in registers, which keeps ten CTAs per SM in
// flight; it is persistent when dw is
// wanted: a thread accumulates dw of its own columns in registers across the rows of its CTA and
// writes one partial row per CTA; a second tiny kernel adds the partial rows in a fixed order, so
// dw is deterministic.
//
// Rounding (solution/rmsnorm.py:28-91 of the reference): the normalised value is rounded to the
// dtype of x before it meets the weight; in backward dy*w is rounded to that dtype too, except on
// the saved-output path, where x is fp32 and nothing is rounded.
#include "common.cuh"
#include "rowpipe.cuh"

namespace soup {
namespace {

constexpr int kMaxWarps = 8;  // TPR <= 256

template <int R>
__device__ __forceinline__ void block_sum(float (&v)[R], float* s_red, int n_warps) {
#pragma unroll
  for (int r = 0; r < R; ++r) v[r] = warp_sum(v[r]);
  if (n_warps == 1) return;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  __syncthreads();  // previous use of s_red is over
  if (lane == 0) {
#pragma unroll
    for (int r = 0; r < R; ++r) s_red[r * kMaxWarps + warp] = v[r];
  }
  __syncthreads();
#pragma unroll
  for (int r = 0; r < R; ++r) {
    float t = 0.f;
    for (int wi = 0; wi < n_warps; ++wi) t += s_red[r * kMaxWarps + wi];
    v[r] = t;
  }
}

template <int VPT, int R>
__global__ void __launch_bounds__(256)
rmsnorm_fwd_kernel(const void* __restrict__ x, const void* __restrict__ w, void* __restrict__ out,
                   float* __restrict__ rstd_out, void* __restrict__ low,
                   const int32_t* __restrict__ slot, void* __restrict__ small, int64_t n_small,
                   int64_t n_rows, int n_cols, float eps, int xdt, int wdt, int odt) {
  __shared__ float s_red[R * kMaxWarps];
  const int n_vec = n_cols >> 3, n_warps = blockDim.x >> 5;
  const int64_t row0 = (int64_t)blockIdx.x * R;
  float xv[R][VPT][8];
  float ss[R];
#pragma unroll
  for (int r = 0; r < R; ++r) {
    ss[r] = 0.f;
    const int64_t row = row0 + r;
#pragma unroll
    for (int j = 0; j < VPT; ++j) {
      const int vi = threadIdx.x + j * blockDim.x;
      if (row < n_rows && vi < n_vec) {
        load8(x, row * n_cols + (vi << 3), xdt, xv[r][j]);
#pragma unroll
        for (int k = 0; k < 8; ++k) ss[r] += xv[r][j][k] * xv[r][j][k];
      }
    }
  }
  block_sum<R>(ss, s_red, n_warps);
#pragma unroll
  for (int j = 0; j < VPT; ++j) {
    const int vi = threadIdx.x + j * blockDim.x;
    if (vi >= n_vec) continue;
    float wv[8];
    load8(w, vi << 3, wdt, wv);
    int sl[8];
    if (low) {
      const int4 a = *reinterpret_cast<const int4*>(slot + (vi << 3));
      const int4 b = *reinterpret_cast<const int4*>(slot + (vi << 3) + 4);
      sl[0] = a.x; sl[1] = a.y; sl[2] = a.z; sl[3] = a.w;
      sl[4] = b.x; sl[5] = b.y; sl[6] = b.z; sl[7] = b.w;
    }
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int64_t row = row0 + r;
      if (row >= n_rows) continue;
      const float rstd = 1.0f / sqrtf(ss[r] / (float)n_cols + eps);
      if (j == 0 && threadIdx.x == 0) rstd_out[row] = rstd;
      float o[8], nrm[8];
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        nrm[k] = round_through(xv[r][j][k] * rstd, xdt);
        o[k] = nrm[k] * wv[k];
      }
      store8(out, row * n_cols + (vi << 3), odt, o);
      if (low) {
        store8(low, row * n_cols + (vi << 3), SOUP_F16, o);
#pragma unroll
        for (int k = 0; k < 8; ++k)
          if (sl[k] >= 0) store1(small, row * n_small + sl[k], SOUP_F16, nrm[k]);
      }
    }
  }
}

// Any n_cols / alignment: one CTA per row, columns re-read from global (L1/L2) for the second pass.
__global__ void __launch_bounds__(256)
rmsnorm_fwd_scalar_kernel(const void* __restrict__ x, const void* __restrict__ w,
                          void* __restrict__ out, float* __restrict__ rstd_out,
                          void* __restrict__ low, const int32_t* __restrict__ slot,
                          void* __restrict__ small, int64_t n_small, int n_cols, float eps, int xdt,
                          int wdt, int odt) {
  __shared__ float s_red[kMaxWarps];
  const int64_t row = blockIdx.x;
  float ss[1] = {0.f};
  for (int c = threadIdx.x; c < n_cols; c += blockDim.x) {
    const float v = load1(x, row * n_cols + c, xdt);
    ss[0] += v * v;
  }
  block_sum<1>(ss, s_red, blockDim.x >> 5);
  const float rstd = 1.0f / sqrtf(ss[0] / (float)n_cols + eps);
  if (threadIdx.x == 0) rstd_out[row] = rstd;
  for (int c = threadIdx.x; c < n_cols; c += blockDim.x) {
    const float nrm = round_through(load1(x, row * n_cols + c, xdt) * rstd, xdt);
    const float o = nrm * load1(w, c, wdt);
    store1(out, row * n_cols + c, odt, o);
    if (low) {
      store1(low, row * n_cols + c, SOUP_F16, o);
      const int s = slot[c];
      if (s >= 0) store1(small, row * n_small + s, SOUP_F16, nrm);
    }
  }
}

// One row of backward for one thread's column vector. Returns the thread's part of sum(gn * n).
__device__ __forceinline__ float bwd_prepare(const float (&dy)[8], const float (&xin)[8],
                                             const float (&wv)[8], const int (&sl)[8],
                                             const void* small, int64_t small_row, float rstd,
                                             int xdt, bool saved_output, float (&gn)[8],
                                             float (&nrm)[8]) {
  float dot = 0.f;
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    if (saved_output) {
      // xin holds fp16((x*rstd)*w); the tiny-|w| columns kept their normalised value aside.
      nrm[k] = sl[k] >= 0 ? load1(small, small_row + sl[k], SOUP_F16) : xin[k] / wv[k];
      gn[k] = dy[k] * wv[k];
    } else {
      nrm[k] = xin[k] * rstd;
      gn[k] = round_through(dy[k] * wv[k], xdt);
    }
    dot += gn[k] * nrm[k];
  }
  return dot;
}

template <int VPT, bool DW>
__global__ void __launch_bounds__(256)
rmsnorm_bwd_kernel(const void* __restrict__ dy, const void* __restrict__ xin,
                   const void* __restrict__ w, const float* __restrict__ rstd_in,
                   void* __restrict__ dx, float* __restrict__ dw_partial,
                   const int32_t* __restrict__ slot, const void* __restrict__ small,
                   int64_t n_small, int64_t n_rows, int n_cols, int ydt, int xdt, int wdt, int dxdt,
                   int saved_output) {
  __shared__ float s_red[kMaxWarps];
  const int n_vec = n_cols >> 3, n_warps = blockDim.x >> 5;
  float wv[VPT][8];
  int sl[VPT][8];
  float dw_acc[VPT][8];
#pragma unroll
  for (int j = 0; j < VPT; ++j) {
    const int vi = threadIdx.x + j * blockDim.x;
#pragma unroll
    for (int k = 0; k < 8; ++k) { wv[j][k] = 0.f; sl[j][k] = -1; dw_acc[j][k] = 0.f; }
    if (vi < n_vec) {
      load8(w, vi << 3, wdt, wv[j]);
      if (saved_output) {
        const int4 a = *reinterpret_cast<const int4*>(slot + (vi << 3));
        const int4 b = *reinterpret_cast<const int4*>(slot + (vi << 3) + 4);
        sl[j][0] = a.x; sl[j][1] = a.y; sl[j][2] = a.z; sl[j][3] = a.w;
        sl[j][4] = b.x; sl[j][5] = b.y; sl[j][6] = b.z; sl[j][7] = b.w;
      }
    }
  }
  // Two passes per row with few live registers, so that many CTAs fit on an SM and their loads
  // overlap: pass 1 reads dy and x for the row's dot product, pass 2 reads them again (they are
  // still in L1/L2, the row is 6 KB) and writes dx.
  for (int64_t row = blockIdx.x; row < n_rows; row += gridDim.x) {
    const float rstd = rstd_in[row];
    float dot[1] = {0.f};
#pragma unroll
    for (int j = 0; j < VPT; ++j) {
      const int vi = threadIdx.x + j * blockDim.x;
      if (vi < n_vec) {
        float yv[8], xv[8], gn[8], nrm[8];
        load8(dy, row * n_cols + (vi << 3), ydt, yv);
        load8(xin, row * n_cols + (vi << 3), xdt, xv);
        dot[0] += bwd_prepare(yv, xv, wv[j], sl[j], small, row * n_small, rstd, xdt,
                              saved_output != 0, gn, nrm);
        if (DW) {
#pragma unroll
          for (int k = 0; k < 8; ++k) dw_acc[j][k] += yv[k] * round_through(nrm[k], xdt);
        }
      }
    }
    block_sum<1>(dot, s_red, n_warps);
    const float mean_dot = dot[0] / (float)n_cols;
#pragma unroll
    for (int j = 0; j < VPT; ++j) {
      const int vi = threadIdx.x + j * blockDim.x;
      if (vi < n_vec) {
        float yv[8], xv[8], gn[8], nrm[8], o[8];
        load8(dy, row * n_cols + (vi << 3), ydt, yv);
        load8(xin, row * n_cols + (vi << 3), xdt, xv);
        bwd_prepare(yv, xv, wv[j], sl[j], small, row * n_small, rstd, xdt, saved_output != 0, gn, nrm);
#pragma unroll
        for (int k = 0; k < 8; ++k) o[k] = (gn[k] - nrm[k] * mean_dot) * rstd;
        store8(dx, row * n_cols + (vi << 3), dxdt, o);
      }
    }
  }
  if (DW) {
#pragma unroll
    for (int j = 0; j < VPT; ++j) {
      const int vi = threadIdx.x + j * blockDim.x;
      if (vi < n_vec) store8(dw_partial, (int64_t)blockIdx.x * n_cols + (vi << 3), SOUP_F32, dw_acc[j]);
    }
  }
}

template <bool DW>
__global__ void __launch_bounds__(256)
rmsnorm_bwd_scalar_kernel(const void* __restrict__ dy, const void* __restrict__ xin,
                          const void* __restrict__ w, const float* __restrict__ rstd_in,
                          void* __restrict__ dx, float* __restrict__ dw_partial,
                          const int32_t* __restrict__ slot, const void* __restrict__ small,
                          int64_t n_small, int64_t n_rows, int n_cols, int ydt, int xdt, int wdt,
                          int dxdt, int saved_output) {
  // dw_partial row of this CTA is accumulated in place in global memory (zeroed first).
  __shared__ float s_red[kMaxWarps];
  if (DW)
    for (int c = threadIdx.x; c < n_cols; c += blockDim.x)
      dw_partial[(int64_t)blockIdx.x * n_cols + c] = 0.f;
  for (int64_t row = blockIdx.x; row < n_rows; row += gridDim.x) {
    const float rstd = rstd_in[row];
    float dot[1] = {0.f};
    for (int c = threadIdx.x; c < n_cols; c += blockDim.x) {
      const float yv = load1(dy, row * n_cols + c, ydt), xv = load1(xin, row * n_cols + c, xdt);
      const float wc = load1(w, c, wdt);
      float nrm, gn;
      if (saved_output) {
        const int s = slot[c];
        nrm = s >= 0 ? load1(small, row * n_small + s, SOUP_F16) : xv / wc;
        gn = yv * wc;
      } else {
        nrm = xv * rstd;
        gn = round_through(yv * wc, xdt);
      }
      dot[0] += gn * nrm;
      if (DW) dw_partial[(int64_t)blockIdx.x * n_cols + c] += yv * round_through(nrm, xdt);
    }
    block_sum<1>(dot, s_red, blockDim.x >> 5);
    const float mean_dot = dot[0] / (float)n_cols;
    for (int c = threadIdx.x; c < n_cols; c += blockDim.x) {
      const float yv = load1(dy, row * n_cols + c, ydt), xv = load1(xin, row * n_cols + c, xdt);
      const float wc = load1(w, c, wdt);
      float nrm, gn;
      if (saved_output) {
        const int s = slot[c];
        nrm = s >= 0 ? load1(small, row * n_small + s, SOUP_F16) : xv / wc;
        gn = yv * wc;
      } else {
        nrm = xv * rstd;
        gn = round_through(yv * wc, xdt);
      }
      store1(dx, row * n_cols + c, dxdt, (gn - nrm * mean_dot) * rstd);
    }
  }
}

// dw[c] = sum over partial rows, fixed order, rounded once to the weight dtype. 32 columns a CTA, every
// sixteenth partial row a warp: a chain of 37 loads for 592 partial rows, where one thread a column had 592
// (11.8 -> 5.0 us at 1536 columns).
constexpr int kReduceWarps = 16;
__global__ void __launch_bounds__(kReduceWarps * 32)
rmsnorm_dw_reduce_kernel(const float* __restrict__ partial, void* __restrict__ dw, int n_partials,
                         int n_cols, int wdt) {
  __shared__ float s_sum[kReduceWarps][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int c = blockIdx.x * 32 + lane;
  float acc = 0.f;
  if (c < n_cols) {
#pragma unroll 8
    for (int p = warp; p < n_partials; p += kReduceWarps) acc += partial[(int64_t)p * n_cols + c];
  }
  s_sum[warp][lane] = acc;
  __syncthreads();
  if (warp != 0 || c >= n_cols) return;
#pragma unroll
  for (int w = 1; w < kReduceWarps; ++w) acc += s_sum[w][lane];
  store1(dw, c, wdt, acc);
}

// ------------------------------------------------------------------------------------------
// Warp-per-row kernels (rows of at most 16 vectors per lane: 2048 fp32 or 4096 16-bit columns).
//
// A warp owns a row: every lane issues all of its 16-byte loads of the row at once, keeps the raw
// bits in registers (4 registers per vector whatever the dtype), reduces with shuffles only (no
// shared memory, no CTA barrier) and streams the results out; then it takes its next row. A lane's
// vector is 16 bytes of the widest streamed input, so every load instruction of the warp covers
// 512 contiguous bytes. With ~50-80 registers per thread 24-36 warps are resident per SM, each
// with a whole row (3-6 KB) in flight, which is what HBM latency x bandwidth asks for.
// ------------------------------------------------------------------------------------------
constexpr int kWarpsPerCta = 8;

template <int EPV>
__device__ __forceinline__ void load_slots(const int32_t* slot, int i, int (&sl)[EPV]) {
#pragma unroll
  for (int q = 0; q < EPV / 4; ++q) {
    const int4 a = *reinterpret_cast<const int4*>(slot + i + 4 * q);
    sl[4 * q] = a.x; sl[4 * q + 1] = a.y; sl[4 * q + 2] = a.z; sl[4 * q + 3] = a.w;
  }
}

// Bit j of the result: vector j of this lane contains a column with a side-buffer slot.
template <int NV, int EPV>
__device__ __forceinline__ uint32_t lane_slot_mask(const int32_t* slot, int n_vec, int lane) {
  uint32_t mask = 0;
  if (!slot) return 0;
#pragma unroll
  for (int j = 0; j < NV; ++j) {
    const int vi = j * 32 + lane;
    if (vi < n_vec) {
      int sl[EPV];
      load_slots<EPV>(slot, vi * EPV, sl);
#pragma unroll
      for (int k = 0; k < EPV; ++k) if (sl[k] >= 0) mask |= 1u << j;
    }
  }
  return mask;
}

// ------------------------------------------------------------------------------------------
// Pipelined warp-per-row kernels: rows arrive in the warp's shared-memory ring (rowpipe.cuh), both
// passes over a row read it from there, results go straight to global memory. Any n_cols whose
// row slot fits the ring; vectors are 16 bytes of the widest streamed input.
// ------------------------------------------------------------------------------------------
template <int EPV, int B>
__device__ __forceinline__ void unpack_smem(const char* row, int vi, int dt, float (&v)[EPV]) {
  unpack<EPV, B>(ld_raw<EPV * B>(row, (int64_t)vi * EPV * B), dt, v);
}

// A dtype that is a template constant (>= 0) is folded by the compiler; -1 takes the run-time code.
template <int C> __device__ __forceinline__ int dt_sel(int rt) { return C >= 0 ? C : rt; }

// ------------------------------------------------------------------------------------------
// One CTA per row (four rows of up to 256 columns), eight columns per thread, everything a row needs
// requested at once: bound by memory when many rows are in flight, by one row's latency when few are.
// The ring kernels below spend the latter on ring set-up, a serial walk of the row by one or two warps
// and, in backward, on the weight's copy in shared memory. With fp32 rows this form was the faster one at 1536
// columns and every row count (10 B and 16 B an element: forward 7.4 -> 5.3 us at 1280 rows, 44.9 -> 41.8 at
// 16384; backward with the residual 14.4 -> 7.6 and 87.6 -> 68.4; 64 rows 5.5 -> 1.9 and 8.1 -> 2.5), and from 8
// to 4096 columns but for: the forward without the fp16 copy at 2048 to 3072 columns and more than 2000 rows,
// 6 % faster to 10 % slower (2048 x 2300 7.9 -> 8.6, x 16384 48.5 -> 46.4; 3072 x 16384 68 -> 71), and the backward without
// the residual at 65536 rows of 64 to 384 columns and 16384 of 2048, 4 to 7 % slower (384 columns 57.5 ->
// 61.5). A 16-bit row is half the bytes for the same threads, and the ring wins once more rows are waiting
// than fit: `row_kernel_covers`. The residual form keeps the 2048 columns it always took: wider rows are
// three launches.
// ------------------------------------------------------------------------------------------
constexpr int kRowMaxThreads = 512;   // rows of up to 4096 columns

// Sum over a row's threads (every thread gets it), in a fixed order; one warp or the whole CTA.
__device__ __forceinline__ float cta_sum(float v, float* s_red) {
  v = warp_sum(v);
  const int warps = (int)(blockDim.x >> 5);
  if (warps == 1) return v;
  if ((threadIdx.x & 31) == 0) s_red[threadIdx.x >> 5] = v;
  __syncthreads();
  float t = 0.f;
  for (int w = 0; w < warps; ++w) t += s_red[w];
  return t;
}

template <int XDT, int WDT, int ODT>
__global__ void __launch_bounds__(kRowMaxThreads)
rmsnorm_fwd_row_kernel(const void* __restrict__ x, const void* __restrict__ w, void* __restrict__ out,
                       float* __restrict__ rstd_out, void* __restrict__ low, const int32_t* __restrict__ slot,
                       void* __restrict__ small, int64_t n_small, int64_t n_rows, int n_cols, float eps,
                       int xdt_rt, int wdt_rt, int odt_rt) {
  __shared__ float s_red[kRowMaxThreads / 32];
  const int xdt = dt_sel<XDT>(xdt_rt), wdt = dt_sel<WDT>(wdt_rt), odt = dt_sel<ODT>(odt_rt);
  const int64_t row = (int64_t)blockIdx.x * blockDim.y + threadIdx.y, at = row * n_cols + threadIdx.x * 8;
  if (row >= n_rows) return;   // only where a warp is a row: nobody waits for it
  const int col = threadIdx.x * 8;
  const bool mine = col < n_cols;
  float xv[8], wv[8];
  int sl[8];
  float ss = 0.f;
  if (mine) {
    load8(x, at, xdt, xv);
    load8(w, col, wdt, wv);
    if (low) load_slots<8>(slot, col, sl);
#pragma unroll
    for (int k = 0; k < 8; ++k) ss += xv[k] * xv[k];
  }
  ss = cta_sum(ss, s_red);
  const float rstd = 1.0f / sqrtf(ss * (1.0f / (float)n_cols) + eps);
  if (threadIdx.x == 0) rstd_out[row] = rstd;
  if (!mine) return;
  float o[8], nrm[8];
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    nrm[k] = round_through(xv[k] * rstd, xdt);
    o[k] = nrm[k] * wv[k];
  }
  store8(out, at, odt, o);
  if (low) {
    store8(low, at, SOUP_F16, o);
#pragma unroll
    for (int k = 0; k < 8; ++k)
      if (sl[k] >= 0) store1(small, row * n_small + sl[k], SOUP_F16, nrm[k]);
  }
}

// The 4-bit model's backward: fp32 dy, the fp16 copy of the forward's output as the saved tensor, fp32
// weight and dx, optionally the residual gradient added and an fp16 copy of the sum written.
__global__ void __launch_bounds__(kRowMaxThreads)
rmsnorm_bwd_saved_row_kernel(const float* __restrict__ dy, const __half* __restrict__ saved,
                             const float* __restrict__ w, const float* __restrict__ rstd_in,
                             const float* __restrict__ add, float* __restrict__ dx, __half* __restrict__ dx16,
                             const int32_t* __restrict__ slot, const __half* __restrict__ small, int64_t n_small,
                             int64_t n_rows, int n_cols) {
  __shared__ float s_red[kRowMaxThreads / 32];
  const int64_t row = (int64_t)blockIdx.x * blockDim.y + threadIdx.y, at = row * n_cols + threadIdx.x * 8;
  if (row >= n_rows) return;   // only where a warp is a row: nobody waits for it
  const int col = threadIdx.x * 8;
  const bool mine = col < n_cols;
  const float rstd = rstd_in[row];
  float yv[8], nrm[8], extra[8];
  float dot = 0.f;
  if (mine) {
    float xv[8], wv[8];
    int sl[8];
    load8(dy, at, SOUP_F32, yv);
    load8(saved, at, SOUP_F16, xv);
    if (add) load8(add, at, SOUP_F32, extra);
    load8(w, col, SOUP_F32, wv);
    load_slots<8>(slot, col, sl);
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      // the normalised value: saved / w, except in the side-buffer columns (|w| tiny)
      nrm[k] = xv[k] * (1.0f / wv[k]);
      if (sl[k] >= 0) nrm[k] = __half2float(small[row * n_small + sl[k]]);
      yv[k] *= wv[k];
      dot += yv[k] * nrm[k];
    }
  }
  const float mean_dot = cta_sum(dot, s_red) * (1.0f / (float)n_cols);
  if (!mine) return;
  float o[8];
#pragma unroll
  for (int k = 0; k < 8; ++k) o[k] = (yv[k] - nrm[k] * mean_dot) * rstd;
  if (add) {   // the gradient that reaches the same tensor along the residual connection
#pragma unroll
    for (int k = 0; k < 8; ++k) o[k] += extra[k];
  }
  store8(dx, at, SOUP_F32, o);
  if (dx16) store8(dx16, at, SOUP_F16, o);   // and its fp16 copy, for the projection backward that receives it next
}

// Backward with a trainable weight, dy, x, weight and dx of one dtype: a CTA walks its rows kDwRows at a
// time, a thread owning eight columns of all of them, so that the weight and the weight gradient's sums are
// eight registers each and one exchange serves kDwRows rows. Bound by memory: four CTAs of 192 threads keep
// 74 KB of it in flight on an SM (four rows spill at that many CTAs). (The warp-per-row kernel below holds
// the sums of a whole row in a warp, 48 registers a thread, and reads dtypes at run time: 101.1 -> 32.3 us
// for 16384 fp16 rows of 1536 columns.)
constexpr int kDwRows = 3;
template <int DT>
__global__ void __launch_bounds__(kRowMaxThreads) __maxnreg__(DT == SOUP_F32 ? 128 : 80)
rmsnorm_bwd_dw_row_kernel(const void* __restrict__ dy, const void* __restrict__ x, const void* __restrict__ w,
                          const float* __restrict__ rstd_in, void* __restrict__ dx,
                          float* __restrict__ dw_partial, int64_t n_rows, int n_cols) {
  constexpr int XB = DT == SOUP_F32 ? 4 : 2, V = XB / 2;   // 16-byte vectors of eight elements
  constexpr int kWarps = kRowMaxThreads / 32;
  __shared__ float s_red[2][kDwRows][kWarps];
  const int col = threadIdx.x * 8, warp = threadIdx.x >> 5, warps = (int)(blockDim.x >> 5);
  const bool mine = col < n_cols;
  const float inv_cols = 1.0f / (float)n_cols;
  float wv[8], dw[8];
#pragma unroll
  for (int k = 0; k < 8; ++k) wv[k] = dw[k] = 0.f;
  if (mine) load8(w, col, DT, wv);
  const int64_t n_steps = (n_rows + kDwRows - 1) / kDwRows;
  int turn = 0;
  for (int64_t step = blockIdx.x; step < n_steps; step += gridDim.x, turn ^= 1) {
    const int64_t row0 = step * kDwRows;
    Raw<16> yr[kDwRows][V], xr[kDwRows][V];
    float rstd[kDwRows], dot[kDwRows];
#pragma unroll
    for (int r = 0; r < kDwRows; ++r) {
      const bool ok = mine && row0 + r < n_rows;
      rstd[r] = row0 + r < n_rows ? rstd_in[row0 + r] : 0.f;
#pragma unroll
      for (int v = 0; v < V; ++v) {
        const int64_t at = ((row0 + r) * n_cols + col) * XB + v * 16;
        yr[r][v].v = xr[r][v].v = make_uint4(0u, 0u, 0u, 0u);
        if (ok) {
          yr[r][v] = ld_raw<16>(dy, at);
          xr[r][v] = ld_raw<16>(x, at);
        }
      }
    }
    auto eight = [](const Raw<16> (&raw)[V], float (&f)[8]) {
#pragma unroll
      for (int v = 0; v < V; ++v) {
        float part[8 / V];
        unpack<8 / V, XB>(raw[v], DT, part);
#pragma unroll
        for (int k = 0; k < 8 / V; ++k) f[v * (8 / V) + k] = part[k];
      }
    };
#pragma unroll
    for (int r = 0; r < kDwRows; ++r) {
      float yv[8], xv[8];
      eight(yr[r], yv);
      eight(xr[r], xv);
      dot[r] = 0.f;
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const float nrm = xv[k] * rstd[r];
        dot[r] += round_through(yv[k] * wv[k], DT) * nrm;
        dw[k] += yv[k] * round_through(nrm, DT);
      }
    }
#pragma unroll
    for (int r = 0; r < kDwRows; ++r) dot[r] = warp_sum(dot[r]);
    if ((threadIdx.x & 31) == 0) {
#pragma unroll
      for (int r = 0; r < kDwRows; ++r) s_red[turn][r][warp] = dot[r];
    }
    __syncthreads();   // one barrier a step: the next one writes the other half of s_red
#pragma unroll
    for (int r = 0; r < kDwRows; ++r) {
      float sum = 0.f;
      for (int i = 0; i < warps; ++i) sum += s_red[turn][r][i];
      if (mine && row0 + r < n_rows) {
        const float mean_dot = sum * inv_cols;
        float yv[8], xv[8], o[8];
        eight(yr[r], yv);
        eight(xr[r], xv);
#pragma unroll
        for (int k = 0; k < 8; ++k)
          o[k] = (round_through(yv[k] * wv[k], DT) - xv[k] * rstd[r] * mean_dot) * rstd[r];
        store8(dx, (row0 + r) * n_cols + col, DT, o);
      }
    }
  }
  if (mine) store8(dw_partial, (int64_t)blockIdx.x * n_cols + col, SOUP_F32, dw);
}

// XDT / WDT / ODT: compile-time dtype codes of the hot combinations, or -1 for "read the argument".
template <int XB, int XDT, int WDT, int ODT>
__global__ void __launch_bounds__(rowpipe::kMaxWarps * 32, 2)
rmsnorm_fwd_pipe_kernel(const void* __restrict__ x, const void* __restrict__ w,
                        void* __restrict__ out, float* __restrict__ rstd_out,
                        void* __restrict__ low, const int32_t* __restrict__ slot,
                        void* __restrict__ small, int64_t n_small, int64_t n_rows, int n_cols,
                        float eps, int xdt_rt, int wdt_rt, int odt_rt, int stages, int team, int* status) {
  constexpr int EPV = 16 / XB;
  const int xdt = dt_sel<XDT>(xdt_rt), wdt = dt_sel<WDT>(wdt_rt), odt = dt_sel<ODT>(odt_rt);
  extern __shared__ __align__(128) char smem[];
  __shared__ int s_abort;
  __shared__ float s_part[2 * rowpipe::kMaxWarps];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
  // a team of `team` (1 or 2) warps shares a row: member m owns vectors [v0, v0 + n_vec)
  const int member = team == 2 ? (warp & 1) : 0;
  const int n_vec = n_cols / EPV / team, v0 = member * n_vec;
  const uint32_t row_bytes = (uint32_t)n_cols * XB / team;   // this member's share of a row
  if (threadIdx.x == 0) s_abort = 0;
  rowpipe::Ring ring;
  ring.init(smem, row_bytes, stages, warp, lane);
  __syncthreads();
  const int64_t row0 = (int64_t)blockIdx.x * (warps / team) + warp / team;
  const int64_t stride = (int64_t)gridDim.x * (warps / team);
  const char* xb = reinterpret_cast<const char*>(x) + (size_t)member * row_bytes;
  const int64_t row_pitch = (int64_t)n_cols * XB;
  int64_t next = row0;   // next row to request
  if (lane == 0) {
    for (int s = 0; s < stages && next < n_rows; ++s, next += stride) {
      umma::mbar_expect_tx(&ring.bars[s], row_bytes);
      rowpipe::bulk_load(ring.slot_ptr(s), xb + next * row_pitch, row_bytes, &ring.bars[s]);
    }
  }
  next = __shfl_sync(0xffffffffu, next, 0);
  // bit v of slot_mask: this lane's v-th vector holds a column with a side-buffer slot
  uint64_t slot_mask = 0;
  if (low) {
    for (int vi = lane, v = 0; vi < n_vec; vi += 32, ++v) {
      int sl[EPV];
      load_slots<EPV>(slot, (v0 + vi) * EPV, sl);
#pragma unroll
      for (int k = 0; k < EPV; ++k) if (sl[k] >= 0) slot_mask |= 1ull << v;
    }
  }
  const float inv_cols = 1.0f / (float)n_cols;
  int iter = 0;
  for (int64_t row = row0; row < n_rows; row += stride, ++iter) {
    if (!ring.wait(&s_abort, status, 11)) {
      ring.drain((int)((next - row) / stride));   // the copies still travelling to this warp's slots
      // a partner already waiting at this row's team barrier is released (it gives up at its next wait)
      if (team == 2) asm volatile("bar.arrive %0, 64;" ::"r"((warp >> 1) + 1) : "memory");
      return;
    }
    const char* src = ring.slot_ptr(ring.slot);
    float ss = 0.f;
#pragma unroll 4
    for (int vi = lane; vi < n_vec; vi += 32) {
      float xv[EPV];
      unpack_smem<EPV, XB>(src, vi, xdt, xv);
#pragma unroll
      for (int k = 0; k < EPV; ++k) ss += xv[k] * xv[k];
    }
    ss = warp_sum(ss);
    if (team == 2) ss = rowpipe::team_sum2(ss, s_part, warp, lane, iter);
    const float rstd = 1.0f / sqrtf(ss * inv_cols + eps);
    if (lane == 0 && member == 0) rstd_out[row] = rstd;
    int v = 0;
#pragma unroll 2
    for (int vi = lane; vi < n_vec; vi += 32, ++v) {
      float xv[EPV], wv[EPV], o[EPV], nrm[EPV];
      unpack_smem<EPV, XB>(src, vi, xdt, xv);
      const int col = (v0 + vi) * EPV;
      loadv<EPV>(w, col, wdt, wv);   // a few KB of weights: L1-resident after the first row
#pragma unroll
      for (int k = 0; k < EPV; ++k) {
        nrm[k] = round_through(xv[k] * rstd, xdt);
        o[k] = nrm[k] * wv[k];
      }
      storev<EPV>(out, row * n_cols + col, odt, o);
      if (low) {
        storev<EPV>(low, row * n_cols + col, SOUP_F16, o);
        if (slot_mask >> v & 1ull) {
          int sl[EPV];
          load_slots<EPV>(slot, col, sl);
#pragma unroll
          for (int k = 0; k < EPV; ++k)
            if (sl[k] >= 0) store1(small, row * n_small + sl[k], SOUP_F16, nrm[k]);
        }
      }
    }
    __syncwarp();
    if (next < n_rows) {
      if (lane == 0) {
        umma::fence_proxy_async_smem();   // the slot's reads are done before the copy overwrites it
        umma::mbar_expect_tx(&ring.bars[ring.slot], row_bytes);
        rowpipe::bulk_load(ring.slot_ptr(ring.slot), xb + next * row_pitch, row_bytes,
                           &ring.bars[ring.slot]);
      }
      next += stride;
    }
    ring.advance();
  }
}

// Backward without dw: a slot holds the dy row followed by the saved row (x, or the fp16 copy of
// the output). YDT .. SAVED: compile-time values of the hot combinations, or -1 for the argument.
template <int YB, int XB, int YDT, int XDT, int WDT, int DXDT, int SAVED>
__global__ void __launch_bounds__(rowpipe::kMaxWarps * 32, 2)
rmsnorm_bwd_pipe_kernel(const void* __restrict__ dy, const void* __restrict__ xin,
                        const void* __restrict__ w, const float* __restrict__ rstd_in,
                        void* __restrict__ dx, const int32_t* __restrict__ slot,
                        const void* __restrict__ small, int64_t n_small, int64_t n_rows, int n_cols,
                        int ydt_rt, int xdt_rt, int wdt_rt, int dxdt_rt, int saved_rt, int stages,
                        int team, int* status) {
  constexpr int EPV = 16 / (YB > XB ? YB : XB);
  const int ydt = dt_sel<YDT>(ydt_rt), xdt = dt_sel<XDT>(xdt_rt), wdt = dt_sel<WDT>(wdt_rt);
  const int dxdt = dt_sel<DXDT>(dxdt_rt), saved_output = dt_sel<SAVED>(saved_rt);
  extern __shared__ __align__(128) char smem[];
  __shared__ int s_abort;
  __shared__ float s_part[2 * rowpipe::kMaxWarps];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
  const int member = team == 2 ? (warp & 1) : 0;
  const int n_vec = n_cols / EPV / team, v0 = member * n_vec;
  // this member's share of a dy row and of a saved row
  const uint32_t y_bytes = (uint32_t)n_cols * YB / team, x_bytes = (uint32_t)n_cols * XB / team;
  const int64_t y_pitch = (int64_t)n_cols * YB, x_pitch = (int64_t)n_cols * XB;
  if (threadIdx.x == 0) s_abort = 0;
  rowpipe::Ring ring;
  ring.init(smem, y_bytes + x_bytes, stages, warp, lane);
  __syncthreads();
  const int64_t row0 = (int64_t)blockIdx.x * (warps / team) + warp / team;
  const int64_t stride = (int64_t)gridDim.x * (warps / team);
  const char* yb = reinterpret_cast<const char*>(dy) + (size_t)member * y_bytes;
  const char* xb = reinterpret_cast<const char*>(xin) + (size_t)member * x_bytes;
  int64_t next = row0;
  if (lane == 0) {
    for (int s = 0; s < stages && next < n_rows; ++s, next += stride) {
      umma::mbar_expect_tx(&ring.bars[s], y_bytes + x_bytes);
      rowpipe::bulk_load(ring.slot_ptr(s), yb + next * y_pitch, y_bytes, &ring.bars[s]);
      rowpipe::bulk_load(ring.slot_ptr(s) + y_bytes, xb + next * x_pitch, x_bytes, &ring.bars[s]);
    }
  }
  next = __shfl_sync(0xffffffffu, next, 0);
  uint64_t slot_mask = 0;
  if (saved_output) {
    for (int vi = lane, v = 0; vi < n_vec; vi += 32, ++v) {
      int sl[EPV];
      load_slots<EPV>(slot, (v0 + vi) * EPV, sl);
#pragma unroll
      for (int k = 0; k < EPV; ++k) if (sl[k] >= 0) slot_mask |= 1ull << v;
    }
  }
  const float inv_cols = 1.0f / (float)n_cols;
  int iter = 0;
  for (int64_t row = row0; row < n_rows; row += stride, ++iter) {
    if (!ring.wait(&s_abort, status, 12)) {
      ring.drain((int)((next - row) / stride));
      if (team == 2) asm volatile("bar.arrive %0, 64;" ::"r"((warp >> 1) + 1) : "memory");
      return;
    }
    const char* ysrc = ring.slot_ptr(ring.slot);
    const char* xsrc = ysrc + y_bytes;
    const float rstd = rstd_in[row];
    float dot = 0.f;
    int v = 0;
#pragma unroll 2
    for (int vi = lane; vi < n_vec; vi += 32, ++v) {
      float yv[EPV], xv[EPV], wv[EPV];
      unpack_smem<EPV, YB>(ysrc, vi, ydt, yv);
      unpack_smem<EPV, XB>(xsrc, vi, xdt, xv);
      const int col = (v0 + vi) * EPV;
      loadv<EPV>(w, col, wdt, wv);
      int sl[EPV];
#pragma unroll
      for (int k = 0; k < EPV; ++k) sl[k] = -1;
      if (slot_mask >> v & 1ull) load_slots<EPV>(slot, col, sl);
#pragma unroll
      for (int k = 0; k < EPV; ++k) {
        float nrm, gn;
        if (saved_output) {
          nrm = sl[k] >= 0 ? load1(small, row * n_small + sl[k], SOUP_F16) : xv[k] / wv[k];
          gn = yv[k] * wv[k];
        } else {
          nrm = xv[k] * rstd;
          gn = round_through(yv[k] * wv[k], xdt);
        }
        dot += gn * nrm;
      }
    }
    dot = warp_sum(dot);
    if (team == 2) dot = rowpipe::team_sum2(dot, s_part, warp, lane, iter);
    const float mean_dot = dot * inv_cols;
    v = 0;
#pragma unroll 2
    for (int vi = lane; vi < n_vec; vi += 32, ++v) {
      float yv[EPV], xv[EPV], wv[EPV], o[EPV];
      unpack_smem<EPV, YB>(ysrc, vi, ydt, yv);
      unpack_smem<EPV, XB>(xsrc, vi, xdt, xv);
      const int col = (v0 + vi) * EPV;
      loadv<EPV>(w, col, wdt, wv);
      int sl[EPV];
#pragma unroll
      for (int k = 0; k < EPV; ++k) sl[k] = -1;
      if (slot_mask >> v & 1ull) load_slots<EPV>(slot, col, sl);
#pragma unroll
      for (int k = 0; k < EPV; ++k) {
        float nrm, gn;
        if (saved_output) {
          nrm = sl[k] >= 0 ? load1(small, row * n_small + sl[k], SOUP_F16) : xv[k] / wv[k];
          gn = yv[k] * wv[k];
        } else {
          nrm = xv[k] * rstd;
          gn = round_through(yv[k] * wv[k], xdt);
        }
        o[k] = (gn - nrm * mean_dot) * rstd;
      }
      storev<EPV>(dx, row * n_cols + col, dxdt, o);
    }
    __syncwarp();
    if (next < n_rows) {
      if (lane == 0) {
        umma::fence_proxy_async_smem();
        umma::mbar_expect_tx(&ring.bars[ring.slot], y_bytes + x_bytes);
        rowpipe::bulk_load(ring.slot_ptr(ring.slot), yb + next * y_pitch, y_bytes,
                           &ring.bars[ring.slot]);
        rowpipe::bulk_load(ring.slot_ptr(ring.slot) + y_bytes, xb + next * x_pitch, x_bytes,
                           &ring.bars[ring.slot]);
      }
      next += stride;
    }
    ring.advance();
  }
}

// YB / XB: bytes per element of dy and of the saved tensor (x, or the fp16 copy of the output).
template <int NV, int YB, int XB, bool DW>
__global__ void __launch_bounds__(kWarpsPerCta * 32)
rmsnorm_bwd_warp_kernel(const void* __restrict__ dy, const void* __restrict__ xin,
                        const void* __restrict__ w, const float* __restrict__ rstd_in,
                        void* __restrict__ dx, float* __restrict__ dw_partial,
                        const int32_t* __restrict__ slot, const void* __restrict__ small,
                        int64_t n_small, int64_t n_rows, int n_cols, int ydt, int xdt, int wdt,
                        int dxdt, int saved_output) {
  constexpr int EPV = 16 / (YB > XB ? YB : XB);
  extern __shared__ float s_dw[];   // DW only: n_cols floats
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int n_vec = n_cols / EPV;
  const int64_t warp0 = (int64_t)blockIdx.x * kWarpsPerCta + warp;
  const int64_t stride = (int64_t)gridDim.x * kWarpsPerCta;
  const uint32_t slot_mask = saved_output ? lane_slot_mask<NV, EPV>(slot, n_vec, lane) : 0u;
  const float inv_cols = 1.0f / (float)n_cols;
  float dw_acc[DW ? NV : 1][EPV];
  if (DW) {
#pragma unroll
    for (int j = 0; j < NV; ++j)
#pragma unroll
      for (int k = 0; k < EPV; ++k) dw_acc[j][k] = 0.f;
  }
  for (int64_t row = warp0; row < n_rows; row += stride) {
    Raw<EPV * YB> yraw[NV];
    Raw<EPV * XB> xraw[NV];
#pragma unroll
    for (int j = 0; j < NV; ++j) {
      const int vi = j * 32 + lane;
      if (vi < n_vec) {
        const int64_t e = row * n_cols + (int64_t)vi * EPV;
        yraw[j] = ld_raw<EPV * YB>(dy, e * YB);
        xraw[j] = ld_raw<EPV * XB>(xin, e * XB);
      }
    }
    const float rstd = rstd_in[row];
    float dot = 0.f;
#pragma unroll
    for (int j = 0; j < NV; ++j) {
      const int vi = j * 32 + lane;
      if (vi < n_vec) {
        float yv[EPV], xv[EPV], wv[EPV];
        unpack<EPV, YB>(yraw[j], ydt, yv);
        unpack<EPV, XB>(xraw[j], xdt, xv);
        loadv<EPV>(w, vi * EPV, wdt, wv);
        int sl[EPV];
#pragma unroll
        for (int k = 0; k < EPV; ++k) sl[k] = -1;
        if (slot_mask >> j & 1u) load_slots<EPV>(slot, vi * EPV, sl);
#pragma unroll
        for (int k = 0; k < EPV; ++k) {
          float nrm, gn;
          if (saved_output) {
            nrm = sl[k] >= 0 ? load1(small, row * n_small + sl[k], SOUP_F16) : xv[k] / wv[k];
            gn = yv[k] * wv[k];
          } else {
            nrm = xv[k] * rstd;
            gn = round_through(yv[k] * wv[k], xdt);
          }
          dot += gn * nrm;
          if (DW) dw_acc[j][k] += yv[k] * round_through(nrm, xdt);
        }
      }
    }
    dot = warp_sum(dot);
    const float mean_dot = dot * inv_cols;
#pragma unroll
    for (int j = 0; j < NV; ++j) {
      const int vi = j * 32 + lane;
      if (vi < n_vec) {
        float yv[EPV], xv[EPV], wv[EPV], o[EPV];
        unpack<EPV, YB>(yraw[j], ydt, yv);
        unpack<EPV, XB>(xraw[j], xdt, xv);
        loadv<EPV>(w, vi * EPV, wdt, wv);
        int sl[EPV];
#pragma unroll
        for (int k = 0; k < EPV; ++k) sl[k] = -1;
        if (slot_mask >> j & 1u) load_slots<EPV>(slot, vi * EPV, sl);
#pragma unroll
        for (int k = 0; k < EPV; ++k) {
          float nrm, gn;
          if (saved_output) {
            nrm = sl[k] >= 0 ? load1(small, row * n_small + sl[k], SOUP_F16) : xv[k] / wv[k];
            gn = yv[k] * wv[k];
          } else {
            nrm = xv[k] * rstd;
            gn = round_through(yv[k] * wv[k], xdt);
          }
          o[k] = (gn - nrm * mean_dot) * rstd;
        }
        storev<EPV>(dx, row * n_cols + (int64_t)vi * EPV, dxdt, o);
      }
    }
  }
  if (DW) {
    // The CTA's warps add their column sums in warp order (deterministic), one partial row per CTA.
    for (int turn = 0; turn < kWarpsPerCta; ++turn) {
      if (warp == turn) {
#pragma unroll
        for (int j = 0; j < NV; ++j) {
          const int vi = j * 32 + lane;
          if (vi < n_vec) {
#pragma unroll
            for (int k = 0; k < EPV; ++k) {
              const int c = vi * EPV + k;
              s_dw[c] = turn == 0 ? dw_acc[j][k] : s_dw[c] + dw_acc[j][k];
            }
          }
        }
      }
      __syncthreads();
    }
    for (int c = threadIdx.x; c < n_cols; c += blockDim.x)
      dw_partial[(int64_t)blockIdx.x * n_cols + c] = s_dw[c];
  }
}

// Vectors per lane the warp kernels are built for; 0: the row is too wide for them.
inline int pick_nv(int n_cols, int epv) {
  const int need = (n_cols / epv + 31) / 32;
  const int options[] = {2, 4, 6, 8, 12, 16};
  for (int o : options) if (need <= o) return o;
  return 0;
}

inline unsigned warp_grid(int64_t n_rows, int ctas_per_sm) {
  const int64_t need = (n_rows + kWarpsPerCta - 1) / kWarpsPerCta;
  const int64_t cap = (int64_t)sm_count() * ctas_per_sm;
  return (unsigned)(need < cap ? (need < 1 ? 1 : need) : cap);
}

struct Shape { int vpt, tpr; };

// Smallest VPT in {1,2,4,8} whose CTA (<= 256 threads) covers the row.
inline Shape pick_shape(int n_cols) {
  const int n_vec = n_cols >> 3;
  int vpt = 1;
  while (vpt < 8 && (n_vec + vpt - 1) / vpt > 256) vpt <<= 1;
  int tpr = (n_vec + vpt - 1) / vpt;
  tpr = ((tpr + 31) / 32) * 32;
  return {vpt, tpr};
}

inline int64_t bwd_ctas(int64_t n_rows) {
  const int64_t cap = (int64_t)sm_count() * 4;
  return n_rows < cap ? (n_rows < 1 ? 1 : n_rows) : cap;
}

// Launch shape of the row kernels: a row's threads, and rows per CTA.
inline dim3 row_block(int64_t n_cols) {
  const unsigned threads = (unsigned)((n_cols / 8 + 31) / 32 * 32);
  return dim3(threads, threads == 32 ? 4 : 1);
}
inline unsigned row_grid(int64_t n_rows, dim3 block) { return (unsigned)((n_rows + block.y - 1) / block.y); }

// Whether the row kernel is the faster one (see there). fp32 rows: always. 16-bit rows: while at most two
// waves of them wait, counted in threads, of which the kernel's registers leave 1152 on an SM (ring and row
// kernel, in us: 1536 columns 4.9 -> 4.1 at 1280 rows but 5.1 -> 5.5 at 2000, 2048 columns 5.1 -> 4.6 at 1200 but
// 5.8 -> 6.9 at 2300, 3584 columns 6.0 -> 7.6 at 1100, 768 columns 4.7 -> 4.4 at 3200 but 4.6 -> 5.6 at 4608).
// Rows of one warp need no barrier and win up to three and a half (128 columns 7.0 -> 5.2 at 16384 rows).
inline bool row_kernel_covers(int64_t n_rows, int64_t n_cols, int dtype) {
  if (n_cols > kRowMaxThreads * 8) return false;
  const unsigned threads = row_block(n_cols).x;
  return dtype == SOUP_F32 || n_rows * threads <= 2ll * sm_count() * (threads == 32 ? 2048 : 1152);
}

// Whether the weight-gradient row kernel is the faster one. Rows of one warp stay with the kernel whose warps take a
// row each. So do many fp32 rows of two or three warps: four CTAs leave an SM 256 or 384 threads, less in flight than
// it takes (warp-per-row and row kernel, in us: 264 columns 22.2 and 17.9 at 8192 rows, 28.5 and 28.9 at 16384, 65.8 and
// 87.0 at 65536; 512 columns 33.5 and 31.3 at 16384, 82.9 and 96.3 at 65536; 576 columns 60.1 and 57.9 at 32768, 99.6 and 106 at
// 65536; 768 columns 69.1 and 63.3 at 32768, 212 and 223 at 131072). Wider rows and 16-bit ones gain at any number of rows:
// fp32 896 x 65536 262 and 129, fp16 264 x 262144 267 and 243, 1024 x 32768 126 and 50.7, bf16 512 x 65536 94.6 and 75.3.
inline bool dw_row_kernel_covers(int64_t n_rows, int64_t n_cols, int dtype) {
  if (n_cols <= 256 || n_cols > kRowMaxThreads * 8) return false;
  if (dtype != SOUP_F32 || n_cols > 768) return true;
  return n_rows <= (n_cols <= 512 ? 16384 : 32768);
}

}  // namespace
}  // namespace soup

extern "C" int soup_rmsnorm_fwd(const void* x, const void* w, void* out, float* rstd, void* low,
                                const int32_t* slot, void* small, int64_t n_small, int64_t n_rows,
                                int64_t n_cols, float eps, int x_dtype, int w_dtype, int out_dtype,
                                void* stream) {
  using namespace soup;
  if (n_rows == 0) return SOUP_OK;
  if (n_rows < 0 || n_cols <= 0 || n_cols > 16384)
    SOUP_FAIL(SOUP_ERR_ARG, "rmsnorm_fwd: need 0 < n_cols <= 16384 (got %lld)", (long long)n_cols);
  if (!x || !w || !out || !rstd) SOUP_FAIL(SOUP_ERR_ARG, "rmsnorm_fwd: null pointer");
  if (!is_float_dtype(x_dtype) || !is_float_dtype(w_dtype) || !is_float_dtype(out_dtype))
    SOUP_FAIL(SOUP_ERR_ARG, "rmsnorm_fwd: unsupported dtype");
  if (low && (!slot || !small || n_small < 1))
    SOUP_FAIL(SOUP_ERR_ARG, "rmsnorm_fwd: low copy needs slot map and side buffer");
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  const bool vec = (n_cols % 8 == 0) && aligned16(x) && aligned16(w) && aligned16(out) &&
                   (!low || (aligned16(low) && aligned16(slot)));
  const int xb = dtype_size(x_dtype);
  // a team of two can split a row whose halves are whole 16-byte vectors
  const rowpipe::Plan plan = vec ? rowpipe::make_plan((size_t)n_cols * xb, 0, (n_cols * xb) % 32 == 0, n_rows)
                                 : rowpipe::Plan{8, 0, 1, 1, 0, 0};
  int* status = plan.stages ? rowpipe::status_word() : nullptr;
  if (!vec) {
    rmsnorm_fwd_scalar_kernel<<<(unsigned)n_rows, 256, 0, s>>>(x, w, out, rstd, low, slot, small,
                                                               n_small, (int)n_cols, eps, x_dtype,
                                                               w_dtype, out_dtype);
  } else if (row_kernel_covers(n_rows, n_cols, x_dtype)) {
    const dim3 block = row_block(n_cols);
#define SOUP_RMS_FWD_R(X_, W_, O_)                                                               \
  rmsnorm_fwd_row_kernel<X_, W_, O_><<<row_grid(n_rows, block), block, 0, s>>>(                  \
      x, w, out, rstd, low, slot, small, n_small, n_rows, (int)n_cols, eps, x_dtype, w_dtype, out_dtype)
    const bool same = x_dtype == w_dtype && x_dtype == out_dtype;
    if (same && x_dtype == SOUP_F32) SOUP_RMS_FWD_R(SOUP_F32, SOUP_F32, SOUP_F32);
    else if (same && x_dtype == SOUP_F16) SOUP_RMS_FWD_R(SOUP_F16, SOUP_F16, SOUP_F16);
    else if (same && x_dtype == SOUP_BF16) SOUP_RMS_FWD_R(SOUP_BF16, SOUP_BF16, SOUP_BF16);
    else SOUP_RMS_FWD_R(-1, -1, -1);
#undef SOUP_RMS_FWD_R
  } else if (plan.stages && status) {
#define SOUP_RMS_FWD_P(XB_, X_, W_, O_)                                                          \
  do {                                                                                            \
    auto kernel = rmsnorm_fwd_pipe_kernel<XB_, X_, W_, O_>;                                       \
    cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)plan.smem);    \
    kernel<<<plan.grid, plan.warps * 32, plan.smem, s>>>(x, w, out, rstd, low, slot, small,       \
                                                         n_small, n_rows, (int)n_cols, eps,       \
                                                         x_dtype, w_dtype, out_dtype, plan.stages, \
                                                         plan.team, status);                      \
  } while (0)
    const bool same = x_dtype == w_dtype && x_dtype == out_dtype;
    if (same && x_dtype == SOUP_F32) SOUP_RMS_FWD_P(4, SOUP_F32, SOUP_F32, SOUP_F32);
    else if (same && x_dtype == SOUP_F16) SOUP_RMS_FWD_P(2, SOUP_F16, SOUP_F16, SOUP_F16);
    else if (same && x_dtype == SOUP_BF16) SOUP_RMS_FWD_P(2, SOUP_BF16, SOUP_BF16, SOUP_BF16);
    else if (xb == 4) SOUP_RMS_FWD_P(4, SOUP_F32, -1, -1);
    else SOUP_RMS_FWD_P(2, -1, -1, -1);
#undef SOUP_RMS_FWD_P
  } else {
    const Shape sh = pick_shape((int)n_cols);
    constexpr int R = 2;  // rows per CTA step (4 measured slower: fewer CTAs fit on an SM)
    const unsigned grid = (unsigned)((n_rows + R - 1) / R);
#define SOUP_RMS_FWD(V_)                                                                       \
  rmsnorm_fwd_kernel<V_, R><<<grid, sh.tpr, 0, s>>>(x, w, out, rstd, low, slot, small, n_small, \
                                                    n_rows, (int)n_cols, eps, x_dtype, w_dtype, \
                                                    out_dtype)
    switch (sh.vpt) {
      case 1: SOUP_RMS_FWD(1); break;
      case 2: SOUP_RMS_FWD(2); break;
      case 4: SOUP_RMS_FWD(4); break;
      default: SOUP_RMS_FWD(8); break;
    }
#undef SOUP_RMS_FWD
  }
  SOUP_CHECK_LAUNCH("rmsnorm_fwd");
  return SOUP_OK;
}

extern "C" int64_t soup_rmsnorm_bwd_partials(int64_t n_rows, int64_t n_cols) {
  (void)n_cols;
  return soup::bwd_ctas(n_rows);
}

namespace soup {
namespace {
int rmsnorm_bwd_any(const void* dy, const void* xin, const void* w, const float* rstd, void* dx,
                    float* dw_partial, void* dw, const int32_t* slot, const void* small,
                    int64_t n_small, int64_t n_rows, int64_t n_cols, int dy_dtype, int xin_dtype,
                    int w_dtype, int dx_dtype, int saved_output, const float* add, __half* dx16,
                    void* stream);
}  // namespace
}  // namespace soup

extern "C" int soup_rmsnorm_bwd(const void* dy, const void* xin, const void* w, const float* rstd,
                                void* dx, float* dw_partial, void* dw, const int32_t* slot,
                                const void* small, int64_t n_small, int64_t n_rows, int64_t n_cols,
                                int dy_dtype, int xin_dtype, int w_dtype, int dx_dtype,
                                int saved_output, void* stream) {
  return soup::rmsnorm_bwd_any(dy, xin, w, rstd, dx, dw_partial, dw, slot, small, n_small, n_rows,
                               n_cols, dy_dtype, xin_dtype, w_dtype, dx_dtype, saved_output, nullptr,
                               nullptr, stream);
}

extern "C" int soup_rmsnorm_bwd_residual(const float* dy, const void* low, const float* w,
                                         const float* rstd, const float* add, float* dx, void* dx16,
                                         const int32_t* slot, const void* small, int64_t n_small,
                                         int64_t n_rows, int64_t n_cols, void* stream) {
  if (add && (reinterpret_cast<uintptr_t>(add) & 15u))
    SOUP_FAIL(SOUP_ERR_ARG, "rmsnorm_bwd_residual: the residual gradient must be 16-byte aligned");
  if (dx16 && (reinterpret_cast<uintptr_t>(dx16) & 7u))
    SOUP_FAIL(SOUP_ERR_ARG, "rmsnorm_bwd_residual: the fp16 copy must be 8-byte aligned");
  return soup::rmsnorm_bwd_any(dy, low, w, rstd, dx, nullptr, nullptr, slot, small, n_small, n_rows,
                               n_cols, SOUP_F32, SOUP_F16, SOUP_F32, SOUP_F32, 1, add,
                               reinterpret_cast<__half*>(dx16), stream);
}

namespace soup {
namespace {
int rmsnorm_bwd_any(const void* dy, const void* xin, const void* w, const float* rstd, void* dx,
                    float* dw_partial, void* dw, const int32_t* slot, const void* small,
                    int64_t n_small, int64_t n_rows, int64_t n_cols, int dy_dtype, int xin_dtype,
                    int w_dtype, int dx_dtype, int saved_output, const float* add, __half* dx16,
                    void* stream) {
  if (n_rows < 0 || n_cols <= 0 || n_cols > 16384)
    SOUP_FAIL(SOUP_ERR_ARG, "rmsnorm_bwd: need 0 < n_cols <= 16384 (got %lld)", (long long)n_cols);
  const bool want_dw = dw != nullptr;
  if (want_dw && !dw_partial) SOUP_FAIL(SOUP_ERR_ARG, "rmsnorm_bwd: dw needs the partial workspace");
  if (want_dw && saved_output)
    SOUP_FAIL(SOUP_ERR_ARG, "rmsnorm_bwd: the saved-output path is for a frozen weight (no dw)");
  if (!is_float_dtype(dy_dtype) || !is_float_dtype(xin_dtype) || !is_float_dtype(w_dtype) ||
      !is_float_dtype(dx_dtype))
    SOUP_FAIL(SOUP_ERR_ARG, "rmsnorm_bwd: unsupported dtype");
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  if (n_rows == 0) {
    if (want_dw) cudaMemsetAsync(dw, 0, (size_t)n_cols * dtype_size(w_dtype), s);
    return SOUP_OK;
  }
  if (!dy || !xin || !w || !rstd || !dx) SOUP_FAIL(SOUP_ERR_ARG, "rmsnorm_bwd: null pointer");
  if (saved_output && (!slot || !small || n_small < 1))
    SOUP_FAIL(SOUP_ERR_ARG, "rmsnorm_bwd: saved-output path needs slot map and side buffer");
  // Rows of moderate width go to the warp-per-row kernel; wider ones to one CTA per row (a
  // persistent grid when dw is accumulated). A 16-bit dy with a 32-bit saved tensor does not occur
  // on the training path and takes the CTA kernel.
  const bool vec = (n_cols % 8 == 0) && aligned16(dy) && aligned16(xin) && aligned16(w) &&
                   aligned16(dx) && (!saved_output || aligned16(slot)) &&
                   (!want_dw || aligned16(dw_partial));
  const int yb = dtype_size(dy_dtype), xb = dtype_size(xin_dtype);
  const int nv = (vec && want_dw && yb >= xb) ? pick_nv((int)n_cols, 16 / yb) : 0;
  const rowpipe::Plan plan = (vec && !want_dw && yb >= xb)
                                 ? rowpipe::make_plan((size_t)n_cols * (yb + xb), 0,
                                                      (n_cols * xb) % 32 == 0, n_rows)
                                 : rowpipe::Plan{8, 0, 1, 1, 0, 0};
  int* status = plan.stages ? rowpipe::status_word() : nullptr;
  unsigned grid = (unsigned)(want_dw ? bwd_ctas(n_rows) : n_rows);
  if ((add || dx16) && !(vec && plan.stages && status))
    SOUP_FAIL(SOUP_ERR_ARG, "rmsnorm_bwd_residual: this shape does not take the residual form");
  if (!vec) {
    if (want_dw)
      rmsnorm_bwd_scalar_kernel<true><<<grid, 256, 0, s>>>(dy, xin, w, rstd, dx, dw_partial, slot,
                                                           small, n_small, n_rows, (int)n_cols,
                                                           dy_dtype, xin_dtype, w_dtype, dx_dtype,
                                                           saved_output);
    else
      rmsnorm_bwd_scalar_kernel<false><<<grid, 256, 0, s>>>(dy, xin, w, rstd, dx, dw_partial, slot,
                                                            small, n_small, n_rows, (int)n_cols,
                                                            dy_dtype, xin_dtype, w_dtype, dx_dtype,
                                                            saved_output);
  } else if (plan.stages && status) {
    grid = plan.grid;
#define SOUP_RMS_BWD_P(YB_, XB_, Y_, X_, W_, DX_, SV_)                                           \
  do {                                                                                            \
    auto kernel = rmsnorm_bwd_pipe_kernel<YB_, XB_, Y_, X_, W_, DX_, SV_>;                        \
    cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)plan.smem);    \
    kernel<<<plan.grid, plan.warps * 32, plan.smem, s>>>(dy, xin, w, rstd, dx, slot, small,       \
                                                         n_small, n_rows, (int)n_cols, dy_dtype,  \
                                                         xin_dtype, w_dtype, dx_dtype,            \
                                                         saved_output, plan.stages, plan.team,    \
                                                         status);                                 \
  } while (0)
    const bool same = dy_dtype == xin_dtype && dy_dtype == w_dtype && dy_dtype == dx_dtype;
    const bool four_bit = saved_output && dy_dtype == SOUP_F32 && xin_dtype == SOUP_F16 &&
                          w_dtype == SOUP_F32 && dx_dtype == SOUP_F32;
    const bool rows = four_bit && row_kernel_covers(n_rows, n_cols, SOUP_F32) && (!dx16 || aligned16(dx16));
    if ((add || dx16) && !(rows && n_cols <= 2048))
      SOUP_FAIL(SOUP_ERR_ARG, "rmsnorm_bwd_residual: this shape does not take the residual form");
    if (rows) {
      const dim3 block = row_block(n_cols);
      rmsnorm_bwd_saved_row_kernel<<<row_grid(n_rows, block), block, 0, s>>>(
          reinterpret_cast<const float*>(dy), reinterpret_cast<const __half*>(xin),
          reinterpret_cast<const float*>(w), rstd, add, reinterpret_cast<float*>(dx), dx16, slot,
          reinterpret_cast<const __half*>(small), n_small, n_rows, (int)n_cols);
    } else if (four_bit)
      SOUP_RMS_BWD_P(4, 2, SOUP_F32, SOUP_F16, SOUP_F32, SOUP_F32, 1);
    else if (!saved_output && same && dy_dtype == SOUP_F16)
      SOUP_RMS_BWD_P(2, 2, SOUP_F16, SOUP_F16, SOUP_F16, SOUP_F16, 0);
    else if (!saved_output && same && dy_dtype == SOUP_BF16)
      SOUP_RMS_BWD_P(2, 2, SOUP_BF16, SOUP_BF16, SOUP_BF16, SOUP_BF16, 0);
    else if (!saved_output && same && dy_dtype == SOUP_F32)
      SOUP_RMS_BWD_P(4, 4, SOUP_F32, SOUP_F32, SOUP_F32, SOUP_F32, 0);
    else if (yb == 4 && xb == 4) SOUP_RMS_BWD_P(4, 4, SOUP_F32, SOUP_F32, -1, -1, -1);
    else if (yb == 4) SOUP_RMS_BWD_P(4, 2, SOUP_F32, -1, -1, -1, -1);
    else SOUP_RMS_BWD_P(2, 2, -1, -1, -1, -1, -1);
#undef SOUP_RMS_BWD_P
  } else if (want_dw && dw_row_kernel_covers(n_rows, n_cols, dy_dtype) && dy_dtype == xin_dtype &&
             dy_dtype == w_dtype && dy_dtype == dx_dtype) {
    const int64_t steps = (n_rows + kDwRows - 1) / kDwRows;
    if (steps < grid) grid = (unsigned)steps;
    const unsigned threads = row_block(n_cols).x;
#define SOUP_RMS_BWD_DW(DT_) \
  rmsnorm_bwd_dw_row_kernel<DT_><<<grid, threads, 0, s>>>(dy, xin, w, rstd, dx, dw_partial, n_rows, (int)n_cols)
    if (dy_dtype == SOUP_F16) SOUP_RMS_BWD_DW(SOUP_F16);
    else if (dy_dtype == SOUP_BF16) SOUP_RMS_BWD_DW(SOUP_BF16);
    else SOUP_RMS_BWD_DW(SOUP_F32);
#undef SOUP_RMS_BWD_DW
  } else if (nv) {
    grid = warp_grid(n_rows, 2);
    const size_t smem = (size_t)n_cols * sizeof(float);
#define SOUP_RMS_BWD_W(NV_, YB_, XB_)                                                            \
  rmsnorm_bwd_warp_kernel<NV_, YB_, XB_, true><<<grid, kWarpsPerCta * 32, smem, s>>>(             \
      dy, xin, w, rstd, dx, dw_partial, slot, small, n_small, n_rows, (int)n_cols, dy_dtype,      \
      xin_dtype, w_dtype, dx_dtype, saved_output)
#define SOUP_RMS_BWD_NV(YB_, XB_)                                                                \
  switch (nv) {                                                                                   \
    case 2: SOUP_RMS_BWD_W(2, YB_, XB_); break;                                                   \
    case 4: SOUP_RMS_BWD_W(4, YB_, XB_); break;                                                   \
    case 6: SOUP_RMS_BWD_W(6, YB_, XB_); break;                                                   \
    case 8: SOUP_RMS_BWD_W(8, YB_, XB_); break;                                                   \
    case 12: SOUP_RMS_BWD_W(12, YB_, XB_); break;                                                 \
    default: SOUP_RMS_BWD_W(16, YB_, XB_); break;                                                 \
  }
    if (yb == 4 && xb == 4) { SOUP_RMS_BWD_NV(4, 4) }
    else if (yb == 4) { SOUP_RMS_BWD_NV(4, 2) }
    else { SOUP_RMS_BWD_NV(2, 2) }
#undef SOUP_RMS_BWD_NV
#undef SOUP_RMS_BWD_W
  } else {
    const Shape sh = pick_shape((int)n_cols);
#define SOUP_RMS_BWD(V_, D_)                                                                     \
  rmsnorm_bwd_kernel<V_, D_><<<grid, sh.tpr, 0, s>>>(dy, xin, w, rstd, dx, dw_partial, slot, small, \
                                                     n_small, n_rows, (int)n_cols, dy_dtype,      \
                                                     xin_dtype, w_dtype, dx_dtype, saved_output)
    if (want_dw) {
      switch (sh.vpt) {
        case 1: SOUP_RMS_BWD(1, true); break;
        case 2: SOUP_RMS_BWD(2, true); break;
        case 4: SOUP_RMS_BWD(4, true); break;
        default: SOUP_RMS_BWD(8, true); break;
      }
    } else {
      switch (sh.vpt) {
        case 1: SOUP_RMS_BWD(1, false); break;
        case 2: SOUP_RMS_BWD(2, false); break;
        case 4: SOUP_RMS_BWD(4, false); break;
        default: SOUP_RMS_BWD(8, false); break;
      }
    }
#undef SOUP_RMS_BWD
  }
  SOUP_CHECK_LAUNCH("rmsnorm_bwd");
  if (want_dw) {
    rmsnorm_dw_reduce_kernel<<<(unsigned)((n_cols + 31) / 32), kReduceWarps * 32, 0, s>>>(
        dw_partial, dw, (int)grid, (int)n_cols, w_dtype);
    SOUP_CHECK_LAUNCH("rmsnorm_dw_reduce");
  }
  return SOUP_OK;
}
}  // namespace
}  // namespace soup


// ------------------------------------------------------------------------------------------
// Backward with the dw workspace inside the library, for callers that cannot allocate.
// ------------------------------------------------------------------------------------------
namespace soup {
namespace {

constexpr int kStaticPartialRows = 640;   // >= 4 CTAs per SM on a 148-SM part (592)
constexpr int kStaticMaxCols = 4096;

// 640 x 4096 fp32 = 10 MiB of device memory per GPU that loads the library, held until exit.
static __device__ __align__(256) float g_dw_scratch[kStaticPartialRows * kStaticMaxCols];

// In host code `g_dw_scratch` is only a handle for the runtime, not a device address; the address
// a kernel can use comes from cudaGetSymbolAddress, asked once per device with that device current.
float* g_dw_scratch_addr[64] = {nullptr};

int static_scratch(float** out) {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return -1;
  if (!g_dw_scratch_addr[dev]) {
    void* p = nullptr;
    const cudaError_t e = cudaGetSymbolAddress(&p, g_dw_scratch);
    if (e != cudaSuccess || !p) {
      set_error("rmsnorm_bwd_noalloc: cudaGetSymbolAddress failed: %s", cudaGetErrorString(e));
      return -2;
    }
    g_dw_scratch_addr[dev] = reinterpret_cast<float*>(p);
  }
  *out = g_dw_scratch_addr[dev];
  return 0;
}

}  // namespace
}  // namespace soup

extern "C" int soup_rmsnorm_bwd_noalloc(const void* dy, const void* xin, const void* w,
                                        const float* rstd, void* dx, void* dw, const int32_t* slot,
                                        const void* small, int64_t n_small, int64_t n_rows,
                                        int64_t n_cols, int dy_dtype, int xin_dtype, int w_dtype,
                                        int dx_dtype, int saved_output, void* stream) {
  using namespace soup;
  if (n_cols > kStaticMaxCols)
    SOUP_FAIL(SOUP_ERR_ARG, "rmsnorm_bwd_noalloc: n_cols %lld exceeds the built-in workspace (max %d); "
              "use soup_rmsnorm_bwd with a caller-provided workspace", (long long)n_cols, kStaticMaxCols);
  if (soup_rmsnorm_bwd_partials(n_rows, n_cols) > kStaticPartialRows)
    SOUP_FAIL(SOUP_ERR_ARG, "rmsnorm_bwd_noalloc: this device needs %lld partial rows, the built-in "
              "workspace has %d", (long long)soup_rmsnorm_bwd_partials(n_rows, n_cols), kStaticPartialRows);
  float* scratch = nullptr;
  if (dw) {
    const int rc = static_scratch(&scratch);
    if (rc == -1) SOUP_FAIL(SOUP_ERR_DEVICE, "rmsnorm_bwd_noalloc: no current CUDA device");
    if (rc != 0) return SOUP_ERR_DEVICE;
  }
  // Every partial row the reduce reads is fully rewritten by its CTA first, so nothing in the
  // workspace has to start at zero even though it keeps the previous call's contents.
  return soup_rmsnorm_bwd(dy, xin, w, rstd, dx, scratch, dw, slot, small, n_small, n_rows, n_cols,
                          dy_dtype, xin_dtype, w_dtype, dx_dtype, saved_output, stream);
}
