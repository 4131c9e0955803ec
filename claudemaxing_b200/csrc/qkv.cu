// The fused block's passes on either side of the attention: the q/k/v projection's output split into
// rotated q (+ adapter), rotated k and v (+ adapter), and the three fp32 gradients of the attention
// rotated back and laid side by side as the fp16 gradient of that projection's output.
//
// A thread owns a pair of 8-element vectors: the matching vectors of a head's two halves, or 16
// neighbouring elements of v. Bound by memory and, at the few thousand tokens of a step, by latency:
// one launch with every pair of the packed row in flight: 4.8 us forward and 5.5 us backward for 1280
// tokens, 12 / 2 heads of 128 (a rotation launch, and a launch of torch's for v's sum or copy, took
// 7.3 + 5.6 and 6.9 + 5.4 us). Arithmetic is fp32 with one rounding, as in qwen_rope_kernel of the
// reference (solution/rope.py:17-43) on the fp32 sum.
#include "common.cuh"

namespace soup {
namespace {

constexpr int kThreads = 256;

struct QkvShape {
  int64_t n;         // tokens
  int hq, hk, d;
  int rot_pairs, v_pairs;   // per token
};

// What pair `i` of a token is: element of the first vector inside the token's [q | k | v] row, the
// distance to the second, and the head dimension's index for the tables (v: distance 8, no tables).
struct Pair {
  int first, apart, angle;
  bool rotated;
};
__device__ __forceinline__ Pair pair_of(const QkvShape& s, int i) {
  Pair p;
  p.rotated = i < s.rot_pairs;
  if (p.rotated) {
    const int per_head = s.d >> 4, h = i / per_head;
    p.angle = (i - h * per_head) << 3;
    p.first = h * s.d + p.angle;
    p.apart = s.d >> 1;
  } else {
    p.angle = 0;
    p.first = (s.hq + s.hk) * s.d + ((i - s.rot_pairs) << 4);
    p.apart = 8;
  }
  return p;
}

struct Tables {
  float c1[8], c2[8], s1[8], s2[8];
  __device__ __forceinline__ void load(const float* cos, const float* sin, int64_t at, int half) {
    load8(cos, at, SOUP_F32, c1);
    load8(cos, at + half, SOUP_F32, c2);
    load8(sin, at, SOUP_F32, s1);
    load8(sin, at + half, SOUP_F32, s2);
  }
};

__global__ void __launch_bounds__(kThreads)
qkv_rope_fwd_kernel(const __half* __restrict__ qkv, int64_t pitch, const __half* __restrict__ add_q,
                    const __half* __restrict__ add_v, const float* __restrict__ cos,
                    const float* __restrict__ sin, __half* __restrict__ q, __half* __restrict__ k,
                    __half* __restrict__ v, const QkvShape s) {
  const int pairs = s.rot_pairs + s.v_pairs;
  const int64_t at = (int64_t)blockIdx.x * kThreads + threadIdx.x, token = at / pairs;
  if (token >= s.n) return;
  const Pair p = pair_of(s, (int)(at - token * pairs));
  const int q_cols = s.hq * s.d, k_cols = s.hk * s.d;
  float x1[8], x2[8];
  load8(qkv, token * pitch + p.first, SOUP_F16, x1);
  load8(qkv, token * pitch + p.first + p.apart, SOUP_F16, x2);
  // the pair's place in its own output, and the adapter term that has the same layout
  const bool in_q = p.first < q_cols;
  __half* out = in_q ? q : p.rotated ? k : v;
  const int64_t to = in_q ? token * q_cols + p.first
                          : token * k_cols + p.first - (p.rotated ? q_cols : q_cols + k_cols);
  const __half* add = in_q ? add_q : p.rotated ? nullptr : add_v;
  Tables t;
  if (p.rotated) t.load(cos, sin, token * s.d + p.angle, s.d >> 1);
  if (add) {
    float y1[8], y2[8];
    load8(add, to, SOUP_F16, y1);
    load8(add, to + p.apart, SOUP_F16, y2);
#pragma unroll
    for (int e = 0; e < 8; ++e) { x1[e] += y1[e]; x2[e] += y2[e]; }
  }
  if (p.rotated) {
#pragma unroll
    for (int e = 0; e < 8; ++e) {   // x*cos + [-x2, x1]*sin
      const float a = x1[e], b = x2[e];
      x1[e] = a * t.c1[e] - b * t.s1[e];
      x2[e] = b * t.c2[e] + a * t.s2[e];
    }
  }
  store8(out, to, SOUP_F16, x1);
  store8(out, to + p.apart, SOUP_F16, x2);
}

__global__ void __launch_bounds__(kThreads)
qkv_rope_bwd_kernel(const float* __restrict__ dq, const float* __restrict__ dk, const float* __restrict__ dv,
                    const float* __restrict__ cos, const float* __restrict__ sin, __half* __restrict__ dqkv,
                    int64_t pitch, const QkvShape s) {
  const int pairs = s.rot_pairs + s.v_pairs;
  const int64_t at = (int64_t)blockIdx.x * kThreads + threadIdx.x, token = at / pairs;
  if (token >= s.n) return;
  const Pair p = pair_of(s, (int)(at - token * pairs));
  const int q_cols = s.hq * s.d, k_cols = s.hk * s.d;
  const bool in_q = p.first < q_cols;
  const float* src = in_q ? dq : p.rotated ? dk : dv;
  const int64_t from = in_q ? token * q_cols + p.first
                            : token * k_cols + p.first - (p.rotated ? q_cols : q_cols + k_cols);
  float x1[8], x2[8];
  load8(src, from, SOUP_F32, x1);
  load8(src, from + p.apart, SOUP_F32, x2);
  if (p.rotated) {
    Tables t;
    t.load(cos, sin, token * s.d + p.angle, s.d >> 1);
#pragma unroll
    for (int e = 0; e < 8; ++e) {   // g*cos + rotate_half^T(g*sin)
      const float a = x1[e], b = x2[e];
      x1[e] = a * t.c1[e] + b * t.s2[e];
      x2[e] = b * t.c2[e] - a * t.s1[e];
    }
  }
  store8(dqkv, token * pitch + p.first, SOUP_F16, x1);
  store8(dqkv, token * pitch + p.first + p.apart, SOUP_F16, x2);
}

inline int qkv_shape(QkvShape& s, int64_t n, int64_t hq, int64_t hk, int64_t d, int64_t pitch) {
  if (n < 0 || hq <= 0 || hk <= 0 || d <= 0 || d % 16 || d > 256 || hq > 4096 || hk > 4096)
    SOUP_FAIL(SOUP_ERR_ARG, "qkv_rope: head_dim must be a multiple of 16 up to 256, with up to 4096 heads");
  if (pitch < (hq + 2 * hk) * d || pitch % 8)
    SOUP_FAIL(SOUP_ERR_ARG, "qkv_rope: the row pitch must cover q, k and v and be a multiple of 8 elements");
  s.n = n;
  s.hq = (int)hq;
  s.hk = (int)hk;
  s.d = (int)d;
  s.rot_pairs = (int)((hq + hk) * d / 16);
  s.v_pairs = (int)(hk * d / 16);
  if (n > (int64_t)INT32_MAX * kThreads / (s.rot_pairs + s.v_pairs))
    SOUP_FAIL(SOUP_ERR_ARG, "qkv_rope: too many tokens");
  return SOUP_OK;
}

inline unsigned qkv_grid(const QkvShape& s) {
  return (unsigned)((s.n * (s.rot_pairs + s.v_pairs) + kThreads - 1) / kThreads);
}

}  // namespace
}  // namespace soup

extern "C" int soup_qkv_rope_fwd(const void* qkv, int64_t qkv_pitch, const void* add_q, const void* add_v,
                                 const float* cos, const float* sin, void* q, void* k, void* v, int64_t n,
                                 int64_t hq, int64_t hk, int64_t d, void* stream) {
  using namespace soup;
  QkvShape s;
  const int rc = qkv_shape(s, n, hq, hk, d, qkv_pitch);
  if (rc != SOUP_OK || n == 0) return rc;
  if (!qkv || !cos || !sin || !q || !k || !v) SOUP_FAIL(SOUP_ERR_ARG, "qkv_rope_fwd: null pointer");
  if (!aligned16(qkv) || !aligned16(add_q) || !aligned16(add_v) || !aligned16(cos) || !aligned16(sin) ||
      !aligned16(q) || !aligned16(k) || !aligned16(v))
    SOUP_FAIL(SOUP_ERR_ARG, "qkv_rope_fwd: pointers must be 16-byte aligned");
  qkv_rope_fwd_kernel<<<qkv_grid(s), kThreads, 0, reinterpret_cast<cudaStream_t>(stream)>>>(
      reinterpret_cast<const __half*>(qkv), qkv_pitch, reinterpret_cast<const __half*>(add_q),
      reinterpret_cast<const __half*>(add_v), cos, sin, reinterpret_cast<__half*>(q), reinterpret_cast<__half*>(k),
      reinterpret_cast<__half*>(v), s);
  SOUP_CHECK_LAUNCH("qkv_rope_fwd");
  return SOUP_OK;
}

extern "C" int soup_qkv_rope_bwd(const float* dq, const float* dk, const float* dv, const float* cos,
                                 const float* sin, void* dqkv, int64_t dqkv_pitch, int64_t n, int64_t hq,
                                 int64_t hk, int64_t d, void* stream) {
  using namespace soup;
  QkvShape s;
  const int rc = qkv_shape(s, n, hq, hk, d, dqkv_pitch);
  if (rc != SOUP_OK || n == 0) return rc;
  if (!dq || !dk || !dv || !cos || !sin || !dqkv) SOUP_FAIL(SOUP_ERR_ARG, "qkv_rope_bwd: null pointer");
  if (!aligned16(dq) || !aligned16(dk) || !aligned16(dv) || !aligned16(cos) || !aligned16(sin) || !aligned16(dqkv))
    SOUP_FAIL(SOUP_ERR_ARG, "qkv_rope_bwd: pointers must be 16-byte aligned");
  qkv_rope_bwd_kernel<<<qkv_grid(s), kThreads, 0, reinterpret_cast<cudaStream_t>(stream)>>>(
      dq, dk, dv, cos, sin, reinterpret_cast<__half*>(dqkv), dqkv_pitch, s);
  SOUP_CHECK_LAUNCH("qkv_rope_bwd");
  return SOUP_OK;
}
