// Pieces shared by the mHC forward and backward kernels.
#pragma once

#include "common.cuh"

namespace hmc {
namespace mhc {

constexpr int STREAMS = 4;
constexpr int MIX = 24;         // 4 pre + 4 post + 16 residual-mix logits
constexpr int BLOCK_COLS = 128;  // columns of the hidden dimension one CTA of the streaming kernels owns

__device__ __forceinline__ void unpack8(const uint4& q, float (&f)[8]) {
  const float2 a = unpack_bf16x2(q.x), b = unpack_bf16x2(q.y), c = unpack_bf16x2(q.z), d = unpack_bf16x2(q.w);
  f[0] = a.x; f[1] = a.y; f[2] = b.x; f[3] = b.y; f[4] = c.x; f[5] = c.y; f[6] = d.x; f[7] = d.y;
}
__device__ __forceinline__ uint4 pack8(const float (&f)[8]) {
  return make_uint4(pack_bf16x2(f[0], f[1]), pack_bf16x2(f[2], f[3]), pack_bf16x2(f[4], f[5]),
                    pack_bf16x2(f[6], f[7]));
}
__device__ __forceinline__ float sigmoid_f(float x) { return 1.0f / (1.0f + expf(-x)); }

// Four consecutive floats; `vec` says that the array is 16-byte aligned (decided once on the host).
__device__ __forceinline__ float4 load4(const float* __restrict__ p, bool vec) {
  if (vec) return __ldg(reinterpret_cast<const float4*>(p));
  return make_float4(__ldg(p), __ldg(p + 1), __ldg(p + 2), __ldg(p + 3));
}

// v = hi + lo with two BF16 parts, 16 mantissa bits
__device__ __forceinline__ void split_pair(float x, float y, uint32_t& hi, uint32_t& lo) {
  hi = pack_bf16x2(x, y);
  const float2 h = unpack_bf16x2(hi);
  lo = pack_bf16x2(x - h.x, y - h.y);
}

// Coefficients of a warp's 16 tokens in its own shared memory, every value twice (both halves of a pair): per token and
// stream i the column mix[0..3][i], post[i], pre[i]. 52 words apart, the eight rows of a read miss no bank.
constexpr int COEF_PITCH = 52;
constexpr int COEF_FLOATS = 16 * COEF_PITCH;

struct CoefLoad {
  float4 v[3];
};
__device__ __forceinline__ CoefLoad fetch_coefficients(const float* __restrict__ mix, const float* __restrict__ post,
                                                       const float* __restrict__ pre, long long first, long long tokens,
                                                       bool vec, int lane) {
  CoefLoad l;
#pragma unroll
  for (int r = 0; r < 3; ++r) {  // 16 tokens x 6 groups of four
    const int item = lane + 32 * r, part = item % 6;
    const long long t = first + item / 6;
    l.v[r] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (t < tokens) l.v[r] = load4(part < 4 ? mix + t * 16 + 4 * part : (part == 4 ? post : pre) + t * 4, vec);
  }
  return l;
}
__device__ __forceinline__ void store_coefficients(float* coef, const CoefLoad& l, int lane) {
  __syncwarp();  // the coefficients before these are no longer read
#pragma unroll
  for (int r = 0; r < 3; ++r) {
    const int item = lane + 32 * r;
    float2* dst = reinterpret_cast<float2*>(coef + item / 6 * COEF_PITCH) + item % 6;
    dst[0] = make_float2(l.v[r].x, l.v[r].x);
    dst[6] = make_float2(l.v[r].y, l.v[r].y);
    dst[12] = make_float2(l.v[r].z, l.v[r].z);
    dst[18] = make_float2(l.v[r].w, l.v[r].w);
  }
  __syncwarp();
}

struct StreamCoef {
  float2 mix[STREAMS], post, pre;
};
__device__ __forceinline__ StreamCoef stream_coef(const float* coef, int token, int stream) {
  const float4* src = reinterpret_cast<const float4*>(coef + token * COEF_PITCH + 12 * stream);
  const float4 a = src[0], b = src[1], c = src[2];
  StreamCoef s;
  s.mix[0] = make_float2(a.x, a.y);
  s.mix[1] = make_float2(a.z, a.w);
  s.mix[2] = make_float2(b.x, b.y);
  s.mix[3] = make_float2(b.z, b.w);
  s.post = make_float2(c.x, c.y);
  s.pre = make_float2(c.z, c.w);
  return s;
}

// Two columns of stream i of the new residual, as stored.
__device__ __forceinline__ uint32_t new_residual_pair(const StreamCoef& c, const float2 (&r)[STREAMS], float2 o) {
  float2 v = mul2(c.mix[0], r[0]);
#pragma unroll
  for (int j = 1; j < STREAMS; ++j) v = fma2(c.mix[j], r[j], v);
  v = fma2(c.post, o, v);
  return pack_bf16x2(v.x, v.y);
}

// D[16 x 8] += A[16 x 16] B[16 x 8], BF16 operands, FP32 accumulation. Lane (g, c) = (lane / 4, lane % 4) holds
// A(g, 2c..), A(g + 8, 2c..), A(g, 2c + 8..), A(g + 8, 2c + 8..); B(2c.., g), B(2c + 8.., g); D(g, 2c..), D(g + 8, 2c..).
__device__ __forceinline__ void mma_16x8x16(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                            uint32_t b1) {
  asm(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// A 4 x 4 matrix in 16 lanes (entry (r, c) in lane 4r + c of each half warp): sums along a row / a column.
__device__ __forceinline__ float row_sum4(float v) {
  v += __shfl_xor_sync(0xffffffffu, v, 1);
  return v + __shfl_xor_sync(0xffffffffu, v, 2);
}
__device__ __forceinline__ float col_sum4(float v) {
  v += __shfl_xor_sync(0xffffffffu, v, 4);
  return v + __shfl_xor_sync(0xffffffffu, v, 8);
}
__device__ __forceinline__ float row_max4(float v) {
  v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, 1));
  return fmaxf(v, __shfl_xor_sync(0xffffffffu, v, 2));
}

constexpr int SINKHORN_MAX_STEPS = 40;  // 2 x 20 iterations

// Sinkhorn forward, one matrix entry per lane. Step 0 = softmax rows (+ eps), odd steps = column normalisation, even
// ones = row normalisation; `emit(step, normaliser, entry)` is called after each. The loop stays rolled: unrolled, its
// 40 steps no longer fit the instruction cache next to what surrounds them.
template <typename Emit>
__device__ __forceinline__ float sinkhorn16(float logit, float eps, int steps, Emit&& emit) {
  const float e = expf(logit - row_max4(logit));
  float s = row_sum4(e);
  float m = e * __frcp_rn(s) + eps;
  emit(0, s, m);
#pragma unroll 1
  for (int step = 1; step < steps; step += 2) {  // the number of steps is even
    s = col_sum4(m) + eps;
    m *= __frcp_rn(s);
    emit(step, s, m);
    if (step + 1 < steps) {
      s = row_sum4(m) + eps;
      m *= __frcp_rn(s);
      emit(step + 1, s, m);
    }
  }
  return m;
}

}  // namespace mhc
}  // namespace hmc
