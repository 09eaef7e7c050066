// MegaGate: FP32 router projection, top-k Route and RouteGrad as single-pass warp kernels.
//
// Route follows MegaGate._torch_forward (hyper_multicore/modules/mega_gate/module.py:189-227) and
// the native 10-stage Route pipeline (hyper_multicore/ops/hyper_mega_gate/op_kernel/
// route_pipeline.h:73-562) but keeps a token's whole expert row in the registers of one warp, so
// nothing round-trips through global memory between stages. RouteGrad follows the autograd of
// the same expression (hyper_multicore/ops/hyper_mega_gate_grad/op_kernel/route_grad_pipeline.h:
// 138-191 plus the library tail hyper_mega_gate_route_grad_post.cpp:59-140).
#include <math.h>

#include "common.cuh"
#include "sm100.cuh"

namespace hmc {
namespace {

constexpr int WARPS_PER_BLOCK = 8;
constexpr float NEG_INF = -INFINITY;

__device__ __forceinline__ float softplus_ref(float x) {
  // torch softplus(beta=1, threshold=20): x > 20 ? x : log1p(exp(x))
  return x > 20.0f ? x : log1pf(expf(x));
}

// argmax over the warp; ties go to the lower expert index
__device__ __forceinline__ void warp_argmax(float& v, int& idx) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const float ov = __shfl_xor_sync(0xffffffffu, v, o);
    const int oi = __shfl_xor_sync(0xffffffffu, idx, o);
    if (ov > v || (ov == v && oi < idx)) {
      v = ov;
      idx = oi;
    }
  }
}

template <int NPL>
__global__ void __launch_bounds__(WARPS_PER_BLOCK * 32)
gate_route_kernel(const float* __restrict__ logits, const float* __restrict__ text_bias,
                  const float* __restrict__ vision_bias, const uint8_t* __restrict__ image_mask,
                  int use_vision_bias, long long tokens, int experts, int top_k, float scale,
                  int scoring, float* __restrict__ weights, long long* __restrict__ indices,
                  float* __restrict__ route_scores, float* __restrict__ selected,
                  float* __restrict__ denominator, int n_group, int topk_group) {
  extern __shared__ float group_stage[];  // [WARPS_PER_BLOCK][experts + n_group], only with n_group > 0
  const int lane = threadIdx.x & 31;
  const long long token = static_cast<long long>(blockIdx.x) * WARPS_PER_BLOCK + (threadIdx.x >> 5);
  if (token >= tokens) return;

  const float* row = logits + token * experts;
  float score[NPL];
  float biased[NPL];
#pragma unroll
  for (int i = 0; i < NPL; ++i) {
    const int e = lane + 32 * i;
    score[i] = e < experts ? row[e] : NEG_INF;
  }
  if (scoring == HMC_SCORE_SOFTMAX) {
    float m = NEG_INF;
#pragma unroll
    for (int i = 0; i < NPL; ++i) m = fmaxf(m, score[i]);
    m = warp_max(m);
    float sum = 0.f;
#pragma unroll
    for (int i = 0; i < NPL; ++i) {
      const int e = lane + 32 * i;
      score[i] = e < experts ? expf(score[i] - m) : 0.f;
      sum += score[i];
    }
    sum = warp_sum(sum);
    const float inv = 1.0f / sum;
#pragma unroll
    for (int i = 0; i < NPL; ++i) score[i] *= inv;
  } else if (scoring == HMC_SCORE_SIGMOID) {
#pragma unroll
    for (int i = 0; i < NPL; ++i) score[i] = 1.0f / (1.0f + expf(-score[i]));
  } else {
#pragma unroll
    for (int i = 0; i < NPL; ++i) score[i] = sqrtf(softplus_ref(score[i]));
  }

  const float* bias = (use_vision_bias && image_mask[token]) ? vision_bias : text_bias;
  float* score_out = route_scores + token * experts;
#pragma unroll
  for (int i = 0; i < NPL; ++i) {
    const int e = lane + 32 * i;
    if (e < experts) {
      score_out[e] = score[i];
      biased[i] = __fadd_rn(score[i], bias[e]);  // never contracted with the softmax scaling: the sum torch rounds
    } else {
      biased[i] = NEG_INF;
    }
  }

  if (n_group > 0) {
    // Group limit: lane g scores group g (sum of its two largest biased scores), the warp picks the
    // topk_group best groups, experts of the other groups leave the selection.
    const int group_size = experts / n_group;
    float* mine = group_stage + (threadIdx.x >> 5) * (experts + n_group);  // a word between the groups: no bank twice
#pragma unroll
    for (int i = 0; i < NPL; ++i) {
      const int e = lane + 32 * i;
      if (e < experts) mine[e + e / group_size] = biased[i];
    }
    __syncwarp();
    float group_score = NEG_INF;
    if (lane < n_group) {
      float first = NEG_INF, second = NEG_INF;
      for (int j = 0; j < group_size; ++j) {
        const float v = mine[lane * (group_size + 1) + j];
        if (v > first) {
          second = first;
          first = v;
        } else if (v > second) {
          second = v;
        }
      }
      group_score = group_size > 1 ? first + second : first;
    }
    uint32_t chosen = 0;
    for (int k = 0; k < topk_group; ++k) {
      float best = (lane < n_group && !((chosen >> lane) & 1u)) ? group_score : NEG_INF;
      int best_idx = (lane < n_group && !((chosen >> lane) & 1u)) ? lane : 0x7fffffff;
      warp_argmax(best, best_idx);
      if (best_idx < 32) chosen |= 1u << best_idx;
    }
#pragma unroll
    for (int i = 0; i < NPL; ++i) {
      const int e = lane + 32 * i;
      if (e < experts && !((chosen >> (e / group_size)) & 1u)) biased[i] = NEG_INF;
    }
  }

  // top-k by repeated warp argmax over the entries not taken yet. NaN orders as +inf (torch.topk treats NaN as the
  // largest value); ties go to the lower expert index. The keys are the biased scores as integers in float order (-0 as
  // +0), so that two integer reductions of the warp find the winner where a float butterfly takes ten shuffles, and one
  // value below every float marks the taken ones. 8192 tokens x 256 experts, top-8 of 4 of 8 groups: 30.5 -> 24.5 us, outputs the same bit for bit.
  constexpr int GONE = static_cast<int>(0x80000000u);
  int key[NPL];
#pragma unroll
  for (int i = 0; i < NPL; ++i) {
    const float b = isnan(biased[i]) ? INFINITY : __fadd_rn(biased[i], 0.f);
    const int bits = __float_as_int(b);
    key[i] = lane + 32 * i < experts ? (bits ^ ((bits >> 31) & 0x7fffffff)) : GONE;
  }
  float* sel_out = selected + token * top_k;
  long long* idx_out = indices + token * top_k;
  float sum = 0.f;
  for (int k = 0; k < top_k; ++k) {
    int best = GONE;
    int best_idx = 0x7fffffff;
#pragma unroll
    for (int i = 0; i < NPL; ++i) {
      if (key[i] > best) {
        best = key[i];
        best_idx = lane + 32 * i;
      }
    }
    const int top = __reduce_max_sync(0xffffffffu, best);
    best_idx = __reduce_min_sync(0xffffffffu, best == top ? best_idx : 0x7fffffff);
    float win_score = 0.f;
#pragma unroll
    for (int i = 0; i < NPL; ++i) {
      if (lane + 32 * i == best_idx) {
        win_score = score[i];
        key[i] = GONE;
      }
    }
    win_score = __shfl_sync(0xffffffffu, win_score, best_idx & 31);
    sum += win_score;  // every lane accumulates the same sequence, in selection order
    if (lane == 0) {
      sel_out[k] = win_score;
      idx_out[k] = best_idx;
    }
  }
  const float denom = sum + 1.0e-20f;
  if (lane == 0) denominator[token] = denom;
  __syncwarp();
  for (int k = lane; k < top_k; k += 32) {
    float w = sel_out[k];
    if (top_k > 1) w = w / denom;
    weights[token * top_k + k] = w * scale;
  }
}

template <int NPL>
__global__ void __launch_bounds__(WARPS_PER_BLOCK * 32)
gate_route_grad_kernel(const float* __restrict__ logits, const float* __restrict__ route_scores,
                       const float* __restrict__ selected, const float* __restrict__ denominator,
                       const long long* __restrict__ indices, const float* __restrict__ grad_weights,
                       long long tokens, int experts, int top_k, float scale, int scoring,
                       float* __restrict__ grad_logits, int* __restrict__ status) {
  const int lane = threadIdx.x & 31;
  const long long token = static_cast<long long>(blockIdx.x) * WARPS_PER_BLOCK + (threadIdx.x >> 5);
  if (token >= tokens) return;

  const float denom = denominator[token];
  const float* sel = selected + token * top_k;
  const float* gw = grad_weights + token * top_k;
  const long long* idx = indices + token * top_k;

  // Gradient of the shared denominator: sum_k -(g_k * scale) * ((sel_k / D) / D), the order in
  // which torch's div backward evaluates it.
  float grad_denom = 0.f;
  if (top_k > 1) {
    for (int k = 0; k < top_k; ++k) grad_denom += -(gw[k] * scale) * ((sel[k] / denom) / denom);
  }
  float grad_score[NPL];
#pragma unroll
  for (int i = 0; i < NPL; ++i) grad_score[i] = 0.f;
  for (int k = 0; k < top_k; ++k) {
    const long long e = idx[k];
    if (e < 0 || e >= experts) {
      if (lane == 0) report_status(status, HMC_STATUS_BAD_INDEX, static_cast<int>(token), k, static_cast<int>(e));
      continue;
    }
    const float g1 = gw[k] * scale;
    const float g = top_k > 1 ? g1 / denom + grad_denom : g1;
#pragma unroll
    for (int i = 0; i < NPL; ++i)
      if (lane + 32 * i == e) grad_score[i] += g;
  }

  const float* x_row = logits + token * experts;
  const float* s_row = route_scores + token * experts;
  float* out = grad_logits + token * experts;
  if (scoring == HMC_SCORE_SOFTMAX) {
    float dot = 0.f;
    float s[NPL];
#pragma unroll
    for (int i = 0; i < NPL; ++i) {
      const int e = lane + 32 * i;
      s[i] = e < experts ? s_row[e] : 0.f;
      dot += grad_score[i] * s[i];
    }
    dot = warp_sum(dot);
#pragma unroll
    for (int i = 0; i < NPL; ++i) {
      const int e = lane + 32 * i;
      if (e < experts) out[e] = (grad_score[i] - dot) * s[i];
    }
  } else if (scoring == HMC_SCORE_SIGMOID) {
#pragma unroll
    for (int i = 0; i < NPL; ++i) {
      const int e = lane + 32 * i;
      if (e < experts) {
        const float s = s_row[e];
        out[e] = grad_score[i] * (1.0f - s) * s;
      }
    }
  } else {
#pragma unroll
    for (int i = 0; i < NPL; ++i) {
      const int e = lane + 32 * i;
      if (e < experts) {
        // sqrt backward: g / (2 * sqrt(sp)); softplus backward: x > 20 ? g : g * z / (z + 1)
        const float g_sp = grad_score[i] / (2.0f * s_row[e]);
        const float x = x_row[e];
        const float z = expf(x);
        out[e] = x > 20.0f ? g_sp : g_sp * z / (z + 1.0f);
      }
    }
  }
}

// ---------------------------------------------------------------------------------------------
// FP32 projection logits[T, E] = float(x[T, H]) . float(W[E, H])^T on CUDA cores with FP32 FMA.
// 64 x 64 output tile per CTA, 4 x 4 per thread, K staged through shared memory in 32-wide slabs. The slabs come in the
// order that the kernels of few tokens below add them in - SLICED: slices of `slice` elements, in a slice `ways` chains
// that take every ways-th slab; otherwise one chain - so that a token's logits are the same bits however many tokens share
// the call and decide between the kernels. The strided order loses the neighbouring half of what a slab fetches, so the
// next slab is in flight while one is multiplied: 8192 tokens x hidden 4096 x 64 experts 310 us in one chain, 423 in this
// order, 248 with the prefetch; 8192 x 7168 x 256 1749, 1715, 1639; BF16 hidden states 8192 x 4096 x 64 277, 408, 253.
// ---------------------------------------------------------------------------------------------
template <typename T>
__device__ __forceinline__ float to_f32(T v);
template <>
__device__ __forceinline__ float to_f32<float>(float v) { return v; }
template <>
__device__ __forceinline__ float to_f32<__nv_bfloat16>(__nv_bfloat16 v) { return __bfloat162float(v); }

template <typename TX, typename TW, bool SLICED>
__global__ void __launch_bounds__(256, SLICED ? 1 : 3)
gate_project_kernel(const TX* __restrict__ x, const TW* __restrict__ w, long long tokens, int hidden,
                    int experts, int slice, int ways, float* __restrict__ logits) {
  constexpr int TM = 64, TN = 64, TK = 32;
  __shared__ float xs[TK][TM + 4];
  __shared__ float ws[TK][TN + 4];
  const long long t0 = static_cast<long long>(blockIdx.x) * TM;
  const int e0 = blockIdx.y * TN;
  const int tx = threadIdx.x & 15;  // expert direction
  const int ty = threadIdx.x >> 4;  // token direction
  TX px[8];
  TW pw[8];
  auto fetch = [&](int k0, int end) {  // 64 rows x 32 k per operand: 256 threads load 8 elements each
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int flat = threadIdx.x + 256 * i;
      const long long t = t0 + (flat >> 5);
      const int e = e0 + (flat >> 5);
      const int k = k0 + (flat & 31);
      px[i] = (t < tokens && k < end) ? x[t * hidden + k] : TX(0.f);
      pw[i] = (e < experts && k < end) ? w[static_cast<long long>(e) * hidden + k] : TW(0.f);
    }
  };
  float acc[4][4] = {}, partial[4][4] = {}, total[4][4] = {};  // of a chain, of a slice, of the row
  int end = SLICED && slice < hidden ? slice : hidden;
  int begin = 0, first = 0, k0 = 0;  // of the slice, of its chain, of the slab
  bool more = true;
  if constexpr (SLICED) fetch(k0, end);
  while (more) {
    if constexpr (!SLICED) fetch(k0, end);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int flat = threadIdx.x + 256 * i;
      xs[flat & 31][flat >> 5] = to_f32<TX>(px[i]);
      ws[flat & 31][flat >> 5] = to_f32<TW>(pw[i]);
    }
    __syncthreads();
    bool chain_done = false, slice_done = false;
    if constexpr (SLICED) {
      k0 += ways * TK;
      chain_done = k0 >= end;
      if (chain_done) {
        first += TK;
        k0 = first;
        slice_done = k0 >= end || first - begin == ways * TK;  // chains that would begin past the end are empty
        if (slice_done) {
          more = end < hidden;
          first = k0 = begin = end;
          end = slice < hidden - begin ? begin + slice : hidden;
        }
      }
      if (more) fetch(k0, end);
    } else {
      k0 += TK;
      more = k0 < hidden;
    }
#pragma unroll
    for (int kk = 0; kk < TK; ++kk) {
      float a[4], b[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) a[i] = xs[kk][ty * 4 + i];
#pragma unroll
      for (int j = 0; j < 4; ++j) b[j] = ws[kk][tx * 4 + j];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
    }
    __syncthreads();
    if (!chain_done) continue;
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        partial[i][j] += acc[i][j];
        acc[i][j] = 0.f;
        if (!slice_done) continue;
        total[i][j] += partial[i][j];
        partial[i][j] = 0.f;
      }
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const long long t = t0 + ty * 4 + i;
    if (t >= tokens) continue;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int e = e0 + tx * 4 + j;
      if (e < experts) logits[t * experts + e] = SLICED ? total[i][j] : acc[i][j];
    }
  }
}

// ---------------------------------------------------------------------------------------------
// The same projection where the 64 x 64 tiling above has too few tiles to fill the chip (decode batches): bound by
// the latency of reading the weight, so the work is cut into 16-token x 16-expert tiles and K into eight slices, one
// per CTA of a cluster, and every warp of a CTA takes its own 32 elements of a 256-element slab. The slabs of the
// next step are in flight while this one is multiplied. A lane owns 4 tokens x 2 experts: per four elements of K six
// 16-byte shared-memory reads without bank conflicts (rows are 260 words apart) feed 32 FMAs. Partial sums meet in
// a fixed order - warps, then slices through distributed shared memory - so results repeat bit for bit.
// ---------------------------------------------------------------------------------------------
constexpr int ROWS_TOKENS = 16;
constexpr int ROWS_EXPERTS = 16;
constexpr int ROWS_SLAB = 256;
constexpr int ROWS_SLICES = 8;
constexpr int ROWS_PITCH = ROWS_SLAB + 4;

// four consecutive elements of row `row` at column k, zeros outside [rows, hidden)
template <typename T, bool VEC>
__device__ __forceinline__ float4 load_four(const T* __restrict__ base, long long row, long long rows, int k, int k_end,
                                            int hidden) {
  float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
  if (row >= rows || k >= k_end) return v;
  const T* src = base + row * hidden + k;
  if constexpr (VEC) {  // hidden and the slice ends are multiples of 4 and the rows aligned: never past the end
    if constexpr (sizeof(T) == 4) {
      v = __ldg(reinterpret_cast<const float4*>(src));
    } else {
      const uint2 q = __ldg(reinterpret_cast<const uint2*>(src));
      const float2 a = unpack_bf16x2(q.x), b = unpack_bf16x2(q.y);
      v = make_float4(a.x, a.y, b.x, b.y);
    }
  } else {
    v.x = to_f32<T>(src[0]);
    if (k + 1 < k_end) v.y = to_f32<T>(src[1]);
    if (k + 2 < k_end) v.z = to_f32<T>(src[2]);
    if (k + 3 < k_end) v.w = to_f32<T>(src[3]);
  }
  return v;
}

// Short rows: one thread per output of the 16 x 16 tile and one chain over K in order, bit for bit the sums of the
// 64 x 64 kernel. 1024 dependent FMAs are about 2 us, what the slices' exchange would cost as well.
constexpr int SHORT_HIDDEN = 1024;

template <typename TX, typename TW, bool VEC>
__global__ void __launch_bounds__(256)
gate_project_short_kernel(const TX* __restrict__ x, const TW* __restrict__ w, long long tokens, int hidden, int experts,
                          float* __restrict__ logits) {
  __shared__ __align__(16) float xs[ROWS_TOKENS * ROWS_PITCH];
  __shared__ __align__(16) float ws[ROWS_EXPERTS * ROWS_PITCH];
  const int tid = threadIdx.x;
  const long long t0 = static_cast<long long>(blockIdx.z) * ROWS_TOKENS;
  const int e0 = static_cast<int>(blockIdx.y) * ROWS_EXPERTS;
  const int tok = tid / ROWS_EXPERTS, e = tid % ROWS_EXPERTS;
  float acc = 0.f;
  for (int k0 = 0; k0 < hidden; k0 += ROWS_SLAB) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int flat = tid + 256 * i;
      const int r = flat >> 6, c = 4 * (flat & 63);
      *reinterpret_cast<float4*>(xs + r * ROWS_PITCH + c) = load_four<TX, VEC>(x, t0 + r, tokens, k0 + c, hidden, hidden);
      *reinterpret_cast<float4*>(ws + r * ROWS_PITCH + c) = load_four<TW, VEC>(w, e0 + r, experts, k0 + c, hidden, hidden);
    }
    __syncthreads();
    const int left = hidden - k0 < ROWS_SLAB ? hidden - k0 : ROWS_SLAB;
#pragma unroll 4
    for (int kk = 0; kk < left; kk += 4) {  // zeros past the end of a row leave the sum as it is
      const float4 a = *reinterpret_cast<const float4*>(xs + tok * ROWS_PITCH + kk);
      const float4 b = *reinterpret_cast<const float4*>(ws + e * ROWS_PITCH + kk);
      acc = fmaf(a.x, b.x, acc);
      acc = fmaf(a.y, b.y, acc);
      acc = fmaf(a.z, b.z, acc);
      acc = fmaf(a.w, b.w, acc);
    }
    __syncthreads();
  }
  if (t0 + tok < tokens && e0 + e < experts) logits[(t0 + tok) * experts + e0 + e] = acc;
}

template <typename TX, typename TW, bool VEC>
__global__ void __cluster_dims__(ROWS_SLICES, 1, 1) __launch_bounds__(256)
gate_project_rows_kernel(const TX* __restrict__ x, const TW* __restrict__ w, long long tokens, int hidden, int experts,
                         int slice, float* __restrict__ logits) {
  __shared__ __align__(16) float xs[ROWS_TOKENS * ROWS_PITCH];
  __shared__ __align__(16) float ws[ROWS_EXPERTS * ROWS_PITCH];
  __shared__ float sums[ROWS_TOKENS * ROWS_EXPERTS];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const long long t0 = static_cast<long long>(blockIdx.z) * ROWS_TOKENS;
  const int e0 = static_cast<int>(blockIdx.y) * ROWS_EXPERTS;
  const uint32_t rank = sm100::cluster_ctarank();
  const long long first = static_cast<long long>(rank) * slice;
  const int k_begin = static_cast<int>(first < hidden ? first : hidden);
  const int k_end = static_cast<int>(first + slice < hidden ? first + slice : hidden);
  const int tg = lane >> 3, eg = lane & 7;
  float acc[4][2] = {};
  float4 px[4], pw[4];
  auto fetch = [&](int k0) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int flat = tid + 256 * i;  // 16 rows of 64 four-element groups
      const int r = flat >> 6, k = k0 + 4 * (flat & 63);
      px[i] = load_four<TX, VEC>(x, t0 + r, tokens, k, k_end, hidden);
      pw[i] = load_four<TW, VEC>(w, e0 + r, experts, k, k_end, hidden);
    }
  };
  fetch(k_begin);
  for (int k0 = k_begin; k0 < k_end; k0 += ROWS_SLAB) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int flat = tid + 256 * i;
      const int at = (flat >> 6) * ROWS_PITCH + 4 * (flat & 63);
      *reinterpret_cast<float4*>(xs + at) = px[i];
      *reinterpret_cast<float4*>(ws + at) = pw[i];
    }
    __syncthreads();
    if (k0 + ROWS_SLAB < k_end) fetch(k0 + ROWS_SLAB);
#pragma unroll
    for (int kk = 0; kk < 32; kk += 4) {
      const int at = warp * 32 + kk;
      float4 a[4], b[2];
#pragma unroll
      for (int i = 0; i < 4; ++i) a[i] = *reinterpret_cast<const float4*>(xs + (tg + 4 * i) * ROWS_PITCH + at);
#pragma unroll
      for (int j = 0; j < 2; ++j) b[j] = *reinterpret_cast<const float4*>(ws + (eg + 8 * j) * ROWS_PITCH + at);
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          acc[i][j] = fmaf(a[i].x, b[j].x, acc[i][j]);
          acc[i][j] = fmaf(a[i].y, b[j].y, acc[i][j]);
          acc[i][j] = fmaf(a[i].z, b[j].z, acc[i][j]);
          acc[i][j] = fmaf(a[i].w, b[j].w, acc[i][j]);
        }
    }
    __syncthreads();
  }
  float* parts = xs;  // [8 warps][256 outputs]
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 2; ++j)
      parts[warp * 256 + (tg + 4 * i) * ROWS_EXPERTS + eg + 8 * j] = acc[i][j];
  __syncthreads();
  float total = 0.f;
#pragma unroll
  for (int v = 0; v < 8; ++v) total += parts[v * 256 + tid];
  sums[tid] = total;
  sm100::cluster_sync_all();
  if (tid < 256 / ROWS_SLICES) {  // this CTA finishes 32 of the tile's outputs
    const int o = static_cast<int>(rank) * (256 / ROWS_SLICES) + tid;
    const uint32_t local = sm100::smem_u32(sums + o);
    float v = 0.f;
#pragma unroll
    for (uint32_t c = 0; c < ROWS_SLICES; ++c) v += sm100::ld_shared_cluster_f32(sm100::map_to_cta(local, c));
    const long long t = t0 + o / ROWS_EXPERTS;
    const int e = e0 + o % ROWS_EXPERTS;
    if (t < tokens && e < experts) logits[t * experts + e] = v;
  }
  sm100::cluster_sync_all();  // no CTA leaves while its sums are still being read
}

template <typename TX, typename TW>
void launch_project(const void* x, const void* w, long long tokens, int hidden, int experts, float* logits,
                    cudaStream_t stream) {
  const TX* px = static_cast<const TX*>(x);
  const TW* pw = static_cast<const TW*>(w);
  const long long tiles = (tokens + 63) / 64 * ((experts + 63) / 64);
  const int slice = ((hidden + ROWS_SLICES - 1) / ROWS_SLICES + 3) / 4 * 4;
  // While the 64 x 64 tiles would leave half of the SMs idle. FP32 weight of 64 experts x hidden 4096: 16 tokens
  // 200 -> 5 us on the device, 512 tokens (8 tiles) 209 -> 25 us; 1024 tokens x 128 experts (32 tiles) 209 -> 75 us.
  // Beyond, the larger tiles' reuse wins: 2048 tokens x 256 experts (128 tiles) took 211 us with them before they had a
  // slab in flight, 271 us here.
  if (2 * tiles <= sm_count()) {
    const dim3 grid(ROWS_SLICES, static_cast<unsigned>((experts + ROWS_EXPERTS - 1) / ROWS_EXPERTS),
                    static_cast<unsigned>((tokens + ROWS_TOKENS - 1) / ROWS_TOKENS));
    const bool vec = hidden % 4 == 0 && reinterpret_cast<uintptr_t>(px) % (4 * sizeof(TX)) == 0 &&
                     reinterpret_cast<uintptr_t>(pw) % (4 * sizeof(TW)) == 0;
    const dim3 short_grid(1, grid.y, grid.z);
    if (hidden <= SHORT_HIDDEN && vec)
      gate_project_short_kernel<TX, TW, true><<<short_grid, 256, 0, stream>>>(px, pw, tokens, hidden, experts, logits);
    else if (hidden <= SHORT_HIDDEN)
      gate_project_short_kernel<TX, TW, false><<<short_grid, 256, 0, stream>>>(px, pw, tokens, hidden, experts, logits);
    else if (vec)
      gate_project_rows_kernel<TX, TW, true><<<grid, 256, 0, stream>>>(px, pw, tokens, hidden, experts, slice, logits);
    else
      gate_project_rows_kernel<TX, TW, false><<<grid, 256, 0, stream>>>(px, pw, tokens, hidden, experts, slice, logits);
    return;
  }
  const dim3 grid(static_cast<unsigned>((tokens + 63) / 64), static_cast<unsigned>((experts + 63) / 64));
  constexpr int WAYS = ROWS_SLAB / 32;
  if (hidden <= SHORT_HIDDEN)
    gate_project_kernel<TX, TW, false><<<grid, 256, 0, stream>>>(px, pw, tokens, hidden, experts, hidden, 1, logits);
  else
    gate_project_kernel<TX, TW, true><<<grid, 256, 0, stream>>>(px, pw, tokens, hidden, experts, slice, WAYS, logits);
}

// FP32 weight [E, H] -> three BF16 parts (hi, mid, lo; hi + mid + lo == w to 24 bits) stacked as
// rows [0, E), [Epad, Epad + E), [2 Epad, 2 Epad + E) of a [3 Epad, H] matrix; other rows zero.
__global__ void gate_split_weight_kernel(const void* __restrict__ w, int w_is_bf16, int experts, int epad, int parts,
                                         long long hidden, __nv_bfloat16* __restrict__ split) {
  const long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= static_cast<long long>(epad) * hidden) return;
  const int e = static_cast<int>(i / hidden);
  float v = 0.f;
  if (e < experts)
    v = w_is_bf16 ? __bfloat162float(static_cast<const __nv_bfloat16*>(w)[i]) : static_cast<const float*>(w)[i];
  const __nv_bfloat16 hi = __float2bfloat16_rn(v);
  split[i] = hi;
  if (parts == 3) {
    const float r1 = v - __bfloat162float(hi);
    const __nv_bfloat16 mid = __float2bfloat16_rn(r1);
    const __nv_bfloat16 lo = __float2bfloat16_rn(r1 - __bfloat162float(mid));
    split[static_cast<long long>(epad) * hidden + i] = mid;
    split[2ll * epad * hidden + i] = lo;
  }
}

// logits[t, e] = sum of the partial products of the weight parts
__global__ void gate_sum_parts_kernel(const float* __restrict__ partial, long long tokens, int experts, int epad,
                                      int parts, float* __restrict__ logits) {
  const long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= tokens * experts) return;
  const long long t = i / experts;
  const int e = static_cast<int>(i % experts);
  const float* row = partial + t * parts * epad;
  float v = row[e];
  if (parts == 3) v = (v + row[epad + e]) + row[2 * epad + e];
  logits[i] = v;
}

template <int NPL>
void launch_route(const hmc_gate_route_args& a, cudaStream_t stream) {
  const unsigned grid = static_cast<unsigned>((a.tokens + WARPS_PER_BLOCK - 1) / WARPS_PER_BLOCK);
  const size_t smem = a.n_group > 0 ? static_cast<size_t>(WARPS_PER_BLOCK) * (a.experts + a.n_group) * sizeof(float) : 0;
  gate_route_kernel<NPL><<<grid, WARPS_PER_BLOCK * 32, smem, stream>>>(
      a.logits, a.text_bias, a.vision_bias, a.image_mask, a.use_vision_bias, a.tokens, a.experts, a.top_k,
      a.scale, a.scoring, a.weights, reinterpret_cast<long long*>(a.indices), a.route_scores, a.selected,
      a.denominator, a.n_group, a.topk_group);
}

template <int NPL>
void launch_route_grad(const hmc_gate_route_grad_args& a, cudaStream_t stream) {
  const unsigned grid = static_cast<unsigned>((a.tokens + WARPS_PER_BLOCK - 1) / WARPS_PER_BLOCK);
  gate_route_grad_kernel<NPL><<<grid, WARPS_PER_BLOCK * 32, 0, stream>>>(
      a.logits, a.route_scores, a.selected, a.denominator, reinterpret_cast<const long long*>(a.indices),
      a.grad_weights, a.tokens, a.experts, a.top_k, a.scale, a.scoring, a.grad_logits, a.status);
}

#define HMC_DISPATCH_NPL(experts, CALL)                    \
  do {                                                     \
    const int npl__ = ((experts) + 31) / 32;               \
    if (npl__ <= 1) { CALL(1); }                           \
    else if (npl__ <= 2) { CALL(2); }                      \
    else if (npl__ <= 4) { CALL(4); }                      \
    else if (npl__ <= 8) { CALL(8); }                      \
    else if (npl__ <= 16) { CALL(16); }                    \
    else { CALL(32); }                                     \
  } while (0)

}  // namespace
}  // namespace hmc

extern "C" int hmc_gate_route(const hmc_gate_route_args* args, void* stream_ptr) {
  using namespace hmc;
  HMC_REQUIRE(args != nullptr, HMC_ERR_INVALID, "hmc_gate_route: null args");
  const hmc_gate_route_args& a = *args;
  // Same argument contract as the reference binding (hyper_multicore/torch/csrc/mega_gate.cpp:40-61).
  HMC_REQUIRE(a.tokens > 0, HMC_ERR_INVALID, "hmc_gate_route: tokens must be positive, got %lld", (long long)a.tokens);
  HMC_REQUIRE(a.experts > 0 && a.experts <= 1024, HMC_ERR_LIMIT,
              "hmc_gate_route: experts must be in [1, 1024], got %d", a.experts);
  HMC_REQUIRE(a.top_k >= 1 && a.top_k <= a.experts, HMC_ERR_INVALID,
              "hmc_gate_route: top_k must be in [1, experts], got %d", a.top_k);
  HMC_REQUIRE(isfinite(a.scale), HMC_ERR_INVALID, "hmc_gate_route: routed scaling factor must be finite");
  HMC_REQUIRE(a.scoring >= HMC_SCORE_SQRTSOFTPLUS && a.scoring <= HMC_SCORE_SIGMOID, HMC_ERR_INVALID,
              "hmc_gate_route: unknown scoring function %d", a.scoring);
  HMC_REQUIRE(a.logits && a.text_bias && a.weights && a.indices && a.route_scores && a.selected && a.denominator,
              HMC_ERR_INVALID, "hmc_gate_route: null tensor pointer");
  HMC_REQUIRE(!a.use_vision_bias || (a.vision_bias && a.image_mask), HMC_ERR_INVALID,
              "hmc_gate_route: vision routing needs vision_bias and image_mask");
  if (a.n_group != 0) {
    HMC_REQUIRE(a.n_group >= 1 && a.n_group <= 32 && a.experts % a.n_group == 0, HMC_ERR_INVALID,
                "hmc_gate_route: n_group (%d) must be in [1, 32] and divide experts (%d)", a.n_group, a.experts);
    HMC_REQUIRE(a.topk_group >= 1 && a.topk_group <= a.n_group, HMC_ERR_INVALID,
                "hmc_gate_route: topk_group (%d) must be in [1, n_group]", a.topk_group);
    HMC_REQUIRE(a.top_k <= a.topk_group * (a.experts / a.n_group), HMC_ERR_INVALID,
                "hmc_gate_route: top_k (%d) exceeds the experts of %d groups", a.top_k, a.topk_group);
  }
  cudaStream_t stream = static_cast<cudaStream_t>(stream_ptr);
#define CALL(N) launch_route<N>(a, stream)
  HMC_DISPATCH_NPL(a.experts, CALL);
#undef CALL
  HMC_LAUNCH_OK();
  return 0;
}

extern "C" int hmc_gate_route_grad(const hmc_gate_route_grad_args* args, void* stream_ptr) {
  using namespace hmc;
  HMC_REQUIRE(args != nullptr, HMC_ERR_INVALID, "hmc_gate_route_grad: null args");
  const hmc_gate_route_grad_args& a = *args;
  // Contract of hyper_multicore/torch/csrc/mega_gate.cpp:132-176.
  HMC_REQUIRE(a.tokens > 0, HMC_ERR_INVALID, "hmc_gate_route_grad: tokens must be positive");
  HMC_REQUIRE(a.experts > 0 && a.experts <= 1024, HMC_ERR_LIMIT,
              "hmc_gate_route_grad: experts must be in [1, 1024], got %d", a.experts);
  HMC_REQUIRE(a.top_k >= 1 && a.top_k <= a.experts, HMC_ERR_INVALID,
              "hmc_gate_route_grad: top_k must be in [1, experts], got %d", a.top_k);
  HMC_REQUIRE(isfinite(a.scale), HMC_ERR_INVALID, "hmc_gate_route_grad: routed scaling factor must be finite");
  HMC_REQUIRE(a.scoring >= HMC_SCORE_SQRTSOFTPLUS && a.scoring <= HMC_SCORE_SIGMOID, HMC_ERR_INVALID,
              "hmc_gate_route_grad: unknown scoring function %d", a.scoring);
  HMC_REQUIRE(a.logits && a.route_scores && a.selected && a.denominator && a.indices && a.grad_weights &&
                  a.grad_logits,
              HMC_ERR_INVALID, "hmc_gate_route_grad: null tensor pointer");
  cudaStream_t stream = static_cast<cudaStream_t>(stream_ptr);
#define CALL(N) launch_route_grad<N>(a, stream)
  HMC_DISPATCH_NPL(a.experts, CALL);
#undef CALL
  HMC_LAUNCH_OK();
  return 0;
}

extern "C" int hmc_gate_project(const void* x, int x_is_bf16, const void* w, int w_is_bf16, int64_t tokens,
                                int64_t hidden, int64_t experts, float* logits, void* stream_ptr) {
  using namespace hmc;
  HMC_REQUIRE(x && w && logits, HMC_ERR_INVALID, "hmc_gate_project: null tensor pointer");
  HMC_REQUIRE(tokens > 0 && hidden > 0 && experts > 0, HMC_ERR_INVALID,
              "hmc_gate_project: extents must be positive");
  HMC_REQUIRE(hidden < (1ll << 31) && experts < 65536 * 64, HMC_ERR_LIMIT, "hmc_gate_project: extent too large");
  cudaStream_t stream = static_cast<cudaStream_t>(stream_ptr);
  const int h = static_cast<int>(hidden), e = static_cast<int>(experts);
  if (x_is_bf16 && w_is_bf16)
    launch_project<__nv_bfloat16, __nv_bfloat16>(x, w, tokens, h, e, logits, stream);
  else if (x_is_bf16)
    launch_project<__nv_bfloat16, float>(x, w, tokens, h, e, logits, stream);
  else if (w_is_bf16)
    launch_project<float, __nv_bfloat16>(x, w, tokens, h, e, logits, stream);
  else
    launch_project<float, float>(x, w, tokens, h, e, logits, stream);
  HMC_LAUNCH_OK();
  return 0;
}

extern "C" int64_t hmc_gate_project_workspace_bytes(int64_t tokens, int64_t hidden, int64_t experts) {
  const int64_t epad = (experts + 7) / 8 * 8;
  return 3 * epad * hidden * 2 + tokens * 3 * epad * 4 + 512;
}

// Tensor-core projection for BF16 hidden states: the FP32 weight is split into three BF16 parts whose
// sum reproduces it to 24 bits, the products with the (exact) BF16 activations accumulate in FP32 on
// tcgen05, and the three partial results are added. FP32 hidden states use hmc_gate_project.
extern "C" int hmc_gate_project_tc(const void* x_bf16, const void* w, int w_is_bf16, int64_t tokens, int64_t hidden,
                                   int64_t experts, float* logits, void* workspace, int64_t workspace_bytes,
                                   void* stream_ptr) {
  using namespace hmc;
  HMC_REQUIRE(x_bf16 && w && logits && workspace, HMC_ERR_INVALID, "hmc_gate_project_tc: null tensor pointer");
  HMC_REQUIRE(tokens > 0 && experts > 0 && hidden > 0 && hidden % 8 == 0, HMC_ERR_INVALID,
              "hmc_gate_project_tc: extents must be positive and hidden a multiple of 8");
  HMC_REQUIRE(workspace_bytes >= hmc_gate_project_workspace_bytes(tokens, hidden, experts), HMC_ERR_INVALID,
              "hmc_gate_project_tc: workspace holds %lld bytes, %lld needed", (long long)workspace_bytes,
              (long long)hmc_gate_project_workspace_bytes(tokens, hidden, experts));
  HMC_REQUIRE(aligned16(x_bf16) && aligned16(workspace), HMC_ERR_INVALID, "hmc_gate_project_tc: 16-byte alignment");
  cudaStream_t stream = static_cast<cudaStream_t>(stream_ptr);
  const int epad = static_cast<int>((experts + 7) / 8 * 8);
  const int parts = w_is_bf16 ? 1 : 3;
  uint8_t* ws = static_cast<uint8_t*>(workspace);
  __nv_bfloat16* split = reinterpret_cast<__nv_bfloat16*>(ws);
  float* partial = reinterpret_cast<float*>(ws + 3ll * epad * hidden * 2);
  long long* ends = reinterpret_cast<long long*>(ws + 3ll * epad * hidden * 2 + tokens * 3ll * epad * 4);
  ends = reinterpret_cast<long long*>((reinterpret_cast<uintptr_t>(ends) + 15) & ~static_cast<uintptr_t>(15));
  const long long split_elems = static_cast<long long>(epad) * hidden;
  gate_split_weight_kernel<<<static_cast<unsigned>((split_elems + 255) / 256), 256, 0, stream>>>(
      w, w_is_bf16, static_cast<int>(experts), epad, parts, hidden, split);
  HMC_LAUNCH_OK();
  HMC_CUDA_OK(cudaMemcpyAsync(ends, &tokens, sizeof(long long), cudaMemcpyHostToDevice, stream));
  hmc_grouped_gemm_args g{};
  g.mode = HMC_GEMM_RAGGED_M;
  g.a_major = HMC_MAJOR_K;
  g.b_major = HMC_MAJOR_K;
  g.epilogue = HMC_EPI_STORE_F32;
  g.groups = 1;
  g.tile_mode = HMC_TILE_SINGLE;
  g.rows = tokens;
  g.n = static_cast<int64_t>(parts) * epad;
  g.k = hidden;
  g.a = x_bf16;
  g.b = split;
  g.c = partial;
  g.group_ends = reinterpret_cast<const int64_t*>(ends);
  int rc = hmc_grouped_gemm(&g, stream);
  if (rc != 0) return rc;
  const long long total = tokens * experts;
  gate_sum_parts_kernel<<<static_cast<unsigned>((total + 255) / 256), 256, 0, stream>>>(
      partial, tokens, static_cast<int>(experts), epad, parts, logits);
  HMC_LAUNCH_OK();
  return 0;
}
