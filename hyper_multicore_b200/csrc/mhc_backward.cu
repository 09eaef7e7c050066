// MegaMHC backward in six launches. The two contractions with the 24-wide gradient of the projection go to the tcgen05
// grouped GEMM, everything that streams over the hidden dimension to a warp per token.
//
// Math is the autograd of the reference's semantic oracle (tests/common/multicore/mega_mhc_grad_golden.py:117-193 over
// mega_mhc_golden.py:29-142; native worker hyper_multicore/ops/hyper_mega_mhc_grad/op_kernel/worker_kernel.cpp).
#include <math.h>

#include "common.cuh"
#include "mhc_shared.cuh"

namespace hmc {

int check_mhc_dims(const char* what, int64_t tokens, int64_t hidden, int32_t num_iters);  // mhc_forward.cu

namespace {

using namespace mhc;

constexpr int MIX_PAD = 32;    // padded width of one BF16 split part
constexpr int WARPS = 8;
constexpr int HEAD_SUMS = 27;  // d bias (24), d alpha (3)
// Four blocks per SM of a B200; the last stage adds one row of 27 sums per block. A constant, so that the size of the
// workspace and the order of these sums follow from the extents alone and not from the device that happens to be current.
constexpr int64_t MAX_HEAD_BLOCKS = 4 * 148;

// ---------------------------------------------------------------------------------------------
// Stage 1, one warp per token: gradients of the mapping head. Walks the Sinkhorn chain forwards and backwards with one
// matrix entry per lane, which keeps its 40 normalisers in shared memory (a thread that walked a whole 4 x 4 matrix had
// 160 of them in local memory: with the splitting of phi 66 us for 1531 tokens, 82 us for 16384; 15 and 55 us this way),
// and emits dq - the gradient of the un-normalised projection - as BF16 parts for the two contractions, the per-token
// coefficient of the RMS term and block sums of d alpha and d bias. Blocks past the tokens split phi for the contraction.
// ---------------------------------------------------------------------------------------------
struct HeadParams {
  const float* hc_before_norm;
  const float* inv_rms;
  const float* alpha;
  const float* bias;
  const float* grad_pre;
  const float* grad_post;
  const float* grad_mix;
  const float* phi;
  long long tokens;
  int hidden;
  int iters;
  float hc_eps;
  __nv_bfloat16* dq_rows;  // [tokens][128]: hi | hi | lo | 0, parts of 32
  __nv_bfloat16* dq_cols;  // [tokens][64] : hi | lo
  __nv_bfloat16* phi_split;  // [128][4 hidden]: hi | lo | hi | 0
  float* rms_coef;
  float* head_parts;       // [token blocks][32]
  long long* ends;
  unsigned token_blocks;
};

// phi [24, K] FP32 -> BF16 split rows [128, K]: rows 0..23 = hi, 32..55 = lo residual (hi + lo carries 16 mantissa
// bits), 64..87 = hi again, every other row zero; the contraction over them meets dq as hi | hi | lo | 0.
__device__ __forceinline__ void split_phi(const HeadParams& p, long long i) {
  const long long k = 4ll * p.hidden;
  if (i >= k) return;
  const __nv_bfloat16 zero = __float2bfloat16_rn(0.f);
#pragma unroll 4
  for (int c = 0; c < MIX_PAD; ++c) {
    __nv_bfloat16 hi = zero, lo = zero;
    if (c < MIX) {
      const float v = p.phi[c * k + i];
      hi = __float2bfloat16_rn(v);
      lo = __float2bfloat16_rn(v - __bfloat162float(hi));
    }
    p.phi_split[c * k + i] = hi;
    p.phi_split[(MIX_PAD + c) * k + i] = lo;
    p.phi_split[(2 * MIX_PAD + c) * k + i] = hi;
    p.phi_split[(3 * MIX_PAD + c) * k + i] = zero;
  }
}

__global__ void __launch_bounds__(256) mhc_head_grad_kernel(const HeadParams p) {
  __shared__ float stage[8][64];
  __shared__ float norms[8][SINKHORN_MAX_STEPS][32];
  if (blockIdx.x >= p.token_blocks) {
    split_phi(p, static_cast<long long>(blockIdx.x - p.token_blocks) * 256 + threadIdx.x);
    return;
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (blockIdx.x == 0 && threadIdx.x == 0) *p.ends = p.tokens;
  float d_bias = 0.f, d_alpha = 0.f;
  for (long long t = static_cast<long long>(blockIdx.x) * 8 + warp; t < p.tokens; t += static_cast<long long>(p.token_blocks) * 8) {
    const float r = p.inv_rms[t];
    const float scale = lane < 4 ? p.alpha[0] : (lane < 8 ? p.alpha[1] : p.alpha[2]);
    const float q = lane < MIX ? p.hc_before_norm[t * MIX + lane] : 0.f;
    const float l = q * r;
    const float a = lane < MIX ? fmaf(l, scale, p.bias[lane]) : 0.f;
    const int entry = lane & 15;
    const int steps = 2 * p.iters;
    float(*norm)[32] = norms[warp];
    float m = sinkhorn16(__shfl_sync(0xffffffffu, a, entry + 8), p.hc_eps, steps,
                         [&](int step, float s, float) { norm[step][lane] = s; });
    float g = p.grad_mix[t * 16 + entry];
    // Each normalisation is out = in / s with s = sum(in) + eps along one axis, so
    // d_in = d_out / s - sum(d_out * out) / s along that axis, and in = out * s. Odd steps are columns, even ones rows.
#pragma unroll 1
    for (int step = steps - 1; step >= 1; step -= 2) {
      float s = norm[step][lane];
      g = (g - col_sum4(g * m)) * __frcp_rn(s);
      m *= s;
      if (step == 1) break;
      s = norm[step - 1][lane];
      g = (g - row_sum4(g * m)) * __frcp_rn(s);
      m *= s;
    }
    m -= p.hc_eps;  // step 0: m = softmax(logit) + eps
    const float d_mix = m * (g - row_sum4(g * m));
    float da = __shfl_sync(0xffffffffu, d_mix, (lane - 8) & 15);
    if (lane < 8) {
      const float sg = sigmoid_f(a);
      da = (lane < 4 ? p.grad_pre[t * 4 + lane] : 2.0f * p.grad_post[t * 4 + lane - 4]) * sg * (1.0f - sg);
    }
    if (lane >= MIX) da = 0.f;
    d_bias += da;
    d_alpha += da * l;
    const float dl = da * scale;
    const float dq = dl * r;
    const float dr = warp_sum(dl * q);
    // r = (S + eps)^-1/2 with S = sum(R^2) / (4H): dR += R * (-r^3 * dr / (4H))
    if (lane == 0) p.rms_coef[t] = -(r * r * r) * dr / static_cast<float>(STREAMS * p.hidden);
    const __nv_bfloat16 hi = __float2bfloat16_rn(dq), lo = __float2bfloat16_rn(dq - __bfloat162float(hi));
    __nv_bfloat16* rows = p.dq_rows + t * 4 * MIX_PAD + lane;
    rows[0] = hi;
    rows[MIX_PAD] = hi;
    rows[2 * MIX_PAD] = lo;
    rows[3 * MIX_PAD] = __float2bfloat16_rn(0.f);
    __nv_bfloat16* cols = p.dq_cols + t * 2 * MIX_PAD + lane;
    cols[0] = hi;
    cols[MIX_PAD] = lo;
  }
  stage[warp][lane] = d_bias;
  stage[warp][32 + lane] = d_alpha;
  __syncthreads();
  if (threadIdx.x < 32) {
    float total = 0.f;
    if (lane < MIX) {
      for (int w = 0; w < 8; ++w) total += stage[w][lane];
    } else if (lane < HEAD_SUMS) {
      const int first = lane == MIX ? 0 : (lane == MIX + 1 ? 4 : 8), last = lane == MIX ? 4 : (lane == MIX + 1 ? 8 : MIX);
      for (int w = 0; w < 8; ++w)
        for (int i = first; i < last; ++i) total += stage[w][32 + i];
    }
    p.head_parts[static_cast<long long>(blockIdx.x) * 32 + lane] = total;
  }
}

// ---------------------------------------------------------------------------------------------
// Stage 5 (one warp per token): everything that streams over the hidden dimension.
// ---------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(WARPS * 32, 2)
mhc_stream_grad_kernel(const uint4* __restrict__ grad_new_residual, const uint4* __restrict__ grad_block_input,
                       const uint4* __restrict__ new_residual, const uint4* __restrict__ mixed_input,
                       const uint4* __restrict__ residual, const uint4* __restrict__ prev_out,
                       const uint4* __restrict__ proj_grad,  // dq . phi, BF16 [tokens, 4H]
                       const uint4* __restrict__ norm_weight, const float* __restrict__ prev_pre,
                       const float* __restrict__ prev_post, const float* __restrict__ prev_mix,
                       const float* __restrict__ rms_rstd, const float* __restrict__ rms_coef, long long tokens,
                       int hidden, uint4* __restrict__ grad_residual, uint4* __restrict__ grad_prev_out,
                       float* __restrict__ grad_prev_pre, float* __restrict__ grad_prev_post,
                       float* __restrict__ grad_prev_mix) {
  const int vec = hidden / 8;
  const int lane = threadIdx.x & 31;
  const int warp = threadIdx.x >> 5;
  for (long long t = static_cast<long long>(blockIdx.x) * WARPS + warp; t < tokens;
       t += static_cast<long long>(gridDim.x) * WARPS) {
    float mix[STREAMS][STREAMS], post[STREAMS], pre[STREAMS];
#pragma unroll
    for (int j = 0; j < STREAMS; ++j) {
      post[j] = prev_post[t * STREAMS + j];
      pre[j] = prev_pre[t * STREAMS + j];
#pragma unroll
      for (int i = 0; i < STREAMS; ++i) mix[j][i] = prev_mix[(t * STREAMS + j) * STREAMS + i];
    }
    const float rstd = rms_rstd[t];
    const float coef = rms_coef[t];
    const uint4* gb_row = grad_block_input + t * vec;
    const uint4* mixed_row = mixed_input + t * vec;
    // pass 1: sum_h (g_block * w) * mixed
    float dot = 0.f;
    for (int v = lane; v < vec; v += 32) {
      float gb[8], w[8], m[8];
      unpack8(ld_16(gb_row + v), gb);
      unpack8(ld_16(norm_weight + v), w);
      unpack8(ld_16(mixed_row + v), m);
#pragma unroll
      for (int e = 0; e < 8; ++e) dot = fmaf(gb[e] * w[e], m[e], dot);
    }
    dot = warp_sum(dot);
    const float back = rstd * rstd * rstd * dot / static_cast<float>(hidden);
    float d_pre[STREAMS] = {0.f, 0.f, 0.f, 0.f}, d_post[STREAMS] = {0.f, 0.f, 0.f, 0.f};
    float d_mix[STREAMS][STREAMS] = {};
    const uint4* new_row = new_residual + t * STREAMS * vec;
    const uint4* gn_row = grad_new_residual + t * STREAMS * vec;
    const uint4* pg_row = proj_grad + t * STREAMS * vec;
    const uint4* res_row = residual + t * STREAMS * vec;
    uint4* gres_row = grad_residual + t * STREAMS * vec;
    for (int v = lane; v < vec; v += 32) {
      float gb[8], w[8], m[8], d_mixed[8];
      unpack8(ld_16(gb_row + v), gb);
      unpack8(ld_16(norm_weight + v), w);
      unpack8(ld_16(mixed_row + v), m);
#pragma unroll
      for (int e = 0; e < 8; ++e) d_mixed[e] = rstd * (gb[e] * w[e]) - m[e] * back;
      float dR[STREAMS][8];
#pragma unroll
      for (int i = 0; i < STREAMS; ++i) {
        float R[8], gn[8], pg[8];
        unpack8(ld_nc_16(new_row + i * vec + v), R);
        unpack8(ld_nc_16(gn_row + i * vec + v), gn);
        unpack8(ld_nc_16(pg_row + i * vec + v), pg);
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          dR[i][e] = gn[e] + pre[i] * d_mixed[e] + coef * R[e] + pg[e];
          d_pre[i] = fmaf(d_mixed[e], R[e], d_pre[i]);
        }
      }
      float o[8], d_out[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
      unpack8(ld_nc_16(prev_out + t * vec + v), o);
#pragma unroll
      for (int i = 0; i < STREAMS; ++i) {
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          d_out[e] = fmaf(post[i], dR[i][e], d_out[e]);
          d_post[i] = fmaf(o[e], dR[i][e], d_post[i]);
        }
      }
      st_cs_16(grad_prev_out + t * vec + v, pack8(d_out));
#pragma unroll
      for (int j = 0; j < STREAMS; ++j) {
        float r[8], d_res[8];
        unpack8(ld_nc_16(res_row + j * vec + v), r);
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          float acc = 0.f;
#pragma unroll
          for (int i = 0; i < STREAMS; ++i) {
            acc = fmaf(mix[j][i], dR[i][e], acc);
            d_mix[j][i] = fmaf(r[e], dR[i][e], d_mix[j][i]);
          }
          d_res[e] = acc;
        }
        st_cs_16(gres_row + j * vec + v, pack8(d_res));
      }
    }
#pragma unroll
    for (int i = 0; i < STREAMS; ++i) {
      d_pre[i] = warp_sum(d_pre[i]);
      d_post[i] = warp_sum(d_post[i]);
#pragma unroll
      for (int j = 0; j < STREAMS; ++j) d_mix[j][i] = warp_sum(d_mix[j][i]);
    }
    if (lane == 0) {
#pragma unroll
      for (int i = 0; i < STREAMS; ++i) {
        grad_prev_pre[t * STREAMS + i] = d_pre[i];
        grad_prev_post[t * STREAMS + i] = d_post[i];
#pragma unroll
        for (int j = 0; j < STREAMS; ++j) grad_prev_mix[(t * STREAMS + j) * STREAMS + i] = d_mix[j][i];
      }
    }
  }
}

// d norm_weight[h] = sum_t grad_block_input[t, h] * mixed_input[t, h] * rstd[t]: a column reduction.
// Block = 32 column vectors x 8 token lanes; every thread keeps 8 FP32 partial sums in registers.
__global__ void __launch_bounds__(256)
mhc_norm_weight_grad_kernel(const uint4* __restrict__ grad_block_input, const uint4* __restrict__ mixed_input,
                            const float* __restrict__ rms_rstd, long long tokens, int vec,
                            float* __restrict__ norm_parts) {
  __shared__ float red[8][32][9];
  const int tx = threadIdx.x & 31;
  const int ty = threadIdx.x >> 5;
  const int v = blockIdx.x * 32 + tx;
  float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  if (v < vec) {
    const long long step = static_cast<long long>(gridDim.y) * 8;
#pragma unroll 4
    for (long long t = static_cast<long long>(blockIdx.y) * 8 + ty; t < tokens; t += step) {
      float gb[8], m[8];
      unpack8(ld_nc_16(grad_block_input + t * vec + v), gb);
      unpack8(ld_nc_16(mixed_input + t * vec + v), m);
      const float r = rms_rstd[t];
#pragma unroll
      for (int e = 0; e < 8; ++e) acc[e] = fmaf(gb[e] * m[e], r, acc[e]);
    }
  }
#pragma unroll
  for (int e = 0; e < 8; ++e) red[ty][tx][e] = acc[e];
  __syncthreads();
  // thread (ty, tx) sums column e = ty of vector tx over the 8 token lanes
  if (v < vec) {
    float total = 0.f;
#pragma unroll
    for (int y = 0; y < 8; ++y) total += red[y][tx][ty];
    norm_parts[(static_cast<long long>(blockIdx.y) * vec + v) * 8 + ty] = total;
  }
}

// ---------------------------------------------------------------------------------------------
// Last stage: the sums over blocks of the stages before, each in a fixed order.
// ---------------------------------------------------------------------------------------------
struct FinishParams {
  const float* norm_parts;  // [norm_rows][hidden]
  const float* head_parts;  // [head_blocks][32]
  const float* phi_parts;   // [64][4 * hidden]: rows 0..23 from the hi part of dq, 32..55 from the lo part
  int hidden;
  int norm_rows;
  int head_blocks;
  unsigned norm_blocks;
  float* grad_norm;
  float* grad_phi;
  float* grad_alpha;
  float* grad_bias;
};

__global__ void __launch_bounds__(256) mhc_finish_grad_kernel(const FinishParams p) {
  unsigned block = blockIdx.x;
  if (block == 0) {  // alpha and bias: the longest chain of the launch starts first
    __shared__ float stage[8][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    float v = 0.f;
#pragma unroll 8
    for (int b = warp; b < p.head_blocks; b += 8) v += __ldcg(p.head_parts + b * 32ll + lane);
    stage[warp][lane] = v;
    __syncthreads();
    if (warp == 0 && lane < HEAD_SUMS) {
      v = 0.f;
#pragma unroll
      for (int w = 0; w < 8; ++w) v += stage[w][lane];
      if (lane < MIX) p.grad_bias[lane] = v;
      else p.grad_alpha[lane - MIX] = v;
    }
    return;
  }
  block -= 1;
  if (block < p.norm_blocks) {
    const int h = static_cast<int>(block) * 256 + threadIdx.x;
    if (h >= p.hidden) return;
    float total = 0.f;
#pragma unroll 8
    for (int r = 0; r < p.norm_rows; ++r) total += __ldcg(p.norm_parts + static_cast<long long>(r) * p.hidden + h);
    p.grad_norm[h] = total;
    return;
  }
  block -= p.norm_blocks;
  const long long k = 4ll * p.hidden;
  const long long i = static_cast<long long>(block) * 256 + threadIdx.x;
  if (i < MIX * k) p.grad_phi[i] = __ldcg(p.phi_parts + i) + __ldcg(p.phi_parts + 32 * k + i);
}

struct GradLayout {
  int norm_rows;
  unsigned head_blocks;
  int64_t ends, phi_split, dq_rows, dq_cols, proj_grad, phi_parts, rms_coef, head_parts, norm_parts, bytes;
};

GradLayout grad_layout(int64_t tokens, int64_t hidden) {
  GradLayout l;
  auto up = [](int64_t v) { return (v + 255) / 256 * 256; };
  const int64_t k = 4 * hidden;
  l.norm_rows = static_cast<int>(tokens >= 4096 ? 64 : (tokens + 63) / 64);
  const int64_t blocks = (tokens + 7) / 8;
  l.head_blocks = static_cast<unsigned>(blocks < MAX_HEAD_BLOCKS ? blocks : MAX_HEAD_BLOCKS);
  l.ends = 0;
  l.phi_split = 256;
  l.dq_rows = l.phi_split + up(128 * k * 2);
  l.dq_cols = l.dq_rows + up(tokens * 128 * 2);
  l.proj_grad = l.dq_cols + up(tokens * 64 * 2);
  l.phi_parts = l.proj_grad + up(tokens * k * 2);
  l.rms_coef = l.phi_parts + up(64 * k * 4);
  l.head_parts = l.rms_coef + up(tokens * 4);
  l.norm_parts = l.head_parts + up(l.head_blocks * 128ll);
  l.bytes = l.norm_parts + up(l.norm_rows * hidden * 4);
  return l;
}

}  // namespace
}  // namespace hmc

using namespace hmc;

extern "C" int64_t hmc_mega_mhc_grad_workspace_bytes(int64_t tokens, int64_t hidden) { return grad_layout(tokens, hidden).bytes; }

extern "C" int hmc_mega_mhc_grad(const hmc_mega_mhc_grad_args* args, void* stream_ptr) {
  HMC_REQUIRE(args != nullptr, HMC_ERR_INVALID, "hmc_mega_mhc_grad: null args");
  const hmc_mega_mhc_grad_args& a = *args;
  int rc = check_mhc_dims("hmc_mega_mhc_grad", a.tokens, a.hidden, a.num_iters);
  if (rc != 0) return rc;
  HMC_REQUIRE(a.grad_new_residual && a.grad_next_pre_mix && a.grad_next_post_mix && a.grad_next_residual_mix &&
                  a.grad_block_input && a.new_residual && a.hc_before_norm && a.inv_rms && a.mixed_input &&
                  a.rms_rstd && a.previous_output && a.residual && a.previous_pre_mix && a.previous_post_mix &&
                  a.previous_residual_mix && a.phi && a.alpha && a.bias && a.norm_weight && a.grad_residual &&
                  a.grad_phi && a.grad_alpha && a.grad_bias && a.grad_previous_output && a.grad_previous_pre_mix &&
                  a.grad_previous_post_mix && a.grad_previous_residual_mix && a.grad_norm_weight && a.workspace,
              HMC_ERR_INVALID, "hmc_mega_mhc_grad: null tensor pointer");
  const GradLayout l = grad_layout(a.tokens, a.hidden);
  HMC_REQUIRE(a.workspace_bytes >= l.bytes, HMC_ERR_INVALID, "hmc_mega_mhc_grad: workspace holds %lld bytes, %lld needed",
              (long long)a.workspace_bytes, (long long)l.bytes);
  HMC_REQUIRE(aligned16(a.grad_new_residual) && aligned16(a.grad_block_input) && aligned16(a.new_residual) &&
                  aligned16(a.mixed_input) && aligned16(a.previous_output) && aligned16(a.residual) &&
                  aligned16(a.norm_weight) && aligned16(a.grad_residual) && aligned16(a.grad_previous_output) &&
                  aligned16(a.workspace),
              HMC_ERR_INVALID, "hmc_mega_mhc_grad: activations must be 16-byte aligned");
  cudaStream_t stream = static_cast<cudaStream_t>(stream_ptr);
  const int hidden = static_cast<int>(a.hidden);
  const long long k = 4ll * a.hidden;
  uint8_t* ws = static_cast<uint8_t*>(a.workspace);

  const int vec = hidden / 8;

  HeadParams h{};
  h.hc_before_norm = a.hc_before_norm;
  h.inv_rms = a.inv_rms;
  h.alpha = a.alpha;
  h.bias = a.bias;
  h.grad_pre = a.grad_next_pre_mix;
  h.grad_post = a.grad_next_post_mix;
  h.grad_mix = a.grad_next_residual_mix;
  h.phi = a.phi;
  h.tokens = a.tokens;
  h.hidden = hidden;
  h.iters = a.num_iters;
  h.hc_eps = a.hc_eps;
  h.dq_rows = reinterpret_cast<__nv_bfloat16*>(ws + l.dq_rows);
  h.dq_cols = reinterpret_cast<__nv_bfloat16*>(ws + l.dq_cols);
  h.phi_split = reinterpret_cast<__nv_bfloat16*>(ws + l.phi_split);
  h.rms_coef = reinterpret_cast<float*>(ws + l.rms_coef);
  h.head_parts = reinterpret_cast<float*>(ws + l.head_parts);
  h.ends = reinterpret_cast<long long*>(ws + l.ends);
  h.token_blocks = l.head_blocks;
  mhc_head_grad_kernel<<<l.head_blocks + static_cast<unsigned>((k + 255) / 256), 256, 0, stream>>>(h);
  HMC_LAUNCH_OK();
  {  // proj_grad[T, 4H] = dq . phi  (contraction over the padded, split 128-wide axis)
    hmc_grouped_gemm_args g{};
    g.mode = HMC_GEMM_RAGGED_M;
    g.a_major = HMC_MAJOR_K;
    g.b_major = HMC_MAJOR_MN;
    g.epilogue = HMC_EPI_STORE_BF16;
    g.groups = 1;
    g.rows = a.tokens;
    g.n = k;
    g.k = 4 * MIX_PAD;
    g.tile_mode = HMC_TILE_SINGLE;  // two k-blocks per tile: the store path decides, and 128-row tiles store by TMA
    g.a = h.dq_rows;
    g.b = h.phi_split;
    g.c = ws + l.proj_grad;
    g.group_ends = reinterpret_cast<const int64_t*>(h.ends);
    g.status = a.status;
    if ((rc = hmc_grouped_gemm(&g, stream)) != 0) return rc;
  }
  {  // phi parts [64, 4H] = dq^T . new_residual, contracted over the tokens
    hmc_grouped_gemm_args g{};
    g.mode = HMC_GEMM_RAGGED_K;
    g.a_major = HMC_MAJOR_MN;
    g.b_major = HMC_MAJOR_MN;
    g.epilogue = HMC_EPI_STORE_F32;
    g.groups = 1;
    g.rows = a.tokens;
    g.m = 2 * MIX_PAD;
    g.n = k;
    g.a = h.dq_cols;
    g.b = a.new_residual;
    g.c = ws + l.phi_parts;
    g.group_ends = reinterpret_cast<const int64_t*>(h.ends);
    g.status = a.status;
    if ((rc = hmc_grouped_gemm(&g, stream)) != 0) return rc;
  }
  mhc_norm_weight_grad_kernel<<<dim3(static_cast<unsigned>((vec + 31) / 32), static_cast<unsigned>(l.norm_rows)), 256, 0, stream>>>(
      static_cast<const uint4*>(a.grad_block_input), static_cast<const uint4*>(a.mixed_input), a.rms_rstd, a.tokens, vec,
      reinterpret_cast<float*>(ws + l.norm_parts));
  HMC_LAUNCH_OK();
  const long long need = (a.tokens + WARPS - 1) / WARPS;
  const int grid = static_cast<int>(need < 4 * sm_count() ? need : 4 * sm_count());
  mhc_stream_grad_kernel<<<grid, WARPS * 32, 0, stream>>>(
      static_cast<const uint4*>(a.grad_new_residual), static_cast<const uint4*>(a.grad_block_input),
      static_cast<const uint4*>(a.new_residual), static_cast<const uint4*>(a.mixed_input),
      static_cast<const uint4*>(a.residual), static_cast<const uint4*>(a.previous_output),
      reinterpret_cast<const uint4*>(ws + l.proj_grad),
      static_cast<const uint4*>(a.norm_weight), a.previous_pre_mix, a.previous_post_mix, a.previous_residual_mix, a.rms_rstd,
      h.rms_coef, a.tokens, hidden, static_cast<uint4*>(a.grad_residual), static_cast<uint4*>(a.grad_previous_output),
      a.grad_previous_pre_mix, a.grad_previous_post_mix, a.grad_previous_residual_mix);
  HMC_LAUNCH_OK();

  FinishParams f{};
  f.norm_parts = reinterpret_cast<const float*>(ws + l.norm_parts);
  f.head_parts = h.head_parts;
  f.phi_parts = reinterpret_cast<const float*>(ws + l.phi_parts);
  f.hidden = hidden;
  f.norm_rows = l.norm_rows;
  f.head_blocks = static_cast<int>(l.head_blocks);
  f.norm_blocks = static_cast<unsigned>((hidden + 255) / 256);
  f.grad_norm = a.grad_norm_weight;
  f.grad_phi = a.grad_phi;
  f.grad_alpha = a.grad_alpha;
  f.grad_bias = a.grad_bias;
  mhc_finish_grad_kernel<<<1 + f.norm_blocks + static_cast<unsigned>((MIX * k + 255) / 256), 256, 0, stream>>>(f);
  HMC_LAUNCH_OK();
  return 0;
}
