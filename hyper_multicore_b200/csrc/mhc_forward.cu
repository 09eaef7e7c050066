// MegaMHC forward: four-stream residual mix, mapping prediction (sigmoid / Sinkhorn) and RMSNorm in two launches.
//
// Math follows the reference's semantic oracle torch_mega_mhc / _predict_mappings / _sinkhorn
// (tests/common/multicore/mega_mhc_golden.py:29-142). Stage order mirrors the native worker
// (hyper_multicore/ops/hyper_mega_mhc/op_kernel/worker_kernel.cpp:92-268): Post, NormCast, Projection (un-normalised
// dot, then scaled by 1/rms), InputMix in BF16, Mapping, RMSNorm.
//
// Bound by memory traffic: 5 rows of `hidden` BF16 values in and 5 out per token, then the mixed row in and the block
// input out. The 24-wide projection against phi is done by the kernel that produces the new residual, while its
// values are in registers; a GEMM of its own would read four of the rows again and, for a handful of tokens, run on
// one SM. A CTA owns 128 columns of the hidden dimension and walks over tokens: its share of phi (two BF16 parts, as
// matrix fragments) then stays in shared memory, and the grid fills the chip for 16 tokens as well as for 16384. The
// contraction is 24 wide, far below what a 128-row tensor-memory tile needs to pay, so it runs as warp-level matrix
// instructions whose A operand is the register fragment the mix leaves behind; nothing is staged for it. What is left
// to do across the columns of a token - 24 dot products, two sums of squares - goes through a small partial buffer
// [column block][token][28], 4% of the traffic (103 MB of scratch at 16384 x 7168).
//
// The bits of a token do not depend on how many share the call: a column block adds its four column steps one after the
// other whether one warp has taken them or four, and the column blocks are added in eight chains whether one warp of the
// second launch walks all of them or eight one each.
//
// Device time, five launches before -> two: 16 tokens x hidden 7168 201 -> 14 us, 1531 x 2560 95 -> 47 us, 4096 x 7168
// 305 -> 180 us, 16384 x 7168 699 -> 599 us. At the large end the first launch takes 489 us for 2.6 GB (5.3 TB/s of what
// it has to move): half of the issue slots are used, and the 12 warps an SM holds at 146 registers wait for the rest.
#include <math.h>

#include "common.cuh"
#include "mhc_shared.cuh"

namespace hmc {
namespace {

using namespace mhc;

constexpr int PART = 28;  // 24 dot products, sum of squares, sum of squares of the mix, padding
constexpr int COL_STEPS = BLOCK_COLS / 32;
constexpr int LANE_SUMS = 16;  // of a lane per column step: 12 dot products, 2 sums of 2 tokens
__host__ __device__ constexpr int stream_warps(int steps) { return steps == 1 ? 4 : 12; }
constexpr int STREAM_ROWS = STREAMS + 1;               // rows read per token
constexpr int SLOT_VECS = 2 * STREAM_ROWS * 32;        // one step of a warp: [token g, token g + 8][row][lane]
constexpr int FRAG_VECS = COL_STEPS * STREAMS * 2 * 3 * 32;  // [column step][stream][k step][8 outputs][lane] hi.b0 hi.b1 lo.b0 lo.b1
constexpr int stream_smem(int steps) {
  return FRAG_VECS * 16 + stream_warps(steps) * (2 * SLOT_VECS * 16 + COEF_FLOATS * 4) +
         (steps == 1 ? COL_STEPS * 32 * LANE_SUMS * 4 : 0);
}
static_assert(stream_smem(COL_STEPS) <= 227 * 1024, "one CTA per SM");

struct StreamParams {
  const uint4* prev_out;
  const uint4* residual;
  const float* prev_pre;
  const float* prev_post;
  const float* prev_mix;
  const float* phi;
  long long tokens;
  int hidden;
  bool phi_vec;   // phi is 16-byte aligned
  bool coef_vec;  // the three coefficient arrays are
  uint4* new_residual;
  uint4* mixed_input;
  float* parts;
};

// A warp takes 16 tokens through STEPS column steps of its CTA's 128 columns. STEPS = 4 for many tokens: it meets no
// other warp on the way, and the sums of its tokens stay in its registers until it writes them. For a few, four warps
// take a step each (STEPS = 1) and meet once per token group to add their steps.
// A lane owns 8 consecutive columns of tokens g and g + 8 of its warp's 16: one 16-byte access per row, four lanes
// cover 64 bytes. The contraction index inside a 16-wide k step is permuted to match (phi's fragments are stored in
// the same order): logical 2c, 2c + 1 | 2c + 8, 2c + 9 of step s are columns 8c + 4s + 0, 1 | 2, 3.
template <int STEPS>
__global__ void __launch_bounds__(32 * stream_warps(STEPS), 1) mhc_stream_kernel(const StreamParams p) {
  extern __shared__ __align__(16) uint8_t smem_raw[];
  uint4* frag = reinterpret_cast<uint4*>(smem_raw);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint4* slots = frag + FRAG_VECS + warp * 2 * SLOT_VECS + lane;  // a lane reads back what it copied itself
  float* const coefs_of_all = reinterpret_cast<float*>(frag + FRAG_VECS + stream_warps(STEPS) * 2 * SLOT_VECS);
  float* const coef = coefs_of_all + warp * COEF_FLOATS;
  // STEPS == 1: [column step][quad of sums][lane]
  float4* const exchange = reinterpret_cast<float4*>(coefs_of_all + stream_warps(STEPS) * COEF_FLOATS);
  const int g = lane >> 2, c = lane & 3;
  const int vec = p.hidden / 8;
  const long long k = 4ll * p.hidden;

  for (int i = threadIdx.x; i < FRAG_VECS; i += 32 * stream_warps(STEPS)) {
    const int l = i & 31;
    int rest = i >> 5;
    const int n = (rest % 3) * 8 + (l >> 2);
    rest /= 3;
    const int s = rest & 1, stream = (rest >> 1) & 3, cs = rest >> 3;
    const long long at = n * k + static_cast<long long>(stream) * p.hidden + blockIdx.x * BLOCK_COLS + cs * 32 + 8 * (l & 3) + 4 * s;
    const float4 v = load4(p.phi + at, p.phi_vec);
    uint4 f;
    split_pair(v.x, v.y, f.x, f.z);
    split_pair(v.z, v.w, f.y, f.w);
    frag[i] = f;
  }
  __syncthreads();

  constexpr int SHARE = COL_STEPS / STEPS;  // warps that share a token group
  const int first_step = (warp % SHARE) * STEPS;
  const int col0 = static_cast<int>(blockIdx.x) * (BLOCK_COLS / 8) + c;  // in vectors of 8
  const long long groups = (p.tokens + 15) / 16;
  const long long stride = static_cast<long long>(gridDim.y) * (stream_warps(STEPS) / SHARE);
  const long long group0 = static_cast<long long>(blockIdx.y) * (stream_warps(STEPS) / SHARE) + warp / SHARE;

  // A step's rows are copied to shared memory while the step before it is worked on: registers could only be refilled
  // once they have been used, and the copies would have a fifth of the time.
  auto fetch = [&](int slot, long long group, int step) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const long long t = group * 16 + 8 * h + g;
      uint4* dst = slots + slot * SLOT_VECS + h * STREAM_ROWS * 32;
      if (t < p.tokens) {
        const uint4* row = p.residual + t * STREAMS * vec + col0 + step * 4;
#pragma unroll
        for (int j = 0; j < STREAMS; ++j) copy_async_16(dst + j * 32, row + j * vec);
        copy_async_16(dst + STREAMS * 32, p.prev_out + t * vec + col0 + step * 4);
      } else {
#pragma unroll
        for (int j = 0; j < STREAM_ROWS; ++j) dst[j * 32] = make_uint4(0, 0, 0, 0);
      }
    }
  };
  int slot = 0;
  CoefLoad next_coef = {};
  if (group0 < groups) {
    fetch(0, group0, first_step);
    next_coef = fetch_coefficients(p.prev_mix, p.prev_post, p.prev_pre, group0 * 16, p.tokens, p.coef_vec, lane);
  }
  copy_async_commit();
  for (long long group = group0; group < groups; group += stride) {
    store_coefficients(coef, next_coef, lane);
    next_coef = fetch_coefficients(p.prev_mix, p.prev_post, p.prev_pre, (group + stride) * 16, p.tokens, p.coef_vec, lane);
    float dot[3][4] = {}, square[4] = {};  // of all steps; square: sums of h = 0, sums of h = 1
#pragma unroll 1
    for (int s0 = 0; s0 < STEPS; ++s0) {
      const int step = first_step + s0;
      if (s0 + 1 < STEPS) fetch(slot ^ 1, group, step + 1);
      else if (group + stride < groups) fetch(slot ^ 1, group + stride, first_step);
      copy_async_commit();
      copy_async_wait<1>();
      const uint4* in = slots + slot * SLOT_VECS;
      slot ^= 1;
      float d[3][4] = {};
      float2 sums[2][2] = {};
      uint32_t a[STREAMS][2][4];  // the new residual, BF16 pairs
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const long long t = group * 16 + 8 * h + g;
        uint32_t mixed_out[4];
        uint4 row[STREAM_ROWS];
#pragma unroll
        for (int j = 0; j < STREAM_ROWS; ++j) row[j] = in[(h * STREAM_ROWS + j) * 32];
#pragma unroll
        for (int q0 = 0; q0 < 4; q0 += 2) {  // two pairs of columns at a time
          float2 r[2][STREAMS], o[2], mixed[2];
#pragma unroll
          for (int q = 0; q < 2; ++q) {
#pragma unroll
            for (int j = 0; j < STREAMS; ++j) r[q][j] = unpack_bf16x2(reinterpret_cast<const uint32_t*>(&row[j])[q0 + q]);
            o[q] = unpack_bf16x2(reinterpret_cast<const uint32_t*>(&row[STREAMS])[q0 + q]);
            mixed[q] = make_float2(0.f, 0.f);
          }
#pragma unroll
          for (int i = 0; i < STREAMS; ++i) {
            const StreamCoef coefs = stream_coef(coef, 8 * h + g, i);
#pragma unroll
            for (int q = 0; q < 2; ++q) {
              a[i][h][q0 + q] = new_residual_pair(coefs, r[q], o[q]);
              const float2 n = unpack_bf16x2(a[i][h][q0 + q]);
              sums[h][0] = fma2(n, n, sums[h][0]);
              mixed[q] = fma2(n, coefs.pre, mixed[q]);
            }
          }
#pragma unroll
          for (int q = 0; q < 2; ++q) {
            sums[h][1] = fma2(mixed[q], mixed[q], sums[h][1]);
            mixed_out[q0 + q] = pack_bf16x2(mixed[q].x, mixed[q].y);
          }
        }
        if (t < p.tokens) {
          uint4* dst = p.new_residual + t * STREAMS * vec + col0 + step * 4;
#pragma unroll
          for (int i = 0; i < STREAMS; ++i) st_16(dst + i * vec, make_uint4(a[i][h][0], a[i][h][1], a[i][h][2], a[i][h][3]));
          st_16(p.mixed_input + t * vec + col0 + step * 4, make_uint4(mixed_out[0], mixed_out[1], mixed_out[2], mixed_out[3]));
        }
      }
      const uint4* my_frag = frag + step * (STREAMS * 2 * 3 * 32) + lane;
#pragma unroll
      for (int i = 0; i < STREAMS; ++i)
#pragma unroll
        for (int s = 0; s < 2; ++s) {
          uint4 f[3];
#pragma unroll
          for (int nt = 0; nt < 3; ++nt) f[nt] = my_frag[((i * 2 + s) * 3 + nt) * 32];
#pragma unroll
          for (int nt = 0; nt < 3; ++nt)
            mma_16x8x16(d[nt], a[i][0][2 * s], a[i][1][2 * s], a[i][0][2 * s + 1], a[i][1][2 * s + 1], f[nt].x, f[nt].y);
#pragma unroll
          for (int nt = 0; nt < 3; ++nt)
            mma_16x8x16(d[nt], a[i][0][2 * s], a[i][1][2 * s], a[i][0][2 * s + 1], a[i][1][2 * s + 1], f[nt].z, f[nt].w);
        }
#pragma unroll
      for (int nt = 0; nt < 3; ++nt)
#pragma unroll
        for (int q = 0; q < 4; ++q) dot[nt][q] += d[nt][q];
#pragma unroll
      for (int q = 0; q < 4; ++q) square[q] += sums[q >> 1][q & 1].x + sums[q >> 1][q & 1].y;
    }
    float* const row = p.parts + (static_cast<long long>(blockIdx.x) * p.tokens + group * 16 + g) * PART;
    const bool stored[2] = {group * 16 + g < p.tokens, group * 16 + 8 + g < p.tokens};
    auto store_dot = [&](int nt, const float(&v)[4]) {
#pragma unroll
      for (int h = 0; h < 2; ++h)
        if (stored[h]) *reinterpret_cast<float2*>(row + 8 * h * PART + nt * 8 + 2 * c) = make_float2(v[2 * h], v[2 * h + 1]);
    };
    auto store_square = [&](const float(&v)[4]) {
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const float x = row_sum4(v[2 * h]), y = row_sum4(v[2 * h + 1]);
        if (stored[h] && c == 0) *reinterpret_cast<float2*>(row + 8 * h * PART + MIX) = make_float2(x, y);
      }
    };
    if constexpr (STEPS == COL_STEPS) {
#pragma unroll
      for (int nt = 0; nt < 3; ++nt) store_dot(nt, dot[nt]);
      store_square(square);
    } else {  // the four warps of the CTA have the same token group, and as many of them
      static_assert(STEPS == 1 && stream_warps(STEPS) == COL_STEPS, "a warp per column step and per quad of sums");
      __syncthreads();  // the sums before these have been read
      float4* mine = exchange + warp * 4 * 32 + lane;
#pragma unroll
      for (int nt = 0; nt < 3; ++nt) mine[nt * 32] = make_float4(dot[nt][0], dot[nt][1], dot[nt][2], dot[nt][3]);
      mine[3 * 32] = make_float4(square[0], square[1], square[2], square[3]);
      __syncthreads();
      float v[4] = {};
#pragma unroll
      for (int s = 0; s < COL_STEPS; ++s) {
        const float4 part = exchange[(s * 4 + warp) * 32 + lane];
        v[0] += part.x;
        v[1] += part.y;
        v[2] += part.z;
        v[3] += part.w;
      }
      if (warp < 3) store_dot(warp, v);
      else store_square(v);
    }
  }
}

struct FinishParams {
  const float* parts;
  const uint4* mixed_input;
  const uint4* norm_weight;
  const float* alpha;
  const float* bias;
  long long tokens;
  int hidden;
  int part_rows;
  float norm_eps;
  float hc_eps;
  int iters;
  uint4* block_input;
  float* inv_rms;
  float* rms_rstd;
  float* next_pre;
  float* next_post;
  float* next_mix;
  float* hc_before_norm;
  float* sum_out;
  float* norm_out;
};

// One token per WARPS warps: adds up the column blocks' partial sums, then RMSNorm of the mixed row and the mapping
// head (Sinkhorn with one matrix entry per lane: two shuffles per step instead of a 4 x 4 walk by one thread).
// Eight warps per token while one warp each would leave SMs without work. Seven lanes read a row of partial sums; row
// 32 i + 4 w + q belongs to chain w of lane group q, and a lane group adds its eight chains in order.
constexpr int CHAINS = 8;
template <int WARPS>
__global__ void __launch_bounds__(256, 4) mhc_finish_kernel(const FinishParams p) {
  static_assert(WARPS == 1 || WARPS == CHAINS, "a warp takes all of the chains or one");
  __shared__ float4 stage[WARPS == 1 ? 1 : CHAINS][28];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int part = WARPS == 1 ? 0 : warp;
  const long long t = WARPS == 1 ? static_cast<long long>(blockIdx.x) * 8 + warp : static_cast<long long>(blockIdx.x);
  if (t >= p.tokens) return;  // whole warps; with WARPS == 8 never taken
  auto add = [](float4& a, const float4& b) { a = make_float4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w); };
  float4 chain[CHAINS / WARPS];
#pragma unroll
  for (int w = 0; w < CHAINS / WARPS; ++w) chain[w] = make_float4(0.f, 0.f, 0.f, 0.f);
  {
    const float4* src = reinterpret_cast<const float4*>(p.parts) + t * (PART / 4) + (lane < 28 ? lane % 7 : 0);
    const long long pitch = p.tokens * (PART / 4);
#pragma unroll 1
    for (int round = part * 4; round < p.part_rows; round += 4 * CHAINS) {
#pragma unroll
      for (int w = 0; w < CHAINS / WARPS; ++w) {
        const int b = round + 4 * w + lane / 7;
        if (lane < 28 && b < p.part_rows) add(chain[w], __ldcg(src + b * pitch));
      }
    }
    __syncwarp();
  }
  float4 sum = make_float4(0.f, 0.f, 0.f, 0.f);
  if constexpr (WARPS == 1) {
#pragma unroll
    for (int w = 0; w < CHAINS; ++w) add(sum, chain[w]);
  } else {
    if (lane < 28) stage[warp][lane] = chain[0];
    __syncthreads();
#pragma unroll
    for (int w = 0; w < CHAINS; ++w) add(sum, stage[w][lane < 28 ? lane : 0]);
  }
#pragma unroll
  for (int o = 14; o >= 7; o -= 7) {  // lane groups 2, 3 onto 0, 1, then 1 onto 0
    sum.x += __shfl_down_sync(0xffffffffu, sum.x, o);
    sum.y += __shfl_down_sync(0xffffffffu, sum.y, o);
    sum.z += __shfl_down_sync(0xffffffffu, sum.z, o);
    sum.w += __shfl_down_sync(0xffffffffu, sum.w, o);
  }
  float v;  // value `lane` of the row
  {
    const int from = lane >> 2;
    const float x = __shfl_sync(0xffffffffu, sum.x, from), y = __shfl_sync(0xffffffffu, sum.y, from),
                z = __shfl_sync(0xffffffffu, sum.z, from), w = __shfl_sync(0xffffffffu, sum.w, from);
    v = (lane & 3) == 0 ? x : ((lane & 3) == 1 ? y : ((lane & 3) == 2 ? z : w));
  }
  const float r4 = rsqrtf(__shfl_sync(0xffffffffu, v, MIX) / static_cast<float>(STREAMS * p.hidden) + p.norm_eps);
  const float rstd = rsqrtf(__shfl_sync(0xffffffffu, v, MIX + 1) / static_cast<float>(p.hidden) + p.norm_eps);
  const int vec = p.hidden / 8;
  const uint4* mixed_row = p.mixed_input + t * vec;
  uint4* block_row = p.block_input + t * vec;
  // four loads in flight before the first store; every lane takes the same number of rounds
  for (int round = part * 32; round < vec; round += 4 * 32 * WARPS) {
    const int first = round + lane;
    uint4 row[4], weight[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int i = first + u * 32 * WARPS;
      row[u] = i < vec ? ld_nc_16(mixed_row + i) : make_uint4(0, 0, 0, 0);
      weight[u] = i < vec ? ld_16(p.norm_weight + i) : make_uint4(0, 0, 0, 0);
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int i = first + u * 32 * WARPS;
      float m[8], w[8], y[8];
      unpack8(row[u], m);
      unpack8(weight[u], w);
#pragma unroll
      for (int e = 0; e < 8; ++e) y[e] = (m[e] * rstd) * w[e];
      if (i < vec) st_cs_16(block_row + i, pack8(y));
    }
  }
  __syncwarp();
  if (part != WARPS - 1) return;  // the last warp of a token has the shortest share of its row
  if (lane == 0) {
    p.inv_rms[t] = r4;
    p.rms_rstd[t] = rstd;
  }
  const float scale = lane < 4 ? p.alpha[0] : (lane < 8 ? p.alpha[1] : p.alpha[2]);
  const float a = lane < MIX ? fmaf(v * r4, scale, p.bias[lane]) : 0.f;
  if (lane < MIX && p.hc_before_norm != nullptr) p.hc_before_norm[t * MIX + lane] = v;
  if (lane < 4) p.next_pre[t * 4 + lane] = sigmoid_f(a) + p.hc_eps;
  else if (lane < 8) p.next_post[t * 4 + lane - 4] = 2.0f * sigmoid_f(a);
  const int entry = lane & 15;
  const float logit = __shfl_sync(0xffffffffu, a, entry + 8);
  float m;
  if (p.sum_out == nullptr && p.norm_out == nullptr) {
    m = sinkhorn16(logit, p.hc_eps, 2 * p.iters, [](int, float, float) {});
  } else {
    m = sinkhorn16(logit, p.hc_eps, 2 * p.iters, [&](int step, float s, float value) {
      if (lane >= 16) return;
      if (p.sum_out != nullptr) {
        if ((step & 1) == 0 && (entry & 3) == 0) p.sum_out[(static_cast<long long>(step) * p.tokens + t) * 4 + (entry >> 2)] = s;
        if ((step & 1) == 1 && entry < 4) p.sum_out[(static_cast<long long>(step) * p.tokens + t) * 4 + entry] = s;
      }
      if (p.norm_out != nullptr) p.norm_out[(static_cast<long long>(step) * p.tokens + t) * 16 + entry] = value;
    });
  }
  if (lane < 16) p.next_mix[t * 16 + lane] = m;
}

}  // namespace

// Token splits of a streaming grid with `col_blocks` column blocks whose CTAs take `groups_per_cta` groups of 16 tokens a
// round, one CTA resident on every SM: the splits with the least waves of the chip times (rounds of a CTA + 1; loading
// phi's fragments costs a CTA about one). One wave alone leaves up to half of the SMs without a CTA: hidden 7168 has 56
// column blocks, so two splits, 112 CTAs.
// This launch, 8192 and 16384 tokens: 7168 283 -> 249 and 544 -> 498 us (two splits -> five), 5120 203 -> 186 and 373 ->
// 360, 4096 152 and 288 -> 282; up to 4096 tokens one wave stays the choice.
static int mhc_token_splits(long long groups, int groups_per_cta, int col_blocks) {
  const long long slots = sm_count();
  const long long rounds = (groups + groups_per_cta - 1) / groups_per_cta;
  const long long most = slots / col_blocks > 64 ? slots / col_blocks : 64;
  long long splits = 1, least = -1, least_waves = 0;
  for (long long s = 1; s <= rounds && s <= most; ++s) {
    const long long waves = (s * col_blocks + slots - 1) / slots;
    const long long cost = waves * ((rounds + s - 1) / s + 1);
    if (least < 0 || cost < least || (cost == least && waves == least_waves)) {  // of equal ones in a wave, the most CTAs
      least = cost;
      least_waves = waves;
      splits = s;
    }
  }
  return static_cast<int>(splits);
}

// Four warps share a token group's columns while one warp each would leave most of the chip without work, which costs
// them a meeting per token group. The whole forward with one warp / four, nothing in L2: hidden 512, 512 tokens (128 pairs
// of a token group and a column block) 27.2 / 18.7 us; 2560, 384 tokens (480) 29.4 / 24.9; 7168, 128 tokens (448) 25.6 /
// 26.0, 200 tokens (728) 30.2 / 30.9, 256 tokens (896) 30.6 / 33.0, 384 tokens (1344) 32.2 / 33.5.
bool mhc_share_columns(long long tokens, long long hidden) {
  return (tokens + 15) / 16 * (hidden / BLOCK_COLS) <= 6ll * sm_count();
}

}  // namespace hmc

using namespace hmc;

extern "C" int64_t hmc_mega_mhc_workspace_bytes(int64_t tokens, int64_t hidden) {
  return hidden / BLOCK_COLS * tokens * PART * 4 + 256;  // partial sums [hidden / 128][tokens][28] f32
}

namespace hmc {
int check_mhc_dims(const char* what, int64_t tokens, int64_t hidden, int32_t num_iters) {
  HMC_REQUIRE(tokens > 0 && tokens < (1ll << 31) / 16, HMC_ERR_INVALID, "%s: token count %lld out of range", what,
              (long long)tokens);
  // hidden % 128 == 0 is the reference's rule (hyper_multicore/modules/mega_mhc_common.py:100-118);
  // its upper bounds on hidden are Ascend buffer limits and do not apply here.
  HMC_REQUIRE(hidden > 0 && hidden % 128 == 0, HMC_ERR_INVALID, "%s: hidden size (%lld) must be a multiple of 128",
              what, (long long)hidden);
  HMC_REQUIRE(num_iters >= 1 && num_iters <= 20, HMC_ERR_INVALID, "%s: num_iters must be in [1, 20], got %d", what,
              num_iters);
  return 0;
}
}  // namespace hmc

extern "C" int hmc_mega_mhc(const hmc_mega_mhc_args* args, void* stream_ptr) {
  HMC_REQUIRE(args != nullptr, HMC_ERR_INVALID, "hmc_mega_mhc: null args");
  const hmc_mega_mhc_args& a = *args;
  int rc = check_mhc_dims("hmc_mega_mhc", a.tokens, a.hidden, a.num_iters);
  if (rc != 0) return rc;
  HMC_REQUIRE(a.previous_output && a.residual && a.previous_pre_mix && a.previous_post_mix &&
                  a.previous_residual_mix && a.phi && a.alpha && a.bias && a.norm_weight && a.new_residual &&
                  a.next_pre_mix && a.next_post_mix && a.next_residual_mix && a.block_input && a.inv_rms &&
                  a.mixed_input && a.rms_rstd && a.workspace,
              HMC_ERR_INVALID, "hmc_mega_mhc: null tensor pointer");
  HMC_REQUIRE(a.workspace_bytes >= hmc_mega_mhc_workspace_bytes(a.tokens, a.hidden), HMC_ERR_INVALID,
              "hmc_mega_mhc: workspace holds %lld bytes, %lld needed", (long long)a.workspace_bytes,
              (long long)hmc_mega_mhc_workspace_bytes(a.tokens, a.hidden));
  HMC_REQUIRE(aligned16(a.previous_output) && aligned16(a.residual) && aligned16(a.new_residual) &&
                  aligned16(a.block_input) && aligned16(a.mixed_input) && aligned16(a.norm_weight) &&
                  aligned16(a.workspace),
              HMC_ERR_INVALID, "hmc_mega_mhc: activations must be 16-byte aligned");
  cudaStream_t stream = static_cast<cudaStream_t>(stream_ptr);
  const int col_blocks = static_cast<int>(a.hidden / BLOCK_COLS);
  StreamParams p{};
  p.prev_out = static_cast<const uint4*>(a.previous_output);
  p.residual = static_cast<const uint4*>(a.residual);
  p.prev_pre = a.previous_pre_mix;
  p.prev_post = a.previous_post_mix;
  p.prev_mix = a.previous_residual_mix;
  p.phi = a.phi;
  p.tokens = a.tokens;
  p.hidden = static_cast<int>(a.hidden);
  p.phi_vec = aligned16(a.phi);
  p.coef_vec = aligned16(a.previous_pre_mix) && aligned16(a.previous_post_mix) && aligned16(a.previous_residual_mix);
  p.new_residual = static_cast<uint4*>(a.new_residual);
  p.mixed_input = static_cast<uint4*>(a.mixed_input);
  p.parts = static_cast<float*>(a.workspace);
  const bool share = mhc_share_columns(a.tokens, a.hidden);
  const int groups_per_cta = share ? stream_warps(1) / COL_STEPS : stream_warps(COL_STEPS);
  const dim3 grid(static_cast<unsigned>(col_blocks),
                  static_cast<unsigned>(mhc_token_splits((a.tokens + 15) / 16, groups_per_cta, col_blocks)));
  static PerDeviceFlag configured{}, configured_share{};
  if (share) {
    if ((rc = allow_dynamic_smem(mhc_stream_kernel<1>, stream_smem(1), configured_share)) != 0) return rc;
    mhc_stream_kernel<1><<<grid, 32 * stream_warps(1), stream_smem(1), stream>>>(p);
  } else {
    if ((rc = allow_dynamic_smem(mhc_stream_kernel<COL_STEPS>, stream_smem(COL_STEPS), configured)) != 0) return rc;
    mhc_stream_kernel<COL_STEPS><<<grid, 32 * stream_warps(COL_STEPS), stream_smem(COL_STEPS), stream>>>(p);
  }
  HMC_LAUNCH_OK();

  FinishParams f{};
  f.parts = p.parts;
  f.mixed_input = static_cast<const uint4*>(a.mixed_input);
  f.norm_weight = static_cast<const uint4*>(a.norm_weight);
  f.alpha = a.alpha;
  f.bias = a.bias;
  f.tokens = a.tokens;
  f.hidden = p.hidden;
  f.part_rows = col_blocks;
  f.norm_eps = a.norm_eps;
  f.hc_eps = a.hc_eps;
  f.iters = a.num_iters;
  f.block_input = static_cast<uint4*>(a.block_input);
  f.inv_rms = a.inv_rms;
  f.rms_rstd = a.rms_rstd;
  f.next_pre = a.next_pre_mix;
  f.next_post = a.next_post_mix;
  f.next_mix = a.next_residual_mix;
  f.hc_before_norm = a.hc_before_norm;
  f.sum_out = a.need_backward ? a.sum_out : nullptr;
  f.norm_out = a.need_backward ? a.norm_out : nullptr;
  // eight warps per token / one, whole forward: hidden 7168, 16 tokens 14.4 / 21.4 us, 512 tokens 37.0 / 41.1, 768 tokens
  // 52.0 / 51.3; hidden 512, 512 tokens 13.2 / 13.6, 768 tokens 19.1 / 15.1
  if (a.tokens <= 4ll * sm_count())
    mhc_finish_kernel<8><<<static_cast<unsigned>(a.tokens), 256, 0, stream>>>(f);
  else
    mhc_finish_kernel<1><<<static_cast<unsigned>((a.tokens + 7) / 8), 256, 0, stream>>>(f);
  HMC_LAUNCH_OK();
  return 0;
}
