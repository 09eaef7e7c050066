// Backward of the router projection, logits[T, E] = float(x[T, H]) . float(W[E, H])^T, for BF16 hidden states:
//   grad_hidden[T, H] = bf16(grad_logits . W)      grad_weight[E, H] = grad_logits^T . float(x)
// (hyper_multicore/modules/mega_gate/function.py:175-178 differentiates the FP32 matmul.)
//
// Both are contractions of 2 T E H operations that FP32 cores would spend a millisecond on at 8192 x 256 x 7168. On the
// tensor cores the FP32 operands travel as BF16 parts:
//  - grad_weight is FP32, so the gradient of the logits is split into three parts (24 bits, every product exact) and
//    the accumulation chain is promoted every 128 tokens, as in the forward projection (gate_promoted.cu);
//  - grad_hidden takes three parts of both operands and every product down to 2^-16 of hi.hi (hi.lo, mid.mid and lo.hi;
//    what is left out, 2^-24, is FP32's own rounding of a product): a gradient whose terms cancel - those of a softmax sum
//    to zero over the experts, which takes out all that the expert rows share - shows the error of the terms and not that
//    of the sum. The parts are stacked along K and go through the grouped GEMM once, the small products first, so that
//    the accumulator is small while it takes them and only the last sixth of the chain rounds at full magnitude.
// At 8192 tokens x 256 experts x hidden 7168 with an FP32 weight: two FP32 matmuls of 587 and 566 us and 212 us of
// conversions before, 142 us (grad_hidden; with two parts each and three products 84 us, at 15 to 28 times the error of
// an FP32 matmul), 125 us (grad_weight) and 21 us of splitting now.
#include "common.cuh"

namespace hmc {

int gate_weight_grad(const void* x_bf16, const void* parts, int64_t tokens, int64_t hidden, int64_t experts, int64_t epad,
                     float* grad_weight, int32_t* status, cudaStream_t stream);  // gate_promoted.cu

namespace {

constexpr int FP32_COPIES = 6, BF16_COPIES = 3;  // products of an FP32 / BF16 weight, stacked along K

// An infinity or a NaN is all in `hi`, and a finite value that would round up to infinity keeps the largest BF16 number
// there. `finite_hi` is what the smaller products are made with: an infinity times a part that is zero is no number, and
// times one of the other sign the wrong infinity, so it may meet nothing but the other side's `hi`.
struct Split3 {
  __nv_bfloat16 hi, mid, lo, finite_hi;
};

__device__ __forceinline__ Split3 split3(float v) {
  Split3 s;
  s.hi = __float2bfloat16_rn(v);
  if (!isfinite(v)) {
    s.mid = s.lo = s.finite_hi = __float2bfloat16_rn(0.f);
    return s;
  }
  if (!isfinite(__bfloat162float(s.hi))) s.hi = __float2bfloat16_rz(v);
  s.finite_hi = s.hi;
  const float r = v - __bfloat162float(s.hi);
  s.mid = __float2bfloat16_rn(r);
  s.lo = __float2bfloat16_rn(r - __bfloat162float(s.mid));
  return s;
}

// One thread per (token, expert of the padded width): the parts of the gradient in the two layouts, each optional.
//   cols [T, 3 * epad] = hi | mid | lo
//   rows [T, copies * e8] = lo | hi | mid | mid | hi | hi, or lo | mid | hi for a BF16 weight
__global__ void __launch_bounds__(256)
gate_grad_parts_kernel(const float* __restrict__ grad, long long tokens, int experts, int epad, int e8, int copies,
                       __nv_bfloat16* __restrict__ cols, __nv_bfloat16* __restrict__ rows, long long* __restrict__ ends) {
  const long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i == 0) *ends = tokens;
  if (i >= tokens * epad) return;
  const long long t = i / epad;
  const int e = static_cast<int>(i - t * epad);
  const Split3 s = split3(e < experts ? grad[t * experts + e] : 0.f);
  if (cols != nullptr) {
    __nv_bfloat16* dst = cols + t * 3 * epad + e;
    dst[0] = s.hi;
    dst[epad] = s.mid;
    dst[2 * epad] = s.lo;
  }
  if (rows != nullptr && e < e8) {
    __nv_bfloat16* dst = rows + t * copies * e8 + e;
    dst[0] = s.lo;
    if (copies == FP32_COPIES) {
      dst[e8] = s.finite_hi;
      dst[2 * e8] = s.mid;
      dst[3 * e8] = s.mid;
      dst[4 * e8] = s.finite_hi;
    } else {
      dst[e8] = s.mid;
    }
    dst[(copies - 1) * e8] = s.hi;
  }
}

// W [E, H] stacked along K to meet `rows` above: hi, lo, mid, hi, mid, hi of an FP32 weight, three times a BF16 one.
__global__ void __launch_bounds__(256)
gate_grad_weight_parts_kernel(const void* __restrict__ w, int w_is_bf16, int experts, int e8, long long hidden,
                              __nv_bfloat16* __restrict__ stacked) {
  const long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= e8 * hidden) return;
  float v = 0.f;
  if (i < experts * hidden)
    v = w_is_bf16 ? __bfloat162float(static_cast<const __nv_bfloat16*>(w)[i]) : static_cast<const float*>(w)[i];
  const Split3 s = split3(v);
  const long long part = e8 * hidden;
  stacked[i] = s.finite_hi;
  stacked[part + i] = w_is_bf16 ? s.finite_hi : s.lo;
  stacked[2 * part + i] = w_is_bf16 ? s.hi : s.mid;
  if (w_is_bf16) return;
  stacked[3 * part + i] = s.finite_hi;
  stacked[4 * part + i] = s.mid;
  stacked[5 * part + i] = s.hi;
}

struct GradLayout {
  int64_t epad, e8, cols, rows, stacked, bytes;
};

GradLayout grad_layout(int64_t tokens, int64_t hidden, int64_t experts) {
  GradLayout l;
  auto up = [](int64_t v) { return (v + 255) / 256 * 256; };
  l.epad = (experts + 63) / 64 * 64;
  l.e8 = (experts + 7) / 8 * 8;
  l.cols = 256;  // the group end sits in front
  l.rows = l.cols + up(tokens * 3 * l.epad * 2);
  l.stacked = l.rows + up(tokens * FP32_COPIES * l.e8 * 2);
  l.bytes = l.stacked + up(FP32_COPIES * l.e8 * hidden * 2);
  return l;
}

}  // namespace
}  // namespace hmc

extern "C" int64_t hmc_gate_project_grad_workspace_bytes(int64_t tokens, int64_t hidden, int64_t experts) {
  return hmc::grad_layout(tokens, hidden, experts).bytes;
}

extern "C" int hmc_gate_project_grad(const float* grad_logits, const void* x_bf16, const void* w, int w_is_bf16,
                                     int64_t tokens, int64_t hidden, int64_t experts, void* grad_hidden_bf16,
                                     float* grad_weight, void* workspace, int64_t workspace_bytes, int32_t* status,
                                     void* stream_ptr) {
  using namespace hmc;
  HMC_REQUIRE(grad_logits && workspace && (x_bf16 || !grad_weight) && (w || !grad_hidden_bf16), HMC_ERR_INVALID,
              "hmc_gate_project_grad: null tensor pointer");
  HMC_REQUIRE(tokens > 0 && experts > 0 && hidden > 0 && hidden % 8 == 0, HMC_ERR_INVALID,
              "hmc_gate_project_grad: extents must be positive and hidden a multiple of 8");
  HMC_REQUIRE(tokens < (1ll << 31) && hidden < (1ll << 31) && experts <= 65536, HMC_ERR_LIMIT,
              "hmc_gate_project_grad: extent too large");
  HMC_REQUIRE(aligned16(x_bf16) && aligned16(grad_hidden_bf16) && aligned16(workspace), HMC_ERR_INVALID,
              "hmc_gate_project_grad: 16-byte alignment");
  const GradLayout l = grad_layout(tokens, hidden, experts);
  HMC_REQUIRE(workspace_bytes >= l.bytes, HMC_ERR_INVALID, "hmc_gate_project_grad: workspace holds %lld bytes, %lld needed",
              (long long)workspace_bytes, (long long)l.bytes);
  cudaStream_t stream = static_cast<cudaStream_t>(stream_ptr);
  uint8_t* ws = static_cast<uint8_t*>(workspace);
  const int copies = w_is_bf16 ? BF16_COPIES : FP32_COPIES;
  __nv_bfloat16* cols = reinterpret_cast<__nv_bfloat16*>(ws + l.cols);
  __nv_bfloat16* rows = reinterpret_cast<__nv_bfloat16*>(ws + l.rows);
  __nv_bfloat16* stacked = reinterpret_cast<__nv_bfloat16*>(ws + l.stacked);
  const long long items = tokens * l.epad;
  gate_grad_parts_kernel<<<static_cast<unsigned>((items + 255) / 256), 256, 0, stream>>>(
      grad_logits, tokens, static_cast<int>(experts), static_cast<int>(l.epad), static_cast<int>(l.e8), copies,
      grad_weight ? cols : nullptr, grad_hidden_bf16 ? rows : nullptr, reinterpret_cast<long long*>(ws));
  HMC_LAUNCH_OK();
  if (grad_hidden_bf16 != nullptr) {
    const long long split = l.e8 * hidden;
    gate_grad_weight_parts_kernel<<<static_cast<unsigned>((split + 255) / 256), 256, 0, stream>>>(
        w, w_is_bf16, static_cast<int>(experts), static_cast<int>(l.e8), hidden, stacked);
    HMC_LAUNCH_OK();
    hmc_grouped_gemm_args g{};
    g.mode = HMC_GEMM_RAGGED_M;
    g.a_major = HMC_MAJOR_K;
    g.b_major = HMC_MAJOR_MN;
    g.epilogue = HMC_EPI_STORE_BF16;
    g.groups = 1;
    g.tile_mode = HMC_TILE_SINGLE;  // few k-blocks per tile: the store path decides, and 128-row tiles store by TMA
    g.rows = tokens;
    g.n = hidden;
    g.k = copies * l.e8;
    g.a = rows;
    g.b = stacked;
    g.c = grad_hidden_bf16;
    g.group_ends = reinterpret_cast<const int64_t*>(ws);
    g.status = status;
    int rc = hmc_grouped_gemm(&g, stream);
    if (rc != 0) return rc;
  }
  if (grad_weight != nullptr) return gate_weight_grad(x_bf16, cols, tokens, hidden, experts, l.epad, grad_weight, status, stream);
  return 0;
}
