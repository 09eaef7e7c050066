"""Typed Python entry points over the C ABI: one function per ``hmc_*`` kernel.

Every function takes CUDA tensors the caller allocated, checks nothing the native side already
checks, and enqueues on torch's current stream.
"""

from __future__ import annotations

import ctypes
import os

import torch

from . import _lib
from ._lib import (HMC_EPI_STORE_BF16, HMC_EPI_STORE_F32, HMC_EPI_SWIGLU, HMC_EPI_SWIGLU_GRAD, HMC_EPI_SWIGLU_GRAD_MXQ, HMC_EPI_SWIGLU_MXQ,
                   HMC_GEMM_RAGGED_K, HMC_GEMM_RAGGED_M, HMC_MAJOR_K, HMC_MAJOR_MN, GroupedGemmArgs)


def _require_cuda(*tensors: torch.Tensor | None) -> torch.device:
    device = None
    for tensor in tensors:
        if tensor is None:
            continue
        if not tensor.is_cuda:
            raise _lib.HmcError("hyper_multicore_b200 kernels need CUDA tensors; there is no CPU path")
        device = tensor.device if device is None else device
        if tensor.device != device:
            raise ValueError("all tensors must be on one CUDA device")
    assert device is not None
    return device


def grouped_gemm(
    a: torch.Tensor,
    b: torch.Tensor,
    c: torch.Tensor,
    group_ends: torch.Tensor,
    *,
    mode: int,
    b_major: int = HMC_MAJOR_MN,
    epilogue: int = HMC_EPI_STORE_BF16,
    aux: torch.Tensor | None = None,
    ready_counters: torch.Tensor | None = None,
    ready_budget_ns: int = 0,
    status: torch.Tensor | None = None,
    max_ctas: int = 0,
    tile_mode: int = 0,
    swiglu_clamp: int = 0,
    swiglu_limit: float = 0.0,
    row_probs: torch.Tensor | None = None,
    row_dot: torch.Tensor | None = None,
    combine: dict | None = None,
    pipe_budget_ns: int = 0,
    dispatch: dict | None = None,
) -> None:
    """Launch the tcgen05 grouped GEMM.

    ``swiglu_clamp`` / ``swiglu_limit`` select the clamped SwiGLU of the SwiGLU epilogues;
    ``row_probs`` (float32 [rows]) weights the activation before FC2 and, in the SwiGLU-grad
    epilogue, ``row_dot`` (float32 [rows], zeroed by the caller) receives the probability gradient.
    ``combine`` (RAGGED_M, BF16 stores) sends the result rows from the epilogue to the routed buffers of
    their source ranks: keys segment_start, combine_target_off (device int64), peer_buffers, peer_ctrl
    (ctypes pointer arrays), ep, local_experts, target_rows_limit; ``c`` may then be None.

    ``dispatch`` (RAGGED_M with ``ready_counters``): the keyword arguments of ``ep_dispatch`` plus ``rank``;
    extra warps of the GEMM then send this rank's rows while its tiles wait for the rows it receives.

    RAGGED_M: ``a`` [rows, k]; ``b`` [groups, k, n_cols] (MN) or [groups, n_cols, k] (K); ``c`` [rows, *].
    RAGGED_K: ``a`` [rows, m]; ``b`` [rows, n]; ``c`` [groups, m, n] BF16 or FP32.
    """
    device = _require_cuda(a, b, c, group_ends, aux, status, row_probs, row_dot)
    if ready_counters is not None and not (ready_counters.is_cuda or ready_counters.is_pinned()):
        raise ValueError("ready_counters must live in device memory or in pinned (device-visible) host memory")
    if c is None and combine is None:
        raise ValueError("grouped_gemm needs an output tensor unless its rows are combined to their sources")
    for name, plane in (("row_probs", row_probs), ("row_dot", row_dot)):
        if plane is not None and (plane.dtype != torch.float32 or not plane.is_contiguous() or plane.numel() < a.shape[0]):
            raise ValueError(f"{name} must be a contiguous float32 tensor with one entry per row")
    args = GroupedGemmArgs()
    args.mode = mode
    args.epilogue = epilogue
    args.groups = group_ends.numel()
    args.max_ctas = max_ctas
    args.tile_mode = tile_mode
    args.rows = a.shape[0]
    if mode == HMC_GEMM_RAGGED_M:
        args.a_major = HMC_MAJOR_K
        args.b_major = b_major
        args.k = a.shape[1]
        n_cols = b.shape[2] if b_major == HMC_MAJOR_MN else b.shape[1]
        args.n = n_cols // 2 if epilogue == HMC_EPI_SWIGLU else n_cols
        args.m = 0
    else:
        args.a_major = HMC_MAJOR_MN
        args.b_major = HMC_MAJOR_MN
        args.m = a.shape[1]
        args.n = b.shape[1]
        args.k = 0
    args.a = a.data_ptr()
    args.b = b.data_ptr()
    args.c = _lib.ptr(c)
    args.aux = _lib.ptr(aux)
    args.group_ends = group_ends.data_ptr()
    args.ready_counters = _lib.ptr(ready_counters)
    args.ready_budget_ns = ready_budget_ns
    args.status = _lib.ptr(status)
    args.swiglu_clamp = swiglu_clamp
    args.swiglu_limit = swiglu_limit
    args.row_probs = _lib.ptr(row_probs)
    args.row_dot = _lib.ptr(row_dot)
    args.pipe_budget_ns = pipe_budget_ns
    fused = None
    if combine is not None:
        fused = _lib.GemmCombine()
        fused.segment_start = combine["segment_start"].data_ptr()
        fused.combine_target_off = combine["combine_target_off"].data_ptr()
        fused.peer_buffers = ctypes.cast(combine["peer_buffers"], ctypes.c_void_p)
        fused.peer_ctrl = ctypes.cast(combine["peer_ctrl"], ctypes.c_void_p)
        fused.ep, fused.local_experts = combine["ep"], combine["local_experts"]
        fused.target_rows_limit = combine["target_rows_limit"]
        args.combine = ctypes.cast(ctypes.pointer(fused), ctypes.c_void_p)
    sending = None
    if dispatch is not None:
        sending = _dispatch_struct(**dispatch)
        args.dispatch = ctypes.cast(ctypes.pointer(sending), ctypes.c_void_p)
    _lib.launch("hmc_grouped_gemm", device, ctypes.byref(args))


def store_words(dst: torch.Tensor, src: torch.Tensor) -> None:
    """dst[:] = src for int32 tensors, by a kernel. ``dst`` may be pinned host memory: the read-back then
    does not wait behind bulk device-to-host copies queued in a copy engine."""
    if dst.dtype != torch.int32 or src.dtype != torch.int32 or dst.numel() < src.numel():
        raise ValueError("store_words copies int32 words into a tensor at least as large")
    if not (dst.is_cuda or dst.is_pinned()):
        raise ValueError("store_words writes device or pinned host memory")
    device = _require_cuda(src)
    _call("hmc_store_words", device, dst.data_ptr(), src.data_ptr(), src.numel())


def grouped_gemm_combine_units(n: int) -> int:
    """Counter increments per result row of a fused-combine GEMM with ``n`` output columns."""
    return int(_lib.load().hmc_grouped_gemm_combine_units(n))


_call = _lib.launch


# ------------------------------------------------------------------------------------------- gate
_GATE_DEFAULT = "1"  # promoted tcgen05 projection for eligible inputs; HMC_GATE_TENSOR_CORES=0 selects FP32 FMAs


def gate_project(x: torch.Tensor, weight: torch.Tensor, use_tensor_cores: bool | str | None = None) -> torch.Tensor:
    """FP32 logits [T, E] = float(x [T, H]) @ float(weight [E, H]).T.

    BF16 hidden states (at least 128 tokens, H a multiple of 8) go through tcgen05 with the weight split
    into three BF16 parts and the accumulation chain of the dominant part cut every 128 elements of K
    ("promoted"); everything else, or ``use_tensor_cores=False`` / HMC_GATE_TENSOR_CORES=0, takes the FP32-FMA
    kernel. ``use_tensor_cores="unpromoted"`` (HMC_GATE_TENSOR_CORES=unpromoted) is the three-GEMM variant
    whose full-length accumulation leaves about 2e-5 absolute error at H = 4096.
    """
    if use_tensor_cores is None:
        use_tensor_cores = {"0": False, "1": True}.get(os.environ.get("HMC_GATE_TENSOR_CORES", _GATE_DEFAULT),
                                                       os.environ.get("HMC_GATE_TENSOR_CORES"))
    device = _require_cuda(x, weight)
    for name, tensor in (("hidden states", x), ("weight", weight)):
        if tensor.dtype not in (torch.bfloat16, torch.float32):
            raise TypeError(f"MegaGate {name} must be BF16 or FP32, got {tensor.dtype}")
    x = x.contiguous()
    weight = weight.contiguous()
    logits = torch.empty((x.shape[0], weight.shape[0]), dtype=torch.float32, device=device)
    eligible = x.dtype == torch.bfloat16 and x.shape[1] % 8 == 0 and x.shape[0] >= 128
    if eligible and use_tensor_cores == "unpromoted":
        need = _lib.load().hmc_gate_project_workspace_bytes(x.shape[0], x.shape[1], weight.shape[0])
        workspace = torch.empty(need, dtype=torch.uint8, device=device)
        _call("hmc_gate_project_tc", device, x.data_ptr(), weight.data_ptr(), int(weight.dtype == torch.bfloat16),
              x.shape[0], x.shape[1], weight.shape[0], logits.data_ptr(), workspace.data_ptr(), need)
        return logits
    if eligible and use_tensor_cores:
        workspace = _gate_weight_parts(x.shape[1], weight.shape[0], device)
        _call("hmc_gate_project_promoted", device, x.data_ptr(), weight.data_ptr(), int(weight.dtype == torch.bfloat16),
              x.shape[0], x.shape[1], weight.shape[0], logits.data_ptr(), workspace.data_ptr(), workspace.numel(), None)
        return logits
    _call("hmc_gate_project", device, x.data_ptr(), int(x.dtype == torch.bfloat16), weight.data_ptr(),
          int(weight.dtype == torch.bfloat16), x.shape[0], x.shape[1], weight.shape[0], logits.data_ptr())
    return logits


def _gate_weight_parts(hidden: int, experts: int, device: torch.device) -> torch.Tensor:
    """Workspace for the BF16 parts of a weight. Every call splits the weight it is given (2.6 us for 64 x 4096): writes
    through ``.data``, as optimisers and sharded training make them, leave no trace on the tensor that would tell parts
    kept from an earlier call from current ones."""
    return torch.empty(_lib.load().hmc_gate_project_promoted_workspace_bytes(hidden, experts), dtype=torch.uint8, device=device)


# The longest chain whose error on the tensor cores is not above the FP32 matmul's: relative error before the rounding to
# BF16 with rows of random numbers / with rows that share a component 100 times as large, tensor cores against matmul:
# 8 experts 4.9e-8 and 5.4e-8 / 1.2e-6 and 3.1e-6, 64 7.7e-8 and 1.4e-7 / 3.3e-6 and 8.5e-6, 256 2.3e-7 and 2.9e-7 /
# 5.9e-6 and 1.7e-5, 512 4.7e-7 and 4.1e-7 / 9.8e-6 and 2.3e-5, 1024 9.9e-7 and 5.7e-7 / 2.1e-5 and 3.3e-5.
_GATE_GRAD_EXPERTS = 256


def gate_project_grad(grad_logits: torch.Tensor, x: torch.Tensor, weight: torch.Tensor, need_hidden: bool, need_weight: bool):
    """Gradients of ``gate_project`` with respect to the hidden states (their dtype) and the weight (its dtype).

    BF16 hidden states take the tensor cores (``hmc_gate_project_grad``); FP32 ones, row lengths that are no multiple of
    8 and HMC_GATE_TENSOR_CORES other than its default the FP32 matmuls, as do a backward that is itself recorded, a
    gradient that is not simply its memory (one batched by vmap, ``is_grads_batched``, or a lazy negation), and the hidden
    states' gradient of more than 256 experts.
    """
    x_rows = x.contiguous()
    functorch = torch._C._functorch  # pylint: disable=protected-access
    plain = not (functorch.is_legacy_batchedtensor(grad_logits) or functorch.is_functorch_wrapped_tensor(grad_logits)
                 or grad_logits.is_neg())
    if not (plain and os.environ.get("HMC_GATE_TENSOR_CORES", _GATE_DEFAULT) == "1" and x.is_cuda and x.dtype == torch.bfloat16
            and x.ndim == 2 and x.shape[1] % 8 == 0 and x_rows.data_ptr() % 16 == 0
            and weight.dtype in (torch.bfloat16, torch.float32) and weight.shape[0] <= 65536 and not torch.is_grad_enabled()):
        return ((grad_logits @ weight.float()).to(x.dtype) if need_hidden else None,
                (grad_logits.t() @ x.float()).to(weight.dtype) if need_weight else None)
    grad_logits = grad_logits.float().contiguous()
    device = _require_cuda(grad_logits, x_rows, weight)
    weight_rows = weight.contiguous()
    (tokens, hidden), experts = x.shape, weight.shape[0]
    if need_hidden and experts > _GATE_GRAD_EXPERTS:
        plain_hidden = (grad_logits @ weight.float()).to(x.dtype)
        return plain_hidden, gate_project_grad(grad_logits, x, weight, False, True)[1] if need_weight else None
    grad_hidden = torch.empty_like(x_rows) if need_hidden else None
    grad_weight = torch.empty(weight.shape, dtype=torch.float32, device=device) if need_weight else None
    need = _lib.load().hmc_gate_project_grad_workspace_bytes(tokens, hidden, experts)
    workspace = torch.empty(need, dtype=torch.uint8, device=device)
    _call("hmc_gate_project_grad", device, grad_logits.data_ptr(), x_rows.data_ptr(), weight_rows.data_ptr(),
          int(weight.dtype == torch.bfloat16), tokens, hidden, experts, _lib.ptr(grad_hidden), _lib.ptr(grad_weight),
          workspace.data_ptr(), need, None)
    return grad_hidden, grad_weight.to(weight.dtype) if need_weight else None


def gate_route_fusable(x: torch.Tensor, weight: torch.Tensor, n_group: int = 0) -> bool:
    """True when projection and Route run as one launch (``gate_project_route``): BF16 hidden states that take
    the promoted tcgen05 projection, at most 64 experts, no group limit."""
    if os.environ.get("HMC_GATE_TENSOR_CORES", _GATE_DEFAULT) != "1" or os.environ.get("HMC_GATE_FUSED_ROUTE", "1") != "1":
        return False
    if not (x.is_cuda and x.dtype == torch.bfloat16 and x.ndim == 2 and x.shape[1] % 8 == 0 and x.shape[0] >= 128):
        return False
    if weight.dtype not in (torch.bfloat16, torch.float32):
        return False
    return bool(_lib.load().hmc_gate_project_route_supported(weight.shape[0], n_group))


def _gate_route_state(tokens: int, experts: int, top_k: int, device: torch.device, keep: bool):
    """The Route's outputs that only its backward reads: route_scores [T, E], selected [T, K], denominator [T, 1]. One
    allocation for a forward that keeps none of them (``keep`` False), whose views the caller drops."""
    f32 = {"dtype": torch.float32, "device": device}
    if keep:
        return torch.empty((tokens, experts), **f32), torch.empty((tokens, top_k), **f32), torch.empty((tokens, 1), **f32)
    return torch.empty(tokens * (experts + top_k + 1), **f32).split((tokens * experts, tokens * top_k, tokens))


def gate_project_route(x, weight, text_bias, vision_bias, image_mask, use_vision_bias, top_k, scale, scoring,
                       keep_state: bool = True):
    """Projection and Route in one launch; the caller checks ``gate_route_fusable`` first.

    Returns (logits [T, E], weights [T, K], indices [T, K] int64, route_scores [T, E], selected [T, K],
    denominator [T, 1]), bit for bit what ``gate_project`` followed by ``gate_route_out`` produce.
    """
    device = _require_cuda(x, weight, text_bias, vision_bias)
    x = x.contiguous()
    weight = weight.contiguous()
    tokens, experts = x.shape[0], weight.shape[0]
    f32 = {"dtype": torch.float32, "device": device}
    logits = torch.empty((tokens, experts), **f32)
    weights = torch.empty((tokens, top_k), **f32)
    indices = torch.empty((tokens, top_k), dtype=torch.int64, device=device)
    scores, selected, denominator = _gate_route_state(tokens, experts, top_k, device, keep_state)
    args = _lib.GateRouteArgs()
    args.logits = None
    args.text_bias = text_bias.data_ptr()
    args.vision_bias = vision_bias.data_ptr()
    args.image_mask = _lib.ptr(image_mask) if use_vision_bias else None
    args.use_vision_bias = int(bool(use_vision_bias))
    args.experts = experts
    args.top_k = top_k
    args.scoring = _lib.HMC_SCORE[scoring]
    args.tokens = tokens
    args.scale = scale
    args.weights = weights.data_ptr()
    args.indices = indices.data_ptr()
    args.route_scores = scores.data_ptr()
    args.selected = selected.data_ptr()
    args.denominator = denominator.data_ptr()
    args.n_group, args.topk_group = 0, 0
    workspace = _gate_weight_parts(x.shape[1], experts, device)
    _call("hmc_gate_project_route", device, x.data_ptr(), weight.data_ptr(), int(weight.dtype == torch.bfloat16), x.shape[1],
          logits.data_ptr(), workspace.data_ptr(), workspace.numel(), ctypes.byref(args), None)
    return logits, weights, indices, scores, selected, denominator


def gate_route_out(logits, text_bias, vision_bias, image_mask, use_vision_bias, top_k, scale, scoring,
                   weights, indices, route_scores, selected, denominator, n_group=0, topk_group=0) -> None:
    """Top-k Route on FP32 logits into caller-owned outputs (``n_group`` > 0: group-limited selection)."""
    device = _require_cuda(logits, text_bias, vision_bias, weights, indices, route_scores, selected, denominator)
    args = _lib.GateRouteArgs()
    args.logits = logits.data_ptr()
    args.text_bias = text_bias.data_ptr()
    args.vision_bias = vision_bias.data_ptr()
    args.image_mask = _lib.ptr(image_mask) if use_vision_bias else None
    args.use_vision_bias = int(bool(use_vision_bias))
    args.experts = logits.shape[1]
    args.top_k = top_k
    args.scoring = _lib.HMC_SCORE[scoring]
    args.tokens = logits.shape[0]
    args.scale = scale
    args.weights = weights.data_ptr()
    args.indices = indices.data_ptr()
    args.route_scores = route_scores.data_ptr()
    args.selected = selected.data_ptr()
    args.denominator = denominator.data_ptr()
    args.n_group, args.topk_group = n_group, topk_group
    _call("hmc_gate_route", device, ctypes.byref(args))


def gate_route_grad_out(logits, route_scores, selected, denominator, indices, grad_weights, top_k, scale,
                        scoring, grad_logits, status=None) -> None:
    """RouteGrad into a caller-owned FP32 [T, E] gradient."""
    device = _require_cuda(logits, route_scores, selected, denominator, indices, grad_weights, grad_logits)
    args = _lib.GateRouteGradArgs()
    args.logits = logits.data_ptr()
    args.route_scores = route_scores.data_ptr()
    args.selected = selected.data_ptr()
    args.denominator = denominator.data_ptr()
    args.indices = indices.data_ptr()
    args.grad_weights = grad_weights.data_ptr()
    args.experts = logits.shape[1]
    args.top_k = top_k
    args.scoring = _lib.HMC_SCORE[scoring]
    args.tokens = logits.shape[0]
    args.scale = scale
    args.grad_logits = grad_logits.data_ptr()
    args.status = _lib.ptr(status)
    _call("hmc_gate_route_grad", device, ctypes.byref(args))


# ------------------------------------------------------------------------------------ route prep
def moe_histogram(indices: torch.Tensor, experts: int, status=None) -> torch.Tensor:
    """INT32 histogram of expert ids."""
    device = _require_cuda(indices)
    flat = indices.reshape(-1).contiguous()
    counts = torch.empty(experts, dtype=torch.int32, device=device)
    _call("hmc_moe_histogram", device, flat.data_ptr(), int(flat.dtype == torch.int64), flat.numel(), experts,
          counts.data_ptr(), _lib.ptr(status))
    return counts


def _carve_words(device: torch.device, *words: int) -> list[torch.Tensor]:
    """Int32 tensors of the given lengths out of one allocation, each on a 256-byte boundary: a call of the route
    preparation has sixteen small tensors, and an allocation costs the host more than a view."""
    padded = [-(-n // 64) * 64 for n in words]
    pieces = torch.empty(sum(padded), dtype=torch.int32, device=device).split(padded)
    return [piece if piece.numel() == n else piece[:n] for piece, n in zip(pieces, words)]


def moe_sort_routes(indices: torch.Tensor, experts: int, *, want_sources: bool = True, status=None):
    """Stable expert-major sort of the flat (token, slot) routes.

    Returns (mapping[T*K] i32, source_of_row[T*K] i32 | None, expert_of_row | None, counts[E] i32,
    cumulative[E] i64).
    """
    device = _require_cuda(indices)
    if indices.dtype not in (torch.int32, torch.int64):
        raise TypeError(f"expert indices must be int32 or int64, got {indices.dtype}")
    flat = indices.reshape(-1).contiguous()
    entries = flat.numel()
    lib = _lib.load()
    need = max(1, lib.hmc_moe_sort_workspace_bytes(entries, experts))
    workspace, mapping, sources, row_experts, counts, cumulative = _carve_words(
        device, -(-need // 4), entries, entries if want_sources else 0, entries if want_sources else 0, experts, 2 * experts)
    cumulative = cumulative.view(torch.int64)
    if not want_sources:
        sources = row_experts = None
    _call("hmc_moe_sort_routes", device, flat.data_ptr(), int(flat.dtype == torch.int64), entries, experts,
          workspace.data_ptr(), 4 * workspace.numel(), mapping.data_ptr(), _lib.ptr(sources), _lib.ptr(row_experts),
          counts.data_ptr(), cumulative.data_ptr(), _lib.ptr(status))
    return mapping, sources, row_experts, counts, cumulative


def moe_sort_routes_local(indices: torch.Tensor, experts: int, mirror: torch.Tensor, status: torch.Tensor):
    """The sort, offsets and read-back of a single-rank call as one launch.

    Returns (mapping, source_of_row, expert_of_row, counts, offsets): the first four as ``moe_sort_routes``, the last as
    ``route_offsets`` of the counts. ``mirror`` (pinned int32 [experts + 8]) receives the counts and the status words.
    """
    device = _require_cuda(indices, status)
    if indices.dtype not in (torch.int32, torch.int64):
        raise TypeError(f"expert indices must be int32 or int64, got {indices.dtype}")
    if not mirror.is_pinned() or mirror.dtype != torch.int32 or mirror.numel() < experts + _lib.HMC_STATUS_WORDS:
        raise ValueError("mirror must be pinned int32 memory of experts + 8 words")
    flat = indices.reshape(-1).contiguous()
    entries = flat.numel()
    need = max(1, _lib.load().hmc_moe_sort_workspace_bytes(entries, experts))
    workspace, mapping, sources, row_experts, counts, ends, starts = _carve_words(
        device, -(-need // 4), entries, entries, entries, experts, 2 * experts, 2 * (experts + 1))
    ends, starts = ends.view(torch.int64), starts.view(torch.int64)
    _call("hmc_moe_sort_routes_local", device, flat.data_ptr(), int(flat.dtype == torch.int64), entries, experts,
          workspace.data_ptr(), 4 * workspace.numel(), mapping.data_ptr(), sources.data_ptr(), row_experts.data_ptr(),
          counts.data_ptr(), ends.data_ptr(), starts.data_ptr(), mirror.data_ptr(), status.data_ptr())
    first = starts[:experts]  # one rank: the source's expert-major order is the owner's
    offsets = {"dispatch_src_off": first, "dispatch_target_off": first, "dispatch_size": counts, "combine_src_off": first,
               "combine_target_off": first, "combine_size": counts, "group_list": ends, "totals": starts[experts:].expand(2),
               "recv_segment_start": first, "send_order_start": starts}
    return mapping, sources, row_experts, counts, offsets


def moe_gather_rows(tokens: torch.Tensor, source_of_row: torch.Tensor, top_k: int, out: torch.Tensor) -> None:
    """out[row] = tokens[source_of_row[row] // top_k]."""
    device = _require_cuda(tokens, source_of_row, out)
    _call("hmc_moe_gather_rows", device, tokens.data_ptr(), source_of_row.data_ptr(), source_of_row.numel(), top_k,
          tokens.shape[1], out.data_ptr())


def moe_permute_from_mapping(tokens, mapping, probs, top_k, out, out_probs, status=None) -> None:
    """out[mapping[t*K+k]] = tokens[t]; out_probs[mapping[t*K+k]] = probs[t, k]."""
    device = _require_cuda(tokens, mapping, out)
    _call("hmc_moe_permute_from_mapping", device, tokens.data_ptr(), mapping.data_ptr(), _lib.ptr(probs),
          tokens.shape[0], top_k, tokens.shape[1], out.data_ptr(), _lib.ptr(out_probs), _lib.ptr(status))


def moe_unpermute(permuted, mapping, probs, num_tokens, top_k, out, status=None) -> None:
    """Weighted K-sum of expert-major rows back to token order."""
    device = _require_cuda(permuted, mapping, out)
    _call("hmc_moe_unpermute", device, permuted.data_ptr(), mapping.data_ptr(), _lib.ptr(probs), num_tokens, top_k,
          permuted.shape[1], permuted.shape[0], out.data_ptr(), _lib.ptr(status))


def moe_unpermute_grad(permuted, grad_out, mapping, probs, top_k, grad_permuted, grad_probs, status=None) -> None:
    """grad_permuted[row] = bf16(grad_out[t] * p); grad_probs[t,k] = <grad_out[t], permuted[row]>."""
    device = _require_cuda(grad_out, mapping, probs, grad_permuted)
    _call("hmc_moe_unpermute_grad", device, _lib.ptr(permuted), grad_out.data_ptr(), mapping.data_ptr(),
          probs.data_ptr(), grad_out.shape[0], top_k, grad_out.shape[1], grad_permuted.data_ptr(),
          _lib.ptr(grad_probs), _lib.ptr(status))


def moe_token_permute_grad(grad_permuted, mapping, num_tokens, top_k, grad_tokens, status=None) -> None:
    """grad_tokens[t] = sum_k grad_permuted[mapping[t*K+k]]."""
    device = _require_cuda(grad_permuted, mapping, grad_tokens)
    _call("hmc_moe_token_permute_grad", device, grad_permuted.data_ptr(), mapping.data_ptr(), num_tokens, top_k,
          grad_permuted.shape[1], grad_tokens.data_ptr(), _lib.ptr(status))


def zero_empty_expert_grad(first, second, cumulative) -> None:
    """Zero the per-expert slices whose cumulative row count did not advance."""
    device = _require_cuda(first, second, cumulative)
    experts = cumulative.numel()
    _call("hmc_zero_empty_expert_grad", device, first.data_ptr(), first.numel() // experts * first.element_size(),
          _lib.ptr(second), 0 if second is None else second.numel() // experts * second.element_size(),
          cumulative.data_ptr(), experts)


def route_offsets(counts_by_source: torch.Tensor, rank: int):
    """Row-unit push-mode descriptors from the gathered [EP, E] INT32 count table."""
    device = _require_cuda(counts_by_source)
    ep, experts = counts_by_source.shape
    local = experts // ep
    sizes = {"dispatch_src_off": 2 * experts, "dispatch_target_off": 2 * experts, "dispatch_size": experts,
             "combine_src_off": 2 * experts, "combine_target_off": 2 * experts, "combine_size": experts,
             "group_list": 2 * local, "totals": 4, "recv_segment_start": 2 * experts, "send_order_start": 2 * (experts + 1)}
    out = {name: words if name in ("dispatch_size", "combine_size") else words.view(torch.int64)
           for name, words in zip(sizes, _carve_words(device, *sizes.values()))}
    _call("hmc_route_offsets", device, counts_by_source.contiguous().data_ptr(), ep, experts, rank,
          *(out[k].data_ptr() for k in ("dispatch_src_off", "dispatch_target_off", "dispatch_size",
                                        "combine_src_off", "combine_target_off", "combine_size", "group_list",
                                        "totals", "recv_segment_start", "send_order_start")))
    return out


# -------------------------------------------------------------------------------------------- mHC
def mega_mhc_out(previous_output, residual, previous_pre_mix, previous_post_mix, previous_residual_mix, phi, alpha,
                 bias, norm_weight, new_residual, next_pre_mix, next_post_mix, next_residual_mix, block_input,
                 hc_before_norm, inv_rms, sum_out, norm_out, mixed_input, rms_rstd, *, hc_eps, norm_eps, num_iters,
                 need_backward, status=None) -> None:
    """Shifted single-pass mHC forward into caller-owned outputs and caches. Where no backward follows, ``mixed_input``
    may be None, and with it every other cache."""
    device = _require_cuda(previous_output, residual, phi, new_residual)
    if mixed_input is None and (need_backward or any(t is not None for t in (hc_before_norm, inv_rms, rms_rstd))):
        raise ValueError("mixed_input may be None only without a backward and together with the other caches")
    hidden = residual.shape[-1]
    tokens = residual.numel() // (4 * hidden)
    need = _lib.load().hmc_mega_mhc_workspace_bytes(tokens, hidden)
    p = _lib.ptr
    if mixed_input is None:  # a forward that keeps nothing: its scratch in one allocation
        rows = 2 * tokens * hidden
        scratch = torch.empty(rows + -(-need // 256) * 256 + 8 * tokens, dtype=torch.uint8, device=device)
        mixed = scratch.data_ptr()  # rows of a multiple of 128 BF16 values: what follows is aligned as well
        workspace = mixed + rows
        rms = workspace + -(-need // 256) * 256
        rstd = rms + 4 * tokens
    else:
        scratch = torch.empty(need, dtype=torch.uint8, device=device)
        mixed, workspace, rms, rstd = p(mixed_input), scratch.data_ptr(), p(inv_rms), p(rms_rstd)
    args = _lib.MegaMhcArgs(
        tokens=tokens, hidden=hidden, previous_output=p(previous_output), residual=p(residual),
        previous_pre_mix=p(previous_pre_mix), previous_post_mix=p(previous_post_mix),
        previous_residual_mix=p(previous_residual_mix), phi=p(phi), alpha=p(alpha), bias=p(bias), norm_weight=p(norm_weight),
        new_residual=p(new_residual), next_pre_mix=p(next_pre_mix), next_post_mix=p(next_post_mix),
        next_residual_mix=p(next_residual_mix), block_input=p(block_input), hc_before_norm=p(hc_before_norm), inv_rms=rms,
        sum_out=p(sum_out), norm_out=p(norm_out), mixed_input=mixed, rms_rstd=rstd, workspace=workspace, workspace_bytes=need,
        hc_eps=hc_eps, norm_eps=norm_eps, num_iters=num_iters, need_backward=int(need_backward), status=p(status))
    _call("hmc_mega_mhc", device, ctypes.byref(args))


def mega_mhc_grad_out(tensors: dict, *, hc_eps: float, num_iters: int, status=None) -> None:
    """mHC backward; ``tensors`` maps every pointer field of ``hmc_mega_mhc_grad_args`` to a tensor."""
    residual = tensors["residual"]
    device = _require_cuda(residual)
    hidden = residual.shape[-1]
    tokens = residual.numel() // (4 * hidden)
    lib = _lib.load()
    workspace = torch.empty(lib.hmc_mega_mhc_grad_workspace_bytes(tokens, hidden), dtype=torch.uint8, device=device)
    args = _lib.MegaMhcGradArgs()
    args.tokens, args.hidden = tokens, hidden
    for name, _ in _lib.MegaMhcGradArgs._fields_:  # pylint: disable=protected-access
        if name in tensors:
            setattr(args, name, _lib.ptr(tensors[name]))
    args.workspace = workspace.data_ptr()
    args.workspace_bytes = workspace.numel()
    args.hc_eps, args.num_iters = hc_eps, num_iters
    args.status = _lib.ptr(status)
    _call("hmc_mega_mhc_grad", device, ctypes.byref(args))


# --------------------------------------------------------------------------------- EP transport
def ep_dispatch(tokens, source_of_row, expert_of_row, dispatch_src_off, dispatch_target_off, *, rows, top_k, ep,
                local_experts, capacity_rows, peer_buffers, peer_ctrl, local_ctrl, generation, status=None,
                budget_ns=0, max_ctas=0, row_values=None, value_index=None, value_plane_offset=0) -> None:
    """Push expert-major rows (or gathered token rows) into their owners' receive buffers.

    ``row_values`` (float32) adds one scalar per row, read at ``value_index[j]`` when an index is
    given, and stored in the float plane ``value_plane_offset`` bytes into each owner's buffer.
    """
    device = _require_cuda(tokens, expert_of_row, dispatch_src_off, dispatch_target_off, local_ctrl, row_values,
                           value_index)
    args = _dispatch_struct(tokens, source_of_row, expert_of_row, dispatch_src_off, dispatch_target_off, rows=rows,
                            top_k=top_k, ep=ep, local_experts=local_experts, capacity_rows=capacity_rows,
                            peer_buffers=peer_buffers, peer_ctrl=peer_ctrl, local_ctrl=local_ctrl,
                            generation=generation, status=status, budget_ns=budget_ns, max_ctas=max_ctas,
                            row_values=row_values, value_index=value_index, value_plane_offset=value_plane_offset)
    _call("hmc_ep_dispatch", device, ctypes.byref(args))


def _dispatch_struct(tokens, source_of_row, expert_of_row, dispatch_src_off, dispatch_target_off, *, rows, top_k, ep,
                     local_experts, capacity_rows, peer_buffers, peer_ctrl, local_ctrl, generation, status=None,
                     budget_ns=0, max_ctas=0, row_values=None, value_index=None, value_plane_offset=0, rank=0,
                     send_order_start=None):
    """``hmc_ep_dispatch_args`` from tensors (``rank`` matters only when the dispatch rides inside a GEMM)."""
    if row_values is not None and (row_values.dtype != torch.float32 or not row_values.is_contiguous()):
        raise ValueError("row_values must be a contiguous float32 tensor")
    args = _lib.EpDispatchArgs()
    args.tokens = tokens.data_ptr()
    args.source_of_row = _lib.ptr(source_of_row)
    args.expert_of_row = expert_of_row.data_ptr()
    args.dispatch_src_off = dispatch_src_off.data_ptr()
    args.dispatch_target_off = dispatch_target_off.data_ptr()
    args.rows, args.top_k, args.hidden = rows, top_k, tokens.shape[1]
    args.ep, args.local_experts, args.capacity_rows = ep, local_experts, capacity_rows
    args.peer_buffers = ctypes.cast(peer_buffers, ctypes.c_void_p)
    args.peer_ctrl = ctypes.cast(peer_ctrl, ctypes.c_void_p)
    args.local_ctrl = local_ctrl.data_ptr()
    args.generation, args.max_ctas, args.budget_ns = generation, max_ctas, budget_ns
    args.status = _lib.ptr(status)
    args.row_values, args.value_index = _lib.ptr(row_values), _lib.ptr(value_index)
    args.value_plane_offset = value_plane_offset
    args.rank = rank
    args.send_order_start = _lib.ptr(send_order_start)
    return args


def ep_combine(results, segment_start, combine_target_off, *, rows, ep, local_experts, target_rows_limit,
               peer_buffers, peer_ctrl, local_ctrl, generation, status=None, budget_ns=0, max_ctas=0,
               result_values=None, value_plane_offset=0) -> None:
    """Return result rows (and optionally one float per row) to the routed buffers of their source ranks."""
    device = _require_cuda(results, segment_start, combine_target_off, local_ctrl, result_values)
    if result_values is not None and (result_values.dtype != torch.float32 or not result_values.is_contiguous()):
        raise ValueError("result_values must be a contiguous float32 tensor")
    args = _lib.EpCombineArgs()
    args.results = results.data_ptr()
    args.segment_start = segment_start.data_ptr()
    args.combine_target_off = combine_target_off.data_ptr()
    args.rows, args.hidden, args.ep, args.local_experts = rows, results.shape[1], ep, local_experts
    args.target_rows_limit = target_rows_limit
    args.peer_buffers = ctypes.cast(peer_buffers, ctypes.c_void_p)
    args.peer_ctrl = ctypes.cast(peer_ctrl, ctypes.c_void_p)
    args.local_ctrl = local_ctrl.data_ptr()
    args.generation, args.max_ctas, args.budget_ns = generation, max_ctas, budget_ns
    args.status = _lib.ptr(status)
    args.result_values = _lib.ptr(result_values)
    args.value_plane_offset = value_plane_offset
    _call("hmc_ep_combine", device, ctypes.byref(args))


def ep_publish_source(peer_ctrl, ep: int, rank: int, generation: int, device: torch.device) -> None:
    """Tell every peer that this rank's source buffer holds the rows of ``generation`` (pull dispatch)."""
    _call("hmc_ep_publish_source", device, peer_ctrl, ep, rank, generation)


def ep_pull(out, segment_start, source_row_off, *, rows, ep, local_experts, source_rows_limit, peer_sources,
            local_ctrl, generation, status=None, budget_ns=0, max_ctas=0, out_values=None,
            value_plane_offset=0) -> None:
    """Fetch this rank's rows from the published source buffers of their source ranks."""
    device = _require_cuda(out, segment_start, source_row_off, local_ctrl, out_values)
    args = _lib.EpPullArgs()
    args.peer_sources = ctypes.cast(peer_sources, ctypes.c_void_p)
    args.source_row_off = source_row_off.data_ptr()
    args.segment_start = segment_start.data_ptr()
    args.out = out.data_ptr()
    args.out_values = _lib.ptr(out_values)
    args.rows, args.hidden, args.ep, args.local_experts = rows, out.shape[1], ep, local_experts
    args.source_rows_limit, args.value_plane_offset = source_rows_limit, value_plane_offset
    args.local_ctrl = local_ctrl.data_ptr()
    args.generation, args.max_ctas, args.budget_ns = generation, max_ctas, budget_ns
    args.status = _lib.ptr(status)
    _call("hmc_ep_pull", device, ctypes.byref(args))


def route_guard(table_block: torch.Tensor, ep: int, experts: int, capacity_rows: int, routed_limit: int, status,
                skip_flag: torch.Tensor, host_mirror: torch.Tensor) -> None:
    """Device-side admission check of one expert-parallel call + mirror of table, status words and decision
    to pinned host memory (``hmc_route_guard``)."""
    device = _require_cuda(table_block, skip_flag, status)
    if not host_mirror.is_pinned() or host_mirror.numel() < ep * (experts + 4) + _lib.HMC_STATUS_WORDS + 1:
        raise ValueError("host_mirror must be pinned int32 memory of ep * (experts + 4) + 9 words")
    _call("hmc_route_guard", device, table_block.data_ptr(), ep, experts, capacity_rows, routed_limit, _lib.ptr(status),
          skip_flag.data_ptr(), host_mirror.data_ptr())


def ep_wait(counter: torch.Tensor, expected: int, status=None, budget_ns: int = 0) -> None:
    """Stream-ordered bounded wait until ``counter[0] >= expected``."""
    device = _require_cuda(counter)
    _call("hmc_ep_wait", device, counter.data_ptr(), expected, budget_ns, _lib.ptr(status))


# ---------------------------------------------------------------------------------------- MXFP8
HMC_MXQ_PLAIN, HMC_MXQ_SWIGLU, HMC_MXQ_SWIGLU_GRAD = 0, 1, 2


def mx_pad_blocks(rows: int, groups: int) -> int:
    """Upper bound of the 128-row blocks of the padded expert-major layout."""
    return (rows + 127) // 128 + groups


def _combine_struct(combine: dict):
    fused = _lib.GemmCombine()
    fused.segment_start = combine["segment_start"].data_ptr()
    fused.combine_target_off = combine["combine_target_off"].data_ptr()
    fused.peer_buffers = ctypes.cast(combine["peer_buffers"], ctypes.c_void_p)
    fused.peer_ctrl = ctypes.cast(combine["peer_ctrl"], ctypes.c_void_p)
    fused.ep, fused.local_experts = combine["ep"], combine["local_experts"]
    fused.target_rows_limit = combine["target_rows_limit"]
    return fused


def mx_gemm_combine_units(n: int) -> int:
    """Counter increments per result row of a fused-combine MX GEMM with ``n`` output columns."""
    return int(_lib.load().hmc_mx_gemm_combine_units(n))


def mx_gemm(a, a_scale, b, b_scale, c, group_ends, *, mode, rows, pad_blocks, n, k=0, m=0,
            b_major=HMC_MAJOR_MN, epilogue=HMC_EPI_STORE_BF16, status=None, max_ctas=0, combine=None,
            tile_mode=0, act: "MxActivations | None" = None, aux=None) -> None:
    """Block-scaled FP8 grouped GEMM; see ``hmc_mx_gemm_args`` for the operand layouts. ``combine`` as in
    ``grouped_gemm``: the rows leave the epilogue for their source ranks and ``c`` may be None. ``tile_mode``:
    0 = 256 x 256 CTA-pair tiles where the shape allows, 1 = 128 x 128 tiles, 2 = pairs or an error.
    ``epilogue=HMC_EPI_SWIGLU_MXQ``: ``c`` = U [rows, n] and ``act`` (an ``MxActivations`` of width n / 2 with both
    axes) receives the quantised bf16(silu(gate) * up). ``epilogue=HMC_EPI_SWIGLU_GRAD_MXQ``: the accumulator is
    dAct [rows, n], ``aux`` = the saved U [rows, 2n], ``act`` (width 2n) receives the quantised dU and ``c`` (dAct)
    may be None."""
    device = _require_cuda(a, a_scale, b, b_scale, c, group_ends, status)
    args = _lib.MxGemmArgs()
    args.mode, args.b_major, args.epilogue = mode, b_major, epilogue
    args.groups, args.max_ctas, args.tile_mode = group_ends.numel(), max_ctas, tile_mode
    args.rows, args.pad_blocks, args.m, args.n, args.k = rows, pad_blocks, m, n, k
    args.a, args.a_scale = a.data_ptr(), a_scale.data_ptr()
    args.b, args.b_scale = b.data_ptr(), b_scale.data_ptr()
    args.c = _lib.ptr(c)
    args.group_ends = group_ends.data_ptr()
    args.status = _lib.ptr(status)
    if act is not None:
        args.act_row_data, args.act_row_scale = act.row_data.data_ptr(), act.row_scale.data_ptr()
        args.act_col_data, args.act_col_scale = _lib.ptr(act.col_data), _lib.ptr(act.col_scale)
    args.aux = _lib.ptr(aux)
    fused = None
    if combine is not None:
        fused = _combine_struct(combine)
        args.combine = ctypes.cast(ctypes.pointer(fused), ctypes.c_void_p)
    _call("hmc_mx_gemm", device, ctypes.byref(args))


def ep_wait_groups(counters: torch.Tensor, group_ends: torch.Tensor, status=None, budget_ns: int = 0) -> None:
    """Stream-ordered bounded wait until every group's arrival counter covers its rows."""
    device = _require_cuda(counters, group_ends)
    _call("hmc_ep_wait_groups", device, counters.data_ptr(), group_ends.data_ptr(), group_ends.numel(), budget_ns,
          _lib.ptr(status))


class MxActivations:
    """Quantised activations in the padded expert-major layout (see ``hmc_mx_quant_args``)."""

    def __init__(self, rows: int, groups: int, width: int, device, *, want_row: bool, want_col: bool) -> None:
        self.rows, self.width = rows, width
        self.pad_blocks = mx_pad_blocks(rows, groups)
        u8 = dict(dtype=torch.uint8, device=device)
        pad_rows = self.pad_blocks * 128
        atoms = self.pad_blocks * (width // 128) * 512
        self.row_data = torch.empty((pad_rows, width), **u8) if want_row else None
        self.row_scale = torch.empty(atoms, **u8) if want_row else None
        self.col_data = torch.empty((pad_rows, width), **u8) if want_col else None
        self.col_scale = torch.empty(atoms, **u8) if want_col else None


def mx_quant(src, group_ends, width, *, kind=HMC_MXQ_PLAIN, aux=None, want_row=True, want_col=False,
             dense=None) -> MxActivations:
    """Quantise expert-major BF16 rows (optionally through SwiGLU / SwiGLU-grad) to MXFP8."""
    device = _require_cuda(src, group_ends, aux, dense)
    rows, groups = src.shape[0], group_ends.numel()
    out = MxActivations(rows, groups, width, device, want_row=want_row, want_col=want_col)
    args = _lib.MxQuantArgs()
    args.kind, args.groups = kind, groups
    args.rows, args.pad_blocks, args.width = rows, out.pad_blocks, width
    args.src, args.aux, args.group_ends = src.data_ptr(), _lib.ptr(aux), group_ends.data_ptr()
    args.row_data, args.row_scale = _lib.ptr(out.row_data), _lib.ptr(out.row_scale)
    args.col_data, args.col_scale = _lib.ptr(out.col_data), _lib.ptr(out.col_scale)
    args.dense = _lib.ptr(dense)
    _call("hmc_mx_quant", device, ctypes.byref(args))
    return out


def mx_quant_weight(weight: torch.Tensor, *, want_col: bool = True, want_row: bool = True) -> dict:
    """BF16 weight [e, m, n] -> the reference's physical MX fields (col_* blocks along m, row_* along n)."""
    device = _require_cuda(weight)
    experts, m, n = weight.shape
    weight = weight.contiguous()
    out = {}
    if want_col:
        out["col_data"] = torch.empty((experts, m, n), dtype=torch.float8_e4m3fn, device=device)
        out["col_scale"] = torch.empty((experts, m // 64, n, 2), dtype=torch.uint8, device=device)
    if want_row:
        out["row_data"] = torch.empty((experts, m, n), dtype=torch.float8_e4m3fn, device=device)
        out["row_scale"] = torch.empty((experts, m, n // 64, 2), dtype=torch.uint8, device=device)
    _call("hmc_mx_quant_weight", device, weight.data_ptr(), experts, m, n, _lib.ptr(out.get("col_data")),
          _lib.ptr(out.get("col_scale")), _lib.ptr(out.get("row_data")), _lib.ptr(out.get("row_scale")))
    return out


def mx_pack_weight_scale(scale: torch.Tensor, axis: int, experts: int, m: int, n: int) -> torch.Tensor:
    """Reference scale tensor (col_scale: axis 0, row_scale: axis 1) -> scale-factor atoms for the GEMM."""
    device = _require_cuda(scale)
    atoms = torch.empty(experts * m * n // 32, dtype=torch.uint8, device=device)
    _call("hmc_mx_pack_weight_scale", device, scale.data_ptr(), axis, experts, m, n, atoms.data_ptr())
    return atoms
