"""Performance cases: one call each of the public modules (MegaGate, MegaMhc, MegaMoeExperts) on one GPU.

Every case goes through the module's own ``forward`` and, for training, through autograd for the gradients of
the activations and of the parameters. Sizes are those of the repository's benchmark configurations, of its
parity configuration, or generic ones between them.
"""

import math

import torch

from hyper_multicore_b200 import MegaGate, MegaMhc, MegaMoeExperts, MegaMoeNumericsOptions
from hyper_multicore_b200.mxfp8 import attach_mx_fields


def listed():
    return [
        # One decode step of a batch of 16 sequences through the router: launches and latency count.
        dict(name="gate_decode", kind="gate", tokens=16, hidden=4096, experts=64, top_k=6, scoring="softmax",
             vision=False, groups=0, kept_groups=0, train=False),
        # The multimodal router of the gate benchmark: a prefill in which part of the tokens are image tokens and
        # take the second correction bias.
        dict(name="gate_prefill_multimodal", kind="gate", tokens=8192, hidden=4096, experts=64, top_k=6,
             scoring="softmax", vision=True, groups=0, kept_groups=0, train=False),
        # Router of the 256-expert configuration in training: group-limited sigmoid top-8, forward and backward.
        dict(name="gate_train_grouped", kind="gate", tokens=8192, hidden=7168, experts=256, top_k=8,
             scoring="sigmoid", vision=False, groups=8, kept_groups=4, train=True),
        # Residual-stream boundary of one decode step.
        dict(name="mhc_decode", kind="mhc", tokens=16, hidden=7168, train=False),
        # Training step on a short, odd number of tokens (what sequence packing leaves over) at a mid hidden size.
        dict(name="mhc_train_ragged", kind="mhc", tokens=1531, hidden=2560, train=True),
        # The mHC benchmark: a full training micro-batch.
        dict(name="mhc_train", kind="mhc", tokens=16384, hidden=7168, train=True),
        # Experts of one decode step: nearly every expert is read for a handful of rows. Weights as [out, in].
        dict(name="moe_decode", kind="moe", precision="bf16", tokens=32, hidden=4096, inter=1536, experts=32, top_k=4,
             layout="EOI", zipf=0.0, limit=0.0, before_fc2=False, train=False),
        # The single-rank parity configuration as a training step: small GEMMs.
        dict(name="moe_train_small", kind="moe", precision="bf16", tokens=512, hidden=1024, inter=2048, experts=16,
             top_k=2, layout="EIO", zipf=0.0, limit=0.0, before_fc2=False, train=True),
        # Prefill of an odd number of tokens with skewed expert load, clamped SwiGLU and probabilities before FC2.
        dict(name="moe_prefill_options", kind="moe", precision="bf16", tokens=3001, hidden=2048, inter=768, experts=64,
             top_k=8, layout="EOI", zipf=1.1, limit=7.0, before_fc2=True, train=False),
        # The headline benchmark: BF16 forward and backward of the expert-parallel configuration's per-rank problem.
        dict(name="moe_train", kind="moe", precision="bf16", tokens=4096, hidden=4096, inter=1536, experts=32, top_k=4,
             layout="EIO", zipf=0.0, limit=0.0, before_fc2=False, train=True),
        # MXFP8 inference on a short odd prefill.
        dict(name="moe_mxfp8_prefill", kind="moe", precision="mxfp8", tokens=1021, hidden=4096, inter=1536, experts=32,
             top_k=4, layout="EIO", zipf=0.0, limit=0.0, before_fc2=False, train=False),
        # Per-rank problem of the MXFP8 expert-parallel configuration: forward and backward under Zipf load.
        dict(name="moe_mxfp8_train", kind="moe", precision="mxfp8", tokens=8192, hidden=7168, inter=2048, experts=32,
             top_k=8, layout="EIO", zipf=1.1, limit=0.0, before_fc2=False, train=True),
    ]


def _log_int(rng, low, high):
    return max(low, min(high, round(math.exp(rng.uniform(math.log(low), math.log(high))))))


def draw(rng):
    """One more case: same modules and options, sizes spread over the whole range."""
    kind = rng.choice(["gate", "mhc", "moe", "moe"])
    train = rng.random() < 0.5
    if kind == "gate":
        groups = rng.choice([0, 0, 4, 8])
        experts = rng.choice([64, 128, 256]) if groups else _log_int(rng, 8, 256)
        return dict(kind=kind, tokens=_log_int(rng, 1, 8192), hidden=64 * _log_int(rng, 16, 112), experts=experts,
                    top_k=rng.randint(1, min(8, experts)), scoring=rng.choice(["softmax", "sigmoid", "sqrtsoftplus"]),
                    vision=rng.random() < 0.3, groups=groups, kept_groups=groups // 2, train=train)
    if kind == "mhc":
        return dict(kind=kind, tokens=_log_int(rng, 1, 16384), hidden=128 * _log_int(rng, 4, 56), train=train)
    precision = rng.choice(["bf16", "bf16", "mxfp8"])
    experts = rng.choice([8, 16, 32, 64])
    hidden, inter = 128 * _log_int(rng, 8, 56), 128 * _log_int(rng, 4, 16)
    top_k = rng.choice([1, 2, 4, 6, 8])
    # no dearer than the largest listed case of its precision
    most = 8192 * 8 * 7168 * 2048 if precision == "mxfp8" else 4096 * 4 * 4096 * 1536 * 2
    tokens = _log_int(rng, 1, max(1, min(8192, most // (top_k * hidden * inter))))
    plain = precision == "mxfp8" or rng.random() < 0.6
    return dict(kind=kind, precision=precision, tokens=tokens, hidden=hidden, inter=inter, experts=experts, top_k=top_k,
                layout="EIO" if precision == "mxfp8" else rng.choice(["EIO", "EOI"]), zipf=rng.choice([0.0, 1.1]),
                limit=0.0 if plain else 7.0, before_fc2=not plain and rng.random() < 0.5, train=train)


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _normal(g, *shape, scale=1.0, dtype=torch.float32):
    return torch.randn(*shape, generator=g, device="cuda").mul_(scale).to(dtype)


def _prepare_gate(case, g):
    tokens, experts = case["tokens"], case["experts"]
    grouped = case["groups"] > 0
    module = MegaGate(hidden_size=case["hidden"], num_experts=experts, top_k=case["top_k"],
                      scoring_func=case["scoring"], routed_scaling_factor=2.5 if grouped else 1.0,
                      vision_enabled=case["vision"], n_group=case["groups"] or None,
                      topk_group=case["kept_groups"] or None).to("cuda")
    with torch.no_grad():
        module.weight.copy_(_normal(g, experts, case["hidden"], scale=0.02))
        module.bias.copy_(_normal(g, experts, scale=0.02))
        if case["vision"]:
            module.bias_vl.copy_(_normal(g, experts, scale=0.02))
    state = dict(module=module, x=_normal(g, 1, tokens, case["hidden"], dtype=torch.bfloat16), mask=None)
    if case["vision"]:
        state["mask"] = torch.arange(tokens, device="cuda").ge(tokens * 3 // 4).unsqueeze(0)
    if case["train"]:
        state["x"].requires_grad_(True)
        state["grad"] = _normal(g, tokens, case["top_k"], scale=0.1)
    return state


def _run_gate(state):
    module, x = state["module"], state["x"]
    if "grad" not in state:
        with torch.no_grad():
            return module(x, state["mask"])
    logits, weights, indices = module(x, state["mask"])
    grads = torch.autograd.grad(weights, (x, module.weight), state["grad"])
    return logits.detach(), weights.detach(), indices, grads


def _prepare_mhc(case, g):
    tokens, hidden = case["tokens"], case["hidden"]
    module = MegaMhc(hidden, device="cuda")
    with torch.no_grad():
        module.phi.copy_(_normal(g, 24, 4 * hidden, scale=0.02))
        module.bias[8:] = (4.0 * torch.eye(4, device="cuda")).flatten()  # residual mix starts near the identity
        module.norm_weight.copy_(1 + _normal(g, hidden, scale=0.02))
    inputs = (_normal(g, tokens, hidden, dtype=torch.bfloat16), _normal(g, tokens, 4, hidden, dtype=torch.bfloat16),
              torch.sigmoid(_normal(g, tokens, 4)), 2 * torch.sigmoid(_normal(g, tokens, 4)),
              torch.softmax(_normal(g, tokens, 4, 4), dim=-1))
    state = dict(module=module, inputs=inputs)
    if case["train"]:
        for value in inputs:
            value.requires_grad_(True)
        state["grads"] = (_normal(g, tokens, 4, hidden, scale=0.1, dtype=torch.bfloat16),
                          _normal(g, tokens, 4, scale=0.1), _normal(g, tokens, 4, scale=0.1),
                          _normal(g, tokens, 4, 4, scale=0.1),
                          _normal(g, tokens, hidden, scale=0.1, dtype=torch.bfloat16))
    return state


def _run_mhc(state):
    module, inputs = state["module"], state["inputs"]
    if "grads" not in state:
        with torch.no_grad():
            return module(*inputs)
    outputs = module(*inputs)
    wanted = (*inputs, module.phi, module.alpha, module.bias, module.norm_weight)
    return tuple(o.detach() for o in outputs), torch.autograd.grad(outputs, wanted, state["grads"])


def _prepare_moe(case, g):
    tokens, hidden, inter = case["tokens"], case["hidden"], case["inter"]
    experts, top_k = case["experts"], case["top_k"]
    options = MegaMoeNumericsOptions(swiglu_limit=case["limit"] or None, apply_probs_before_fc2=case["before_fc2"])
    module = MegaMoeExperts(hidden_size=hidden, intermediate_size=inter, num_experts=experts, top_k=top_k,
                            precision=case["precision"], numerics_options=options)
    if case["layout"] == "EIO":
        shapes = (experts, hidden, 2 * inter), (experts, inter, hidden)
    else:
        shapes = (experts, 2 * inter, hidden), (experts, hidden, inter)
    weights = [_normal(g, *shape, scale=0.02, dtype=torch.bfloat16) for shape in shapes]
    if case["zipf"]:
        # expert popularity falls as a power law; Gumbel noise turns it into a draw without replacement per token
        logits = -case["zipf"] * torch.log(torch.randperm(experts, generator=g, device="cuda") + 1.0)
        logits = logits - torch.log(-torch.log(torch.rand(tokens, experts, generator=g, device="cuda").clamp(1e-9, 1 - 1e-6)))
        probs, ids = torch.topk(torch.sigmoid(logits), top_k, dim=-1)
        probs = probs / probs.sum(dim=-1, keepdim=True)
    else:
        logits = torch.rand(tokens, experts, generator=g, device="cuda") * 2 - 1
        probs, ids = torch.topk(torch.softmax(logits, dim=-1), top_k, dim=-1)
    state = dict(module=module, x=_normal(g, tokens, hidden, dtype=torch.bfloat16), ids=ids, probs=probs.contiguous(),
                 weights=weights)
    if case["train"]:
        for value in (state["x"], state["probs"], *weights):
            value.requires_grad_(True)
        state["grad"] = _normal(g, tokens, hidden, dtype=torch.bfloat16)
    if case["precision"] == "mxfp8":
        for weight in weights:
            attach_mx_fields(weight)
    return state


def _run_moe(state):
    module, x, probs, weights = state["module"], state["x"], state["probs"], state["weights"]
    if "grad" not in state:
        with torch.no_grad():
            return module(x, state["ids"], probs, expert_weights=tuple(weights))
    out = module(x, state["ids"], probs, expert_weights=tuple(weights))
    return out.detach(), torch.autograd.grad(out, (x, probs, *weights), state["grad"])


def prepare(case, seed):
    return {"gate": _prepare_gate, "mhc": _prepare_mhc, "moe": _prepare_moe}[case["kind"]](case, _generator(seed)) \
        | {"kind": case["kind"]}


def run(state):
    return {"gate": _run_gate, "mhc": _run_mhc, "moe": _run_moe}[state["kind"]](state)


def _exact_gate(case, state):
    """The logits alone: the rest follows a Top-K selection, which jumps where two scores are close, so that it has
    no 64-bit counterpart."""
    logits = state["x"].detach().double().flatten(0, 1) @ state["module"].weight.detach().double().t()
    return (logits, None, None, None) if case["train"] else (logits, None, None)


def _mhc_double(previous_output, residual, pre, post, mix, phi, alpha, bias, norm_weight, eps=1e-6):
    new = torch.einsum("tji,tjh->tih", mix, residual) + post.unsqueeze(-1) * previous_output.unsqueeze(1)
    # what follows is a function of the stored BF16 streams
    new = new + (new.detach().float().bfloat16().double() - new.detach())
    normed = new * torch.rsqrt(new.square().mean(dim=(1, 2), keepdim=True) + eps)
    pre_l, post_l, mix_l = torch.split(normed.flatten(1) @ phi.t(), (4, 4, 16), dim=-1)
    pre_b, post_b, mix_b = torch.split(bias, (4, 4, 16))
    current = torch.softmax((mix_l * alpha[2] + mix_b).view(-1, 4, 4), dim=-1) + eps
    current = current / (current.sum(dim=1, keepdim=True) + eps)
    for _ in range(19):
        current = current / (current.sum(dim=2, keepdim=True) + eps)
        current = current / (current.sum(dim=1, keepdim=True) + eps)
    mixed = (new * pre.unsqueeze(-1)).sum(dim=1)
    block = mixed * torch.rsqrt(mixed.square().mean(dim=-1, keepdim=True) + eps) * norm_weight
    return (new, torch.sigmoid(pre_l * alpha[0] + pre_b) + eps, 2 * torch.sigmoid(post_l * alpha[1] + post_b), current,
            block)


def _exact_mhc(case, state):
    module = state["module"]
    weights = [p.detach().double() for p in (module.phi, module.alpha, module.bias, module.norm_weight)]
    outputs, rows, totals = [], [], None
    for first in range(0, case["tokens"], 2048):
        part = slice(first, first + 2048)
        leaves = [v.detach()[part].double() for v in state["inputs"]] + weights
        if not case["train"]:
            outputs.append(_mhc_double(*leaves))
            continue
        leaves = [v.clone().requires_grad_(True) for v in leaves]
        out = _mhc_double(*leaves)
        grads = torch.autograd.grad(out, leaves, [g[part].double() for g in state["grads"]])
        outputs.append([o.detach() for o in out])
        rows.append(grads[:5])
        totals = grads[5:] if totals is None else [a + b for a, b in zip(totals, grads[5:])]
    result = tuple(torch.cat(v) for v in zip(*outputs))
    return (result, (*(torch.cat(v) for v in zip(*rows)), *totals)) if case["train"] else result


def _exact_moe(case, state):
    """Without any rounding of what lies between, and for MXFP8 without the quantisation."""
    x, probs, ids = state["x"].detach().double(), state["probs"].detach().double(), state["ids"]
    weights = [w.detach() for w in state["weights"]]
    out = torch.zeros_like(x)
    grads = [torch.zeros_like(x), torch.zeros_like(probs)] + [torch.zeros(w.shape, dtype=torch.float64, device="cuda")
                                                              for w in weights] if case["train"] else None
    for expert in range(case["experts"]):
        rows, slots = torch.where(ids == expert)
        if rows.numel() == 0:
            continue
        leaves = [v.requires_grad_(case["train"]) for v in (x[rows], probs[rows, slots], *(w[expert].double() for w in weights))]
        w1, w2 = leaves[2:] if case["layout"] == "EIO" else (leaves[2].t(), leaves[3].t())
        gate, up = (leaves[0] @ w1).chunk(2, dim=-1)
        if case["limit"]:
            gate, up = gate.clamp(max=case["limit"]), up.clamp(-case["limit"], case["limit"])
        y = (torch.nn.functional.silu(gate) * up) @ w2 * leaves[1].unsqueeze(-1)
        out.index_add_(0, rows, y.detach())
        if case["train"]:
            got = torch.autograd.grad(y, leaves, state["grad"][rows].double())
            grads[0].index_add_(0, rows, got[0])
            grads[1][rows, slots] = got[1]
            grads[2][expert], grads[3][expert] = got[2], got[3]
    return (out, tuple(grads)) if case["train"] else out


def exact(case, seed):
    """``run``'s outputs in 64 bits, by plain torch."""
    state = prepare(case, seed)
    return {"gate": _exact_gate, "mhc": _exact_mhc, "moe": _exact_moe}[case["kind"]](case, state)


def work(case):
    t, h = case["tokens"], case["hidden"]
    if case["kind"] == "gate":
        e, k = case["experts"], case["top_k"]
        read = 2 * t * h + 4 * e * h
        total = read + 4 * t * e + 12 * t * k
        if case["train"]:  # x and the weight again, grad_weights in; the two gradients out
            total += read + 4 * t * k + read
        return {"bytes": total, "flops": (6 if case["train"] else 2) * t * h * e}
    if case["kind"] == "mhc":
        row = 2 * t * h
        phi = 4 * 24 * 4 * h
        maps = 4 * 24 * t
        total = 10 * row + 2 * maps + phi  # residual and previous output in; new residual and block input out
        if case["train"]:  # mixed input is kept; 15 rows in and 5 out in the backward
            total += row + 20 * row + 3 * maps + 2 * phi
        return {"bytes": total, "flops": (6 if case["train"] else 2) * t * 4 * h * 24}
    e, k, i = case["experts"], case["top_k"], case["inter"]
    touched = min(e, t * k) * 3 * h * i * (1 if case["precision"] == "mxfp8" else 2)
    row, inner = 2 * t * h, 2 * t * k * i
    total = 2 * row + 12 * t * k + touched
    if case["train"]:  # gate | up kept and read again; dY in, dX out, weights in and their BF16 gradients out
        total += 4 * inner + 3 * row + 8 * t * k + touched + 2 * 3 * e * h * i
    return {"bytes": total, "flops": (18 if case["train"] else 6) * t * k * h * i}


def tolerance(case):
    """About four times the difference measured against an evaluation in 64 bits (gate, mHC) or with the sums of
    another GEMM and the golden's summation order (experts). The largest terms are one BF16 rounding of a stored
    intermediate (2^-9): the mixed row of mHC, the rows of the Top-K sums, an E4M3 step of a quantised activation."""
    if case["kind"] == "gate":
        # FP32 logits and weights: 2e-6 at most; training adds a hidden-state gradient rounded to BF16
        return {"rel": 2.5e-4, "max": 3.2e-2, "differ": 1e-3} if case["train"] else {"rel": 8e-6, "max": 4e-5, "differ": 1e-3}
    if case["kind"] == "mhc":
        return {"rel": 1.8e-2, "max": 0.12} if case["train"] else {"rel": 1.2e-2, "max": 3.2e-2}
    if case["precision"] == "mxfp8":
        return {"rel": 1.6e-2, "max": 0.55} if case["train"] else {"rel": 1.5e-3, "max": 0.16}
    return {"rel": 1.6e-2, "max": 0.14} if case["train"] else {"rel": 1e-3, "max": 0.08}
