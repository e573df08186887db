"""The work this framework is used for, as cases that can be timed and compared.

A case is one pass of the MoE layer through the calls an engine or a script makes:

  infer       forward_inference: generation, a few tokens per call or a whole context
  train       forward + backward: one micro-batch of a training step
  checkpoint  forward, save_routing, recompute, backward: the same under activation checkpointing
  block       block_forward + block_backward: RMSNorm, layer and skip connection around the same products
  adamw       adamw_step: the optimiser over the layer's parameters, after which the layer is ready for forward

Token counts, widths and expert counts are those of the repository's workloads (mgpt_b200/synth.py) and ragged
neighbours of them.  Parameters and gradients live in one flat FP32 buffer each, as in an engine's arena.
"""
import ctypes
import math

import torch

from mgpt_b200 import MoELayer
from mgpt_b200 import _lib


def _case(name, kind, n, C, H, E, k, mode="bf16", io="bf16", skew=False, store=False):
    return {"name": name, "kind": kind, "n": n, "C": C, "H": H, "E": E, "k": k,
            "mode": mode,      # arithmetic of the layer: "bf16" (tensor cores) or "fp32" (the reference's dtype)
            "io": io,          # dtype of the tokens
            "skew": skew,      # router bias 2*ln(1/(e+1)): a few experts take most tokens
            "store": store}    # weight gradients stored (first micro-batch of a step) instead of accumulated


def listed():
    return [
        # one sequence being generated: a single new token, the smallest call
        _case("decode_1", "infer", 1, 1024, 2816, 32, 2),
        # batched serving, one new token per sequence
        _case("decode_64", "infer", 64, 1024, 2816, 32, 2),
        _case("decode_256", "infer", 256, 1024, 2816, 32, 2),
        # the context of a prompt, a ragged number of tokens (the generator runs the whole context forward)
        _case("prefill_1777", "infer", 1777, 1024, 2816, 32, 2),
        # the reference's own default model, batch 16 x 64 tokens, all FP32
        _case("default_fp32", "train", 1024, 128, 512, 8, 2, mode="fp32", io="fp32"),
        # a medium model, the first micro-batch after zero_grad
        _case("medium", "train", 8192, 512, 1376, 16, 2, store=True),
        # the same model driven by an engine whose tensors are FP32, at a ragged batch
        _case("medium_f32_tokens", "train", 5003, 512, 1376, 16, 2, io="fp32"),
        # skewed routing: most experts empty, one with every token
        _case("skewed", "train", 16384, 1024, 512, 64, 4, skew=True),
        # the 64-expert model, the largest batch
        _case("large", "train", 32768, 2048, 1408, 64, 2),
        # a checkpointed block's share of a step
        _case("checkpoint", "checkpoint", 4096, 1024, 1408, 32, 2),
        # the whole feed-forward half of a transformer block
        _case("block", "block", 6000, 768, 2048, 16, 2),
        # the optimiser step of the decode model's layer
        _case("adamw", "adamw", 0, 1024, 2816, 32, 2),
    ]


def _log(rng, lo, hi, step=1):
    v = math.exp(rng.uniform(math.log(lo), math.log(hi + step)))
    return max(lo, min(hi, int(v) // step * step))


def draw(rng):
    kind = rng.choice(["infer", "infer", "infer", "train", "train", "train", "fp32", "checkpoint", "block", "adamw"])
    if kind == "fp32":          # small models in the reference's dtype
        return _unnamed(_case("", "train", _log(rng, 64, 2048), _log(rng, 64, 256, 8), _log(rng, 128, 1024, 8),
                              rng.randint(4, 16), rng.randint(1, 2), mode="fp32", io="fp32"))
    C = _log(rng, 256, 2048, 64)
    H = max(256, min(2816, _log(rng, max(256, C // 2), 4 * C, 8)))
    E = _log(rng, 4, 64)
    k = rng.randint(1, 4)
    # no larger than the largest listed case: parameters (fewer where an optimiser walks them), rows x widths, tokens
    while E > 4 and E * C * H > (32 * 1024 * 2816 if kind == "adamw" else 64 * 2048 * 1408):
        E = max(4, E // 2)
    if kind == "adamw":
        return _unnamed(_case("", "adamw", 0, C, H, E, k))
    n = _log(rng, 1, 4096) if kind == "infer" else _log(rng, 256, 32768)
    most = 32768 * 2 * 2048 * 1408 * (3 if kind == "checkpoint" else 4) // 4
    while n * k * C * H > most or n * C > 32768 * 2048:
        n = max(1, n // 2)
    io = "bf16" if rng.random() < 0.8 else "fp32"
    return _unnamed(_case("", kind, n, C, H, E, k, io=io, skew=rng.random() < 0.25,
                          store=kind != "infer" and rng.random() < 0.4))


def _unnamed(case):
    del case["name"]
    return case


def _flat_views(layer):
    """One flat FP32 buffer and a view of it per parameter, every view on a 256-byte boundary."""
    sizes = [(p.numel() + 63) // 64 * 64 for p in layer.get_parameters()]
    flat = torch.zeros(sum(sizes), dtype=torch.float32, device=layer.device)
    views, at = [], 0
    for p, s in zip(layer.get_parameters(), sizes):
        views.append(flat[at: at + p.numel()].view(p.shape))
        at += s
    return flat, views


def _pointers(views):
    return (ctypes.c_void_p * len(views))(*[v.data_ptr() for v in views])


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    C, E, n = case["C"], case["E"], case["n"]
    layer = MoELayer(C, case["H"], E, case["k"], mode=case["mode"])
    s = {"kind": case["kind"], "layer": layer}
    w, w_views = _flat_views(layer)
    g, g_views = _flat_views(layer)
    # weights ~ N(0, 0.02), biases as small as a trained model's; the router's bias skewed where the case says so
    for p, wv, gv in zip(layer.get_parameters(), w_views, g_views):
        p.grad = None
        p.data = wv
        p.grad = gv
    w.normal_(0.0, 0.02, generator=gen)
    if case["skew"]:
        w_views[1].add_(-2.0 * torch.log(torch.arange(1, E + 1, device="cuda", dtype=torch.float32)))
    lib = _lib.load()
    _lib.check(lib.mgpt_moe_bind_params(layer._h, _pointers(w_views), _pointers(g_views), len(w_views)))
    layer.sync_weights()
    if case["store"]:
        layer.set_weight_grad_overwrite(True)
    s["weights"], s["grads"] = w, g
    if case["kind"] == "adamw":
        g.normal_(0.0, 0.01, generator=gen)
        m, m_views = _flat_views(layer)
        v, v_views = _flat_views(layer)
        m.normal_(0.0, 0.01, generator=gen)
        v.uniform_(1e-6, 1e-3, generator=gen)
        layer.opt_m, layer.opt_v = m_views, v_views
        _lib.check(lib.mgpt_moe_bind_optimizer_state(layer._h, _pointers(m_views), _pointers(v_views), len(m_views)))
        s["m"], s["v"] = m, v
        return s
    dt = torch.bfloat16 if case["io"] == "bf16" else torch.float32
    s["x"] = torch.randn(n, C, generator=gen, device="cuda").to(dt)
    if case["kind"] != "infer":
        s["dy"] = torch.randn(n, C, generator=gen, device="cuda").to(dt)
    if case["kind"] == "block":
        s["scale"] = 1.0 + 0.1 * torch.randn(C, generator=gen, device="cuda")
        s["d_scale"] = torch.zeros(C, device="cuda")
    return s


def run(state):
    layer, kind = state["layer"], state["kind"]
    if kind == "infer":
        return layer.forward_inference(state["x"])
    if kind == "adamw":
        layer.adamw_step(10)
        return {"w": state["weights"], "m": state["m"], "v": state["v"]}
    if kind == "block":
        y = layer.block_forward(state["x"], state["scale"])
        dx = layer.block_backward(state["scale"], state["dy"], state["d_scale"])
        return {"y": y, "dx": dx, "grads": state["grads"], "d_scale": state["d_scale"]}
    y = layer.forward(state["x"])
    if kind == "checkpoint":
        routing = layer.save_routing()
        layer.recompute_into(state["x"], y, routing)
    dx = layer.backward(state["dy"])
    return {"y": y, "dx": dx, "grads": state["grads"]}


def _touched(case):
    """Experts that receive a row: expected number under uniform routing; a quarter of them under the skewed bias."""
    E, rows = case["E"], case["n"] * case["k"]
    t = E * (1.0 - (1.0 - 1.0 / E) ** rows)
    return min(t, max(case["k"], E / 4)) if case["skew"] else t


def work(case):
    n, C, H, E, k = (case[x] for x in ("n", "C", "H", "E", "k"))
    per_expert = 3 * C * H + 2 * H + C
    params = C * E + E + E * per_expert
    if case["kind"] == "adamw":
        # w, g, m, v in, w, m, v out, one BF16 copy of the weights for the products
        return {"bytes": params * (16 + 12 + 2), "flops": 15 * params}
    wb = 2 if case["mode"] == "bf16" else 4
    io = 2 if case["io"] == "bf16" else 4
    weights = _touched(case) * per_expert * wb + C * E * 4
    rows = n * k
    flops = 6 * rows * C * H + 2 * n * C * E
    if case["kind"] == "infer":
        return {"bytes": weights + 2 * n * C * io, "flops": flops}
    forwards = 2 if case["kind"] == "checkpoint" else 1
    grads = (E if case["store"] else 2 * _touched(case)) * per_expert * 4 + 2 * C * E * 4
    return {"bytes": weights + grads + 4 * n * C * io,
            "flops": flops * forwards + 12 * rows * C * H + 4 * n * C * E}


def tolerance(case):
    if case["kind"] == "adamw":
        return "exact"                  # the reference's FP32 operations, one by one
    if case["mode"] == "fp32":
        return {"rel": 1e-5}            # FP32 operands, FP32 sums in another order
    return {"rel": 1e-2}                # BF16 operands and activations, FP32 sums
