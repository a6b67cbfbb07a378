"""The work a user of this framework has it do, as timed cases.

Three kinds of case, each through the public entry points:

``blocks``   torch MoE blocks rewritten by ``zmlx_b200.patch.patch`` and called one after the other, as a decoder
             calls them: router, top-k, gate/up + SwiGLU, down, combine, shared expert.  One token per sequence is
             decode, many tokens are a batch of sequences or a prompt (prefill).
``ops``      the operator surface (``zmlx_b200.kernels``) for a user who keeps their own block: gating, fused
             gate/up + SwiGLU over the selected experts, down projection with the weighted combine.
``model``    ``zmlx_b200.model.StackedDecoder``: a decode step against a filled KV cache, or a prompt from position 0.

The block shapes are the ones ``zmlx_b200.synthetic.CONFIGS`` names, the decoder is ``DECODER_CONFIGS["c4"]``; of its 48
equal layers a case runs ``layers``.  Weights and activations follow ``zmlx_b200.synthetic``.
"""

from __future__ import annotations

from dataclasses import replace

import torch

from zmlx_b200 import nn, synthetic
from zmlx_b200.kernels import fused_moe, moe
from zmlx_b200.model import DECODER_CONFIGS, StackedDecoder
from zmlx_b200.patch import patch

_DEV = "cuda"


def listed() -> list[dict]:
    return [
        # one interactive sequence, one token: the smallest calls, several blocks deep so that weights come from HBM
        {"name": "decode_qwen3_t1", "kind": "blocks", "config": "c2", "layers": 12, "tokens": 1},
        {"name": "decode_glm_mxfp4_t1", "kind": "blocks", "config": "c3", "layers": 8, "tokens": 1},
        {"name": "decode_deepseek_t1", "kind": "blocks", "config": "c5", "layers": 1, "tokens": 1},
        # a few sequences decoded together
        {"name": "decode_deepseek_t6", "kind": "blocks", "config": "c5", "layers": 1, "tokens": 6},
        # a serving batch: a few rows per expert
        {"name": "batch_qwen3_t32", "kind": "blocks", "config": "c2", "layers": 4, "tokens": 32},
        {"name": "batch_deepseek_t64", "kind": "blocks", "config": "c5", "layers": 1, "tokens": 64},
        # prompts: tens to hundreds of rows per expert, with a ragged length
        {"name": "prefill_glm_mxfp4_t300", "kind": "blocks", "config": "c3", "layers": 2, "tokens": 300},
        {"name": "prefill_deepseek_t512", "kind": "blocks", "config": "c5", "layers": 1, "tokens": 512},
        {"name": "prefill_qwen3_t4096", "kind": "blocks", "config": "c2", "layers": 1, "tokens": 4096},
        # the operators called one by one on an odd number of tokens
        {"name": "ops_qwen3_t19", "kind": "ops", "config": "c2", "tokens": 19},
        # the stacked decoder: a decode step of four sequences, and a prompt
        {"name": "model_decode_b4", "kind": "model", "layers": 4, "batch": 4, "context": 3000, "tokens": 1},
        {"name": "model_prefill_s1500", "kind": "model", "layers": 4, "batch": 1, "context": 0, "tokens": 1500},
    ]


def _log_int(rng, lo: int, hi: int) -> int:
    return min(hi, max(lo, round(lo * (hi / lo) ** rng.random())))


def draw(rng) -> dict:
    kind = rng.choices(("blocks", "ops", "model"), weights=(8, 2, 2))[0]
    if kind == "model":
        if rng.random() < 0.5:
            return {"kind": "model", "layers": rng.randint(2, 4), "batch": rng.randint(1, 8),
                    "context": _log_int(rng, 16, 4200), "tokens": 1}
        return {"kind": "model", "layers": rng.randint(2, 4), "batch": 1, "context": 0,
                "tokens": _log_int(rng, 32, 1500)}
    config = rng.choice(("c1", "c2", "c3", "c5") if kind == "blocks" else ("c1", "c2", "c3"))
    if kind == "ops":
        return {"kind": "ops", "config": config, "tokens": _log_int(rng, 1, 500)}
    if config == "c5":
        return {"kind": "blocks", "config": config, "layers": 1, "tokens": _log_int(rng, 1, 512)}
    tokens = _log_int(rng, 1, 4000)
    return {"kind": "blocks", "config": config, "layers": 12 if tokens <= 8 else (4 if tokens <= 64 else 1),
            "tokens": tokens}


# ------------------------------------------------------------------ inputs


class _Stack(torch.nn.Module):
    def __init__(self, blocks):
        super().__init__()
        self.layers = torch.nn.ModuleList(blocks)


def _randn(gen: torch.Generator, shape, std: float) -> torch.Tensor:
    return torch.empty(shape, dtype=torch.bfloat16, device=_DEV).normal_(0.0, std, generator=gen)


def _decoder(case: dict, seed: int) -> StackedDecoder:
    cfg = replace(DECODER_CONFIGS["c4"], n_layers=case["layers"])
    gen = torch.Generator(device=_DEV)
    gen.manual_seed(seed)
    d, hq, hk, hd = cfg.d_model, cfg.n_heads, cfg.n_kv_heads, cfg.head_dim

    def ones(n):
        return torch.ones(n, dtype=torch.bfloat16, device=_DEV)

    params = {"embed": _randn(gen, (cfg.vocab, d), 1.0), "lm_head": _randn(gen, (cfg.vocab, d), 0.02),
              "final_norm": ones(d), "layers": []}
    for i in range(cfg.n_layers):
        params["layers"].append({
            "attn_norm": ones(d), "ffn_norm": ones(d), "q_norm": ones(hd), "k_norm": ones(hd),
            "q_w": _randn(gen, (hq * hd, d), 0.02), "k_w": _randn(gen, (hk * hd, d), 0.02),
            "v_w": _randn(gen, (hk * hd, d), 0.02), "o_w": _randn(gen, (d, hq * hd), 0.02),
            "moe": synthetic.make_layer(cfg.moe, layer=16 * seed + i, device=_DEV),
        })
    model = StackedDecoder(cfg, params, max_batch=case["batch"], max_seq=case["context"] + case["tokens"] + 256)
    # what a prompt leaves behind: unit-variance keys (they are RMS-normed) and values of about that size
    model.k_cache[:, :, :, :case["context"]].normal_(0.0, 1.0, generator=gen)
    model.v_cache[:, :, :, :case["context"]].normal_(0.0, 0.9, generator=gen)
    return model


def prepare(case: dict, seed: int):
    if case["kind"] == "model":
        model = _decoder(case, seed)
        gen = torch.Generator(device=_DEV)
        gen.manual_seed(seed + 1)
        ids = torch.randint(0, model.cfg.vocab, (case["batch"], case["tokens"]), generator=gen, device=_DEV)
        return {"case": case, "model": model, "ids": ids}
    cfg = synthetic.CONFIGS[case["config"]]
    n = case["tokens"]
    if case["kind"] == "ops":
        p = synthetic.make_layer(cfg, layer=16 * seed, device=_DEV)
        x = synthetic.make_tokens(cfg, n, step=seed, device=_DEV)
        return {"case": case, "cfg": cfg, "p": p, "x": x, "logits": x @ p["router_w"].T}
    blocks = [nn.block_from_params(cfg, synthetic.make_layer(cfg, layer=16 * seed + i, device=_DEV))
              for i in range(case["layers"])]
    model = patch(_Stack(blocks), patterns=["moe_mlp"])
    xs = [synthetic.make_tokens(cfg, n, step=16 * seed + i, device=_DEV) for i in range(case["layers"])]
    return {"case": case, "model": model, "xs": xs}


# ------------------------------------------------------------------ one pass


def _run_ops(state):
    cfg, p, x = state["cfg"], state["p"], state["x"]
    weights, indices = moe.topk_gating_softmax(state["logits"], cfg.top_k)
    kw = {"group_size": cfg.group_size, "mode": cfg.mode}
    act = fused_moe.gather_qmm_swiglu(x[:, None, None, :], p["gate_w"], p["gate_s"], p["gate_b"], p["up_w"], p["up_s"],
                                      p["up_b"], rhs_indices=indices, **kw)
    act = act.squeeze(-2)
    out = moe.gather_qmm_combine_quantized(act, p["down_w"], p["down_s"], p["down_b"], weights, indices, **kw)
    return {"weights": weights, "indices": indices, "act": act, "out": out}


@torch.no_grad()
def run(state):
    case = state["case"]
    if case["kind"] == "ops":
        return _run_ops(state)
    if case["kind"] == "blocks":
        return [block(x) for block, x in zip(state["model"].layers, state["xs"])]
    model, c, n = state["model"], case["context"], case["tokens"]
    model.pos = c
    logits = model.forward(state["ids"])
    return {"logits": logits, "k": model.k_cache[:, :, :, c:c + n], "v": model.v_cache[:, :, :, c:c + n]}


# ------------------------------------------------------------------ what a pass cannot do without


def _block_work(cfg, tokens: int) -> tuple[float, float]:
    """Bytes and operations of one block: the experts that this many tokens touch (in expectation, for routing as good
    as uniform) once each, the router, the token rows in and out."""
    distinct = cfg.n_experts * (1.0 - (1.0 - cfg.top_k / cfg.n_experts) ** tokens)
    nbytes = (distinct + cfg.n_shared) * cfg.expert_bytes + cfg.router_bytes + tokens * cfg.d_model * 2 * 2
    flops = 2.0 * tokens * (3 * cfg.d_model * cfg.d_ff * (cfg.top_k + cfg.n_shared) + cfg.n_experts * cfg.d_model)
    return nbytes, flops


def work(case: dict) -> dict:
    if case["kind"] == "model":
        cfg = DECODER_CONFIGS["c4"]
        d, hq, hk, hd = cfg.d_model, cfg.n_heads, cfg.n_kv_heads, cfg.head_dim
        B, S, c = case["batch"], case["tokens"], case["context"]
        nbytes, flops = _block_work(cfg.moe, B * S)
        proj = d * (2 * hq + 2 * hk) * hd
        keys = S * c + S * (S + 1) // 2  # query-key pairs per sequence
        nbytes += proj * 2 + B * 2 * hk * hd * 2 * (c + S)
        flops += 2.0 * B * S * proj + 4.0 * B * hq * hd * keys
        nbytes = case["layers"] * nbytes + cfg.vocab * d * 2 + B * S * d * 2 + B * cfg.vocab * 4
        return {"bytes": nbytes, "flops": case["layers"] * flops + 2.0 * B * cfg.vocab * d}
    cfg = synthetic.CONFIGS[case["config"]]
    nbytes, flops = _block_work(cfg, case["tokens"])
    if case["kind"] == "ops":  # the router linear is the user's; activations and results of each operator move
        rows = case["tokens"] * cfg.top_k
        nbytes += rows * (cfg.d_ff * 2 * 2 + 8) + case["tokens"] * cfg.n_experts * 2
        nbytes -= cfg.n_shared * cfg.expert_bytes + cfg.router_bytes
        flops -= 2.0 * case["tokens"] * cfg.d_model * (3 * cfg.d_ff * cfg.n_shared + cfg.n_experts)
        return {"bytes": nbytes, "flops": flops}
    return {"bytes": case["layers"] * nbytes, "flops": case["layers"] * flops}


def tolerance(case: dict) -> dict:
    if case["kind"] == "model":
        # four layers through other kernels and another order of the attention sums: 0.005 on the logits, 0.007 on
        # the keys and values of a prompt (every bfloat16 rounding of the residual stream, and the few tokens whose
        # last expert is decided by a tie)
        return {"rel": 0.03}
    if case["kind"] == "ops":
        # against float64 sums with the same bfloat16 roundings: 2e-4 to 5e-4; ranking on given logits is exact up to ties
        return {"rel": 0.002, "differ": 0.002}
    # the same 2e-4 to 5e-4; with many tokens, one in some thousands has its last expert decided by the rounding of a
    # router logit to bfloat16 (summed in another order: 1 token in 24576 of c2, 2 in 3072 of c5)
    return {"rel": 0.002 if case["tokens"] < 256 else 0.01}


# ------------------------------------------------------------------ the same in 64 bits


_E2M1 = (0.0, 0.5, 1.0, 1.5, 2.0, 3.0, 4.0, 6.0, -0.0, -0.5, -1.0, -1.5, -2.0, -3.0, -4.0, -6.0)


def _bf(v: torch.Tensor) -> torch.Tensor:
    """Where the path keeps bfloat16 between its steps, so does this: the rest is float64."""
    return v.to(torch.bfloat16).to(torch.float64)


def _matrix(cfg, p: dict, name: str, e: int) -> torch.Tensor:
    """Expert ``e``'s (N, K) weights, float64."""
    w = p[f"{name}_w"].view(torch.int32)[e]
    code = (w.unsqueeze(-1) >> torch.arange(0, 32, 4, device=w.device, dtype=torch.int32)) & 15
    code = code.reshape(w.shape[0], -1)
    s = p[f"{name}_s"][e]
    if cfg.mode == "mxfp4":
        v = torch.tensor(_E2M1, dtype=torch.float64, device=w.device)[code]
        return (v.reshape(*s.shape, -1) * torch.exp2(s.to(torch.float64) - 127.0)[..., None]).reshape(code.shape)
    v = code.to(torch.float64).reshape(*s.shape, -1) * s.to(torch.float64)[..., None]
    return (v + p[f"{name}_b"][e].to(torch.float64)[..., None]).reshape(code.shape)


def _silu_mul(g: torch.Tensor, u: torch.Tensor, per_op: bool) -> torch.Tensor:
    g, u = _bf(g), _bf(u)
    if not per_op:
        return _bf(g * torch.sigmoid(g) * u)
    y = _bf(1.0 / _bf(1.0 + _bf(torch.exp(g.abs()))))
    return _bf(_bf(g * torch.where(g < 0, y, _bf(1.0 - y))) * u)


def _experts(cfg, p: dict, x: torch.Tensor, idx: torch.Tensor, per_op: bool):
    """(h, y) of every (token, slot) pair."""
    T, K = idx.shape
    h = torch.empty((T, K, cfg.d_ff), dtype=torch.float64, device=x.device)
    y = torch.empty((T, K, cfg.d_model), dtype=torch.float64, device=x.device)
    for e in torch.unique(idx).tolist():
        t, k = (idx == e).nonzero(as_tuple=True)
        h[t, k] = _silu_mul(x[t] @ _matrix(cfg, p, "gate", e).T, x[t] @ _matrix(cfg, p, "up", e).T, per_op)
        y[t, k] = _bf(h[t, k] @ _matrix(cfg, p, "down", e).T)
    return h, y


def _largest(v: torch.Tensor, k: int) -> torch.Tensor:
    return torch.sort(v, dim=-1, descending=True, stable=True).indices[..., :k]


def _route(cfg, logits: torch.Tensor, bias):
    """(weights, indices) of the block's router on bfloat16 logits."""
    if cfg.family in ("glm", "deepseek"):
        aff = torch.sigmoid(logits)
        score = aff + bias.to(torch.float64)
        if cfg.n_group > 1:
            g = score.reshape(score.shape[0], cfg.n_group, -1)
            best = _largest(g.topk(2, dim=-1).values.sum(-1), cfg.topk_group)
            keep = torch.zeros(g.shape[:2], dtype=torch.bool, device=g.device).scatter_(1, best, True)
            score = torch.where(keep[..., None], g, torch.zeros_like(g)).reshape(score.shape)
        idx = _largest(score, cfg.top_k)
        w = aff.gather(1, idx)
        return w / w.sum(-1, keepdim=True) * cfg.routed_scaling_factor, idx
    idx = _largest(logits, cfg.top_k)
    return torch.softmax(logits.gather(1, idx), dim=-1), idx  # the same as renormalised probabilities


def exact(case: dict, seed: int):
    """What :func:`run` returns, in float64 with the path's bfloat16 hand-overs.  A decoder has none: its rounding
    travels from layer to layer."""
    if case["kind"] == "model":
        return None
    cfg, n = synthetic.CONFIGS[case["config"]], case["tokens"]
    if case["kind"] == "ops":
        p = synthetic.make_layer(cfg, layer=16 * seed, device=_DEV)
        x = synthetic.make_tokens(cfg, n, step=seed, device=_DEV)
        logits = (x @ p["router_w"].T).to(torch.float64)  # an input of the path
        idx = _largest(logits, cfg.top_k)
        w = torch.softmax(logits.gather(1, idx), dim=-1)
        h, y = _experts(cfg, p, x.to(torch.float64), idx, False)
        return {"weights": w, "indices": None, "act": h, "out": _bf((y * w[..., None]).sum(1))}
    outs = []
    for i in range(case["layers"]):
        p = synthetic.make_layer(cfg, layer=16 * seed + i, device=_DEV)
        x = synthetic.make_tokens(cfg, n, step=16 * seed + i, device=_DEV).to(torch.float64)
        w, idx = _route(cfg, _bf(x @ p["router_w"].to(torch.float64).T), p["expert_bias"])
        y = _bf((_experts(cfg, p, x, idx, cfg.mode == "mxfp4")[1] * w[..., None]).sum(1))
        if cfg.n_shared:
            zero = torch.zeros((n, 1), dtype=torch.int64, device=_DEV)
            y = _bf(y + _experts(cfg, p["shared"], x, zero, True)[1][:, 0])
        outs.append(y)
    return outs
