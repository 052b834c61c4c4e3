"""The work whose speed this repository tracks, as cases over the framework's public entry points.

A reinforcement-learning step of this framework consists of a rollout (prompts in, sampled tokens and their log-probs out), passes
that score the sampled sequences under the old and the reference policy, the advantage estimate, and the policy update: forward,
backward, optimizer.  Every case below is one such piece with the layer sizes of a preset of ``verl_b200.models.config``, cut to a few
layers where the whole model would not leave room for several states on one card, with random weights and ragged sequences.

``listed()`` names the cases, ``draw(rng)`` gives others of the same ranges, ``prepare`` / ``run`` are what a user's program does,
``work`` is what a pass cannot do without, ``tolerance`` how far another correct implementation may be off, and ``exact`` the same
outputs in 64 bits from plain torch.
"""

from __future__ import annotations

import math

import numpy as np
import torch
import torch.nn.functional as F

from verl_b200.models import DecoderModel, FlatParams
from verl_b200.models.config import get_preset
from verl_b200.ops import functional as OF
from verl_b200.ops import native
from verl_b200.trainer.ppo.prefix_grouper_utils import pack_shared_prefix_batch
from verl_b200.workers.engine.native.engine import pack_padded_batch
from verl_b200.workers.rollout.native.engine import RolloutEngine, SamplingParams

DEVICE = "cuda"


# ------------------------------------------------------------------------------------------------ the cases
def listed() -> list[dict]:
    return [
        # policy update of a group-relative method: the samples of a prompt share its tokens (the headline workload's micro-batch)
        dict(name="update 7b groups", kind="update", model="qwen2.5-7b", layers=4, groups=2, samples=5, prompt=1024, response=1024,
             recompute="none"),
        # update of a whole small model (heads of 64), single samples, gradient checkpointing
        dict(name="update 0.5b", kind="update", model="qwen2.5-0.5b", layers=24, groups=12, samples=1, prompt=512, response=1024,
             recompute="full"),
        # update of a mixture-of-experts model: router, grouped expert products, query / key norms
        dict(name="update moe", kind="update", model="qwen3-30b-a3b", layers=2, groups=8, samples=1, prompt=512, response=1024,
             recompute="none"),
        # log-probs of the old / reference policy over a large micro-batch: forward only
        dict(name="score 7b groups", kind="score", model="qwen2.5-7b", layers=4, groups=4, samples=5, prompt=1024, response=1024),
        # one short sequence scored (a teacher or a reward model that answers single requests): latency
        dict(name="score 0.5b one row", kind="score", model="qwen2.5-0.5b", layers=24, groups=1, samples=1, prompt=40, response=23),
        # greedy validation rollout, groups of samples, prefill and captured decode steps
        dict(name="generate 7b", kind="generate", model="qwen2.5-7b", layers=4, groups=16, samples=4, prompt=512, new=64, fp8=False),
        # a few prompts through a whole small model: decode steps bound by launches
        dict(name="generate 0.5b few", kind="generate", model="qwen2.5-0.5b", layers=24, groups=4, samples=1, prompt=96, new=32, fp8=False),
        # mixture-of-experts rollout with block-scaled fp8 weights (the rollout precision of that recipe)
        dict(name="generate moe fp8", kind="generate", model="qwen3-30b-a3b", layers=2, groups=32, samples=1, prompt=256, new=32, fp8=True),
        # the sampler of one decode step over a full batch of slots
        dict(name="sample", kind="sample", rows=320, vocab=152064, temperature=1.0, top_k=-1, top_p=1.0),
        # advantages with a critic: reverse scan over time, whitening over the batch
        dict(name="gae", kind="gae", rows=512, length=1024),
        # group-relative advantages: the smallest call of a step
        dict(name="group advantage", kind="group_advantage", rows=320, samples=5, length=2048),
        # the optimizer's pass over a shard: gradient norm, clipping, AdamW, refreshed bf16 weights
        dict(name="optimizer", kind="optimizer", numel=(1 << 28) + 24),
    ]


def _log_int(rng, lo: int, hi: int) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng) -> dict:
    kind = rng.choice(["update", "update", "score", "score", "generate", "generate", "sample", "gae", "group_advantage", "optimizer"])
    if kind == "sample":
        top = rng.choice([(-1, 1.0), (-1, 1.0), (rng.randint(2, 200), 1.0), (-1, round(rng.uniform(0.5, 0.99), 3))])
        return dict(kind=kind, rows=_log_int(rng, 1, 512), vocab=8 * _log_int(rng, 64, 19008),
                    temperature=rng.choice([0.0, 1.0, round(rng.uniform(0.5, 1.5), 3)]), top_k=top[0], top_p=top[1])
    if kind == "gae":
        return dict(kind=kind, rows=_log_int(rng, 1, 2048), length=_log_int(rng, 17, 2048))
    if kind == "group_advantage":
        samples = rng.randint(1, 16)
        return dict(kind=kind, rows=samples * _log_int(rng, 1, 128), samples=samples, length=_log_int(rng, 17, 4096))
    if kind == "optimizer":
        return dict(kind=kind, numel=8 * _log_int(rng, 1 << 10, 1 << 25))
    model, most_layers, most_tokens = rng.choice([("qwen2.5-7b", 4, 12000), ("llama-3.1-8b", 4, 12000), ("qwen2.5-0.5b", 24, 16000),
                                                  ("qwen3-30b-a3b", 2, 8000)])
    samples = rng.choice([1, rng.randint(2, 8)])
    case = dict(kind=kind, model=model, layers=rng.randint(max(1, most_layers // 2), most_layers))
    if kind == "generate":
        groups = _log_int(rng, 1, max(1, 64 // samples))
        prompt = _log_int(rng, 16, 512)
        return dict(case, groups=groups, samples=samples, prompt=prompt, new=rng.randint(8, 64),
                    fp8=model == "qwen3-30b-a3b" and rng.random() < 0.5)
    prompt, response = _log_int(rng, 16, 1024), _log_int(rng, 16, 1024)
    groups = _log_int(rng, 1, max(1, most_tokens // (samples * (prompt + response))))
    case.update(groups=groups, samples=samples, prompt=prompt, response=response)
    if kind == "update":
        case["recompute"] = rng.choice(["none", "full"])
    return case


# ------------------------------------------------------------------------------------------------ inputs
def _config(case: dict):
    cfg = get_preset(case["model"])
    cfg.num_hidden_layers = case["layers"]
    return cfg


def _params(case: dict, seed: int, with_grad: bool = False) -> FlatParams:
    params = FlatParams(_config(case), dtype=torch.bfloat16, device=DEVICE, with_main_grad=with_grad)
    params.init_weights(seed=seed % (1 << 30), std=0.02)
    return params


def _make_decided(params: FlatParams, model: str, seed: int):
    """Weights whose greedy next token is decided clearly, as a trained model's mostly is: the sublayers add little to the stream and the head
    reads the embedding of the token that follows in a fixed random cycle (the token itself where head and embedding are one table).
    Returns the successor of every token."""
    cfg = params.cfg
    g = torch.Generator(device=DEVICE).manual_seed(seed % (1 << 30) + 77)
    share = {"qwen2.5-7b": 0.05, "llama-3.1-8b": 0.05, "qwen2.5-0.5b": 0.4, "qwen3-30b-a3b": 0.35}[model]
    for i in range(cfg.num_hidden_layers):
        for name, w in params.layer(i).items():
            if "o_proj" in name or "down_proj" in name:
                w.mul_(share / math.sqrt(2 * cfg.num_hidden_layers))
    embed = params["embed_tokens.weight"]
    successor = torch.arange(cfg.vocab_size, device=DEVICE)
    embed.mul_(1.0 / (0.02 * math.sqrt(cfg.hidden_size)))
    if not cfg.tie_word_embeddings:
        successor = torch.randperm(cfg.vocab_size, device=DEVICE, generator=g)
        params.lm_head_weight[successor] = embed
    return successor


def _lengths(case: dict):
    """Random numbers for the ragged lengths: a matter of the case and not of the seed, so that outputs of all seeds have one shape."""
    return np.random.RandomState(sum(case.get(k, 0) * f for k, f in zip(("groups", "samples", "prompt", "response", "new", "layers"),
                                                                         (1, 31, 977, 3001, 7919, 65537))) % (1 << 31))


def _rows(case: dict, seed: int, vocab: int):
    """A padded micro-batch as the trainer hands it out: left-padded prompts, right-padded responses, ragged lengths."""
    rs = np.random.RandomState(seed % (1 << 31))
    P, R, n = case["prompt"], case["response"], case["samples"]
    lengths = _lengths(case)
    plen = np.repeat(lengths.randint(max(1, P // 2), P + 1, case["groups"]), n)
    rlen = lengths.randint(max(1, R // 4), R + 1, case["groups"] * n)
    ids = rs.randint(3, vocab, (case["groups"] * n, P + R))
    ids[:, :P] = np.repeat(ids[::n, :P], n, axis=0)
    at = np.arange(P + R)[None]
    mask = (at >= P - plen[:, None]) & (at < P + rlen[:, None])
    ids[~mask] = 0
    dev = lambda x: torch.from_numpy(x).to(DEVICE)
    return dev(ids), dev(mask.astype(np.int64)), [int(v) for v in plen], [int(v) for v in rlen]


def prepare(case: dict, seed: int) -> dict:
    kind = case["kind"]
    g = torch.Generator(device=DEVICE).manual_seed(seed % (1 << 30))
    randn = lambda *s: torch.randn(*s, device=DEVICE, generator=g)
    st = dict(case=case, kind=kind)
    if kind in ("update", "score"):
        params = _params(case, seed, with_grad=kind == "update")
        st.update(params=params, model=DecoderModel(params.cfg, params, recompute=case.get("recompute", "none"),
                                                    max_positions=case["prompt"] + case["response"] + 1))
        st["ids"], st["mask"], st["plen"], st["rlen"] = _rows(case, seed, params.cfg.vocab_size)
        n_tok = sum(st["rlen"])
        # upstream gradients of a token-mean policy loss with an entropy bonus: one advantage per row
        adv = torch.repeat_interleave(randn(len(st["rlen"])), torch.tensor(st["rlen"], device=DEVICE))
        st["g_lp"] = -adv * (1.0 + 0.1 * randn(n_tok)) / n_tok
        st["g_ent"] = torch.full((n_tok,), -0.01 / n_tok, device=DEVICE)
    elif kind == "generate":
        params = _params(case, seed)
        st["successor"] = _make_decided(params, case["model"], seed)
        rs = np.random.RandomState(seed % (1 << 31))
        n, bs = case["samples"], 64
        lens = _lengths(case).randint(max(1, case["prompt"] // 2), case["prompt"] + 1, case["groups"])
        st["prompts"] = [rs.randint(3, params.cfg.vocab_size, L).tolist() for L in lens]
        st["prompts"] = [p for p in st["prompts"] for _ in range(n)]
        pages = -(-(case["prompt"] + case["new"]) // bs)
        st["params"] = params
        st["engine"] = RolloutEngine(params.cfg, params, max_num_seqs=len(st["prompts"]), max_num_batched_tokens=8192,
                                     max_model_len=pages * bs, block_size=bs, num_blocks=len(st["prompts"]) * pages + 1, eos_token_id=-1,
                                     quantization="fp8" if case["fp8"] else None)
        st["sampling"] = SamplingParams(temperature=0.0, max_tokens=case["new"], ignore_eos=True)
    elif kind == "sample":
        st["logits"] = (randn(case["rows"], case["vocab"]) * 2.5).bfloat16()
        st["seeds"] = torch.randint(1 << 40, (case["rows"],), device=DEVICE, generator=g)
    elif kind in ("gae", "group_advantage"):
        B, L = case["rows"], case["length"]
        length = torch.randint(max(1, L // 4), L + 1, (B, 1), device=DEVICE, generator=g)
        at = torch.arange(L, device=DEVICE)[None]
        st["mask"] = (at < length).float()
        score = (torch.rand(B, 1, device=DEVICE, generator=g) * 7).floor() / 7
        st["rewards"] = torch.where(at == length - 1, score, torch.zeros_like(score)).contiguous()
        if kind == "gae":
            st["rewards"] = st["rewards"] - 0.001 * randn(B, L).abs() * st["mask"]  # a divergence penalty on every token
            st["values"] = 0.3 + 0.2 * randn(B, L)
        else:
            st["group"] = torch.arange(B, device=DEVICE) // case["samples"]
    else:
        n = case["numel"]
        st["master"] = randn(n) * 0.02
        st["grad"] = randn(n) * 1e-3
        st["m"], st["v"] = randn(n) * 1e-3, randn(n).square() * 1e-6
        st["out"] = st["master"].bfloat16()
        st["ctrl"] = torch.zeros(4, device=DEVICE)
    return st


# ------------------------------------------------------------------------------------------------ one pass
def _score(st: dict, need_grad: bool):
    case = st["case"]
    if case["samples"] > 1:
        gids = [i // case["samples"] for i in range(len(st["rlen"]))]
        batch, positions, labels, _ = pack_shared_prefix_batch(st["ids"], st["mask"], None, case["response"], gids, st["plen"], st["rlen"])
        return st["model"].forward_logprobs(batch, None, 1.0, need_grad=need_grad, positions=positions, position_labels=labels)
    lens = [p + r for p, r in zip(st["plen"], st["rlen"])]
    batch, labels, index, valid = pack_padded_batch(st["ids"], st["mask"], None, case["response"], lens)
    return st["model"].forward_logprobs(batch, labels, 1.0, need_grad=need_grad, positions=index[valid])


def run(st: dict):
    case, kind = st["case"], st["kind"]
    if kind == "score":
        with torch.no_grad():
            lp, ent = _score(st, False)
        return {"log_probs": lp, "entropy": ent}
    if kind == "update":
        params = st["params"]
        params.zero_grad()
        lp, ent = _score(st, True)
        torch.autograd.backward([lp, ent], [st["g_lp"], st["g_ent"]])
        return {"log_probs": lp.detach(), "entropy": ent.detach(), "grads": _units(params, params.main_grad)}
    if kind == "generate":
        outs = st["engine"].generate(st["prompts"], st["sampling"])
        return {"tokens": np.array([o.token_ids for o in outs]), "log_probs": np.array([o.log_probs for o in outs], dtype=np.float32)}
    if kind == "sample":
        tok, lp = OF.sample_tokens(st["logits"], case["temperature"], st["seeds"], 3, 0, case["top_k"], case["top_p"])
        return {"tokens": tok, "log_probs": lp}
    if kind == "gae":
        adv, ret = OF.gae_advantage(st["rewards"], st["values"], st["mask"], 1.0, 0.95, whiten=True)
        return {"advantages": adv, "returns": ret}
    if kind == "group_advantage":
        adv, score = OF.grpo_advantage(st["rewards"], st["mask"], st["group"], case["rows"] // case["samples"])
        return {"advantages": adv, "scores": score}
    ops = native.ops()
    st["ctrl"].zero_()
    ops.sumsq_(st["grad"], st["ctrl"])
    ops.clip_coef_(st["ctrl"], 1.0)
    ops.adamw_(st["master"], st["grad"], st["m"], st["v"], st["out"], st["ctrl"], 1e-4, 0.9, 0.999, 1e-8, 0.01, 10, 1.0, False)
    return {"weights": st["master"], "m": st["m"], "v": st["v"], "bf16": st["out"], "norm": st["ctrl"][3]}


def _units(params: FlatParams, flat: torch.Tensor) -> list[torch.Tensor]:
    """The gradient buffer cut into embedding, layers, final norm and head."""
    return [flat[slice(*params.layer_range(i))] for i in range(-1, params.cfg.num_hidden_layers + 1)]


# ------------------------------------------------------------------------------------------------ what a pass cannot do without
def _layer_weights(cfg) -> tuple[float, float]:
    """(weights of a layer, weights that a token meets in it)."""
    attn = cfg.hidden_size * (cfg.qkv_size + cfg.q_size)
    if cfg.is_moe:
        one = 3 * cfg.hidden_size * cfg.moe_intermediate_size
        router = cfg.hidden_size * cfg.num_experts
        return attn + router + cfg.num_experts * one, attn + router + cfg.num_experts_per_tok * one
    mlp = 3 * cfg.hidden_size * cfg.intermediate_size
    return attn + mlp, attn + mlp


def work(case: dict) -> dict:
    kind = case["kind"]
    if kind == "sample":
        return {"bytes": 2.0 * case["rows"] * case["vocab"], "flops": 0.0}
    if kind in ("gae", "group_advantage"):
        n = case["rows"] * case["length"]
        return {"bytes": (20.0 if kind == "gae" else 12.0) * n, "flops": 0.0}
    if kind == "optimizer":
        return {"bytes": 30.0 * case["numel"], "flops": 0.0}
    cfg = _config(case)
    L, H, V = cfg.num_hidden_layers, cfg.hidden_size, cfg.vocab_size
    stored, met = _layer_weights(cfg)
    head = float(H * V)
    p = 0.75 * case["prompt"]  # mean lengths of the ragged rows
    if kind == "generate":
        rows, new, wb = case["groups"] * case["samples"], case["new"], 1.0 if case["fp8"] else 2.0
        flops = 2.0 * L * met * case["groups"] * p + 2.0 * head * case["groups"] + (2.0 * L * met + 2.0 * head) * rows * (new - 1)
        kv = 4.0 * L * cfg.kv_size
        used = stored if not cfg.is_moe else met + (stored - met) * (1 - (1 - cfg.num_experts_per_tok / cfg.num_experts) ** rows)
        ctx = case["groups"] * p + rows * new / 2  # the samples of a prompt share its cached tokens
        bytes_ = wb * L * stored + 2.0 * head + (new - 1) * (wb * L * used + 2.0 * head + kv * ctx)
        return {"bytes": bytes_, "flops": flops}
    r = 0.625 * case["response"]
    rows = case["groups"] * case["samples"]
    tokens, predicted = case["groups"] * p + rows * r, rows * r
    pairs = case["groups"] * p * p / 2 + rows * (r * p + r * r / 2)
    passes = 3.0 if kind == "update" else 1.0
    flops = passes * (2.0 * L * met * tokens + 2.0 * head * predicted) + L * cfg.q_size * pairs * 4.0 * (3.5 if kind == "update" else 1.0)
    weights = L * stored + head + (0 if cfg.tie_word_embeddings else tokens * H)
    bytes_ = 2.0 * weights + (4.0 * (L * stored + head * (1 if cfg.tie_word_embeddings else 2)) if kind == "update" else 0.0)
    return {"bytes": bytes_, "flops": flops}


def tolerance(case: dict):
    kind = case["kind"]
    if kind == "update":
        return {"rel": 0.03, "max": 0.9}
    if kind == "score":
        return {"rel": 0.01, "max": 0.1}
    if kind == "generate":
        return {"rel": 0.02, "max": 0.3, "differ": 0.005}
    if kind == "sample":
        return {"rel": 1e-4, "max": 0.01, "differ": 0.01}
    return {"rel": 2e-5, "max": 1e-3}


# ------------------------------------------------------------------------------------------------ 64 bits, plain torch
def _norm(x, w, eps):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + eps) * w


def _rotary(cfg, n: int):
    half = torch.arange(0, cfg.head_dim, 2, dtype=torch.float64, device=DEVICE)
    inv = cfg.rope_theta ** (-half / cfg.head_dim)
    s = cfg.rope_scaling
    if s:  # long wavelengths slowed down by the factor, short ones kept, a ramp between
        turns = s["original_max_position_embeddings"] * inv / (2 * math.pi)
        keep = ((turns - s["low_freq_factor"]) / (s["high_freq_factor"] - s["low_freq_factor"])).clamp(0, 1)
        inv = keep * inv + (1 - keep) * inv / s["factor"]
    ang = torch.arange(n, dtype=torch.float64, device=DEVICE)[:, None] * inv
    return ang.cos()[:, None], ang.sin()[:, None]


def _rotate(x, cos, sin):
    a, b = x.chunk(2, -1)
    return torch.cat([a * cos - b * sin, b * cos + a * sin], -1)


def _decoder_layer(cfg, W: dict, x, cos, sin):
    T, D = x.shape[0], cfg.head_dim
    qkv = _norm(x, W["input_layernorm.weight"], cfg.rms_norm_eps) @ W["self_attn.qkv_proj.weight"].T
    if "self_attn.qkv_proj.bias" in W:
        qkv = qkv + W["self_attn.qkv_proj.bias"]
    q, k, v = (t.view(T, -1, D) for t in qkv.split([cfg.q_size, cfg.kv_size, cfg.kv_size], -1))
    if cfg.qk_norm:
        q, k = _norm(q, W["self_attn.q_norm.weight"], cfg.rms_norm_eps), _norm(k, W["self_attn.k_norm.weight"], cfg.rms_norm_eps)
    q, k = _rotate(q, cos, sin), _rotate(k, cos, sin)
    heads = []
    later = torch.ones(T, T, dtype=torch.bool, device=DEVICE).triu(1)
    per = cfg.num_attention_heads // cfg.num_key_value_heads
    for h in range(cfg.num_key_value_heads):
        s = torch.einsum("tgd,sd->gts", q[:, h * per : (h + 1) * per], k[:, h]) / math.sqrt(D)
        heads.append(torch.einsum("gts,sd->tgd", s.masked_fill(later, -math.inf).softmax(-1), v[:, h]))
    x = x + torch.cat(heads, 1).reshape(T, cfg.q_size) @ W["self_attn.o_proj.weight"].T
    h = _norm(x, W["post_attention_layernorm.weight"], cfg.rms_norm_eps)
    if not cfg.is_moe:
        gate, up = (h @ W["mlp.gate_up_proj.weight"].T).chunk(2, -1)
        return x + (F.silu(gate) * up) @ W["mlp.down_proj.weight"].T
    w, chosen = torch.topk((h @ W["mlp.gate.weight"].T).softmax(-1), cfg.num_experts_per_tok, dim=-1)
    if cfg.norm_topk_prob:
        w = w / w.sum(-1, keepdim=True)
    out = torch.zeros_like(x)
    for e in range(cfg.num_experts):
        t, j = (chosen == e).nonzero(as_tuple=True)
        if len(t):
            gate, up = (h[t] @ W["mlp.experts.gate_up_proj"][e].T).chunk(2, -1)
            y = (F.silu(gate) * up) @ W["mlp.experts.down_proj"][e].T
            out = out.index_add(0, t, y * w[t, j, None])
    return x + out


def _decoder(cfg, W: dict, ids, first: int):
    """Log-softmax of the logits at positions ``first`` .. of one sequence."""
    cos, sin = _rotary(cfg, len(ids))
    x = W["embed_tokens.weight"][ids]
    for i in range(cfg.num_hidden_layers):
        p = f"layers.{i}."
        x = _decoder_layer(cfg, {k[len(p):]: v for k, v in W.items() if k.startswith(p)}, x, cos, sin)
    x = _norm(x[first:], W["norm.weight"], cfg.rms_norm_eps)
    return F.log_softmax(x @ W.get("lm_head.weight", W["embed_tokens.weight"]).T, -1)


def _exact_rows(st: dict, grad: bool):
    case, params = st["case"], st["params"]
    cfg, P = params.cfg, case["prompt"]
    W = {}
    for n, w in params.views.items():
        w = w.double()
        W[n] = w.requires_grad_(grad) if not n.endswith(("gate_up_proj", "experts.down_proj")) else [e.clone().requires_grad_(grad) for e in w]
    lps, ents, at = [], [], 0
    for row, (p, r) in enumerate(zip(st["plen"], st["rlen"])):
        ids = st["ids"][row, P - p : P + r]
        with torch.set_grad_enabled(grad):
            logp = _decoder(cfg, W, ids[:-1], p - 1)
            lp = logp.gather(-1, ids[p:, None])[:, 0]
            ent = -(logp.exp() * logp).sum(-1)
            if grad:
                torch.autograd.backward([lp, ent], [st["g_lp"][at : at + r].double(), st["g_ent"][at : at + r].double()])
        lps.append(lp.detach())
        ents.append(ent.detach())
        at += r
    out = {"log_probs": torch.cat(lps), "entropy": torch.cat(ents)}
    if grad:
        flat = torch.zeros(params.numel, dtype=torch.float64, device=DEVICE)
        for n, w in W.items():
            o = params.offsets[n]
            for part in w if isinstance(w, list) else [w]:
                if part.grad is not None:
                    flat[o : o + part.numel()] = part.grad.reshape(-1)
                o += part.numel()
        out["grads"] = _units(params, flat)
    return out


def _exact_sample(st: dict):
    """The log-prob of the greedy token. (Which token a draw picks is the sampler's own stream of random numbers.)"""
    x = st["logits"].double()
    best = x.max(-1)
    return {"tokens": best.indices, "log_probs": best.values - x.logsumexp(-1)} if st["case"]["temperature"] == 0 else None


@torch.no_grad()
def _exact_generate(st: dict):
    case, params = st["case"], st["params"]
    W = {n: w.double() for n, w in params.views.items()}
    toks, lps = [], []
    for prompt in st["prompts"][:: case["samples"]]:
        ids = list(prompt)
        for _ in range(case["new"]):
            ids.append(int(st["successor"][ids[-1]]))
        logp = _decoder(params.cfg, W, torch.tensor(ids[:-1], device=DEVICE), len(prompt) - 1)
        best = logp.max(-1)
        toks += [best.indices] * case["samples"]
        lps += [best.values] * case["samples"]
    return {"tokens": torch.stack(toks), "log_probs": torch.stack(lps)}


def exact(case: dict, seed: int):
    kind, st = case["kind"], prepare(case, seed)
    if kind in ("update", "score"):
        return _exact_rows(st, kind == "update")
    if kind == "generate":
        return _exact_generate(st)
    if kind == "sample":
        return _exact_sample(st)
    if kind == "gae":
        r, v, m = (st[k].double() for k in ("rewards", "values", "mask"))
        gamma, lam = 1.0, 0.95
        adv, nextv, last = torch.zeros_like(r), torch.zeros_like(r[:, 0]), torch.zeros_like(r[:, 0])
        for t in reversed(range(r.shape[1])):  # a masked token hands the later value and advantage through
            step = r[:, t] + gamma * nextv - v[:, t] + gamma * lam * last
            nextv = torch.where(m[:, t] > 0, v[:, t], nextv)
            last = torch.where(m[:, t] > 0, step, last)
            adv[:, t] = last
        mean = (adv * m).sum() / m.sum()
        var = ((adv - mean).square() * m).sum() / m.sum() * (m.sum() / (m.sum() - 1).clamp(min=1))
        return {"advantages": (adv - mean) * torch.rsqrt(var + 1e-8), "returns": adv + v}
    if kind == "group_advantage":
        score = st["rewards"].double().sum(-1)
        s = score.view(-1, case["samples"])
        adv = s if case["samples"] == 1 else s - s.mean(-1, keepdim=True)
        adv = adv / ((s.std(-1, keepdim=True) if case["samples"] > 1 else 1.0) + 1e-6)
        return {"advantages": adv.reshape(-1, 1) * st["mask"].double(), "scores": score}
    p, gr, m, v = (st[k].double() for k in ("master", "grad", "m", "v"))
    norm = gr.square().sum().sqrt()
    gr = gr * (1.0 / (norm + 1e-6)).clamp(max=1.0)
    m, v = 0.9 * m + 0.1 * gr, 0.999 * v + 0.001 * gr.square()
    p = p * (1 - 1e-4 * 0.01) - 1e-4 * (m / (1 - 0.9**10)) / ((v / (1 - 0.999**10)).sqrt() + 1e-8)
    return {"weights": p, "m": m, "v": v, "bf16": p, "norm": norm}
