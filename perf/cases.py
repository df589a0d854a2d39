"""What is measured of this framework: the passes that its users spend their time on, at the sizes of the shipped recipes.

* training: one micro-batch through a pipeline stage of the decoder, forward and backward with full recomputation, gradients
  into the flat buffers of the data-parallel wrapper (``GPTModel.hidden_states``, ``DistributedDataParallel``);
* scoring and the LM head: log-probabilities of given tokens on the last stage, without gradients (reference pass) and with
  them (``GPTModel.forward_logprob``);
* rollout: prompts and decode steps over the paged cache (``ModelRunner.prefill`` / ``decode``, decode from CUDA graphs);
* serving of a layer-by-layer decoder: prompts and following tokens through ``LLMEngine.replay``.

All in bf16, which is what every recipe runs.  A stage has one to four layers of the model's own width: the layers of a stage
repeat, and so does their time.
"""
import math
import random

import torch
import torch.utils.checkpoint

from mindspeed_rl_b200 import ops
from mindspeed_rl_b200.models.gpt import GPTModel, PackedMeta
from mindspeed_rl_b200.models.transformer_config import TransformerConfig
from mindspeed_rl_b200.parallel.ddp import DistributedDataParallel
from mindspeed_rl_b200.reshard.alias import alias_rollout_weights
from mindspeed_rl_b200.rollout import serve_bench
from mindspeed_rl_b200.rollout.engine import LLMEngine
from mindspeed_rl_b200.rollout.model_runner import KVCache, ModelRunner

BLOCK = 16            # tokens of a cache block

# architectures of configs/model
MODELS = {
    "qwen25_7b": dict(num_layers=28, hidden_size=3584, ffn_hidden_size=18944, num_attention_heads=28, num_query_groups=4,
                      vocab_size=152064, add_qkv_bias=True),
    "qwen3_8b": dict(num_layers=36, hidden_size=4096, ffn_hidden_size=12288, num_attention_heads=32, num_query_groups=8,
                     vocab_size=151936, kv_channels=128, qk_layernorm=True, max_position_embeddings=40960),
    "qwen3_30b_a3b": dict(num_layers=48, hidden_size=2048, ffn_hidden_size=8192, num_attention_heads=32, num_query_groups=4,
                          vocab_size=151936, kv_channels=128, qk_layernorm=True, max_position_embeddings=40960, num_experts=128,
                          moe_router_topk=8, moe_ffn_hidden_size=768, norm_topk_prob=True, moe_aux_loss_coeff=0.001),
}


def listed():
    return [
        # a micro-batch of one short answer per row (micro_batch_size 1-4, a few hundred tokens): the smallest update
        dict(name="train_8b_short", kind="train", model="qwen3_8b", layers=2, lengths="257,611,93,520"),
        # the GRPO recipe's micro-batch: prompts of 1024 with answers of 256 to 2048 tokens, packed
        dict(name="train_7b_grpo", kind="train", model="qwen25_7b", layers=2, lengths="1280,3072,1863,2201"),
        # long-answer recipes (packing budget 32768): one near-full sequence and what fits beside it
        dict(name="train_7b_long", kind="train", model="qwen25_7b", layers=1, lengths="22528,7361,2879"),
        # expert layers at the sequence length of the larger expert recipes (8192)
        dict(name="train_30b_moe", kind="train", model="qwen3_30b_a3b", layers=1, lengths="8192,5003,3189"),
        # the last stage of an update: LM head, log-probability and entropy, and back
        dict(name="head_7b", kind="head", model="qwen25_7b", layers=1, lengths="1280,1783,1033"),
        # the reference pass: forward only, larger micro-batches
        dict(name="score_7b", kind="score", model="qwen25_7b", layers=2, lengths="1280,3072,1863,2201,2500,1517,3001,950"),
        # rollout prompts of the GRPO recipe
        dict(name="prefill_7b", kind="prefill", model="qwen25_7b", layers=4, lengths="1024,1024,1024,1024,1024,1024,1024,1024", cached=0),
        # portions of long prompts behind what is cached already (chunked prefill, multi-turn continuation)
        dict(name="prefill_8b_portion", kind="prefill", model="qwen3_8b", layers=4, lengths="2048,2048", cached=8192),
        # decode at the recipe's batch: 8 samples of each of 32 prompts, answers at different lengths
        dict(name="decode_7b_b256", kind="decode", model="qwen25_7b", layers=4, batch=256, samples=8, prompt=1024, least=1, most=1024),
        # the end of a rollout: one long sequence left
        dict(name="decode_7b_b1", kind="decode", model="qwen25_7b", layers=4, batch=1, samples=1, prompt=1024, least=1900, most=1900),
        # expert model, the tail of a rollout without shared prompts
        dict(name="decode_30b_b48", kind="decode", model="qwen3_30b_a3b", layers=2, batch=48, samples=1, prompt=700, least=1, most=3000),
        # layer-by-layer decoder: recurrent layers, latent attention, experts by table; prompts and four following tokens
        dict(name="serve_mixed", kind="serve", size="2k", lengths="2048,1531,777,3001", steps=4),
    ]


def _split(rng, total, parts):
    cuts = [rng.random() + 0.15 for _ in range(parts)]
    got = [max(1, int(total * c / sum(cuts))) for c in cuts]
    return ",".join(str(n) for n in got)


def _log(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    kind = rng.choice(["train", "train", "train", "head", "score", "prefill", "prefill", "decode", "decode", "decode", "serve"])
    if kind == "train":
        model = rng.choice(list(MODELS))
        total = _log(rng, 400, 24000)
        return dict(kind=kind, model=model, layers=1 if total > 8000 else rng.choice([1, 2]), lengths=_split(rng, total, rng.choice([1, 2, 3, 5, 8])))
    if kind == "head":
        return dict(kind=kind, model=rng.choice(["qwen25_7b", "qwen3_8b"]), layers=1, lengths=_split(rng, _log(rng, 500, 4500), rng.choice([1, 2, 4])))
    if kind == "score":
        return dict(kind=kind, model=rng.choice(["qwen25_7b", "qwen3_8b", "qwen3_30b_a3b"]), layers=rng.choice([1, 2]),
                    lengths=_split(rng, _log(rng, 1000, 16384), rng.choice([1, 3, 8])))
    if kind == "prefill":
        return dict(kind=kind, model=rng.choice(list(MODELS)), layers=2, lengths=_split(rng, _log(rng, 64, 8192), rng.choice([1, 2, 4, 8])),
                    cached=rng.choice([0, 0, 1000, 4096, 8192]))
    if kind == "decode":
        samples, prompts = rng.choice([1, 1, 4, 8]), _log(rng, 1, 32)
        least = rng.randint(1, 1000)
        return dict(kind=kind, model=rng.choice(list(MODELS)), layers=2, batch=samples * prompts, samples=samples, prompt=rng.randint(100, 1200),
                    least=least, most=least + rng.randint(0, 1500))
    return dict(kind="serve", size=rng.choice(["1k", "2k"]), lengths=_split(rng, _log(rng, 300, 7000), rng.choice([1, 2, 4])), steps=rng.randint(1, 4))


# ------------------------------------------------------------------------------------------------------------------
# states and passes
# ------------------------------------------------------------------------------------------------------------------
def _config(case, **more):
    return TransformerConfig(**{**MODELS[case["model"]], **more})


def _lengths(case):
    return [int(n) for n in case["lengths"].split(",")]


def _generator(seed, device="cuda"):
    return torch.Generator(device=device).manual_seed(int(seed) + 1)


@torch.no_grad()
def _as_trained(model):
    """Fresh weights are smaller than trained ones in two places that matter to rounding: a router's logits spread over several
    units, so that the last of the chosen experts weighs little, and the residual stream is of the order of one."""
    for layer in model.decoder.layers:
        if hasattr(layer.mlp, "router"):
            layer.mlp.router.weight.mul_(4.0)
    if model.embedding is not None:
        model.embedding.word_embeddings.weight.mul_(50.0)
    return model


def _contexts(case):
    """Keys each decoding sequence sees, its new token included: answers spread over their range, in a fixed random order."""
    b = case["batch"]
    own = [case["least"] + (case["most"] - case["least"]) * i // max(b - 1, 1) for i in range(b)]
    random.Random(3).shuffle(own)
    return [case["prompt"] + n for n in own]


def prepare(case, seed):
    g = _generator(seed)
    kind = case["kind"]
    if kind == "serve":
        size = next(s for s in serve_bench.SIZES if s.name == case["size"])
        cfg, weights = serve_bench.build(size, "mixed", torch.device("cuda"))
        lengths = _lengths(case)
        eng = LLMEngine(cfg, "cuda", max_num_seqs=len(lengths), max_num_batched_tokens=16384, max_model_len=8192, block_size=BLOCK,
                        enforce_eager=False, graph_batch_sizes=(1, 2, 4))
        eng.runner.bind_weights(weights)
        eng.init_cache(sum((n + case["steps"]) // BLOCK + 2 for n in lengths))
        ids = [torch.randint(0, size.vocab, (n + case["steps"],), generator=g, device="cuda").tolist() for n in lengths]
        return dict(kind=kind, engine=eng, ids=ids, lengths=lengths, steps=case["steps"])
    if kind in ("train", "head", "score"):
        cfg = _config(case)
        last = kind != "train"
        first = cfg.num_layers - case["layers"] if last else cfg.num_layers // 2
        model = _as_trained(GPTModel(cfg, pre_process=False, post_process=last, layer_numbers=list(range(first, first + case["layers"])),
                                     device="cuda", seed=seed))
        lengths = _lengths(case)
        t = sum(lengths)
        state = dict(kind=kind, model=model, meta=PackedMeta.from_lengths(lengths, "cuda"),
                     h=torch.randn(t, cfg.hidden_size, generator=g, device="cuda").bfloat16())
        if last:
            state["labels"] = torch.randint(0, cfg.vocab_size, (t,), generator=g, device="cuda")
        if kind != "score":
            state["ddp"] = DistributedDataParallel(model)
        if kind == "train":
            state["grad"] = (torch.randn(t, cfg.hidden_size, generator=g, device="cuda") * 0.1).bfloat16()
        if kind == "head":
            # policy-gradient weights: advantages of either sign over the number of tokens, and an entropy bonus
            state["dlogp"] = torch.randn(t, generator=g, device="cuda") / t
            state["dent"] = torch.full((t,), -0.01 / t, device="cuda")
        return state
    cfg = _config(case, num_layers=case["layers"])
    model = _as_trained(GPTModel(cfg, device="cuda", seed=seed))
    if kind == "prefill":
        lengths, cached = _lengths(case), case["cached"]
        contexts = [cached + n for n in lengths]
    else:
        contexts = _contexts(case)
    longest = max(contexts)
    blocks = [(n + BLOCK - 1) // BLOCK for n in contexts]
    width = max(blocks)
    runner = ModelRunner(cfg, "cuda", max_model_len=max(4096, (longest + 1023) // 1024 * 1024), enforce_eager=kind == "prefill",
                         graph_batch_sizes=() if kind == "prefill" else (case["batch"],))
    runner.bind_weights(alias_rollout_weights(model))
    cache = KVCache(cfg.num_layers, sum(blocks), BLOCK, cfg.num_query_groups, cfg.head_dim, cfg.params_dtype, "cuda")
    for layer in range(cfg.num_layers):
        for half in (cache.k, cache.v):
            half[layer].copy_(torch.randn(half.shape[1:], generator=g, device="cuda"))
    runner.bind_cache(cache)
    order = torch.randperm(sum(blocks), generator=g, device="cuda").to(torch.int32)
    table = torch.zeros(len(contexts), width, dtype=torch.int32, device="cuda")
    at = 0
    for i, n in enumerate(blocks):
        table[i, :n] = order[at:at + n]
        at += n
    state = dict(kind=kind, model=model, runner=runner, cfg=cfg, contexts=contexts, table=table)
    if kind == "prefill":
        pos = torch.cat([torch.arange(cached, n, device="cuda") for n in contexts])
        seq = torch.repeat_interleave(torch.arange(len(lengths), device="cuda"), torch.tensor(lengths, device="cuda"))
        state.update(ids=torch.randint(0, cfg.vocab_size, (sum(lengths),), generator=g, device="cuda"), positions=pos.to(torch.int32),
                     slots=table[seq, pos // BLOCK].long() * BLOCK + pos % BLOCK, cu_q=_cu(lengths), max_q=max(lengths), lengths=lengths,
                     last=(_cu(lengths)[1:] - 1).long(), prefix=None)
        if cached:
            key_seq = torch.repeat_interleave(torch.arange(len(contexts), device="cuda"), torch.tensor(contexts, device="cuda"))
            key_pos = torch.cat([torch.arange(n, device="cuda") for n in contexts])
            state["prefix"] = dict(block_tables=table, token_seq=key_seq.to(torch.int32), token_pos=key_pos.to(torch.int32), cu_k=_cu(contexts))
        return state
    b, samples = case["batch"], case["samples"]
    length = torch.tensor(contexts, device="cuda")
    state.update(ids=torch.randint(0, cfg.vocab_size, (b,), generator=g, device="cuda"), positions=(length - 1).to(torch.int32),
                 lens=length.to(torch.int32), longest=longest, groups=None)
    if samples > 1:
        tile = ops.decode_prefix_tile(cfg.num_attention_heads, cfg.num_query_groups, cfg.head_dim, BLOCK)
        runner.prefix_tile = tile
        start, rows, shared, any_shared = ops.build_decode_groups(
            [i // samples for i in range(b)], [case["prompt"]] * b,
            ops.decode_group_max(cfg.num_attention_heads, cfg.num_query_groups, tile), multiple=max(1, tile))
        if any_shared:
            whole = case["prompt"] // BLOCK                       # blocks that the samples of a prompt share
            table[:, :whole] = table[torch.arange(b, device="cuda") // samples * samples, :whole]
            state["groups"] = tuple(torch.tensor(x, dtype=torch.int32, device="cuda") for x in (start, rows, shared)) + (
                sum(1 for r in rows if r[0] >= 0),)
    row = torch.arange(b, device="cuda")
    state["slots"] = table[row, (length - 1) // BLOCK].long() * BLOCK + (length - 1) % BLOCK
    return state


def _cu(lengths):
    cu = [0]
    for n in lengths:
        cu.append(cu[-1] + n)
    return torch.tensor(cu, dtype=torch.int32, device="cuda")


def _gradients(model):
    return {name: p.main_grad for name, p in model.named_parameters()}


def run(s):
    kind = s["kind"]
    if kind in ("train", "head"):
        s["ddp"].zero_grad_buffer()
        h = s["h"].detach().requires_grad_(True)
        if kind == "train":
            out = s["model"].hidden_states(h, s["meta"])
            torch.autograd.backward([out], [s["grad"]])
            return {"out": out.detach(), "dh": h.grad, "grads": _gradients(s["model"])}
        logp, entropy = s["model"].forward_logprob(h, s["labels"], s["meta"], want_entropy=True)
        torch.autograd.backward([logp, entropy], [s["dlogp"], s["dent"]])
        return {"logp": logp.detach(), "entropy": entropy.detach(), "dh": h.grad, "grads": _gradients(s["model"])}
    if kind == "score":
        with torch.no_grad():
            return s["model"].forward_logprob(s["h"], s["labels"], s["meta"])[0]
    if kind == "prefill":
        return s["runner"].prefill(s["ids"], s["positions"], s["slots"], s["cu_q"], s["max_q"], s["last"], s["prefix"])
    if kind == "decode":
        return s["runner"].decode(s["ids"], s["positions"], s["slots"], s["table"], s["lens"], s["longest"], s["groups"])
    ids, names = s["ids"], [str(i) for i in range(len(s["ids"]))]
    out = [s["engine"].replay([(r, x[:n], [n - 1]) for r, x, n in zip(names, ids, s["lengths"])])]
    for k in range(s["steps"]):
        out.append(s["engine"].replay([(r, [x[n + k]], [0]) for r, x, n in zip(names, ids, s["lengths"])], names if k == s["steps"] - 1 else ()))
    return out


# ------------------------------------------------------------------------------------------------------------------
# what a pass cannot do without
# ------------------------------------------------------------------------------------------------------------------
def _layer_size(c):
    """(weights of a layer that a token meets, all weights of a layer)."""
    width = (c.num_attention_heads + 2 * c.num_query_groups) * c.head_dim
    attn = c.hidden_size * (width + c.num_attention_heads * c.head_dim)
    if c.is_moe:
        expert = 3 * c.hidden_size * c.moe_ffn_hidden_size
        return attn + c.moe_router_topk * expert + c.num_experts * c.hidden_size, attn + c.num_experts * (expert + 2 * c.hidden_size)
    return attn + 3 * c.hidden_size * c.ffn_hidden_size, attn + 3 * c.hidden_size * c.ffn_hidden_size


def work(case):
    kind = case["kind"]
    if kind == "serve":
        size = next(s for s in serve_bench.SIZES if s.name == case["size"])
        w, hd, t = size.width, size.heads * 128, sum(_lengths(case)) + case["steps"] * len(_lengths(case))
        delta = w * hd * 4 + 2 * 128 * (w + hd)
        latent = w * size.heads * (size.dn + size.dr) + w * (size.rank + size.dr) + size.rank * size.heads * (size.dn + size.dv) + w * hd
        expert = 3 * w * size.expert_ff
        per_token = 3 * delta + latent + 3 * w * size.ff + 3 * (size.top + 1) * expert
        weights = 3 * delta + latent + 3 * w * size.ff + 3 * (size.experts + 1) * expert + size.vocab * w
        pairs = sum(n * (n + 1) / 2 for n in _lengths(case))
        recurrence = 3 * t * size.heads * 8 * 128 * 128
        return {"bytes": 2.0 * weights * (1 + case["steps"]), "flops": 2.0 * t * per_token + 2.0 * pairs * size.heads * (size.dn + size.dr + size.dv) + recurrence}
    c = _config(case)
    met, whole = _layer_size(c)
    n_layers, heads = case["layers"], c.num_attention_heads * c.head_dim
    if kind == "decode":
        contexts, b = _contexts(case), case["batch"]
        seen = sum(n - case["prompt"] for n in contexts) + case["prompt"] * ((b + case["samples"] - 1) // case["samples"])
        touched = whole if not c.is_moe else whole * min(1.0, b * c.moe_router_topk / c.num_experts)
        return {"bytes": 2.0 * (n_layers * (touched + 2 * seen * c.num_query_groups * c.head_dim) + c.vocab_size * (c.hidden_size + b)),
                "flops": 2.0 * b * (n_layers * met + c.vocab_size * c.hidden_size) + 4.0 * n_layers * sum(contexts) * heads}
    lengths = _lengths(case)
    t = sum(lengths)
    cached = case.get("cached", 0)
    pairs = sum(n * cached + n * (n + 1) / 2 for n in lengths)
    layer = 2.0 * t * met + 4.0 * pairs * heads
    if kind == "prefill":
        kv = 2 * c.num_query_groups * c.head_dim * sum(cached + n for n in lengths)
        return {"bytes": 2.0 * (n_layers * (whole + kv) + c.vocab_size * c.hidden_size + t * c.hidden_size),
                "flops": n_layers * layer + 2.0 * len(lengths) * c.vocab_size * c.hidden_size}
    head = 2.0 * t * c.vocab_size * c.hidden_size
    if kind == "score":
        return {"bytes": 2.0 * (n_layers * whole + c.vocab_size * c.hidden_size + t * c.hidden_size), "flops": n_layers * layer + head}
    back = 2.0 * t * met * 2 + 10.0 * pairs * heads
    flops = n_layers * (layer + back) + (3 * head if kind == "head" else 0)
    weights = n_layers * whole + (c.vocab_size * c.hidden_size if kind == "head" else 0)
    return {"bytes": 2.0 * (2 * weights + 4 * t * c.hidden_size), "flops": flops}


def tolerance(case):
    # bf16 activations and matrix operands, 32-bit sums.  An expert whose routing weight is nearly another's may be chosen by one
    # implementation and not by the other, which moves single tokens.
    if case.get("model") == "qwen3_30b_a3b":
        return {"rel": 0.03, "max": 0.99}
    return {"rel": 0.02, "max": 0.5}


# ------------------------------------------------------------------------------------------------------------------
# the same in 64 bits, plain torch
# ------------------------------------------------------------------------------------------------------------------
def _rms(x, weight, eps):
    return x / torch.sqrt(x.square().mean(-1, keepdim=True) + eps) * weight


def _turn(x, pos, base):
    """Rotary positions, first half of a head paired with the second; ``x [T, heads, d]``."""
    d = x.shape[-1]
    a = pos.double()[:, None] * base ** (-torch.arange(0, d, 2, device=x.device, dtype=torch.float64) / d)
    cos, sin = torch.cos(a)[:, None], torch.sin(a)[:, None]
    u, v = x[..., :d // 2], x[..., d // 2:]
    return torch.cat([u * cos - v * sin, v * cos + u * sin], -1)


def _attend(q, k, v, offset, scale=None):
    """Causal attention of one sequence, ``q [n, heads, d]`` behind ``offset`` earlier keys; queries in portions."""
    rep, scale = q.shape[1] // k.shape[1], scale or q.shape[-1] ** -0.5
    kh, vh = k.transpose(0, 1), v.transpose(0, 1)                                   # [groups, keys, d]

    def part(qp, kp, vp, first):
        n, g = qp.shape[0], kp.shape[0]
        s = torch.einsum("nghd,gkd->ghnk", qp.reshape(n, g, rep, -1), kp) * scale
        hidden = torch.arange(kp.shape[1], device=q.device)[None] > torch.arange(first, first + n, device=q.device)[:, None]
        p = torch.softmax(s.masked_fill(hidden, -math.inf), -1)
        return torch.einsum("ghnk,gkd->nghd", p, vp).reshape(n, g * rep, -1)

    out, step = [], max(64, min(1024, 2 ** 28 // (q.shape[1] * k.shape[0])))
    for a in range(0, q.shape[0], step):
        b = min(a + step, q.shape[0])
        args = (q[a:b], kh[:, :offset + b], vh[:, :offset + b], offset + a)
        out.append(torch.utils.checkpoint.checkpoint(part, *args, use_reentrant=False) if torch.is_grad_enabled() else part(*args))
    return torch.cat(out)


def _experts(x, p, c, with_aux):
    scores = torch.softmax(x @ p["mlp.router.weight"].t(), -1)
    top, idx = scores.topk(c.moe_router_topk, -1)
    weight = top / (top.sum(-1, keepdim=True) + 1e-20)
    f = c.moe_ffn_hidden_size
    w1, w2 = p["mlp.experts.weight1"].view(c.hidden_size, c.num_experts, 2 * f), p["mlp.experts.weight2"].view(c.num_experts, f, c.hidden_size)
    out = torch.zeros_like(x)
    for e in range(c.num_experts):
        tok, slot = torch.nonzero(idx == e, as_tuple=True)
        if tok.numel():
            gu = x[tok] @ w1[:, e]
            y = (torch.nn.functional.silu(gu[:, :f]) * gu[:, f:]) @ w2[e]
            out = out.index_add(0, tok, y * weight[tok, slot, None])
    if not with_aux:
        return out, 0.0
    share = torch.bincount(idx.reshape(-1), minlength=c.num_experts).double() / idx.numel()
    return out, c.moe_aux_loss_coeff * c.num_experts * (share * scores.mean(0)).sum()


def _layer64(p, c, h, pos, attend, with_aux=False):
    """One layer; ``attend(q, k, v)`` gets the heads of all tokens."""
    eps, nh, nkv, d = c.norm_epsilon, c.num_attention_heads, c.num_query_groups, c.head_dim
    qkv = _rms(h, p["input_layernorm.weight"], eps) @ p["self_attention.linear_qkv.weight"].t()
    if c.add_qkv_bias:
        qkv = qkv + p["self_attention.linear_qkv.bias"]
    parts = qkv.view(-1, nkv, nh // nkv + 2, d)
    q, k, v = parts[:, :, :-2].reshape(-1, nh, d), parts[:, :, -2], parts[:, :, -1]
    if c.qk_layernorm:
        q, k = _rms(q, p["self_attention.q_layernorm.weight"], eps), _rms(k, p["self_attention.k_layernorm.weight"], eps)
    o = attend(_turn(q, pos, c.rotary_base), _turn(k, pos, c.rotary_base), v)
    h = h + o.reshape(h.shape[0], -1) @ p["self_attention.linear_proj.weight"].t()
    x = _rms(h, p["pre_mlp_layernorm.weight"], eps)
    if c.is_moe:
        out, aux = _experts(x, p, c, with_aux)
        return h + out, aux
    gu = x @ p["mlp.linear_fc1.weight"].t()
    f = c.ffn_hidden_size
    return h + (torch.nn.functional.silu(gu[:, :f]) * gu[:, f:]) @ p["mlp.linear_fc2.weight"].t(), 0.0


def _layer_weights(weights, i):
    lead = f"decoder.layers.{i}."
    return {n[len(lead):]: w for n, w in weights.items() if n.startswith(lead)}


def _exact_stage(case, s):
    c = s["model"].cfg
    lengths = _lengths(case)
    grads = case["kind"] != "score"
    weights = {n: p.detach().double().requires_grad_(grads) for n, p in s["model"].named_parameters()}
    h0 = s["h"].double().requires_grad_(grads)
    h, pos, loss = h0, torch.cat([torch.arange(n, device="cuda") for n in lengths]), 0.0

    def attend(q, k, v):
        return torch.cat([_attend(*x, 0) for x in zip(q.split(lengths), k.split(lengths), v.split(lengths))])

    with torch.set_grad_enabled(grads):
        for i in range(case["layers"]):
            h, aux = _layer64(_layer_weights(weights, i), c, h, pos, attend, grads)
            loss = loss + aux
        result = {}
        if case["kind"] == "train":
            result["out"] = h.detach()
            loss = loss + (h * s["grad"].double()).sum()
        else:
            x = _rms(h, weights["decoder.final_layernorm.weight"], c.norm_epsilon)
            logp, ent = [], []
            for a in range(0, x.shape[0], 2048):
                z = torch.log_softmax(x[a:a + 2048] @ weights["output_layer.weight"].t(), -1)
                logp.append(z.gather(-1, s["labels"][a:a + 2048, None])[:, 0])
                if grads:
                    ent.append(-(z.exp() * z).sum(-1))
                del z
            logp = torch.cat(logp)
            if not grads:
                return logp
            ent = torch.cat(ent)
            result.update(logp=logp.detach(), entropy=ent.detach())
            loss = loss + (logp * s["dlogp"].double()).sum() + (ent * s["dent"].double()).sum()
        names = list(weights)
        got = torch.autograd.grad(loss, [h0] + [weights[n] for n in names])
    return {**result, "dh": got[0], "grads": dict(zip(names, got[1:]))}


@torch.no_grad()
def _exact_rollout(s):
    c, model, cache = s["cfg"], s["model"], s["runner"].cache
    weights = {n: p.detach().double() for n, p in model.named_parameters() if n.startswith("decoder.")}
    new = s.get("lengths") or [1] * len(s["contexts"])
    h, pos = model.embedding.word_embeddings.weight[s["ids"]].double(), s["positions"]
    for i in range(c.num_layers):
        def attend(q, k, v):
            out = []
            for j, (n, m, qs, ks, vs) in enumerate(zip(s["contexts"], new, q.split(new), k.split(new), v.split(new))):
                rows = s["table"][j, :(n + BLOCK - 1) // BLOCK].long()
                old_k, old_v = (half[i][rows].flatten(0, 1)[:n - m].double() for half in (cache.k, cache.v))
                out.append(_attend(qs, torch.cat([old_k, ks]), torch.cat([old_v, vs]), n - m))
            return torch.cat(out)

        h, _ = _layer64(_layer_weights(weights, i), c, h, pos, attend)
    if "last" in s:
        h = h[s["last"]]
    return _rms(h, weights["decoder.final_layernorm.weight"], c.norm_epsilon) @ model.output_weight().double().t()


def _short_conv(x, w):
    """Causal convolution per channel over the token axis of ``x [B, T, C]``, ``w [C, taps]``, then silu."""
    taps = w.shape[1]
    padded = torch.nn.functional.pad(x, (0, 0, taps - 1, 0))
    return torch.nn.functional.silu(sum(padded[:, i:i + x.shape[1]] * w[:, i] for i in range(taps)))


def _delta64(h, w, m, eps):
    """Gated delta rule with a decay per key channel, token by token; ``h [B, T, W]``."""
    b, t, _ = h.shape
    hn, d, dv = m.heads, m.dim, m.vdim

    def unit(x):
        return x / torch.sqrt(x.square().sum(-1, keepdim=True) + 1e-6)

    q, k, v = (_short_conv(h @ w[n].t(), w[n + ".conv"]).view(b, t, hn, -1) for n in "qkv")
    q, k = unit(q) * d ** -0.5, unit(k)
    beta = torch.sigmoid(h @ w["b"].t())
    rate = torch.nn.functional.softplus(h @ w["a1"].t() @ w["a2"].t() + w["dt_bias"]).view(b, t, hn, d)
    decay = torch.exp(-torch.exp(w["A_log"]).view(hn, 1) * rate)
    state, out = torch.zeros(b, hn, d, dv, dtype=h.dtype, device=h.device), torch.empty_like(v)
    for i in range(t):
        state = state * decay[:, i, :, :, None]
        u = beta[:, i, :, None] * (v[:, i] - (state * k[:, i, :, :, None]).sum(2))
        state = state + k[:, i, :, :, None] * u[:, :, None]
        out[:, i] = (state * q[:, i, :, :, None]).sum(2)
    gate = torch.sigmoid(h @ w["g1"].t() @ w["g2"].t()).view(b, t, hn, dv)
    return (_rms(out, w["norm"], eps) * gate).reshape(b, t, hn * dv) @ w["o"].t()


def _latent64(h, w, m, eps):
    b, t, _ = h.shape
    pos = torch.arange(t, device=h.device)

    def turn(x):                                                                     # neighbours of [T, heads, d] are a pair
        a = pos.double()[:, None, None] * m.rot.base ** (-torch.arange(0, m.rot_dim, 2, device=h.device).double() / m.rot_dim)
        u, v = x[..., 0::2], x[..., 1::2]
        return torch.stack([u * a.cos() - v * a.sin(), v * a.cos() + u * a.sin()], -1).flatten(-2)

    out = []
    for x in h:
        q = (x @ w["q"].t()).view(t, m.heads, m.dim + m.rot_dim)
        row = x @ w["dkv"].t()
        c = _rms(row[:, :m.kv_rank], w["dkv.norm"], eps)
        kr = turn(row[:, None, m.kv_rank:]).expand(-1, m.heads, -1)
        k = torch.cat([(c @ w["uk"].t()).view(t, m.heads, m.dim), kr], -1)
        q = torch.cat([q[..., :m.dim], turn(q[..., m.dim:])], -1)
        out.append(_attend(q, k, (c @ w["uv"].t()).view(t, m.heads, m.vdim), 0, m.scale).reshape(t, -1) @ w["o"].t())
    return torch.stack(out)


def _glu64(x, gate, up, down, spec):
    g, u = x @ gate.t(), x @ up.t()
    if spec.act == "gelu_tanh":
        return (torch.nn.functional.gelu(g, approximate="tanh") * u) @ down.t()
    g, u = g.clamp(max=spec.limit), u.clamp(-spec.limit, spec.limit)
    return (g * torch.sigmoid(spec.alpha * g) * (u + 1)) @ down.t()


def _table_experts64(x, ids, w, m):
    out = torch.sigmoid(x @ w["shared.sg"].t()) * _glu64(x, w["shared.gate"], w["shared.up"], w["shared.down"], m.shared)
    chosen = w["table"][ids]
    for e in range(m.experts):
        tok = torch.nonzero((chosen == e).any(-1))[:, 0]
        if tok.numel():
            out = out.index_add(0, tok, _glu64(x[tok], w[f"e{e}.gate"], w[f"e{e}.up"], w[f"e{e}.down"], m.expert) / m.top)
    return out


@torch.no_grad()
def _exact_serve(case, s):
    size = next(z for z in serve_bench.SIZES if z.name == case["size"])
    cfg = s["engine"].cfg
    stored = {n: x if n.endswith(".table") else x.double() for n, x in serve_bench.random_state(cfg, torch.device("cuda")).items()}
    longest, b = max(s["lengths"]) + s["steps"], len(s["ids"])
    ids = torch.tensor([x + [0] * (longest - len(x)) for x in s["ids"]], device="cuda")   # what follows a sequence does not reach it
    h = stored["embed"][ids] * cfg.embedding_scale

    def under(lead):
        return {n[len(lead):]: x for n, x in stored.items() if n.startswith(lead)}

    for i, layer in enumerate(cfg.layers):
        mixer = _latent64 if layer.type == "latent_attention" else _delta64
        h = h + mixer(_rms(h, 1 + stored[f"l{i}.norm1"], cfg.norm_epsilon), under(f"l{i}.mix."), layer.mixer, cfg.norm_epsilon)
        x, w = _rms(h, 1 + stored[f"l{i}.norm2"], cfg.norm_epsilon).view(b * longest, size.width), under(f"l{i}.mlp.")
        if "table" in w:
            y = _table_experts64(x, ids.view(-1), w, layer.mlp)
        else:
            y = _glu64(x, w["gate"], w["up"], w["down"], layer.mlp)
        h = h + y.view_as(h)
    x = _rms(h, 1 + stored["final.norm"], cfg.norm_epsilon)
    row = torch.arange(b, device="cuda")
    return [x[row, torch.tensor(s["lengths"], device="cuda") - 1 + k] @ stored["embed"].t() for k in range(1 + s["steps"])]


def exact(case, seed):
    s = prepare(case, seed)
    if case["kind"] == "serve":
        return _exact_serve(case, s)
    if case["kind"] in ("prefill", "decode"):
        return _exact_rollout(s)
    return _exact_stage(case, s)
