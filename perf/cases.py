"""The work that the framework's speed is measured on: steps of the models it serves, as the engine runs them.

A pass is one step of a model whose weights, paged caches and recurrent states are on the GPU: embedding, decoder layers,
final norm and the logits of the rows that would be sampled.  Steps of decode rows only replay the CUDA graph that the engine
captures for them (``ModelRunner.capture_graphs``, batch rounded up to its bucket); steps with prompt tokens run eagerly
through the model under a forward context, as the engine and ``engine/static_workload.py`` do.  Prompts are uniform-random
tokens, weights are the loader's seeded random ones, caches hold random context, pages lie in random order.

Models, at the widths of the configurations that the benchmark and the hybrid benchmark name and with their full
vocabularies, but with 2 to 4 layers, since a layer's time does not depend on how many there are (the head of 128 k to
152 k rows weighs more here than in the whole model):

* ``llama``    Llama-3.1-8B, bf16
* ``llama70b`` Llama-3.1-70B, bf16 weights, int8 cache with a scale per token and head
* ``moe``      Qwen3-30B-A3B style, 128 experts, top 8, bf16
* ``deepseek`` DeepSeek-V3 (latent attention, grouped sigmoid routing, shared expert), fp8 weights in 128 x 128 blocks; a
               dense and two expert layers with 64 of its 256 experts, a share under expert parallelism
* ``next``     Qwen3-Next: three gated-delta-rule layers and one of gated attention (head size 256), 64 experts, top 8

``listed`` and ``draw`` speak of a step by its rows: ``decodes`` rows of one token with up to ``context`` cached tokens, and
``prompts`` portions of up to ``tokens`` tokens behind up to ``past`` cached ones (a prompt cut by the scheduler).  ``even``
rows are all as long as the largest; the others are spread between a sixteenth of it and all of it.
"""
from __future__ import annotations

import math
import random

import torch

BLOCK = 64
_MAX_POSITION = 65536

_LLAMA = dict(architecture="LlamaForCausalLM", vocab_size=128256, rms_norm_eps=1e-5, rope_theta=500000.0, num_key_value_heads=8,
              head_dim=128, max_position_embeddings=_MAX_POSITION)
MODELS = {
    "llama": dict(_LLAMA, hidden_size=4096, intermediate_size=14336, num_hidden_layers=4, num_attention_heads=32),
    "llama70b": dict(_LLAMA, hidden_size=8192, intermediate_size=28672, num_hidden_layers=2, num_attention_heads=64),
    "moe": dict(architecture="Qwen3MoeForCausalLM", vocab_size=151936, hidden_size=2048, intermediate_size=6144,
                num_hidden_layers=4, num_attention_heads=32, num_key_value_heads=4, head_dim=128, rms_norm_eps=1e-6,
                rope_theta=1000000.0, max_position_embeddings=_MAX_POSITION, qk_norm=True, num_experts=128,
                num_experts_per_tok=8, moe_intermediate_size=768, norm_topk_prob=True),
    "deepseek": dict(architecture="DeepseekV3ForCausalLM", vocab_size=129280, hidden_size=7168, intermediate_size=18432,
                     num_hidden_layers=3, num_attention_heads=128, num_key_value_heads=128, rms_norm_eps=1e-6,
                     rope_theta=10000.0, max_position_embeddings=_MAX_POSITION, q_lora_rank=1536, kv_lora_rank=512,
                     qk_nope_head_dim=128, qk_rope_head_dim=64, v_head_dim=128, first_k_dense_replace=1, num_experts=64,
                     num_experts_per_tok=8, moe_intermediate_size=2048, n_shared_experts=1, scoring_func="sigmoid", n_group=8,
                     topk_group=4, routed_scaling_factor=2.5, topk_method="noaux_tc", norm_topk_prob=True, quantization="fp8",
                     quant_config={"quant_method": "fp8", "weight_block_size": [128, 128]}),
    "next": dict(architecture="Qwen3NextForCausalLM", vocab_size=151936, hidden_size=2048, intermediate_size=5440,
                 num_hidden_layers=4, num_attention_heads=16, num_key_value_heads=2, head_dim=256, rms_norm_eps=1e-6,
                 rope_theta=10000000.0, max_position_embeddings=_MAX_POSITION, qk_norm=True, num_experts=64,
                 num_experts_per_tok=8, moe_intermediate_size=512, n_shared_experts=1, shared_expert_intermediate_size=512,
                 norm_topk_prob=True,
                 hf_config=dict(linear_num_value_heads=32, linear_num_key_heads=16, linear_key_head_dim=128,
                                linear_value_head_dim=128, linear_conv_kernel_dim=4, full_attention_interval=4)),
}


def _case(model, decodes=0, context=0, prompts=0, tokens=0, past=0, even=False, name=None):
    c = dict(model=model, decodes=decodes, context=context, prompts=prompts, tokens=tokens, past=past, even=even)
    return c if name is None else dict(c, name=name)


def listed():
    return [
        # one user in a chat: the smallest step there is, every weight read for one token
        _case("llama", 1, 900, name="llama_decode_1"),
        # a server under light load, requests of all ages
        _case("llama", 40, 2048, name="llama_decode_40"),
        # the headline benchmark's decode step: 256 requests of 1024 + 128 tokens, half way through
        _case("llama", 256, 1088, even=True, name="llama_decode_256"),
        # the headline benchmark's prefill step
        _case("llama", prompts=8, tokens=1024, even=True, name="llama_prompts_8x1024"),
        # chunked prefill under load: decode rows beside new prompts and the rest of longer ones
        _case("llama", 37, 1500, 3, 777, 1000, name="llama_mixed"),
        # long contexts from a quantised cache
        _case("llama70b", 16, 32768, name="llama70b_int8_decode_16"),
        # expert models: decode, and prompts
        _case("moe", 64, 2048, name="moe_decode_64"),
        _case("moe", prompts=4, tokens=2048, even=True, name="moe_prompts_4x2048"),
        # latent attention and block-scaled fp8: decode, and prompts
        _case("deepseek", 64, 4096, name="deepseek_decode_64"),
        _case("deepseek", prompts=3, tokens=1000, name="deepseek_prompts_3x1000"),
        # recurrent layers: decode, and prompts
        _case("next", 64, 2048, name="next_decode_64"),
        _case("next", prompts=4, tokens=2048, name="next_prompts_4x2048"),
    ]


# the most of a drawn case: decode rows, cached tokens of all decode rows, prompt tokens, cached tokens before a portion
_LIMITS = {"llama": (256, 278528, 8192, 2048), "llama70b": (32, 300000, 2048, 2048), "moe": (256, 278528, 8192, 2048),
           "deepseek": (128, 150000, 3000, 1024), "next": (128, 150000, 8192, 2048)}


def draw(rng):
    model = rng.choice(["llama", "llama", "llama70b", "moe", "moe", "deepseek", "next"])
    rows, cached, toks, past = _LIMITS[model]
    log = lambda lo, hi: int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    c = _case(model, even=False)
    kind = rng.choice(["decode", "decode", "prompt", "prompt", "mixed"])
    if kind != "prompt":
        c["decodes"] = log(1, rows if kind == "decode" else rows // 4)
        c["context"] = min(32768, log(16, cached // c["decodes"]) if c["decodes"] < cached // 16 else 16)
    if kind != "decode":
        total = log(33, toks if kind == "prompt" else toks // 2)
        c["prompts"] = min(log(1, 16), max(1, total // 24))
        c["tokens"] = max(1, total // c["prompts"])
        c["past"] = rng.choice([0, 0, log(16, past)])
    return c


# ------------------------------------------------------------------------------------------------ rows of a step
def _rows(case):
    """``[(cached tokens, new tokens)]``, decode rows first; the same for every seed."""
    rng = random.Random("%(model)s %(decodes)s %(context)s %(prompts)s %(tokens)s %(past)s" % case)
    size = lambda top: top if case["even"] or top <= 1 else rng.randint(max(1, top // 16), top)
    rows = [(size(case["context"]), 1) for _ in range(case["decodes"])]
    rows += [(size(case["past"]) if case["past"] else 0, size(case["tokens"])) for _ in range(case["prompts"])]
    return rows


def _bucket(n):
    """Rows of the captured graph that the engine would replay for ``n`` decode rows."""
    for b in (1, 2, 4, 8):
        if n <= b:
            return b
    return -(-n // 16) * 16 if n <= 128 else -(-n // 32) * 32


# ------------------------------------------------------------------------------------------------ what a program holds
def _config(case, seed):
    from vllm_metax_b200 import ModelConfig

    return ModelConfig(dtype=torch.bfloat16, seed=seed, **MODELS[case["model"]])


@torch.no_grad()
def prepare(case, seed):
    from vllm_metax_b200 import LLM
    from vllm_metax_b200.attention.metadata import AttentionMetadata

    rows = _rows(case)
    graph = case["prompts"] == 0
    B = _bucket(len(rows)) if graph else len(rows)
    longest = max(a + b for a, b in rows)
    T = B if graph else sum(b for _, b in rows)
    pages = [-(-(a + b) // BLOCK) for a, b in rows]
    model_len = max(2048, 1 << (longest - 1).bit_length())
    llm = LLM(_config(case, seed), device="cuda", block_size=BLOCK, max_model_len=model_len, max_num_seqs=B,
              max_num_batched_tokens=max(T, B), num_gpu_blocks=sum(pages) + 1, load_format="dummy", enforce_eager=True, seed=seed,
              kv_cache_dtype="int8_per_token_head" if case["model"] == "llama70b" else "auto")
    r = llm.engine.runner
    dev = r.device
    g = torch.Generator(device=dev).manual_seed(seed)
    for name, p in r.model.named_parameters():
        if name.endswith(".dt_bias"):          # step sizes between 1e-3 and 0.1, decay rates between 1 and 16
            dt = torch.exp(torch.rand(p.shape, generator=g, device=dev) * math.log(100.0) + math.log(1e-3))
            p.data.copy_(torch.log(torch.expm1(dt)))
        elif name.endswith(".A_log"):
            p.data.copy_(torch.log(torch.rand(p.shape, generator=g, device=dev) * 15 + 1))
        elif name.endswith("embed_tokens.weight"):
            p.data.mul_(50.0)                  # a stream as large as what a layer adds to it, with a direction all tokens share;
            p.data.add_(_shared(p))            # where codes of 8 bits turn every rounding into one of theirs, as deep in a model,
            if case["model"] == "deepseek":    # where it is much larger
                p.data.mul_(8.0)
        elif name.endswith(".gate.weight"):
            _decided(p, case["model"])
        elif name.endswith(".e_score_correction_bias"):
            p.data.mul_(0.1)
    for c in r.kv_caches:                      # what earlier steps left: context
        t, scales = (c["mla"], None) if isinstance(c, dict) else c
        if t.dtype == torch.int8:
            t.copy_(torch.randint(-127, 128, t.shape, generator=g, device=dev, dtype=torch.int8))
            scales.uniform_(0.004, 0.016, generator=g)
        else:
            t.normal_(generator=g)
    for conv, ssm in _states(r.model):
        conv.normal_(generator=g)
        ssm.normal_(generator=g).mul_(0.1)
    table = torch.zeros(B, r.max_blocks_per_seq, dtype=torch.int32)
    order = (torch.randperm(sum(pages), generator=g, device=dev) + 1).to(torch.int32).cpu()      # (page 0: rows that pad a graph)
    at, slots, pos = 0, [], []
    for i, (a, b) in enumerate(rows):
        table[i, : pages[i]] = order[at: at + pages[i]]
        at += pages[i]
        p = torch.arange(a, a + b)
        pos.append(p)
        slots.append(table[i, p // BLOCK].long() * BLOCK + p % BLOCK)
    pad = B - len(rows)
    pos = torch.cat(pos + [torch.zeros(pad, dtype=torch.int64)]).to(dev)
    slots = torch.cat(slots + [torch.full((pad,), -1)]).to(dev)
    lens = torch.tensor([a + b for a, b in rows] + [1] * pad, dtype=torch.int32)
    starts = torch.tensor([0] + [b for _, b in rows] + [1] * pad, dtype=torch.int32).cumsum(0).to(torch.int32)
    ids = torch.randint(0, r.cfg.model.vocab_size, (T,), generator=g, device=dev)
    state = {"llm": llm, "runner": r, "rows": rows, "ids": ids, "pos": pos, "slots": slots, "table": table.to(dev),
             "caches": [[c["mla"]] if isinstance(c, dict) else [t for t in c if t is not None] for c in r.kv_caches],
             "states": [list(s) for s in _states(r.model)]}
    if graph:
        r.use_graphs = True
        r.capture_graphs([B])
        r.input_ids[:B], r.positions[:B], r.slot_mapping[:B] = ids, pos, slots
        r.seq_lens[:B], r.block_table[:B] = lens.to(dev), state["table"]
        r.query_start_loc[: B + 1] = starts.to(dev)
        if r.state_slots is not None:
            scratch = r.max_seqs
            idx = torch.tensor(list(range(len(rows))) + [scratch] * pad, dtype=torch.int32)
            r.state_dev[:B] = idx.to(dev)
            r.state_dev[scratch: scratch + B] = torch.tensor([1] * len(rows) + [0] * pad, dtype=torch.int32, device=dev)
        state["graph"], state["logits"], _ = r.graphs[B]
        return state
    n = case["decodes"]
    md = AttentionMetadata(
        num_tokens=T, num_reqs=B, num_decodes=n, num_decode_tokens=n, query_start_loc=starts.to(dev), seq_lens=lens.to(dev),
        block_table=state["table"], slot_mapping=slots, max_query_len=max(b for _, b in rows), max_seq_len=longest,
        block_size=BLOCK, query_start_loc_cpu=starts, seq_lens_cpu=lens,
        prefill_query_start_loc=(starts[n:] - n).to(dev), max_prefill_query_len=max(b for _, b in rows))
    md.extra["prefill_no_context"] = all(a == 0 for a, _ in rows[n:])
    if r.state_slots is not None:
        md.extra["state_indices"] = torch.arange(B, dtype=torch.int32, device=dev)
        md.extra["state_has_init"] = torch.tensor([int(a > 0) for a, _ in rows], dtype=torch.int32, device=dev)
    state["metadata"] = md
    state["last"] = (starts[1:] - 1).long().to(dev)
    return state


def _shared(p):
    """The direction that all hidden states share: entries of one size and of alternating sign."""
    d = torch.ones(p.shape[-1], dtype=p.dtype, device=p.device)
    d[1::2] = -1
    return d


def _decided(p, model):
    """A router that prefers some experts clearly, as trained ones do (with the loader's, the chosen experts weigh about the
    same and the last of them is a toss-up): logits spread by 3, and for sigmoid scores low on average."""
    d, w = _shared(p).float(), p.data.float()
    w -= (w @ d)[:, None] * d / d.numel()
    w *= 3.0 / w.std() / math.sqrt(d.numel())
    if model == "deepseek":
        w -= 8.0 / d.numel() * d
    p.data.copy_(w)


def _states(model):
    """The convolution carry and the matrix state of every recurrent layer."""
    if not hasattr(model, "allocate_state"):
        return []
    return [(l.linear_attn.conv_state, l.linear_attn.ssm_state) for l in model.model.layers.values() if hasattr(l, "linear_attn")]


@torch.no_grad()
def run(state):
    from vllm_metax_b200.attention.metadata import ForwardContext, set_forward_context

    out = {"caches": state["caches"], "states": state["states"]}
    if "graph" in state:
        state["graph"].replay()
        out["logits"] = state["logits"][: len(state["rows"])]
        return out
    r = state["runner"]
    with set_forward_context(ForwardContext(state["metadata"], r.kv_caches, state["pos"])):
        h = r.model(state["ids"], state["pos"])
    out["hidden"] = h
    out["logits"] = r.model.compute_logits(h.index_select(0, state["last"]))
    return out


# ------------------------------------------------------------------------------------------------ what a pass costs
def work(case):
    m, rows = MODELS[case["model"]], _rows(case)
    T, R = sum(b for _, b in rows), len(rows)
    W, V, L, H, D = m["hidden_size"], m["vocab_size"], m["num_hidden_layers"], m["num_attention_heads"], m.get("head_dim", 128)
    Hkv = m["num_key_value_heads"]
    pairs = sum(b * a + b * (b + 1) // 2 for a, b in rows)              # (query, key) pairs under the causal mask
    cached, total = sum(a for a, _ in rows), sum(a + b for a, b in rows)
    E, k = m.get("num_experts", 0), m.get("num_experts_per_tok", 0)
    hit = E * (1 - (1 - k / E) ** T) if E else 0
    by = 2.0 * V * W + 2.0 * T * W + 2.0 * R * V + 10.0 * T             # head, embedding rows, logits, ids
    fl = 2.0 * V * W * R
    if case["prompts"]:
        by += 2.0 * T * W                                               # hidden states are handed out
    for i in range(L):
        if case["model"] == "deepseek":
            q, kv, nope, rope, v = m["q_lora_rank"], m["kv_lora_rank"], 128, 64, 128
            fp8 = W * (q + kv + rope) + q * H * (nope + rope) + H * v * W
            by += fp8 + 2.0 * kv * H * (nope + v) + 2.0 * (kv + rope) * total
            fl += 2.0 * T * (fp8 + kv * H * (nope + v))
            fresh = case["decodes"] == 0 and cached == 0
            fl += 2.0 * H * pairs * ((nope + rope + v) if fresh else (2 * kv + rope))
            ff, one, shared = m["intermediate_size"], 1.0, m["moe_intermediate_size"]
        elif case["model"] == "next" and (i + 1) % 4:
            nk, nv, d = 16, 32, 128
            w = W * (2 * nk * d + 2 * nv * d + 2 * nv) + nv * d * W
            by += 2.0 * w + 2 * 4.0 * R * nv * d * d + 2 * 2.0 * R * 3 * (2 * nk + nv) * d
            fl += 2.0 * T * w + 6.0 * T * nv * d * d
            one, shared = 2.0, m["shared_expert_intermediate_size"]
        else:
            gate = H * D if case["model"] == "next" else 0
            w = W * (H * D + gate + 2 * Hkv * D) + H * D * W
            per = Hkv * (2 * D + 8) if case["model"] == "llama70b" else 4.0 * Hkv * D
            by += 2.0 * w + per * total
            fl += 2.0 * T * w + 4.0 * H * D * pairs
            ff, one, shared = m["intermediate_size"], 2.0, m.get("shared_expert_intermediate_size", 0)
        if E and i >= m.get("first_k_dense_replace", 0):
            I = m["moe_intermediate_size"]
            by += one * 3 * W * (hit * I + shared) + 2.0 * E * W
            fl += 2.0 * T * (3 * W * (k * I + shared) + E * W)
        else:
            by += one * 3 * W * ff
            fl += 2.0 * T * 3 * W * ff
    return {"bytes": by, "flops": fl}


def tolerance(case):
    """Another order of sums at the same precision: bf16 activations between the kernels (fp8 ones in front of the products of
    ``deepseek``), and the experts that a rounded router logit picks differently."""
    return {"llama": {"rel": 0.02, "max": 0.2}, "llama70b": {"rel": 0.02, "max": 0.2, "differ": 0.01},
            "moe": {"rel": 0.02, "max": 0.5}, "deepseek": {"rel": 0.03, "max": 0.5},
            "next": {"rel": 0.02, "max": 0.5}}[case["model"]]


# ------------------------------------------------------------------------------------------------ the same in 64 bits
def _rms(x, w, eps):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + eps) * w.double()


def _rope(x, pos, theta, rot, pairs=False):
    """``x [T, H, D]``: rotates its first ``rot`` entries, halves against each other or (``pairs``) neighbours."""
    inv = theta ** (-torch.arange(0, rot, 2, dtype=torch.float64, device=x.device) / rot)
    ang = pos.double()[:, None, None] * inv
    c, s = ang.cos(), ang.sin()
    a, b = (x[..., 0:rot:2], x[..., 1:rot:2]) if pairs else (x[..., : rot // 2], x[..., rot // 2: rot])
    a, b = a * c - b * s, b * c + a * s
    y = torch.stack([a, b], -1).flatten(-2) if pairs else torch.cat([a, b], -1)
    return torch.cat([y, x[..., rot:]], -1)


def _linear(x, layer):
    """``x W^T``; before fp8 weights ``x`` is rounded as the format says."""
    w = layer.weight.double()
    if layer.weight.dtype != torch.float8_e4m3fn:
        return x @ w.T
    return _e4m3(x) @ _blocks(w, layer.weight_scale_inv).T


def _e4m3(x):
    g = x.view(x.shape[0], -1, 128)
    s = g.abs().amax(-1, keepdim=True).clamp_min(1e-10) / 448.0
    return ((g / s).to(torch.float8_e4m3fn).double() * s).view_as(x)


def _blocks(w, s):
    return w * s.double().repeat_interleave(128, -2)[..., : w.shape[-2], :].repeat_interleave(128, -1)[..., : w.shape[-1]]


def _attend(q, k, v, scale, first):
    """``q [n, H, D]`` at positions ``first ..`` over ``k [S, Hk, D]``, ``v [S, Hk, Dv]``; heads in groups share keys."""
    n, H, D = q.shape
    S, Hk = k.shape[0], k.shape[1]
    out = []
    for i in range(0, n, 512):
        x = q[i: i + 512]
        c = x.shape[0]
        end = first + i + c
        s = torch.einsum("nhgd,shd->hgns", x.view(c, Hk, H // Hk, D), k[:end]) * scale
        s.masked_fill_(torch.arange(end, device=q.device)[None, :] > (first + i + torch.arange(c, device=q.device))[:, None],
                       float("-inf"))
        out.append(torch.einsum("hgns,shd->nhgd", s.softmax(-1), v[:end]).reshape(c, H, v.shape[-1]))
    return torch.cat(out)


def _swiglu(y, interleaved):
    g, u = (y[:, 0::2], y[:, 1::2]) if interleaved else y.chunk(2, -1)
    return torch.nn.functional.silu(g) * u


def _mlp(x, mlp):
    """Unquantised gate and up rows alternate; in fp8 they follow one another."""
    return _linear(_swiglu(_linear(x, mlp.gate_up_proj), mlp.gate_up_proj.weight.dtype != torch.float8_e4m3fn), mlp.down_proj)


def _moe(x, mlp, m):
    ex = mlp.experts
    logits = x @ mlp.gate.weight.double().T
    k = m["num_experts_per_tok"]
    if m.get("scoring_func") == "sigmoid":
        s = logits.sigmoid()
        pick = s + ex.e_score_correction_bias.double()
        groups = pick.view(x.shape[0], m["n_group"], -1)
        best = groups.topk(2, -1)[0].sum(-1).topk(m["topk_group"], -1)[1]
        keep = torch.zeros(groups.shape[:2], dtype=torch.bool, device=x.device).scatter_(1, best, True)
        ids = groups.masked_fill(~keep[..., None], float("-inf")).flatten(1).topk(k, -1)[1]
        w = s.gather(1, ids)
    else:
        w, ids = logits.softmax(-1).topk(k, -1)
    w = w / w.sum(-1, keepdim=True) * m.get("routed_scaling_factor", 1.0)
    y = torch.zeros_like(x)
    fp8 = ex.w13_weight.dtype == torch.float8_e4m3fn
    for e in ids.unique().tolist():
        t, j = (ids == e).nonzero(as_tuple=True)
        w13, w2 = ex.w13_weight[e].double(), ex.w2_weight[e].double()
        if fp8:
            w13, w2 = _blocks(w13, ex.w13_weight_scale_inv[e]), _blocks(w2, ex.w2_weight_scale_inv[e])
            z = _e4m3(_swiglu(_e4m3(x[t]) @ w13.T, False)) @ w2.T
        else:
            z = _swiglu(x[t] @ w13.T, True) @ w2.T
        y.index_add_(0, t, z * w[t, j][:, None])
    shared = getattr(mlp, "shared_experts", None) or getattr(mlp, "shared_expert", None)
    if shared is not None:
        z = _mlp(x, shared)
        if getattr(mlp, "shared_expert_gate", None) is not None:
            z = z * (x @ mlp.shared_expert_gate.weight.double().T).sigmoid()
        y += z
    return y


def _delta(lin, x, rows, conv, ssm, m):
    """Gated delta rule; ``conv`` and ``ssm`` (64 bits) are updated."""
    nk, nv, d, rep = lin.nk, lin.nv, lin.dk, lin.rep
    T = x.shape[0]
    p = _linear(x, lin.in_proj_qkvz).view(T, nk, -1)
    ba = _linear(x, lin.in_proj_ba).view(T, nk, 2 * rep)
    q, k, v, z = p.split([d, d, rep * d, rep * d], -1)
    b, a = ba.split([rep, rep], -1)
    beta = b.reshape(T, nv).sigmoid()
    decay = torch.exp(-torch.exp(lin.A_log.double()) * torch.nn.functional.softplus(a.reshape(T, nv) + lin.dt_bias.double()))
    mixed = torch.cat([q.reshape(T, -1), k.reshape(T, -1), v.reshape(T, -1)], -1)
    taps, K = lin.conv1d.weight.double(), lin.K
    starts = [0]
    for _, n in rows:
        starts.append(starts[-1] + n)
    out = torch.empty_like(mixed)
    for i, (past, n) in enumerate(rows):
        ext = torch.cat([conv[i] if past else torch.zeros_like(conv[i]), mixed[starts[i]: starts[i + 1]]])
        out[starts[i]: starts[i + 1]] = torch.nn.functional.silu((ext.unfold(0, K, 1) * taps).sum(-1))
        conv[i] = ext[-(K - 1):]
        if not past:
            ssm[i] = 0
    q, k, v = out.split([nk * d, nk * d, nv * d], -1)
    unit = lambda t: t * torch.rsqrt(t.square().sum(-1, keepdim=True) + 1e-6)
    q = (unit(q.view(T, nk, d)) * d ** -0.5).repeat_interleave(rep, 1)
    k = unit(k.view(T, nk, d)).repeat_interleave(rep, 1)
    v = v.view(T, nv, d)
    o = torch.empty(T, nv, d, dtype=torch.float64, device=x.device)
    order = sorted(range(len(rows)), key=lambda i: -rows[i][1])          # sequences side by side, the longest first
    first = torch.tensor([starts[i] for i in order], device=x.device)
    S = ssm[torch.tensor(order, device=x.device)]
    for t in range(max(n for _, n in rows)):
        c = sum(rows[i][1] > t for i in order)
        at = first[:c] + t
        s, kt = S[:c], k[at]
        s *= decay[at][..., None, None]
        u = beta[at][..., None] * (v[at] - torch.einsum("bhkv,bhk->bhv", s, kt))
        s += kt[..., None] * u[..., None, :]
        o[at] = torch.einsum("bhkv,bhk->bhv", s, q[at])
    ssm[torch.tensor(order, device=x.device)] = S
    o = _rms(o, lin.norm.weight, m["rms_norm_eps"]) * torch.nn.functional.silu(z.reshape(T, nv, d))
    return _linear(o.reshape(T, -1), lin.out_proj)


@torch.no_grad()
def exact(case, seed):
    """Outputs of ``run`` from the same weights, caches and tokens; none for the 8-bit cache, whose values are whole numbers."""
    st, m = prepare(case, seed), MODELS[case["model"]]
    net, rows, eps, theta = st["runner"].model, st["rows"], m["rms_norm_eps"], m["rope_theta"]
    T = sum(b for _, b in rows)
    ids, pos, slots = st["ids"][:T], st["pos"][:T], st["slots"][:T]
    H, Hkv, D = m["num_attention_heads"], m["num_key_value_heads"], m.get("head_dim", 128)
    x = net.model.embed_tokens.weight[ids].double()
    caches, states, kv = [], [], 0
    for i, layer in enumerate(net.model.layers.values()):
        h = _rms(x, layer.input_layernorm.weight, eps)
        if hasattr(layer, "linear_attn"):
            conv, ssm = (t.double() for t in st["states"][len(states)])
            y = _delta(layer.linear_attn, h, rows, conv, ssm, m)
            states.append([conv, ssm])
        else:
            at, cache = layer.self_attn, st["caches"][kv]
            kv += 1
            gate = None
            if case["model"] == "deepseek":
                ql, kl, nope, rd = m["q_lora_rank"], m["kv_lora_rank"], 128, 64
                p = _linear(h, at.fused_qkv_a_proj)
                q = _linear(_rms(p[:, :ql], at.q_a_layernorm.weight, eps), at.q_b_proj).view(T, H, nope + rd)
                q_pe = _rope(q[..., nope:], pos, theta, rd, True)
                up = at.kv_b_proj.weight.double().view(H, -1, kl)
                q = torch.cat([torch.einsum("thn,hnl->thl", q[..., :nope], up[:, :nope]), q_pe], -1)
                new = torch.cat([_rms(p[:, ql: ql + kl], at.kv_a_layernorm.weight, eps),
                                 _rope(p[:, None, ql + kl:], pos, theta, rd, True)[:, 0]], -1)
                c = cache[0].double()
                c.view(-1, kl + rd)[slots] = new
                flat = c.view(-1, 1, kl + rd)
                k_all, v_all, scale = flat, flat[..., :kl], (nope + rd) ** -0.5
                caches.append([c])
            else:
                p = _linear(h, at.qkv_proj)
                q, k, v = p.split([p.shape[1] - 2 * Hkv * D, Hkv * D, Hkv * D], -1)
                if case["model"] == "next":
                    q, gate = q.view(T, H, 2, D).unbind(2)
                q, k, v = q.reshape(T, H, D), k.view(T, Hkv, D), v.view(T, Hkv, D)
                if hasattr(at, "q_norm"):
                    q, k = _rms(q, at.q_norm.weight, eps), _rms(k, at.k_norm.weight, eps)
                rot = D // 4 if case["model"] == "next" else D
                q, k, scale = _rope(q, pos, theta, rot), _rope(k, pos, theta, rot), D ** -0.5
                c = cache[0].double()
                if len(cache) > 1:
                    c *= cache[1].double()[..., None]
                c[slots // BLOCK, 0, slots % BLOCK], c[slots // BLOCK, 1, slots % BLOCK] = k, v
                k_all, v_all = c[:, 0].reshape(-1, Hkv, D), c[:, 1].reshape(-1, Hkv, D)
                caches.append([c] if len(cache) == 1 else [None, None])
            o, t = [], 0
            for j, (past, n) in enumerate(rows):
                p = torch.arange(past + n, device=x.device)
                where = st["table"][j, p // BLOCK].long() * BLOCK + p % BLOCK
                o.append(_attend(q[t: t + n], k_all[where], v_all[where], scale, past))
                t += n
            o = torch.cat(o)
            if case["model"] == "deepseek":
                o = torch.einsum("thl,hvl->thv", o, up[:, nope:])
            if gate is not None:
                o = o * gate.sigmoid()
            y = _linear(o.reshape(T, -1), at.o_proj)
            del k_all, v_all, c
        x = x + y
        h = _rms(x, layer.post_attention_layernorm.weight, eps)
        if hasattr(layer.mlp, "experts"):
            x = x + _moe(h, layer.mlp, m)
        else:
            x = x + _mlp(h, layer.mlp)
    h = _rms(x, net.model.norm.weight, eps)
    out = {"caches": caches, "states": states}
    last = torch.arange(T, device=x.device) if case["prompts"] == 0 else st["last"]
    if case["prompts"]:
        out["hidden"] = h
    out["logits"] = h[last] @ net.lm_head.weight[: m["vocab_size"]].double().T
    return out
