"""Workloads whose speed is measured, through the public entry points a user's program calls.

Kinds of case, and what each stands for:

``generate``    plain autoregressive decode of one request (:meth:`JetSpecEngine.generate`): one row per forward, the smallest
                calls, where launches and the latency of every kernel count.
``tree``        tree-speculative decode of one request (:meth:`JetSpecEngine.generate_tree`): the framework's main path, from
                the API's default tree (15 nodes) to the headline's (depth 20, width 7, 128 nodes, a real draft head in every
                round); bf16 and NVFP4 weights.
``tree_batch``  tree-speculative decode of several requests (:meth:`JetSpecEngine.generate_tree_batch`) with a drafter that is
                conditioned on the target's tapped hidden states: ragged prompts, verify forwards of up to 16 x 128 rows, dense
                and mixture-of-experts targets; with one long prompt and a few new tokens it is a prefill.
``batch``       continuous batching without speculation (:meth:`JetSpecEngine.generate_batch`).
``step``        a serving loop of its own that replays token ids (:meth:`JetSpecEngine.step`): portions of prompts beside single
                decoded tokens, logits of chosen rows; Qwen3 and a decoder of mixed layers (retention, window attention, latent
                attention).
``attention``   the paged tree attention op alone, as the Hugging Face backend calls it, over long contexts.

Decoding entry points return token ids and nothing else of what the model computed, so the models of those cases have the wide
margins of ``init="stable"`` (the greedy token after ``t`` is ``t + 1``); what the same kernels compute in numbers comes back
from ``tree_batch`` (hidden states of five layers), ``step`` (logits) and ``attention``.  Weights are random, made from the seed.
"""
from __future__ import annotations

import gc
import math

import torch

from jetspec_b200 import (DraftHeadTreeDrafter, JetSpecEngine, OracleOverrideDrafter, OracleTreeDrafter, SamplingParams,
                          TreeDrafter, ops)
from jetspec_b200.models import (BandScaling, DraftHeadModel, KizezenConfig, KizezenForCausalLM, KizezenLayerConfig,
                                 LatentAttentionConfig, Qwen3ForCausalLM, RampScaling, RetentionConfig, RotaryConfig,
                                 WindowAttentionConfig, draft_head_config, qwen3_8b_config)
from jetspec_b200.models.config import qwen3_30b_a3b_config

BF16 = torch.bfloat16
MEAN_ACCEPT = 7.0


def listed():
    return [
        # a short chat turn without speculation: one row per forward
        dict(name="generate_short", kind="generate", model="qwen3-8b", layers=36, weights="bf16", prompt=33, new=16),
        # the API's default tree (block of 4, width 2, budget 15), a model-free drafter
        dict(name="tree_default", kind="tree", model="qwen3-8b", layers=36, weights="bf16", prompt=96, new=32, depth=3, width=2,
             budget=15, head=False),
        # the headline: draft head in every round, 128-node trees
        dict(name="tree_headline", kind="tree", model="qwen3-8b", layers=36, weights="bf16", prompt=512, new=96, depth=20, width=7,
             budget=128, head=True),
        # the same on 4-bit weights, 64-node trees
        dict(name="tree_nvfp4", kind="tree", model="qwen3-8b", layers=36, weights="nvfp4", prompt=512, new=64, depth=15, width=4,
             budget=64, head=False),
        # time to the first tokens of one long prompt
        dict(name="prefill_long", kind="tree_batch", model="qwen3-8b", layers=36, weights="bf16", n=1, lo=6001, hi=6001, new=8,
             depth=7, width=2, budget=16),
        # sixteen requests of mixed length, 16 x 128 rows per verify forward (a third of the depth)
        dict(name="tree_batch_16", kind="tree_batch", model="qwen3-8b", layers=12, weights="bf16", n=16, lo=256, hi=2048, new=24,
             depth=20, width=7, budget=128),
        # eight requests on the mixture-of-experts target, 8 x 128 rows (a twelfth of the depth)
        dict(name="tree_batch_moe", kind="tree_batch", model="qwen3-30b-a3b", layers=4, weights="bf16", n=8, lo=256, hi=1024,
             new=24, depth=20, width=7, budget=128),
        # many short requests decoded together without speculation
        dict(name="batch_24", kind="batch", model="qwen3-8b", layers=36, weights="bf16", n=24, lo=16, hi=128, new=12),
        # a serving loop: prompts in portions beside decoded tokens (a third of the depth)
        dict(name="step_qwen3", kind="step", model="qwen3-8b", layers=12, n=5, lo=40, hi=700, chunk=256, new=6),
        # the same loop on mixed layers
        dict(name="step_mixed", kind="step", model="kizezen", layers=8, n=4, lo=60, hi=1500, chunk=512, new=8),
        # the attention op over long contexts
        dict(name="attention_long", kind="attention", heads=32, kv_heads=8, n=4, nodes=128, lo=2048, hi=12000, causal=False),
    ]


def _spread(rng, lo, hi):
    """A whole number of [lo, hi], even over its logarithm."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["generate", "tree", "tree", "tree_batch", "tree_batch", "batch", "step", "attention"])
    if kind == "attention":
        heads, kv = rng.choice([(32, 8), (32, 4), (16, 8), (64, 8)])
        lo = _spread(rng, 1, 4000)
        causal = rng.random() < 0.3
        return dict(kind=kind, heads=heads, kv_heads=kv, n=_spread(rng, 1, 16), nodes=_spread(rng, 1, 600 if causal else 256), lo=lo,
                    hi=_spread(rng, lo, 12000), causal=causal)
    model = "qwen3-30b-a3b" if rng.random() < 0.2 else "qwen3-8b"
    layers = rng.choice([4, 6, 8, 12]) if model == "qwen3-8b" else 4
    if kind == "step":
        model = rng.choice(["qwen3-8b", "kizezen"])
        lo = _spread(rng, 1, 300)
        return dict(kind=kind, model=model, layers=rng.choice([4, 8, 12] if model == "qwen3-8b" else [4, 8]), n=rng.randint(1, 8),
                    lo=lo, hi=_spread(rng, lo, 1600), chunk=_spread(rng, 64, 1024), new=rng.randint(2, 10))
    if kind == "generate":
        return dict(kind=kind, model=model, layers=layers, weights="bf16", prompt=_spread(rng, 2, 2000), new=rng.randint(8, 32))
    if kind == "batch":
        lo = _spread(rng, 1, 200)
        return dict(kind=kind, model=model, layers=layers, weights="bf16", n=_spread(rng, 2, 40), lo=lo, hi=_spread(rng, lo, 600),
                    new=rng.randint(6, 16))
    width, depth = rng.randint(2, 8), rng.randint(3, 20)
    if kind == "tree":
        weights = rng.choice(["bf16", "bf16", "nvfp4"]) if model == "qwen3-8b" else "bf16"
        return dict(kind=kind, model=model, layers=layers, weights=weights, prompt=_spread(rng, 3, 3000), new=rng.randint(24, 96),
                    depth=depth, width=width, budget=_spread(rng, 12, 256), head=weights == "bf16" and rng.random() < 0.5)
    lo = _spread(rng, 8, 800)
    return dict(kind=kind, model=model, layers=layers, weights="bf16", n=rng.randint(1, 16), lo=lo, hi=_spread(rng, lo, 2048),
                new=rng.randint(12, 32), depth=depth, width=width, budget=_spread(rng, 12, 128))


# ------------------------------------------------------------------ what a case is made of
def _qwen_config(case):
    make = {"qwen3-8b": qwen3_8b_config, "qwen3-30b-a3b": qwen3_30b_a3b_config}[case["model"]]
    return make(num_hidden_layers=case["layers"])


def _kizezen_config(case):
    """Width 2048, 16 heads; layers repeat (retention, window attention, latent attention, window attention)."""
    heads, kv = 16, 8
    win = WindowAttentionConfig(heads, kv, 128, 128, 1024, 128, 5e5, 128 ** -0.5, sink=False, qk_norm=False, bias=True, keep_first=4,
                                sink_logits=True, proj_norm=True, o_bias=False, gate=True,
                                rot=RotaryConfig(128, 5e5, "half", BandScaling(8.0, 1.0, 4.0, 8192)))
    lat = LatentAttentionConfig(heads, 96, 128, 0, 512, 128 ** -0.5, rot=RotaryConfig(32, 1e4, "next", RampScaling(40.0, 4096, 32.0, 1.0)),
                                sink_logits=True, gate=True)
    n = heads // 2
    ret = RetentionConfig(n, 128, 256, [1.0 - 2.0 ** (-5 - 7 * i / (n - 1)) for i in range(n)], RotaryConfig(128, 1e4))
    return KizezenConfig(vocab_size=32768, hidden_size=2048, layers=[KizezenLayerConfig((ret, win, lat, win)[i % 4], 9216)
                                                                     for i in range(case["layers"])])


def _model(case, seed):
    if case["model"] == "kizezen":
        m = KizezenForCausalLM.random_init(_kizezen_config(case), seed=seed, dtype=BF16, device="cuda")
        g = torch.Generator(device="cuda").manual_seed(seed)
        with torch.no_grad():
            for name, p in m.named_parameters():
                if name.endswith(("bias", "sink", "sink_logits")):
                    p.normal_(0.0, 0.5, generator=g)
        return m
    return Qwen3ForCausalLM.random_init(_qwen_config(case), seed=seed, dtype=BF16, device="cuda", init="stable")


def _lengths(case):
    """Prompt (or context) lengths: part of the case, the same for every seed; the longest comes first."""
    g = torch.Generator().manual_seed(1000 * case["n"] + case["hi"])
    return [case["hi"]] + torch.randint(case["lo"], case["hi"] + 1, (case["n"] - 1,), generator=g).tolist()


def _prompts(case, seed, vocab):
    g = torch.Generator().manual_seed(seed + 2)
    lengths = _lengths(case) if "n" in case else [case["prompt"]]
    return [torch.randint(0, vocab, (1, n), generator=g) for n in lengths]


def _continuation(prompt, new, vocab):
    """What a model with ``init="stable"`` decodes after a prompt: it counts upwards."""
    return [(int(prompt[0, -1]) + 1 + i) % vocab for i in range(new)]


def _script(case, prompt, vocab, seed):
    """A drafter whose accepted lengths are drawn from a geometric distribution, for one prompt; ``seed`` picks the draw."""
    most = max(1, min(case["depth"], (case["budget"] - 2) // case["width"] + 1))
    return OracleTreeDrafter(prompt[0].tolist() + _continuation(prompt, case["new"], vocab), vocab, tree_width=case["width"],
                             mean_accept=MEAN_ACCEPT, max_accept=most, seed=seed)


class _Conditioned(TreeDrafter):
    """A drafter that is handed the target's hidden states each round; it keeps the last ones for its caller."""

    def __init__(self, script):
        self.script, self.hidden = script, None

    def propose_logits(self, context_ids, depth, target_hidden=None, **kwargs):
        self.hidden = target_hidden
        return self.script.propose_logits(context_ids, depth)

    def propose_topk(self, context_ids, depth, width=None, target_hidden=None, **kwargs):
        self.hidden = target_hidden
        tok, lp = self.script.propose_topk_at(int(context_ids.shape[-1]), depth, width)
        return torch.from_numpy(tok).long(), torch.tensor(lp, dtype=torch.float32)


def _taps(case):
    return sorted({1, case["layers"] // 3, case["layers"] // 2, case["layers"] - 2, case["layers"] - 1})


# ------------------------------------------------------------------ prepare and run
def prepare(case, seed):
    if case["kind"] == "attention":
        return _prepare_attention(case, seed)
    gc.collect()                      # engines of earlier states hold their graphs in reference cycles
    model = _model(case, seed)
    cfg, vocab = model.config, model.config.vocab_size
    if case.get("weights") == "nvfp4":
        from jetspec_b200.models.nvfp4 import quantize_model_nvfp4
        quantize_model_nvfp4(model)
    prompts = _prompts(case, seed, vocab)
    longest = max(int(p.shape[1]) for p in prompts)
    state = {"case": case, "prompts": prompts}
    if case["kind"] == "step":
        tokens = [p[0].tolist() + torch.randint(0, vocab, (case["new"],), generator=torch.Generator().manual_seed(seed + 3 + i)).tolist()
                  for i, p in enumerate(prompts)]
        eng = JetSpecEngine(model, device="cuda", dtype=BF16)
        eng.reserve_pool(sum((len(t) + 15) // 16 * 16 for t in tokens), case["n"])
        state.update(engine=eng, steps=_schedule(case, tokens))
    else:
        room = longest + case["new"] + 320
        eng = JetSpecEngine(model, device="cuda", dtype=BF16, max_seq_len=(room + 255) // 256 * 256)
        state.update(engine=eng, sampling=SamplingParams(0.0, case["new"]))
        if case["kind"] == "tree":
            draft = script = _script(case, prompts[0], vocab, 0)
            if case["head"]:
                bs = case["depth"] + 1
                head = DraftHeadModel.random_init(draft_head_config(cfg, num_layers=1, block_size=bs, num_taps=5), seed=seed + 1,
                                                  dtype=BF16, device="cuda")
                draft = OracleOverrideDrafter(DraftHeadTreeDrafter(head, model, block_size=bs), script)
            state["drafter"] = draft
        elif case["kind"] == "tree_batch":
            state["drafters"] = [_Conditioned(_script(case, p, vocab, i)) for i, p in enumerate(prompts)]
    run(state)                        # a server warms its engine up: pool, captured graphs
    return state


def _schedule(case, tokens):
    """The steps of a replay: request ``i`` enters at step ``i``, its prompt goes in by portions of ``chunk``, then its remaining
    tokens one by one; the logits behind each prompt and of each decoded token are wanted."""
    at = [0] * len(tokens)
    steps = []
    while any(a < len(t) for a, t in zip(at, tokens)):
        entries = []
        for i, t in enumerate(tokens):
            if i > len(steps) or at[i] >= len(t):
                continue
            prompt = len(t) - case["new"]
            n = min(case["chunk"], prompt - at[i]) if at[i] < prompt else 1
            at[i] += n
            entries.append((i, t[at[i] - n:at[i]], [n - 1] if at[i] >= prompt else []))
        steps.append(entries)
    return steps


def run(state):
    case = state["case"]
    if case["kind"] == "attention":
        return ops.paged_tree_attention(*state["args"], scale=128 ** -0.5, causal=case["causal"], max_q=case["nodes"])
    eng = state["engine"]
    if case["kind"] == "generate":
        return torch.tensor(eng.generate(state["prompts"][0], state["sampling"])["token_ids"])
    if case["kind"] == "batch":
        return torch.tensor([o["token_ids"] for o in eng.generate_batch(state["prompts"], state["sampling"])])
    if case["kind"] == "tree":
        out = eng.generate_tree(state["prompts"][0], state["drafter"], tree_depth=case["depth"], tree_width=case["width"],
                                budget=case["budget"], sampling_params=state["sampling"], return_stats=True)
        return {"tokens": torch.tensor(out["token_ids"]), "accepted": torch.tensor(out["accept_lengths"]),
                "sizes": torch.tensor(out["tree_sizes"])}
    if case["kind"] == "tree_batch":
        outs = eng.generate_tree_batch(state["prompts"], state["drafters"], block_size=case["depth"] + 1, tree_width=case["width"],
                                       budget=case["budget"], sampling_params=state["sampling"], target_layer_ids=_taps(case),
                                       return_stats=True)
        return {"tokens": torch.tensor([o["token_ids"] for o in outs]),
                "accepted": torch.tensor([a for o in outs for a in o["accept_lengths"]]),
                "hidden": [d.hidden for d in state["drafters"]]}
    logits, live = [], {}
    last = {i: k for k, entries in enumerate(state["steps"]) for i, _, _ in entries}
    for k, entries in enumerate(state["steps"]):
        got = eng.step([(i + 1, toks, want) for i, toks, want in entries])
        if got is not None:
            logits.append(got)
        for i, _, _ in entries:
            if last[i] == k:
                eng.pool.free(i + 1)
    return torch.cat(logits)


# ------------------------------------------------------------------ the attention op
def _prepare_attention(case, seed):
    n, nodes, H, G = case["n"], case["nodes"], case["heads"], case["kv_heads"]
    g = torch.Generator(device="cuda").manual_seed(seed)
    past = _lengths(case)
    page = 16
    pages = [(p + nodes + page - 1) // page for p in past]
    total, S = sum(pages), (sum(pages) + 8) * page
    order = torch.randperm(total, generator=torch.Generator().manual_seed(seed))
    width = max(pages) * page
    table = torch.zeros(n, width, dtype=torch.int32)
    first = 0
    for i, c in enumerate(pages):
        ids = order[first:first + c]
        table[i, :c * page] = (ids[:, None] * page + torch.arange(page)[None]).reshape(-1).to(torch.int32)
        first += c
    normal = lambda *s: torch.randn(*s, device="cuda", generator=g, dtype=torch.float32)
    q = (normal(n * nodes, H, 128) * 1.5).to(BF16)
    k, v = normal(G, S, 128).to(BF16), normal(G, S, 128).to(BF16)
    i32 = dict(dtype=torch.int32, device="cuda")
    bits = None if case["causal"] else ops.pack_ancestor_bits(_ancestors(case, seed), (nodes + 31) // 32).cuda()
    return {"case": case, "args": (q, k, v, table.cuda(), torch.arange(n, **i32), torch.arange(n + 1, **i32) * nodes,
                                   torch.tensor(past, **i32), bits)}


def _ancestors(case, seed):
    """Which nodes of its own tree each node sees, ``(n * nodes, nodes)``: random trees, every node below an earlier one."""
    n, nodes = case["n"], case["nodes"]
    g = torch.Generator().manual_seed(seed + 5)
    up = (torch.rand(n, nodes, generator=g) * torch.arange(nodes)).long()
    seen = torch.zeros(n, nodes, nodes, dtype=torch.bool)
    rows = torch.arange(n)
    for i in range(nodes):
        if i:
            seen[:, i] = seen[rows, up[:, i]]
        seen[:, i, i] = True
    return seen.view(n * nodes, nodes)


# ------------------------------------------------------------------ what a pass cannot do without
def _forward_cost(cfg, rows, sequences, scored, nvfp4=False):
    """``(weight bytes, other bytes, flops)`` of one forward of ``rows`` rows, attention left out, ``scored`` of which meet the
    vocabulary."""
    H, V = cfg.hidden_size, cfg.vocab_size
    attn = H * (cfg.num_attention_heads * 2 + cfg.num_key_value_heads * 2) * cfg.head_dim
    if cfg.is_moe:
        one = 3 * H * cfg.moe_intermediate_size
        used = cfg.num_experts * (1.0 - (1.0 - cfg.num_experts_per_tok / cfg.num_experts) ** rows)
        stored, active = attn + used * one + H * cfg.num_experts, attn + cfg.num_experts_per_tok * one + H * cfg.num_experts
    else:
        stored = active = attn + 3 * H * cfg.intermediate_size
    L = cfg.num_hidden_layers
    weights = L * stored * (0.5625 if nvfp4 else 2) + V * H * 2
    return weights, rows * H * 2, 2.0 * (L * active * rows + V * H * scored)


def _rounds(case, prompt_len, seed):
    """``(rounds, hidden rows the drafter sees in the last one)`` of a scripted request."""
    most = max(1, min(case["depth"], (case["budget"] - 2) // case["width"] + 1))
    script = OracleTreeDrafter([0], 2 ** 20, tree_width=case["width"], mean_accept=MEAN_ACCEPT, max_accept=most, seed=seed)
    end = prompt_len + case["new"]
    at, n, seen = prompt_len + 1, 0, 0
    while at < end:
        seen = at - 1
        # depths behind the end of the script propose nothing true
        at += min(script.planned_accept(at, case["depth"]), max(0, end - at)) + 1
        n += 1
    return n, seen


def work(case):
    if case["kind"] == "attention":
        past = _lengths(case)
        keys = sum(past) + case["n"] * case["nodes"]
        rows = case["n"] * case["nodes"]
        seen = case["nodes"] * sum(past) + case["n"] * case["nodes"] ** 2 / 2
        return {"bytes": keys * case["kv_heads"] * 512 + rows * case["heads"] * 512, "flops": 4.0 * seen * case["heads"] * 128}
    if case["model"] == "kizezen":
        cfg = _kizezen_config(case)
        W, F, rows = cfg.hidden_size, 9216, sum(_lengths(case)) + case["n"] * case["new"]
        per = {"retention": W * 2 * 1024 + W * 3 * 2048 + W * 2048, "attention": W * (2048 * 2 + 1024 * 2),
               "latent_attention": W * (16 * 128 + 544 + 2048) + 512 * 16 * 224}
        weights = sum(per[l.mixer_type] + 2 * W * F for l in cfg.layers)
        wanted = case["n"] * (case["new"] + 1)
        steps = len(_schedule(case, [[0] * (n + case["new"]) for n in _lengths(case)]))
        return {"bytes": steps * (weights + cfg.vocab_size * W) * 2.0 + wanted * cfg.vocab_size * 4,
                "flops": 2.0 * (weights * rows + cfg.vocab_size * W * wanted)}
    cfg = _qwen_config(case)
    lengths = _lengths(case) if "n" in case else [case["prompt"]]
    kv = cfg.num_hidden_layers * cfg.num_key_value_heads * 512            # bytes of keys and values of one token
    pair = cfg.num_hidden_layers * cfg.num_attention_heads * 512          # flops of one query and one key
    total = sum(lengths)
    if case["kind"] == "step":
        steps = _schedule(case, [[0] * (n + case["new"]) for n in lengths])
        b = f = 0.0
        at = [0] * len(lengths)
        for entries in steps:
            rows = sum(len(t) for _, t, _ in entries)
            w, o, fl = _forward_cost(cfg, rows, len(entries), sum(len(x) for _, _, x in entries))
            b, f = b + w + o, f + fl
            for i, t, _ in entries:
                at[i] += len(t)
                b, f = b + at[i] * kv, f + pair * len(t) * (at[i] - len(t) / 2)
        return {"bytes": b, "flops": f}
    fp4 = case["weights"] == "nvfp4"
    w, o, f = _forward_cost(cfg, total, len(lengths), len(lengths), fp4)
    b, f = w + o + total * kv, f + pair * sum(n * n / 2 for n in lengths)
    if case["kind"] in ("generate", "batch"):
        rounds, rows = case["new"] - 1, len(lengths)
    else:
        rounds, rows = max(_rounds(case, n, i)[0] for i, n in enumerate(lengths)), case["budget"] * len(lengths)
    w, o, fl = _forward_cost(cfg, rows, len(lengths), rows, fp4)
    b, f = b + rounds * (w + o + total * kv), f + rounds * (fl + pair * (rows / len(lengths)) * total)
    if case.get("head"):
        H, draft = cfg.hidden_size, case["depth"] + 1
        layer = H * (cfg.num_attention_heads * 2 + cfg.num_key_value_heads * 2) * cfg.head_dim + 3 * H * cfg.intermediate_size
        own = layer + 5 * H * H + cfg.vocab_size * H
        b, f = b + rounds * own * 2.0, f + rounds * 2.0 * own * draft
    return {"bytes": b, "flops": f}


def tolerance(case):
    if case["kind"] in ("generate", "batch", "tree"):
        return "exact"
    if case["kind"] == "attention":
        return {"rel": 0.01, "max": 0.1}
    # two bf16 forwards of 36 layers, each about 0.015 off the 64-bit one; a routed expert that flips moves a row by more
    return {"rel": 0.03, "max": 0.6}


# ------------------------------------------------------------------ the same in 64 bits
def _rms(x, w, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps) * w


def _turn(x, angles, amp=1.0, neighbours=False):
    """Rotates the pairs of ``x (T, heads, 2 * n)`` by ``angles (T, n)``."""
    c, s = amp * torch.cos(angles)[:, None], amp * torch.sin(angles)[:, None]
    if neighbours:
        a, b = x[..., 0::2], x[..., 1::2]
        return torch.stack((a * c - b * s, b * c + a * s), -1).flatten(-2)
    a, b = x.chunk(2, -1)
    return torch.cat((a * c - b * s, b * c + a * s), -1)


def _attend(q, k, v, scale, seen=None, sink=None):
    """Softmax attention of ``q (T, H, D)`` over ``k, v (S, G, D)``; causal unless ``seen (T, S)`` says otherwise."""
    T, H, G = q.shape[0], q.shape[1], k.shape[1]
    out = torch.empty(T, H, v.shape[2], dtype=q.dtype, device=q.device)
    if seen is None:
        seen = torch.ones(T, k.shape[0], dtype=torch.bool, device=q.device).tril()
    for n in range(H):
        s = (q[:, n] @ k[:, n * G // H].T * scale).masked_fill_(~seen, -math.inf)
        top = s.amax(-1, keepdim=True)
        if sink is not None:
            top = torch.clamp(top, min=float(sink[n]))
        s = s.sub_(top).exp_()
        z = s.sum(-1, keepdim=True)
        out[:, n] = (s @ v[:, n * G // H]) / (z + torch.exp(sink[n] - top) if sink is not None else z)
    return out


def _qwen_64(model, ids, taps):
    """Hidden rows behind the layers ``taps`` and the logits' input, in 64 bits, for one sequence."""
    cfg, w = model.config, lambda p: p.detach().double()
    T, D = len(ids), cfg.head_dim
    ids = torch.as_tensor(ids, device="cuda")
    angles = torch.arange(T, device="cuda").double()[:, None] * (
        cfg.rope_theta ** (-torch.arange(0, D, 2, device="cuda").double() / D))[None]
    x, kept = w(model.model.embed_tokens.weight[ids]), {}
    for i, layer in enumerate(model.model.layers):
        a = layer.self_attn
        h = _rms(x, w(layer.input_layernorm.weight), cfg.rms_norm_eps)
        q, k, v = ((h @ w(p.weight).T).view(T, -1, D) for p in (a.q_proj, a.k_proj, a.v_proj))
        q = _turn(_rms(q, w(a.q_norm.weight), cfg.rms_norm_eps), angles)
        k = _turn(_rms(k, w(a.k_norm.weight), cfg.rms_norm_eps), angles)
        x = x + _attend(q, k, v, D ** -0.5).flatten(1) @ w(a.o_proj.weight).T
        h = _rms(x, w(layer.post_attention_layernorm.weight), cfg.rms_norm_eps)
        silu = torch.nn.functional.silu
        if cfg.is_moe:
            m = layer.mlp
            p = torch.softmax(h @ w(m.gate.weight).T, -1)
            best, which = p.topk(cfg.num_experts_per_tok, -1)
            if cfg.norm_topk_prob:
                best = best / best.sum(-1, keepdim=True)
            y = torch.zeros_like(x)
            for e in range(cfg.num_experts):
                t, j = (which == e).nonzero(as_tuple=True)
                if t.numel():
                    g, u = (h[t] @ w(m.w_gate_up[e]).T).chunk(2, -1)
                    y.index_add_(0, t, (silu(g) * u) @ w(m.w_down[e]).T * best[t, j][:, None])
            x = x + y
        else:
            m = layer.mlp
            x = x + (silu(h @ w(m.gate_proj.weight).T) * (h @ w(m.up_proj.weight).T)) @ w(m.down_proj.weight).T
        kept[i] = x
    last = _rms(x, w(model.model.norm.weight), cfg.rms_norm_eps)
    kept[cfg.num_hidden_layers - 1] = last
    return torch.cat([kept[i] for i in taps], -1) if taps else None, last


def _kizezen_64(model, ids):
    """The logits' input in 64 bits for one sequence."""
    cfg, w, eps = model.config, lambda p: p.detach().double(), model.config.norm_eps
    T = len(ids)
    pos = torch.arange(T, device="cuda").double()
    back = pos[:, None] - pos[None]
    x = w(model.model.embed_tokens.weight[torch.as_tensor(ids, device="cuda")]) * cfg.embed_scale
    for layer, l in zip(model.model.layers, cfg.layers):
        m, c = layer.mixer, l.mixer
        h = _rms(x, w(layer.norm1.weight), eps)
        of = lambda p: h @ w(p.weight).T + (w(p.bias) if p.bias is not None else 0.0)
        if l.mixer_type == "retention":
            ang = pos[:, None] * torch.tensor(_frequencies(c.rot), device="cuda", dtype=torch.float64)[None]
            q, k = (_turn(of(p).view(T, c.heads, c.dim), ang) for p in (m.q_proj, m.k_proj))
            v, y = of(m.v_proj).view(T, c.heads, c.vdim), []
            for n in range(c.heads):
                fade = torch.where(back >= 0, c.decay[n] ** back.clamp(min=0), 0.0)
                y.append((q[:, n] @ k[:, n].T * c.dim ** -0.5 * fade) @ v[:, n])
            y = _rms(torch.stack(y, 1), 1.0, eps).flatten(1) * torch.nn.functional.silu(of(m.gate_proj))
        elif l.mixer_type == "attention":
            ang = pos[:, None] * torch.tensor(_frequencies(c.rot), device="cuda", dtype=torch.float64)[None]
            q = _turn(_rms(of(m.q_proj), w(m.q_norm), eps).view(T, c.heads, c.dim), ang)
            k = _turn(_rms(of(m.k_proj), w(m.k_norm), eps).view(T, c.kv_heads, c.dim), ang)
            seen = (back >= 0) & ((back < c.window) | (pos[None] < c.keep_first))
            y = _attend(q, k, of(m.v_proj).view(T, c.kv_heads, c.vdim), c.scale, seen, w(m.sink_logits))
            y = (y * torch.sigmoid(of(m.gate_proj))[..., None]).flatten(1)
        else:
            ang = pos[:, None] * torch.tensor(_frequencies(c.rot), device="cuda", dtype=torch.float64)[None]
            amp = 0.1 * math.log(c.rot.scaling.factor) + 1.0
            q, down = of(m.q_proj).view(T, c.heads, -1), of(m.kv_down)
            lat = _rms(down[:, :c.kv_rank], w(m.kv_norm), eps)
            shared = _turn(down[:, None, c.kv_rank:], ang, amp, True).expand(T, c.heads, -1)
            q = torch.cat((q[..., :c.dim], _turn(q[..., c.dim:], ang, amp, True)), -1)
            k = torch.cat(((lat @ w(m.k_up.weight).T).view(T, c.heads, c.dim), shared), -1)
            y = _attend(q, k, (lat @ w(m.v_up.weight).T).view(T, c.heads, c.vdim), c.scale, back >= 0, w(m.sink))
            y = (y * torch.sigmoid(of(m.gate_proj))[..., None]).flatten(1)
        x = x + y @ w(m.o_proj.weight).T
        h = _rms(x, w(layer.norm2.weight), eps)
        x = x + torch.nn.functional.gelu(h @ w(layer.mlp.up_proj.weight).T) @ w(layer.mlp.down_proj.weight).T
    return _rms(x, w(model.model.norm.weight), eps)


def _frequencies(rot):
    """Radians per position of a rotation's pairs, with the two scalings of the configuration above."""
    s, out = rot.scaling, []
    n = rot.dims // 2
    if isinstance(s, RampScaling):
        at = lambda turns: rot.dims * math.log(s.original / (2.0 * math.pi * turns)) / (2.0 * math.log(rot.base))
        lo, hi = max(math.floor(at(s.fast)), 0), min(math.ceil(at(s.slow)), rot.dims - 1)
    for i in range(n):
        f = rot.base ** (-i / n)
        if isinstance(s, BandScaling):
            wave = 2.0 * math.pi / f
            t = min(1.0, max(0.0, (s.original / wave - s.low) / (s.high - s.low)))
            f = (1.0 - t) * f / s.factor + t * f
        elif isinstance(s, RampScaling):
            r = min(max((i - lo) / max(hi - lo, 0.001), 0.0), 1.0)
            f = f / s.factor * r + f * (1.0 - r)
        out.append(f)
    return out


@torch.no_grad()
def exact(case, seed):
    if case["kind"] in ("generate", "batch", "tree"):
        return None                   # token ids only
    if case["kind"] == "attention":
        q, k, v, table, rows, cu_q, past, _ = _prepare_attention(case, seed)["args"]
        n, nodes = case["n"], case["nodes"]
        own = torch.ones(n * nodes, nodes, dtype=torch.bool).tril() if case["causal"] else _ancestors(case, seed)
        if case["causal"]:
            own = torch.ones(nodes, nodes, dtype=torch.bool).tril().repeat(n, 1)
        out = []
        for i, p in enumerate(past.tolist()):
            at = table[i, :p + nodes].long()
            seen = torch.cat((torch.ones(nodes, p, dtype=torch.bool), own[i * nodes:(i + 1) * nodes]), 1).cuda()
            out.append(_attend(q[i * nodes:(i + 1) * nodes].double(), k[:, at].double().transpose(0, 1), v[:, at].double().transpose(0, 1),
                               128 ** -0.5, seen))
        return torch.cat(out).flatten(1)
    model = _model(case, seed)
    vocab = model.config.vocab_size
    prompts = _prompts(case, seed, vocab)
    if case["kind"] == "tree_batch":
        hidden = []
        for i, p in enumerate(prompts):
            ids = p[0].tolist() + _continuation(p, case["new"], vocab)
            seen = _rounds(case, int(p.shape[1]), i)[1]
            hidden.append(_qwen_64(model, ids[:seen], _taps(case))[0][None])
        return {"tokens": None, "accepted": None, "hidden": hidden}
    tokens = [p[0].tolist() + torch.randint(0, vocab, (case["new"],), generator=torch.Generator().manual_seed(seed + 3 + i)).tolist()
              for i, p in enumerate(prompts)]
    rows = [_kizezen_64(model, t) if case["model"] == "kizezen" else _qwen_64(model, t, None)[1] for t in tokens]
    steps, at, wanted = _schedule(case, tokens), [0] * len(tokens), []
    for entries in steps:
        for i, toks, want in entries:
            wanted += [rows[i][at[i] + k] for k in want]
            at[i] += len(toks)
    head = model.lm_head.weight
    rows = torch.stack(wanted)
    return torch.cat([rows @ head[a:a + 16384].detach().double().T for a in range(0, vocab, 16384)], -1)
