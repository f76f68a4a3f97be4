"""The calls whose speed is tracked: what a user of the framework has it do, from one token of one request to a packed
training sequence.

``listed()`` names the cases, ``draw(rng)`` gives one more of the same ranges, ``prepare`` builds what a program holds before
the call, ``run`` makes the call through the public entry points, ``work`` counts the bytes and operations it cannot do
without, ``exact`` computes the same outputs in 64 bits with plain tensor code.

Kinds: ``train`` (forward and backward of a decoder stack with full recomputation), ``moe`` (forward and backward of routed
experts), ``serve`` (one serving step of a decoder stack over paged keys and values: prefill portions, or a decode step that
is replayed from a CUDA graph as the engine does), ``sample`` (the token sampler), ``delta`` and ``ssd`` (the recurrences of
hybrid stacks), ``latent`` (decode attention over latent pages).
"""

from __future__ import annotations

import math
import random

import torch

BF = torch.bfloat16
PAGE = 128
THETA = 500000.0
EPS = 1e-5
#: width, feed-forward, query heads, key heads, head size of the decoder stacks
STACKS = {"small": (1024, 2816, 8, 2, 128), "medium": (2048, 6144, 16, 4, 128), "large": (4096, 14336, 32, 8, 128),
          "shard": (8192, 3584, 8, 1, 128), "narrow": (1024, 2816, 16, 4, 64)}


# ------------------------------------------------------------------------------------------------------------ the cases
def listed():
    return [
        # one packed sequence of the headline fine-tuning run, two of its layers
        dict(name="train 1x8192", kind="train", stack="large", layers=2, vocab=32000, rows=1, length=8192, docs=False),
        # a small model on short padded rows of a few documents each
        dict(name="train 3x1021 packed", kind="train", stack="narrow", layers=2, vocab=4096, rows=3, length=1021, docs=True),
        # the experts of one mixture layer, a training sequence
        dict(name="experts 4096", kind="moe", tokens=4096, width=2048, ff=768, experts=128, top=8),
        # prompts of several requests in one step, some behind a cached prefix, running requests with their next token
        dict(name="prefill 5+3 requests", kind="serve", stack="large", layers=4, vocab=32000, seqs=5, tokens=3900, singles=3,
             past=1100, quant="none"),
        # one user waiting for the next token
        dict(name="decode 1x300", kind="serve", stack="large", layers=4, vocab=32000, seqs=0, tokens=0, singles=1, past=300,
             quant="none"),
        # an ordinary load
        dict(name="decode 48x2500", kind="serve", stack="large", layers=4, vocab=32000, seqs=0, tokens=0, singles=48,
             past=2500, quant="none"),
        # a full engine
        dict(name="decode 256x1400", kind="serve", stack="large", layers=4, vocab=32000, seqs=0, tokens=0, singles=256,
             past=1400, quant="none"),
        # weight-only quantised serving of a few requests
        dict(name="decode nf4 4x900", kind="serve", stack="large", layers=4, vocab=32000, seqs=0, tokens=0, singles=4,
             past=900, quant="nf4"),
        # sampled (not greedy) requests of one step
        dict(name="sample 64", kind="sample", rows=64, vocab=128256, dtype="bf16", penalties=False),
        # the recurrent layers of a delta-rule hybrid, prompts of one step
        dict(name="delta rule 8192", kind="delta", seqs=2, tokens=8192, heads=32, dk=128, dv=128, channel_gate=False),
        # the recurrent layers of a state-space hybrid, prompts of one step
        dict(name="state space 6000", kind="ssd", seqs=3, tokens=6000, heads=64, dim=64, groups=1, state=128),
        # a decode step of a latent-attention model
        dict(name="latent decode 32x2000", kind="latent", seqs=32, keys=2000, heads=128),
    ]


def _log(rng: random.Random, lo: float, hi: float) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng: random.Random):
    kind = rng.choice(["train", "moe", "prefill", "decode", "decode", "quant", "sample", "delta", "ssd", "latent"])
    if kind == "train":
        length = _log(rng, 130, 8192)
        stack = rng.choice(["small", "medium", "large", "narrow"])
        return dict(kind="train", stack=stack, layers=rng.randint(1, 2), vocab=rng.choice([4096, 32000]),
                    rows=rng.randint(1, max(1, min(4, 6000 // length))), length=length, docs=rng.random() < 0.5)
    if kind == "moe":
        width, ff, experts, top = rng.choice([(2048, 768, 128, 8), (1024, 512, 16, 2), (2048, 1408, 64, 6)])
        return dict(kind="moe", tokens=_log(rng, 64, 4096), width=width, ff=ff, experts=experts, top=top)
    if kind == "prefill":
        seqs = rng.randint(1, 8)
        return dict(kind="serve", stack=rng.choice(["small", "medium", "large", "shard"]), layers=rng.randint(2, 4), vocab=32000,
                    seqs=seqs, tokens=max(seqs * 2, _log(rng, 20, 4096)), singles=rng.choice([0, 0, rng.randint(1, 40)]),
                    past=rng.choice([0, _log(rng, 16, 4000)]), quant="none")
    if kind == "decode":
        n = _log(rng, 1, 256)
        return dict(kind="serve", stack=rng.choice(["small", "medium", "large", "shard"]), layers=rng.randint(2, 4), vocab=32000,
                    seqs=0, tokens=0, singles=n, past=_log(rng, 16, min(8000, 350000 // n)), quant="none")
    if kind == "quant":
        n = _log(rng, 1, 64)
        return dict(kind="serve", stack=rng.choice(["small", "medium", "large"]), layers=rng.randint(2, 4), vocab=32000, seqs=0,
                    tokens=0, singles=n, past=_log(rng, 16, 2000), quant=rng.choice(["nf4", "int8", "a4bit", "mxfp4"]))
    if kind == "sample":
        return dict(kind="sample", rows=_log(rng, 1, 256), vocab=rng.choice([32000, 50257, 128256, 151936]),
                    dtype=rng.choice(["bf16", "f32"]), penalties=rng.random() < 0.3)
    if kind == "delta":
        seqs = _log(rng, 1, 64)
        dk, dv = rng.choice([(128, 128), (128, 128), (64, 64), (128, 256)])
        return dict(kind="delta", seqs=seqs, tokens=max(seqs, _log(rng, 1, 8192)), heads=rng.choice([4, 16, 32]), dk=dk, dv=dv,
                    channel_gate=rng.random() < 0.25)
    if kind == "ssd":
        seqs = _log(rng, 1, 64)
        return dict(kind="ssd", seqs=seqs, tokens=max(seqs, _log(rng, 1, 8192)), heads=rng.choice([8, 24, 64]),
                    dim=rng.choice([64, 64, 128]), groups=rng.choice([1, 1, 4]), state=rng.choice([16, 64, 128]))
    n = _log(rng, 1, 128)
    return dict(kind="latent", seqs=n, keys=_log(rng, 16, min(16000, 200000 // n)), heads=rng.choice([16, 64, 128]))


# --------------------------------------------------------------------------------------------------------------- inputs
def _gen(seed: int) -> torch.Generator:
    return torch.Generator(device="cuda").manual_seed(seed)


def _rn(g, *shape, std=1.0, dtype=BF):
    return torch.randn(shape, generator=g, device="cuda", dtype=dtype).mul_(std)


def _split(total: int, parts: int, key: str, least: int = 1) -> list[int]:
    """``parts`` ragged lengths of at least ``least`` that add up to ``total``: the same for every seed."""
    r = random.Random(key)
    w = [r.uniform(0.2, 1.0) for _ in range(parts)]
    free = total - least * parts
    out = [least + int(free * x / sum(w)) for x in w]
    out[0] += total - sum(out)
    return out


def _weights(case, g) -> dict[str, torch.Tensor]:
    """Weights of a decoder stack, by the framework's parameter names."""
    H, F, hq, hk, d = STACKS[case["stack"]]
    V = case["vocab"]
    std = H ** -0.5 if H < 2048 else 0.02
    w = {"model.embed_tokens.weight": _rn(g, V, H)}
    for i in range(case["layers"]):
        p = f"model.layers.{i}."
        w[p + "self_attn.qkv_proj.weight"] = _rn(g, (hq + 2 * hk) * d, H, std=std)
        w[p + "self_attn.o_proj.weight"] = _rn(g, H, hq * d, std=std)
        w[p + "mlp.gate_up_proj.weight"] = _rn(g, 2 * F, H, std=std)
        w[p + "mlp.down_proj.weight"] = _rn(g, H, F, std=std)
        w[p + "input_layernorm.weight"] = _rn(g, H, std=0.1).add_(1.0)
        w[p + "post_attention_layernorm.weight"] = _rn(g, H, std=0.1).add_(1.0)
    w["model.norm.weight"] = _rn(g, H, std=0.1).add_(1.0)
    w["lm_head.weight"] = _rn(g, V, H, std=std)
    return w


def _model(case, weights, positions: int):
    from easydel_b200.modules.llama import LlamaConfig, LlamaForCausalLM

    H, F, hq, hk, d = STACKS[case["stack"]]
    cfg = LlamaConfig(vocab_size=case["vocab"], hidden_size=H, intermediate_size=F, num_hidden_layers=case["layers"],
                      num_attention_heads=hq, num_key_value_heads=hk, head_dim=d, rms_norm_eps=EPS, rope_theta=THETA,
                      max_position_embeddings=positions, tie_word_embeddings=False,
                      gradient_checkpointing="nothing_saveable", lmhead_chunksize=2048)
    model = LlamaForCausalLM.sequential_init(cfg, dtype=BF, param_dtype=BF, device="cuda", seed=0)
    params = dict(model.named_parameters())
    assert params.keys() == weights.keys()
    with torch.no_grad():
        for n, p in params.items():
            p.copy_(weights[n])
    return model


def _train_batch(case, g):
    B, T = case["rows"], case["length"]
    ids = torch.randint(0, case["vocab"], (B, T), generator=g, device="cuda")
    labels, seg = ids.clone(), None
    if case["docs"]:
        rows = []
        for b in range(B):      # a few documents per row, then padding (segment 0)
            lens = _split(T - T // 16, 3, f"{T}/{b}", 8)
            rows.append(sum(([i + 1] * n for i, n in enumerate(lens)), []) + [0] * (T // 16))
        seg = torch.tensor(rows, dtype=torch.int32, device="cuda")
        first = torch.ones_like(seg, dtype=torch.bool)
        first[:, 1:] = seg[:, 1:] != seg[:, :-1]
        labels[first | (seg == 0)] = -100      # no document predicts the next one's first token
    return ids, labels, seg


def _moe_inputs(case, g):
    T, H, F, E, k = case["tokens"], case["width"], case["ff"], case["experts"], case["top"]
    logits = _rn(g, T, E, dtype=torch.float32) + _rn(g, E, std=0.7, dtype=torch.float32)     # some experts are popular
    p, idx = torch.softmax(logits, -1).topk(k, -1)
    return dict(x=_rn(g, T, H), gu=_rn(g, E, 2 * F, H, std=H ** -0.5), down=_rn(g, E, H, F, std=F ** -0.5),
                p=p / p.sum(-1, keepdim=True), idx=idx, dy=_rn(g, T, H))


def _serve_spans(case) -> list[tuple[int, int]]:
    """(new tokens, cached keys before them) of every request: single tokens first, as the scheduler orders a step."""
    r = random.Random(f"{case['singles']}/{case['seqs']}/{case['tokens']}/{case['past']}")
    out = [(1, max(1, int(case["past"] * r.uniform(0.3, 1.0)))) for _ in range(case["singles"])]
    if case["seqs"]:
        for n in _split(case["tokens"], case["seqs"], f"p{case['tokens']}/{case['seqs']}"):
            out.append((n, int(case["past"] * r.choice([0, 0, 1, r.random()]))))
    return out


def _serve_inputs(case, seed):
    g = _gen(seed)
    spans = _serve_spans(case)
    _, _, _, hk, d = STACKS[case["stack"]]
    w = _weights(case, g)
    need = [-(-(a + p) // PAGE) for a, p in spans]
    pages = sum(need) + 1
    perm = (torch.randperm(pages - 1, generator=g, device="cuda") + 1).tolist()      # page 0 is the null page
    width = max(64, max(need))
    table = torch.zeros(len(spans), width, dtype=torch.int32)
    slots, pos, at = [], [], 0
    for b, (a, p) in enumerate(spans):
        mine = perm[at:at + need[b]]
        at += need[b]
        table[b, :need[b]] = torch.tensor(mine, dtype=torch.int32)
        where = range(p, p + a)
        pos += where
        slots += [mine[i // PAGE] * PAGE + i % PAGE for i in where]
    L = case["layers"]
    k, v = _rn(g, L, pages, PAGE, hk, d), _rn(g, L, pages, PAGE, hk, d)
    ids = torch.randint(0, case["vocab"], (len(pos),), generator=g, device="cuda")
    return dict(spans=spans, weights=w, k=k, v=v, table=table.cuda(), pages=pages, ids=ids,
                pos=torch.tensor(pos, dtype=torch.int32, device="cuda"), slots=torch.tensor(slots, dtype=torch.int32, device="cuda"))


def _delta_inputs(case, seed):
    g = _gen(seed)
    T, H, dk, dv, B = case["tokens"], case["heads"], case["dk"], case["dv"], case["seqs"]
    unit = lambda x: (x.float() * torch.rsqrt(x.float().pow(2).sum(-1, keepdim=True) + 1e-6)).to(BF)  # noqa: E731
    act = torch.nn.functional.silu
    gate = (T, H, dk) if case["channel_gate"] else (T, H)
    rate = torch.rand(H, generator=g, device="cuda") * 15.9 + 0.1
    rate = rate[None, :, None] if case["channel_gate"] else rate[None]
    return dict(q=unit(act(_rn(g, T, H, dk))), k=unit(act(_rn(g, T, H, dk))), v=act(_rn(g, T, H, dv)),
                g=-rate * torch.nn.functional.softplus(_rn(g, *gate, dtype=torch.float32) - 4.0),
                beta=torch.sigmoid(_rn(g, T, H, dtype=torch.float32)), cu=_cu(case),
                state=torch.zeros(B, H, dk, dv, device="cuda"))


def _ssd_inputs(case, seed):
    g = _gen(seed)
    T, H, P, G, N = case["tokens"], case["heads"], case["dim"], case["groups"], case["state"]
    f32 = torch.float32
    return dict(x=torch.nn.functional.silu(_rn(g, T, H, P)), dt=_rn(g, T, H), A=-(torch.rand(H, generator=g, device="cuda") * 15 + 1),
                B=torch.nn.functional.silu(_rn(g, T, G, N)), C=torch.nn.functional.silu(_rn(g, T, G, N)),
                D=_rn(g, H, std=0.1, dtype=f32) + 1, bias=_rn(g, H, dtype=f32) - 4.0, cu=_cu(case),
                state=torch.zeros(case["seqs"], H, P, N, device="cuda"))


def _lens(case) -> list[int]:
    return _split(case["tokens"], case["seqs"], f"{case['tokens']}/{case['seqs']}")


def _cu(case) -> torch.Tensor:
    return torch.tensor([0] + _lens(case), device="cuda").cumsum(0).to(torch.int32)


def _latent_inputs(case, seed):
    g = _gen(seed)
    r = random.Random(f"{case['seqs']}/{case['keys']}")
    lens = [max(1, int(case["keys"] * r.uniform(0.3, 1.0))) for _ in range(case["seqs"])]
    need = [-(-n // PAGE) for n in lens]
    perm = torch.randperm(sum(need), generator=g, device="cuda").add_(1).to(torch.int32)
    table = torch.zeros(len(lens), max(need), dtype=torch.int32, device="cuda")
    at = 0
    for b, n in enumerate(need):
        table[b, :n] = perm[at:at + n]
        at += n
    return dict(q=_rn(g, len(lens), case["heads"], 576, std=0.6), pages=_rn(g, sum(need) + 1, PAGE, 1, 576), table=table,
                lens=torch.tensor(lens, dtype=torch.int32, device="cuda"), host_lens=lens)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "train":
        from easydel_b200.infra.base_state import EasyDeLState
        from easydel_b200.optimizers import OptimizerFactory, SchedulerConfig

        g = _gen(seed)
        model = _model(case, _weights(case, g), case["length"]).train()
        ids, labels, seg = _train_batch(case, g)
        tx, _ = OptimizerFactory.create("adamw", SchedulerConfig(None, learning_rate=1e-5), weight_decay=0.01)
        state = EasyDeLState.create(model=model, tx=tx, init_opt_state=True)
        batch = dict(input_ids=ids, labels=labels, **({} if seg is None else {"segment_ids": seg}))
        return dict(kind=kind, model=model, state=state, batch=batch)
    if kind == "moe":
        i = _moe_inputs(case, _gen(seed))
        for n in ("gu", "down"):
            i[n] = torch.nn.Parameter(i[n])
            i[n].main_grad = torch.zeros(i[n].shape, dtype=torch.float32, device="cuda")
        return dict(kind=kind, **i)
    if kind == "serve":
        return _prepare_serve(case, seed)
    if kind == "sample":
        g = _gen(seed)
        R, V = case["rows"], case["vocab"]
        u = lambda *s: torch.rand(*s, generator=g, device="cuda")  # noqa: E731
        kw = dict(temperature=torch.where(u(R) < 0.1, torch.zeros(R, device="cuda"), 0.5 + 0.7 * u(R)),
                  top_k=torch.where(u(R) < 0.5, torch.zeros(R, device="cuda"), 1 + 63 * u(R)).to(torch.int32),
                  top_p=0.7 + 0.3 * u(R), min_p=torch.where(u(R) < 0.7, torch.zeros(R, device="cuda"), 0.1 * u(R)),
                  seeds=torch.randint(0, 1 << 31, (R,), generator=g, device="cuda"),
                  steps=torch.randint(0, 1000, (R,), generator=g, device="cuda").to(torch.int32))
        if case["penalties"]:
            counts = torch.zeros(R, V, dtype=torch.int32, device="cuda")
            seen = torch.randint(0, V, (R, 300), generator=g, device="cuda")
            counts.scatter_add_(1, seen, torch.ones_like(seen, dtype=torch.int32))
            kw.update(counts=counts, presence=0.5 * u(R), frequency=0.5 * u(R), repetition=1.0 + 0.3 * u(R))
        logits = _rn(g, R, V, std=2.5, dtype=BF if case["dtype"] == "bf16" else torch.float32)
        return dict(kind=kind, logits=logits, kw=kw)
    if kind == "delta":
        return dict(kind=kind, **_delta_inputs(case, seed))
    if kind == "ssd":
        return dict(kind=kind, **_ssd_inputs(case, seed))
    if kind == "latent":
        from easydel_b200.ops import latent

        i = _latent_inputs(case, seed)
        splits = latent.decode_splits(case["seqs"], case["heads"], None, case["keys"], _sms())
        return dict(kind=kind, splits=splits, **i)
    raise ValueError(kind)


def _sms() -> int:
    return torch.cuda.get_device_properties(0).multi_processor_count


def _prepare_serve(case, seed):
    from easydel_b200.caching.paged import PagedBatchMeta, PagedKVCache
    from easydel_b200.layers.quantization import EasyQuantizer

    i = _serve_inputs(case, seed)
    _, _, _, hk, d = STACKS[case["stack"]]
    spans, B, T = i["spans"], len(i["spans"]), len(i["pos"])
    model = _model(case, i.pop("weights"), 16384).eval()
    if case["quant"] != "none":
        model = EasyQuantizer(case["quant"]).apply_quantization(model)
    cache = PagedKVCache(case["layers"], i["pages"], hk, d, device="cuda")
    cache.k.copy_(i.pop("k"))
    cache.v.copy_(i.pop("v"))
    news = torch.tensor([a for a, _ in spans], device="cuda")
    cu = torch.cat([news.new_zeros(1), news.cumsum(0)]).to(torch.int32)
    decode = case["seqs"] == 0
    units, width = B * hk, i["table"].shape[1]
    splits = 1 if not decode or units * 2 > _sms() else int(min(8, width // 4, max(1, _sms() // units)))
    meta = PagedBatchMeta(cu_q=cu, kv_lens=torch.tensor([a + p for a, p in spans], dtype=torch.int32, device="cuda"),
                          page_table=i["table"], slot_mapping=i["slots"], max_q=max(a for a, _ in spans), num_seqs=B,
                          last_token_index=cu[1:] - 1, request_distribution=(case["singles"], B, B), num_splits=splits,
                          slot_ids=torch.arange(B, dtype=torch.int32, device="cuda"),
                          spans=None if decode else [(a, a + p) for a, p in spans])
    cache.step_meta = meta
    s = dict(kind="serve", model=model, cache=cache, meta=meta, ids=i["ids"][None], pos=i["pos"][None], graph=None)
    if decode:      # the engine captures the decode step of a batch size once and replays it from then on
        with torch.no_grad():
            _serve_step(s)
            torch.cuda.synchronize()
            s["graph"] = torch.cuda.CUDAGraph()
            with torch.cuda.graph(s["graph"]):
                s["logits"] = _serve_step(s)
    return s


def _serve_step(s):
    from easydel_b200.ops import serving

    m = s["meta"]
    res = s["model"](input_ids=s["ids"], position_ids=s["pos"], past_key_values=s["cache"], cache_metadata=m,
                     apply_lm_head=False)
    return s["model"].apply_lm_head(serving.gather_rows(res.last_hidden_state[0], m.last_token_index))


# ---------------------------------------------------------------------------------------------------------------- calls
def run(s):
    kind = s["kind"]
    if kind == "train":
        s["state"].zero_grad()
        _, metrics = s["model"].compute_loss(**s["batch"])
        metrics.loss.backward()
        return dict(loss=metrics.loss.detach(), grads={n: p.main_grad for n, p in s["model"].named_parameters()})
    if kind == "moe":
        from easydel_b200.ops.moe_kernels import moe_ffn

        s["gu"].main_grad.zero_()
        s["down"].main_grad.zero_()
        x, p = s["x"].detach().requires_grad_(), s["p"].detach().requires_grad_()
        y = moe_ffn(x, s["gu"], s["down"], p, s["idx"])
        y.backward(s["dy"])
        return dict(y=y.detach(), dx=x.grad, dp=p.grad, gu=s["gu"].main_grad, down=s["down"].main_grad)
    if kind == "serve":
        if s["graph"] is not None:
            s["graph"].replay()
            logits = s["logits"]
        else:
            with torch.no_grad():
                logits = _serve_step(s)
        return dict(logits=logits, k=s["cache"].k, v=s["cache"].v)
    if kind == "sample":
        from easydel_b200.ops import serving

        tokens, logprobs = serving.sample(s["logits"], want_logprob=True, **s["kw"])
        return dict(tokens=tokens, logprobs=logprobs)
    if kind == "delta":
        from easydel_b200.ops import ssm

        s["state"].zero_()      # new prompts start from an empty state
        o = ssm.gated_delta_rule(s["q"], s["k"], s["v"], s["g"], s["beta"], None, s["cu"], s["state"])
        return dict(o=o, state=s["state"])
    if kind == "ssd":
        from easydel_b200.ops import ssm

        s["state"].zero_()
        y = ssm.ssd_scan(s["x"], s["dt"], s["A"], s["B"], s["C"], s["D"], s["bias"], True, s["cu"], s["state"])
        return dict(y=y, state=s["state"])
    if kind == "latent":
        from easydel_b200.ops import serving

        return serving.mla_decode_attention(s["q"], s["pages"], s["lens"], s["table"], scale=192 ** -0.5, num_splits=s["splits"])
    raise ValueError(kind)


# ----------------------------------------------------------------------------------------------------------------- work
def work(case):
    kind = case["kind"]
    if kind == "train":
        H, F, hq, hk, d = STACKS[case["stack"]]
        B, T, L, V = case["rows"], case["length"], case["layers"], case["vocab"]
        layer = (hq + 2 * hk) * d * H + H * hq * d + 3 * H * F
        pairs = B * T * (T + 1) / 2
        if case["docs"]:
            pairs = sum(n * (n + 1) / 2 for b in range(B) for n in _split(T - T // 16, 3, f"{T}/{b}", 8) + [T // 16])
        flops = 6.0 * B * T * (L * layer + V * H) + L * 3.5 * 4 * pairs * hq * d     # without the recomputation
        params = L * layer + 2 * V * H
        return dict(flops=flops, bytes=6.0 * params)           # weights read, gradients written
    if kind == "moe":
        T, H, F, E, k = case["tokens"], case["width"], case["ff"], case["experts"], case["top"]
        used = E * (1 - (1 - k / E) ** T)
        return dict(flops=18.0 * T * k * H * F, bytes=3 * H * F * (2.0 * used + 4 * E) + 8.0 * T * H)
    if kind == "serve":
        H, F, hq, hk, d = STACKS[case["stack"]]
        L, V, spans = case["layers"], case["vocab"], _serve_spans(case)
        T, B = sum(a for a, _ in spans), len(spans)
        layer = (hq + 2 * hk) * d * H + H * hq * d + 3 * H * F
        pairs = sum(a * p + a * (a + 1) / 2 for a, p in spans)
        keys = sum(a + p for a, p in spans)
        per = {"none": 2.0, "nf4": 0.5 + 2 / 64, "a4bit": 0.5 + 4 / 64, "mxfp4": 0.5 + 2 / 32, "int8": 1 + 2 / 128}[case["quant"]]
        return dict(flops=2.0 * T * L * layer + 2.0 * B * V * H + 4.0 * L * pairs * hq * d,
                    bytes=per * L * layer + 2.0 * V * H + 4.0 * L * keys * hk * d + 2.0 * T * H + 2.0 * B * V)
    if kind == "sample":
        n = case["rows"] * case["vocab"]
        return dict(flops=0, bytes=n * ((2 if case["dtype"] == "bf16" else 4) + (4 if case["penalties"] else 0)))
    if kind == "delta":
        T, H, dk, dv = case["tokens"], case["heads"], case["dk"], case["dv"]
        gate = 4 * dk if case["channel_gate"] else 4
        return dict(flops=8.0 * T * H * dk * dv, bytes=T * H * (4.0 * dk + 4 * dv + gate + 4) + 8.0 * case["seqs"] * H * dk * dv)
    if kind == "ssd":
        T, H, P, G, N = case["tokens"], case["heads"], case["dim"], case["groups"], case["state"]
        return dict(flops=6.0 * T * H * P * N, bytes=T * (4.0 * H * P + 2 * H + 4 * G * N) + 8.0 * case["seqs"] * H * P * N)
    if kind == "latent":
        r = random.Random(f"{case['seqs']}/{case['keys']}")
        keys = sum(max(1, int(case["keys"] * r.uniform(0.3, 1.0))) for _ in range(case["seqs"]))
        return dict(flops=2.0 * keys * case["heads"] * (576 + 512), bytes=2.0 * keys * 576 + 2.0 * case["seqs"] * case["heads"] * 1088)
    raise ValueError(kind)


def tolerance(case):
    # bf16 operands and results with fp32 sums: about 2e-3 per rounding, more through a stack of layers
    kind = case["kind"]
    if kind in ("train", "serve"):
        return {"rel": 0.03, "max": 0.9}
    if kind == "sample":
        return {"rel": 1e-5, "max": 1e-3, "differ": 0.01}
    if kind == "moe":
        return {"rel": 0.02, "max": 0.5}
    return {"rel": 0.01, "max": 0.3}


# ------------------------------------------------------------------------------------------------------------- 64 bits
def _norm64(x, w):
    return x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + EPS) * w


def _rope64(x, pos):
    d = x.shape[-1]
    f = THETA ** (-torch.arange(0, d, 2, device="cuda", dtype=torch.float64) / d)
    a = pos.double()[:, None, None] * f
    x1, x2 = x[..., :d // 2], x[..., d // 2:]
    return torch.cat([x1 * a.cos() - x2 * a.sin(), x2 * a.cos() + x1 * a.sin()], -1)


def _layer64(x, w, p, case, pos, attend):
    """One decoder layer over token rows ``x``; ``attend(q, k, v)`` is the attention over the rows."""
    _, F, hq, hk, d = STACKS[case["stack"]]
    h = _norm64(x, w[p + "input_layernorm.weight"]) @ w[p + "self_attn.qkv_proj.weight"].t()
    q, k, v = (t.reshape(len(x), -1, d) for t in h.split([hq * d, hk * d, hk * d], -1))
    x = x + attend(_rope64(q, pos), _rope64(k, pos), v).reshape(len(x), -1) @ w[p + "self_attn.o_proj.weight"].t()
    gu = _norm64(x, w[p + "post_attention_layernorm.weight"]) @ w[p + "mlp.gate_up_proj.weight"].t()
    return x + (torch.nn.functional.silu(gu[:, :F]) * gu[:, F:]) @ w[p + "mlp.down_proj.weight"].t()


def _head64(q, k, v, mask):
    s = q @ k.t() * q.shape[-1] ** -0.5
    return torch.softmax(s.masked_fill(~mask, -math.inf), -1) @ v


def _exact_train(case, seed):
    from torch.utils.checkpoint import checkpoint

    g = _gen(seed)
    w = {n: t.double().requires_grad_() for n, t in _weights(case, g).items()}
    ids, labels, seg = _train_batch(case, g)
    _, _, hq, hk, _ = STACKS[case["stack"]]
    T, loss = case["length"], 0.0
    causal = torch.ones(T, T, dtype=torch.bool, device="cuda").tril()
    target = torch.full_like(labels, -100)
    target[:, :-1] = labels[:, 1:]
    count = (target != -100).sum()
    for b in range(case["rows"]):
        mask, pos = causal, torch.arange(T, device="cuda")
        if seg is not None:
            mask = causal & (seg[b][:, None] == seg[b][None])
            start = torch.ones_like(seg[b], dtype=torch.bool)
            start[1:] = seg[b][1:] != seg[b][:-1]
            pos = pos - (pos * start).cummax(0).values

        def attend(q, k, v, mask=mask):
            return torch.stack([checkpoint(_head64, q[:, h], k[:, h * hk // hq], v[:, h * hk // hq], mask, use_reentrant=False)
                                for h in range(hq)], 1)

        x = w["model.embed_tokens.weight"][ids[b]]
        for i in range(case["layers"]):
            x = checkpoint(_layer64, x, w, f"model.layers.{i}.", case, pos, attend, use_reentrant=False)
        logits = _norm64(x, w["model.norm.weight"]) @ w["lm_head.weight"].t()
        part = torch.nn.functional.cross_entropy(logits, target[b], ignore_index=-100, reduction="sum") / count
        part.backward()
        loss = loss + part.detach()
        del logits, part, x
    return dict(loss=loss, grads={n: t.grad for n, t in w.items()})


def _exact_moe(case, seed):
    i = _moe_inputs(case, _gen(seed))
    F = case["ff"]
    x, p = i["x"].double().requires_grad_(), i["p"].double().requires_grad_()
    gu, down, idx = i["gu"].double().requires_grad_(), i["down"].double().requires_grad_(), i["idx"]
    y = torch.zeros_like(x)
    for e in range(case["experts"]):
        t, j = (idx == e).nonzero(as_tuple=True)
        h = x[t] @ gu[e].t()
        y = y.index_add(0, t, (torch.nn.functional.silu(h[:, :F]) * h[:, F:]) @ down[e].t() * p[t, j][:, None])
    grads = torch.autograd.grad(y, [x, p, gu, down], i["dy"].double())
    return dict(zip(("y", "dx", "dp", "gu", "down"), (y.detach(), *grads)))


def _exact_serve(case, seed):
    i = _serve_inputs(case, seed)
    w = {n: t.double() for n, t in i["weights"].items() if n != "model.embed_tokens.weight"}
    w["model.embed_tokens.weight"] = i["weights"]["model.embed_tokens.weight"]
    if case["quant"] != "none":      # the weights are what their codes say: read off the prepared model's buffers
        s = prepare(case, seed)
        for n, m in s["model"].named_modules():
            if hasattr(m, "codes"):
                c = m.codes.long()
                if m.bits == 4:
                    c = torch.stack([c & 15, c >> 4], -1).reshape(c.shape[0], -1)
                wide = lambda t: t.double().repeat_interleave(m.group, 1)  # noqa: B023, E731
                w[n + ".weight"] = m.lut.double()[c] * wide(m.scales) + (0 if m.zeros is None else wide(m.zeros))
        del s
    _, _, hq, hk, d = STACKS[case["stack"]]
    x = w["model.embed_tokens.weight"][i["ids"]].double()
    ks, vs = [], []
    for layer in range(case["layers"]):
        kc, vc = i["k"][layer].double().view(-1, hk, d), i["v"][layer].double().view(-1, hk, d)

        def attend(q, k, v, kc=kc, vc=vc):
            kc[i["slots"].long()], vc[i["slots"].long()] = k, v
            out, at = torch.empty_like(q), 0
            for b, (a, p) in enumerate(i["spans"]):
                pages = i["table"][b, :-(-(a + p) // PAGE)].long()
                rows = (pages[:, None] * PAGE + torch.arange(PAGE, device="cuda")).view(-1)[:a + p]
                kk, vv = kc[rows].repeat_interleave(hq // hk, 1), vc[rows].repeat_interleave(hq // hk, 1)
                sc = torch.einsum("ahd,khd->hak", q[at:at + a], kk) * d ** -0.5
                see = torch.arange(a + p, device="cuda")[None] <= torch.arange(p, p + a, device="cuda")[:, None]
                out[at:at + a] = torch.einsum("hak,khd->ahd", torch.softmax(sc.masked_fill(~see, -math.inf), -1), vv)
                at += a
            return out

        x = _layer64(x, w, f"model.layers.{layer}.", case, i["pos"], attend)
        ks.append(kc.view(i["k"][layer].shape))
        vs.append(vc.view(i["v"][layer].shape))
    last = torch.tensor([a for a, _ in i["spans"]], device="cuda").cumsum(0) - 1
    return dict(logits=_norm64(x[last], w["model.norm.weight"]) @ w["lm_head.weight"].t(), k=torch.stack(ks), v=torch.stack(vs))


def _padded(t, lens, fill=0.0):
    """Packed token rows -> ``[longest, sequences, ...]`` in 64 bits."""
    out = torch.full((max(lens), len(lens), *t.shape[1:]), fill, dtype=torch.float64, device="cuda")
    at = 0
    for b, n in enumerate(lens):
        out[:n, b] = t[at:at + n].double()
        at += n
    return out


def _exact_delta(case, seed):
    i, lens = _delta_inputs(case, seed), _lens(case)
    q, k, v, beta = (_padded(i[n], lens) for n in ("q", "k", "v", "beta"))
    beta = _padded(i["beta"].to(BF), lens)      # the recurrence takes 16-bit update gates
    decay = _padded(i["g"], lens).exp()
    decay = decay[..., None] if case["channel_gate"] else decay[..., None, None]
    S = i["state"].double()
    o = torch.empty_like(v)
    for t in range(max(lens)):
        S *= decay[t]
        r = (v[t] - torch.einsum("bhk,bhkv->bhv", k[t], S)) * beta[t][..., None]
        S += k[t][..., None] * r[:, :, None]
        o[t] = torch.einsum("bhk,bhkv->bhv", q[t], S)
    return dict(o=torch.cat([o[:n, b] for b, n in enumerate(lens)]) * case["dk"] ** -0.5, state=S)


def _exact_ssd(case, seed):
    i, lens = _ssd_inputs(case, seed), _lens(case)
    rep = case["heads"] // case["groups"]
    x, B, C = (_padded(i[n], lens) for n in ("x", "B", "C"))
    dt = _padded(torch.nn.functional.softplus(i["dt"].double() + i["bias"].double()), lens)
    decay = (dt * i["A"].double()).exp()[..., None, None]
    S, y = i["state"].double(), torch.empty_like(x)
    for t in range(max(lens)):
        S *= decay[t]
        S += (dt[t][..., None] * x[t])[..., None] * B[t].repeat_interleave(rep, 1)[:, :, None]
        y[t] = torch.einsum("bhpn,bhn->bhp", S, C[t].repeat_interleave(rep, 1)) + i["D"].double()[:, None] * x[t]
    return dict(y=torch.cat([y[:n, b] for b, n in enumerate(lens)]), state=S)


def _exact_latent(case, seed):
    i = _latent_inputs(case, seed)
    out = []
    for b, n in enumerate(i["host_lens"]):
        rows = i["pages"][i["table"][b, :-(-n // PAGE)].long()].view(-1, 576)[:n].double()
        out.append(torch.softmax(i["q"][b].double() @ rows.t() * 192 ** -0.5, -1) @ rows[:, :512])
    return torch.stack(out)


def exact(case, seed):
    f = {"train": _exact_train, "moe": _exact_moe, "serve": _exact_serve, "delta": _exact_delta, "ssd": _exact_ssd,
         "latent": _exact_latent}.get(case["kind"])      # sampled tokens come out of a random draw: no such value
    if f is None:
        return None
    if case["kind"] == "train":
        return f(case, seed)
    with torch.enable_grad() if case["kind"] == "moe" else torch.no_grad():
        return f(case, seed)
