"""Workloads that stand for what a user of this framework runs on one GPU, through its public entry points.

Kinds of case
  rollout   ``Generator.generate``: prompts in, tokens and their log-probs out (prefill, then captured decode steps)
  logprobs  ``algorithms.sequence_logprobs``: the frozen reference policy's pass over finished rollouts
  update    one policy update: ``zero_grad``, ``policy_train_step`` (forward and backward over the microbatches), ``AdamW.step``
  prompt    ``Session.feed``: requests bring whole prompts and want the logits of their last token

Models have the real layer sizes of the repository's configurations (Llama-7B, Qwen3-8B and the served "2b" and "7b" shapes of the serving
benchmark) and few layers: a layer costs the same however many there are. Weights are random. Their output heads are shaped so that greedy
decoding has a clear favourite, as trained models have, and so that an update is nearly on-policy, as in training.
"""
import math

import torch

DEVICE = "cuda:0"
EOS = 2
F64 = torch.float64

#: Served shapes: width, heads, KV heads, experts, chosen ones, groups, groups kept, hidden units of an expert and of the shared one, query rank
SERVED = {"2b": (2048, 16, 4, 32, 4, 4, 2, 1024, 1024, 768), "7b": (4096, 32, 8, 64, 6, 8, 3, 1408, 2816, 1536)}
SERVED_VOCAB = 32000


def listed():
    return [
        # one interactive request: launches and latency
        dict(name="rollout_1", kind="rollout", model="llama7b", layers=4, rows=1, group=1, longest=33, new=16, forced=False, dtype="bfloat16"),
        # a small evaluation batch of unlike prompts
        dict(name="rollout_16", kind="rollout", model="llama7b", layers=4, rows=16, group=1, longest=419, new=32, forced=False, dtype="bfloat16"),
        # the generation phase of GRPO: 32 prompts, eight samples each, all rows decoding at once, rows ending at different lengths
        dict(name="rollout_grpo", kind="rollout", model="llama7b", layers=4, rows=256, group=8, longest=512, new=48, forced=True, dtype="bfloat16"),
        # the reference pass over a microbatch of finished rollouts of up to 2560 tokens
        dict(name="logprobs_16k", kind="logprobs", model="llama7b", layers=2, rows=12, longest=2560, dtype="bfloat16"),
        # a small update: a few short samples
        dict(name="update_small", kind="update", model="llama7b", layers=2, rows=4, longest=211, recompute="none", micro=8192, dtype="bfloat16"),
        # the update phase of GRPO: rollouts of up to 2560 tokens, two microbatches, activations recomputed
        dict(name="update_16k", kind="update", model="llama7b", layers=2, rows=12, longest=2560, recompute="full", micro=8192, dtype="bfloat16"),
        # an update of a model with grouped queries, normalised heads and a large vocabulary
        dict(name="update_gqa", kind="update", model="qwen3_8b", layers=2, rows=6, longest=1501, recompute="none", micro=8192, dtype="bfloat16"),
        # serving: prompts of a mixture-of-experts model, several requests at once
        dict(name="prompt_dulisun", kind="prompt", model="dulisun-7b", layers=4, rows=8, longest=1024, dtype="bfloat16"),
        # serving: decoding a batch of a mixture-of-experts model
        dict(name="rollout_dulisun", kind="rollout", model="dulisun-7b", layers=4, rows=64, group=1, longest=200, new=48, forced=False, dtype="bfloat16"),
        # serving in true fp32, as recorded runs are replayed
        dict(name="rollout_f32", kind="rollout", model="dulisun-2b", layers=2, rows=4, group=1, longest=90, new=16, forced=False, dtype="float32"),
        # serving: one long prompt of a latent-attention model
        dict(name="prompt_zafopel", kind="prompt", model="zafopel-7b", layers=4, rows=1, longest=8000, dtype="bfloat16"),
        # serving: decoding a few requests of a latent-attention model
        dict(name="rollout_zafopel", kind="rollout", model="zafopel-7b", layers=4, rows=8, group=1, longest=600, new=32, forced=False, dtype="bfloat16"),
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(("rollout", "rollout", "logprobs", "update", "update", "prompt"))
    if kind == "rollout":
        model = rng.choice(("llama7b", "llama7b", "qwen3_8b", "dulisun-7b", "zafopel-7b", "dulisun-2b", "zafopel-2b"))
        dtype = rng.choice(("bfloat16", "float32")) if model.endswith("-2b") else "bfloat16"
        if dtype == "float32":
            return dict(kind=kind, model=model, layers=2, rows=log(1, 8), group=1, longest=log(8, 120), new=log(4, 16), forced=False, dtype=dtype)
        group = rng.choice((1, 1, 4, 8)) if model == "llama7b" else 1
        rows = max(1, log(1, 256) // group) * group
        longest = min(log(16, 1024), max(16, 16384 * group // rows))
        return dict(kind=kind, model=model, layers=rng.choice((2, 4)), rows=rows, group=group, longest=longest, new=log(8, 48), forced=rng.random() < 0.5, dtype=dtype)
    if kind == "prompt":
        model = rng.choice(("dulisun-7b", "zafopel-7b", "dulisun-2b", "zafopel-2b", "llama7b"))
        rows = log(1, 16)
        return dict(kind=kind, model=model, layers=rng.choice((2, 4)), rows=rows, longest=log(16, 8192 // rows), dtype="bfloat16")
    rows = log(1, 24)
    longest = min(log(24, 2560), 16384 // rows)
    if kind == "logprobs":
        return dict(kind=kind, model=rng.choice(("llama7b", "llama7b", "qwen3_8b")), layers=2, rows=rows, longest=longest, dtype="bfloat16")
    model = rng.choice(("llama7b", "llama7b", "llama7b", "qwen3_8b"))
    longest = min(longest, 8192 // rows) if model == "qwen3_8b" else longest
    return dict(kind=kind, model=model, layers=2, rows=rows, longest=longest, recompute=rng.choice(("full", "none")), micro=rng.choice((4096, 8192)), dtype="bfloat16")


# ---------------------------------------------------------------------------------------------------- shapes of a case
def _spread(n, lo, hi):
    """``n`` unlike lengths from ``lo`` to ``hi``, the largest first."""
    return [hi] + [lo + int((hi - lo) * ((0.6180339887 * i) % 1.0)) for i in range(1, n)]


def _prompt_lens(c):
    """Length of every row's prompt (rollout, prompt), equal inside a group."""
    if c["kind"] == "rollout" and c["group"] > 1:
        return [c["longest"]] * c["rows"]
    return _spread(c["rows"], max(1, c["longest"] // 3), c["longest"])


def _new_lens(c):
    """Tokens that every row generates."""
    return _spread(c["rows"], max(1, c["new"] // 4), c["new"]) if c["forced"] else [c["new"]] * c["rows"]


def _train_lens(c):
    """(prompt, response) length of every row (logprobs, update)."""
    total = _spread(c["rows"], max(8, c["longest"] // 4), c["longest"])
    return [(max(2, t // 5), t - max(2, t // 5)) for t in total]


def _llama_config(c):
    import dataclasses
    from rpeg_b200.models.llama import LlamaConfig
    base = LlamaConfig.llama7b(max_pos=4096) if c["model"] == "llama7b" else LlamaConfig.qwen3_8b(max_pos=4096)
    return dataclasses.replace(base, n_layers=c["layers"])


def _is_llama(c):
    return c["model"] in ("llama7b", "qwen3_8b")


def _served_config(c):
    from rpeg_b200.models.dulisun import AttentionMixer, DecoderLayer, DulisunConfig, ExpertMixture
    from rpeg_b200.models.zafopel import InputScaledMixture, LatentMixer, ParallelLayer, ZafopelConfig
    family, size = c["model"].split("-")
    width, heads, kv, experts, top, groups, keep, ff, shared, q_rank = SERVED[size]
    if family == "dulisun":
        layer = DecoderLayer(AttentionMixer(heads, kv, 128, 128 ** -0.5, 8192, 64, 10000.0), ExpertMixture(experts, top, ff, shared, groups, keep))
        return DulisunConfig(width, SERVED_VOCAB, (layer,) * c["layers"], max_pos=9216)
    made = []
    for i in range(c["layers"]):
        common = dict(heads=heads, dim=128, rot_dim=64, vdim=128, kv_rank=512, scale=192 ** -0.5)
        m = LatentMixer(**common, window=8192, kv_from=i - 2 if i % 4 == 3 else None) if i % 2 else LatentMixer(**common, q_rank=q_rank, sink=True)
        made.append(ParallelLayer(m, InputScaledMixture(experts, top, 1024)))
    return ZafopelConfig(width, SERVED_VOCAB, tuple(made), max_pos=9216)


# ---------------------------------------------------------------------------------------------------- models and inputs from a seed
def _rng(seed, what):
    g = torch.Generator(device=DEVICE)
    g.manual_seed(seed * 16 + what)
    return g


def _successor(vocab, seed):
    """The token that greedy decoding is to choose after each one: a permutation that leads to no token below 3."""
    nxt = torch.arange(vocab, device=DEVICE)
    nxt[3:] = 3 + torch.randperm(vocab - 3, generator=_rng(seed, 1), device=DEVICE)
    return nxt


def _model(c, seed):
    """The model, and the token that follows each one under greedy decoding."""
    dtype = getattr(torch, c["dtype"])
    if _is_llama(c):
        from rpeg_b200.models.llama import LlamaModel
        cfg = _llama_config(c)
        train = c["kind"] == "update"
        m = LlamaModel(cfg, DEVICE, trainable=train, recompute=c["recompute"] if train else "full", seed=seed)
        g = _rng(seed, 2)

        def rows(scale):
            return torch.randn((cfg.vocab, cfg.d_model), generator=g, device=DEVICE) * scale

        if c["kind"] in ("logprobs", "update"):
            # trained embeddings are not vanishingly small; an update is nearly on-policy: no log-prob is far from -ln(vocab)
            m.p["embed"].copy_(rows(1.0))
            m.p["lm_head"].copy_(rows(6e-4 if train else 0.02))
            return m, None
        embed = rows(1.0)
        m.p["embed"].copy_(embed)
        nxt = _successor(cfg.vocab, seed)
        head = rows(0.35 / math.sqrt(cfg.d_model))
        # the favourite's logit is about 7: a layer adds about 2.6 to the mean square of a stream that starts at 1
        head[nxt] += embed * (7.0 * math.sqrt(1 + 2.6 * cfg.n_layers) / cfg.d_model)
        m.p["lm_head"].copy_(head)
        return m, nxt
    cfg = _served_config(c)
    g = _rng(seed, 3)
    if cfg.family == "dulisun":
        from rpeg_b200.models.dulisun import DulisunModel
        m = DulisunModel(cfg, DEVICE, dtype=dtype, seed=seed)
        # the embedding is the output head too: the favourite is the token itself, its logit set by the last norm's weight
        favourite = math.sqrt(cfg.width) / math.sqrt(1 + 2 * cfg.n_layers)
        m.p["final_norm"].copy_(8.0 / favourite - 1.0 + 0.03 * torch.randn(cfg.width, generator=g, device=DEVICE))
        return m, torch.arange(cfg.vocab, device=DEVICE)
    from rpeg_b200.models.zafopel import ZafopelModel
    m = ZafopelModel(cfg, DEVICE, dtype=dtype, seed=seed)
    nxt = _successor(cfg.vocab, seed)
    head = torch.randn((cfg.vocab, cfg.width), generator=g, device=DEVICE) * (0.8 / math.sqrt(cfg.width))
    head[nxt] += torch.tanh(0.5 * m.p["embed"].float()) * (50.0 / cfg.width)
    m.p["head"].copy_(head)
    return m, nxt


def _prompts(c, vocab, seed):
    g, lens = _rng(seed, 4), _prompt_lens(c)
    made = [torch.randint(3, vocab, (n,), generator=g, device=DEVICE, dtype=torch.int32) for n in lens]
    if c["kind"] == "rollout" and c["group"] > 1:
        made = [made[i // c["group"] * c["group"]] for i in range(len(made))]
    return made


def _rollout(c, vocab, seed):
    """Finished rollouts of a policy whose log-probs lie near -ln(vocab), a little above the reference's: dictionary of tensors, padded to
    the longest."""
    g, lens = _rng(seed, 5), _train_lens(c)
    n, s, t = len(lens), max(p for p, _ in lens), max(r for _, r in lens)
    f32 = dict(generator=g, device=DEVICE)
    r_len = torch.tensor([r for _, r in lens], device=DEVICE)
    mask = (torch.arange(t, device=DEVICE)[None, :] < r_len[:, None]).float()
    scores = torch.randn(n, **f32)
    return dict(prompt_ids=torch.randint(3, vocab, (n, s), dtype=torch.int32, **f32), resp_ids=torch.randint(3, vocab, (n, t), dtype=torch.int32, **f32),
                old_logp=(-math.log(vocab) + 0.01 * torch.randn((n, t), **f32)) * mask, ref_logp=(-math.log(vocab) - 0.05 + 0.01 * torch.randn((n, t), **f32)) * mask,
                mask=mask, adv=((scores + 0.5)[:, None] * mask).contiguous())


def _algo(c):
    from rpeg_b200.engine import algorithms as A
    return A.AlgoConfig(kl_coef=0.04, micro_tokens=c.get("micro", 16384), head_chunk=8192)


def prepare(case, seed):
    c = case
    model, _ = _model(c, seed)
    if c["kind"] in ("logprobs", "update"):
        from rpeg_b200.engine import algorithms as A
        from rpeg_b200.engine.optimizer import AdamW
        d, lens = _rollout(c, model.cfg.vocab, seed), _train_lens(c)
        ro = A.Rollout(d["prompt_ids"], [p for p, _ in lens], d["resp_ids"], [r for _, r in lens], d["old_logp"], d["mask"], ref_logp=d["ref_logp"], adv=d["adv"])
        return dict(c=c, model=model, rollout=ro, algo=_algo(c), opt=AdamW(model) if c["kind"] == "update" else None)
    from rpeg_b200.engine.generation import Generator
    prompts = _prompts(c, model.cfg.vocab, seed)
    new = c["new"] if c["kind"] == "rollout" else 1
    gen = Generator(model, max_slots=c["rows"], max_seq_len=c["longest"] + new, kv_budget_bytes=24e9, eos_id=EOS)
    if c["kind"] == "prompt":
        from rpeg_b200.engine.session import Session
        lists = [p.tolist() for p in prompts]
        return dict(c=c, session=Session(gen), entries=[(i, p, [len(p) - 1]) for i, p in enumerate(lists)])
    if c["group"] > 1:
        prompts = torch.stack(prompts)
    forced = [n if n < c["new"] else 0 for n in _new_lens(c)] if c["forced"] else None
    return dict(c=c, gen=gen, prompts=prompts, forced=forced)


def run(state):
    c = state["c"]
    if c["kind"] == "rollout":
        r = state["gen"].generate(state["prompts"], c["new"], greedy=True, forced_lens=state["forced"], group_size=c["group"])
        return dict(tokens=r.tokens, logprobs=r.logprobs, lengths=r.lengths)
    if c["kind"] == "prompt":
        out = state["session"].feed(state["entries"])
        for rid, _, _ in state["entries"]:
            state["session"].end(rid)
        return out
    from rpeg_b200.engine import algorithms as A
    model = state["model"]
    if c["kind"] == "logprobs":
        return dict(logprobs=A.sequence_logprobs(model, state["rollout"], state["algo"]))
    model.zero_grad()
    metrics = A.policy_train_step(model, state["rollout"], state["algo"])
    opt = state["opt"]
    opt.step()
    return dict(loss=metrics["loss"], kl=metrics["kl_sum"], grads=model.g, weights=model.w, master=opt.master, m=opt.m, v=opt.v)


# ---------------------------------------------------------------------------------------------------- what a pass cannot do without
def _pairs(n, window=0):
    return n * (n + 1) / 2


def _layer_costs(c):
    """Per layer: parameters that every token meets, parameters of one expert, chosen experts, experts, FLOPs per (query, visible key) pair,
    cached bytes per token."""
    size = 4 if c["dtype"] == "float32" else 2
    if c["model"] == "llama7b":
        return 4 * 4096 * 4096 + 3 * 4096 * 11008, 0, 0, 0, 4 * 4096, 2 * 4096 * size
    if c["model"] == "qwen3_8b":
        return (2 * 4096 + 2 * 1024) * 4096 + 3 * 4096 * 12288, 0, 0, 0, 4 * 4096, 2 * 1024 * size
    family, s = c["model"].split("-")
    width, heads, kv, experts, top, _, _, ff, shared, q_rank = SERVED[s]
    if family == "dulisun":
        return width * 128 * (2 * heads + kv) + width * (experts + 2 * shared), 2 * width * ff, top, experts, 4 * 128 * heads, 2 * kv * 128 * size
    maps = heads * 256 * 512
    q = (width * q_rank + q_rank * heads * 192 + width * heads * 192) // 2           # half of the layers have a query latent
    return q + width * 576 + maps + heads * 128 * width + width * experts, 3 * width * 1024, top, experts, 2 * heads * (192 + 128), 576 * size


def work(case):
    c = case
    vocab, width = (151936, 4096) if c["model"] == "qwen3_8b" else (32000, 4096 if not c["model"].endswith("2b") else 2048)
    base, expert, top, experts, pair, cached = _layer_costs(c)
    size = 4 if c["dtype"] == "float32" else 2
    L, head = c["layers"], vocab * width

    def weights(tokens):                       # bytes of the weights that a step of so many tokens must read
        used = experts * (1 - (1 - top / experts) ** tokens) if experts else 0
        return size * (L * (base + used * expert) + head)

    per_token = 2 * L * (base + top * expert)
    if c["kind"] in ("logprobs", "update"):
        lens = _train_lens(c)
        tokens, heads = sum(p + r for p, r in lens), sum(r for _, r in lens)
        flops = tokens * per_token + 2 * head * heads + L * pair * sum(_pairs(p + r) for p, r in lens)
        if c["kind"] == "logprobs":
            return dict(bytes=weights(tokens) + 2 * tokens * width + 4 * heads, flops=flops)
        params = L * base + 2 * head
        # weights read and written, gradients written and read, three fp32 states read and written
        return dict(bytes=params * (2 + 2 + 4 + 4 + 24) + 2 * tokens * width, flops=3 * flops)
    prompts = _prompt_lens(c)
    if c["kind"] == "prompt":
        t = sum(prompts)
        return dict(bytes=weights(t) + t * L * cached + 2 * vocab * len(prompts), flops=t * per_token + 2 * head * len(prompts) + L * pair * sum(_pairs(p) for p in prompts))
    new = _new_lens(c)
    first = prompts[::c["group"]]
    flops = sum(first) * per_token + 2 * head * len(first) + L * pair * sum(_pairs(p) for p in first)
    nbytes = weights(sum(first)) + sum(first) * L * cached
    for step in range(1, max(new)):
        live = [i for i in range(c["rows"]) if new[i] > step]
        seen = sum(prompts[i] + step for i in live)
        shared = sum(prompts[i] // 64 * 64 for i in live) if c["group"] > 1 else 0
        own = seen - shared + (sum(prompts[i] // 64 * 64 for i in {j // c["group"] * c["group"] for j in live}) if shared else 0)
        nbytes += weights(len(live)) + L * cached * own
        flops += len(live) * (per_token + 2 * head) + L * pair * seen
    return dict(bytes=nbytes, flops=flops)


def tolerance(case):
    c = case
    if c["dtype"] == "float32":
        return {"rel": 1e-5, "max": 1e-4, "differ": 0.0}
    if c["kind"] == "update":
        return {"rel": 0.03, "max": 0.9}
    if c["kind"] == "logprobs":
        return {"rel": 0.004, "max": 0.05}
    return {"rel": 0.03, "max": 0.5, "differ": 0.0}


# ---------------------------------------------------------------------------------------------------- the same in 64 bits, plain torch
def _rms(x, eps):
    return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + eps)


def _causal(q, k, v, scale, sink=None):
    """``q [n, H, d]``, ``k [n, G, d]``, ``v [n, G, e]`` -> ``[n, H, e]``, a block of queries at a time."""
    n, heads, _ = q.shape
    rep = heads // k.shape[1]
    k, v = k.repeat_interleave(rep, 1).transpose(0, 1), v.repeat_interleave(rep, 1).transpose(0, 1)
    out = []
    for s in range(0, n, 1024):
        e = min(n, s + 1024)
        w = (q[s:e].transpose(0, 1) @ k[:, :e].transpose(1, 2)) * scale
        w = w.masked_fill(torch.arange(e, device=q.device)[None, None, :] > torch.arange(s, e, device=q.device)[None, :, None], -math.inf)
        if sink is not None:
            w = torch.cat([w, sink[:, None, None].expand(heads, e - s, 1)], 2)
        out.append((torch.softmax(w, 2)[:, :, :e] @ v[:, :e]).transpose(0, 1))
    return torch.cat(out)


def _half_rotate(x, base):
    """Rotation of the pairs (i, i + d / 2) of every head, ``x [n, H, d]``."""
    n, d = x.shape[0], x.shape[2]
    a = torch.arange(n, dtype=F64, device=x.device)[:, None] * base ** (-torch.arange(0, d, 2, dtype=F64, device=x.device) / d)
    cos, sin = a.cos()[:, None], a.sin()[:, None]
    lo, hi = x[..., : d // 2], x[..., d // 2:]
    return torch.cat([lo * cos - hi * sin, hi * cos + lo * sin], -1)


def _pair_rotate(x, base, dims):
    """Rotation of the pairs (2 i, 2 i + 1) of the first ``dims`` entries of every head."""
    n = x.shape[0]
    a = torch.arange(n, dtype=F64, device=x.device)[:, None] * base ** (-torch.arange(0, dims, 2, dtype=F64, device=x.device) / dims)
    cos, sin = a.cos()[:, None], a.sin()[:, None]
    u, v = x[..., 0:dims:2], x[..., 1:dims:2]
    return torch.cat([torch.stack([u * cos - v * sin, v * cos + u * sin], -1).flatten(-2), x[..., dims:]], -1)


def _llama_hidden(cfg, p, tokens):
    x, hd, n = p["embed"][tokens.long()], cfg.head_dim, tokens.numel()
    for i in range(cfg.n_layers):
        h = _rms(x, cfg.rms_eps) * p[f"l{i}.attn_norm"]
        q, k, v = (h @ p[f"l{i}.wqkv"].T).view(n, -1, hd).split([cfg.n_heads, cfg.n_kv_heads, cfg.n_kv_heads], 1)
        if cfg.qk_norm:
            q, k = _rms(q, cfg.rms_eps) * p[f"l{i}.q_norm"], _rms(k, cfg.rms_eps) * p[f"l{i}.k_norm"]
        o = _causal(_half_rotate(q, cfg.rope_theta), _half_rotate(k, cfg.rope_theta), v, hd ** -0.5)
        x = x + o.reshape(n, -1) @ p[f"l{i}.wo"].T
        gate, up = ((_rms(x, cfg.rms_eps) * p[f"l{i}.mlp_norm"]) @ p[f"l{i}.w_gate_up"].T).chunk(2, 1)
        x = x + (torch.nn.functional.silu(gate) * up) @ p[f"l{i}.w_down"].T
    return _rms(x, cfg.rms_eps) * p["final_norm"]


def _expert_sum(h, chosen, scale, one):
    """Sum over the chosen experts of ``one(expert, rows of h, their factors)``."""
    out = torch.zeros_like(h)
    for e in chosen.unique().tolist():
        row, col = (chosen == e).nonzero(as_tuple=True)
        out.index_add_(0, row, one(e, h[row], scale[row, col][:, None]))
    return out


def _dulisun_hidden(cfg, m, tokens):
    p, eps, n = m.p, cfg.norm_eps, tokens.numel()

    def w(name):
        return p[name].to(F64)

    def norm(x, name):
        return _rms(x, eps) * (1 + w(name))

    x = norm(p["embed"][tokens.long()].to(F64), "embed_norm")
    for i, layer in enumerate(cfg.layers):
        a, e = layer.mixer, layer.mlp
        q, k = (x @ w(f"l{i}.wqk").T).view(n, -1, a.dim).split([a.heads, a.kv_heads], 1)
        v = k
        q, k = (_rms(_pair_rotate(t, a.rot_base, a.rot_dims), eps) for t in (q, k))
        x = x + norm(_causal(q, k, v, a.scale, m.sink[i].to(F64)).reshape(n, -1) @ w(f"l{i}.wo").T, f"l{i}.norm1")
        s = torch.softmax((x @ w(f"l{i}.router").T)[:, : e.experts], -1)
        best = s.view(n, e.groups, -1).amax(2).topk(e.keep, 1).indices
        allowed = torch.zeros((n, e.groups), dtype=torch.bool, device=s.device).scatter_(1, best, True).repeat_interleave(e.experts // e.groups, 1)
        chosen = s.masked_fill(~allowed, -1).topk(e.top, 1).indices

        def expert(j, rows, factor):
            return factor * (torch.nn.functional.gelu(rows @ p[f"l{i}.w_up"][j].to(F64).T) @ p[f"l{i}.w_down"][j].to(F64).T)

        out = _expert_sum(x, chosen, s.gather(1, chosen), expert)
        for j in range(e.experts, e.segments):
            out += expert(j, x, 1.0)
        x = x + norm(out, f"l{i}.norm2")
    return norm(x, "final_norm")


def _zafopel_hidden(cfg, m, tokens):
    p, eps, n = m.p, cfg.norm_eps, tokens.numel()

    def w(name):
        return p[name].to(F64)

    def norm(x, i, name):
        return torch.tanh(m.alpha[i].to(F64) * x) * w(name) + w(name + ".b")

    x, latents = p["embed"][tokens.long()].to(F64), {}
    for i, layer in enumerate(cfg.layers):
        a, e = layer.mixer, layer.mlp
        h = norm(x, i, f"l{i}.norm1")
        proj = h @ w(f"l{i}.w_in").T
        if a.kv_from is None:
            c, r = proj[:, a.q_in:a.q_in + a.kv_in].split([a.kv_rank, a.rot_dim], 1)
            latents[i] = _rms(c, eps) * w(f"l{i}.kv_norm"), _pair_rotate(r[:, None], a.rot_base, a.rot_dim)
        c, r = latents[i if a.kv_from is None else a.kv_from]
        q = proj[:, : a.q_in]
        if a.q_rank:
            q = (_rms(q, eps) * w(f"l{i}.q_norm")) @ w(f"l{i}.w_uq").T
        q0, q1 = q.view(n, a.heads, -1).split([a.dim, a.rot_dim], 2)
        uk, uv = w(f"l{i}.w_ukv").split([a.heads * a.dim, a.heads * a.vdim])
        k = torch.cat([(c @ uk.T).view(n, a.heads, -1), r.expand(n, a.heads, a.rot_dim)], 2)
        o = _causal(torch.cat([q0, _pair_rotate(q1, a.rot_base, a.rot_dim)], 2), k, (c @ uv.T).view(n, a.heads, -1), a.scale,
                    None if m.sink[i] is None else m.sink[i].to(F64))
        s = torch.sigmoid(proj[:, a.q_in + a.kv_in:][:, : e.experts])
        chosen = s.topk(e.top, 1).indices

        def expert(j, rows, factor):
            gate, up = ((factor * rows) @ p[f"l{i}.w_gate_up"][j].to(F64).T).chunk(2, 1)
            return (torch.nn.functional.silu(gate) * up) @ p[f"l{i}.w_down"][j].to(F64).T

        x = x + o.reshape(n, -1) @ w(f"l{i}.wo").T + _expert_sum(h, chosen, s.gather(1, chosen), expert)
    return norm(x, cfg.n_layers, "final_norm")


def _exact_update(c, model, d):
    """Loss, gradients and the state after one step of AdamW, in the flat order of the parameters."""
    cfg, layout = model.cfg, model.layout
    w = model.w.to(F64).requires_grad_()
    lens, t_max = _train_lens(c), d["resp_ids"].shape[1]
    denom, loss, kl = sum(r for _, r in lens), 0.0, 0.0
    for i, (pl, rl) in enumerate(lens):
        p = {name: layout.view(w, name) for name in layout.entries}
        tokens = torch.cat([d["prompt_ids"][i, :pl], d["resp_ids"][i, :rl]])
        x = _llama_hidden(cfg, p, tokens)[pl - 1:pl - 1 + rl]
        lp = torch.log_softmax(x @ p["lm_head"].T, -1).gather(1, d["resp_ids"][i, :rl].long()[:, None])[:, 0]
        old, ref, adv = (d[k][i, :rl].to(F64) for k in ("old_logp", "ref_logp", "adv"))
        ratio = torch.exp(lp - old)
        part = (0.04 * (lp - ref) - torch.minimum(ratio * adv, ratio.clamp(0.8, 1.2) * adv)).sum() / denom
        part.backward()
        loss, kl = loss + part.item(), kl + (lp - ref).sum().item()
    g = w.grad
    with torch.no_grad():
        w = w.detach()
        gc = g * min(1.0, 1.0 / (g.norm().item() + 1e-6))
        m, v = 0.1 * gc, 0.001 * gc * gc
        after = w - 1e-6 * gc / (gc.abs() + 1e-8)
    return dict(loss=loss, kl=kl, grads=g, weights=after, master=after, m=m, v=v)


def exact(case, seed):
    c = case
    model, nxt = _model(c, seed)
    cfg = model.cfg
    with torch.set_grad_enabled(c["kind"] == "update"):
        if c["kind"] == "update":
            model.g = None
            model.gp = {}
            return _exact_update(c, model, _rollout(c, cfg.vocab, seed))
        if _is_llama(c):
            p = {name: t.to(F64) for name, t in model.p.items()}
            head = p["lm_head"]
            hidden = lambda tokens: _llama_hidden(cfg, p, tokens)  # noqa: E731
        else:
            head = (model.p["embed"] if cfg.family == "dulisun" else model.p["head"]).to(F64)
            hidden = lambda tokens: (_dulisun_hidden if cfg.family == "dulisun" else _zafopel_hidden)(cfg, model, tokens)  # noqa: E731
        if c["kind"] == "logprobs":
            d = _rollout(c, cfg.vocab, seed)
            out = torch.zeros(d["mask"].shape, dtype=F64, device=DEVICE)
            for i, (pl, rl) in enumerate(_train_lens(c)):
                tokens = torch.cat([d["prompt_ids"][i, :pl], d["resp_ids"][i, :rl]])
                logits = hidden(tokens)[pl - 1:pl - 1 + rl] @ head.T
                out[i, :rl] = torch.log_softmax(logits, -1).gather(1, d["resp_ids"][i, :rl].long()[:, None])[:, 0]
            return dict(logprobs=out)
        prompts = _prompts(c, cfg.vocab, seed)
        if c["kind"] == "prompt":
            return [hidden(p_)[-1:] @ head.T for p_ in prompts]
        new = _new_lens(c)
        tokens = torch.zeros((c["rows"], c["new"]), dtype=torch.int32, device=DEVICE)
        logp = torch.zeros((c["rows"], c["new"]), dtype=F64, device=DEVICE)
        for i in range(0, c["rows"], c["group"]):
            chain = [prompts[i][-1].long()]
            for _ in range(c["new"]):
                chain.append(nxt[chain[-1]])
            full = torch.cat([prompts[i], torch.stack(chain[1:]).int()])
            n = prompts[i].numel()
            lp = torch.log_softmax(hidden(full[:-1])[n - 1:] @ head.T, -1)
            for r in range(i, i + c["group"]):
                tok = lp.argmax(-1)
                if new[r] < c["new"]:
                    tok[new[r] - 1] = EOS
                tokens[r, : new[r]] = tok[: new[r]].int()
                logp[r, : new[r]] = lp.gather(1, tok[:, None])[: new[r], 0]
        return dict(tokens=tokens, logprobs=logp, lengths=torch.tensor(new, dtype=torch.int32, device=DEVICE))
