"""What the framework is timed on: steps of the served models, training-side operators, and the operator suite.

Sizes are those of the model shapes, tests and benchmark of this repository, and ragged ones around them.  Models run with
the number of layers one pipeline stage holds, with embedding and head.  Inputs come from the seed alone."""
from __future__ import annotations

import dataclasses
import math
import random
from types import SimpleNamespace as NS

import torch

import vexact_b200 as vb
from vexact_b200 import inferencer as inf

BF = torch.bfloat16
PAGE = 16                      # tokens of a KV page
HYBRID_PAGE = 64
# layers of one stage: four stages of the dense models, eight of the others, rounded up
STAGE_LAYERS = {"qwen3-1.7b-shape": 7, "qwen2-1.5b-shape": 7, "qwen3-30b-a3b-shape": 6, "moonlight-16b-a3b-shape": 3}
# (query heads, KV heads, key dim, value dim) of the packed attention calls
HEADS = {"qwen3-30b-a3b-shape": (32, 4, 128, 128), "qwen3-1.7b-shape": (16, 8, 128, 128),
         "qwen2-1.5b-shape": (12, 2, 128, 128), "moonlight-16b-a3b-shape": (16, 16, 192, 128)}
HYBRID = dict(width=2048, vocab=32768, streams=4, mult=0.3, eps=1e-5, ff=8192, heads=64, p=64, state=128, groups=8, taps=4,
              lat_heads=16, dim=128, rot=64, vdim=128, rank=512, base=50000.0, kinds=("ssm", "ssm", "latent", "ssm"))
PROJ_N, PROJ_K, VOCAB = 6144, 2048, 151936     # the operator suite's projection and vocabulary


def listed():
    return [
        # the operator suite at a handful of tokens: eager calls, where launches and host work count
        dict(name="operator suite 7 rows", kind="suite", rows=7),
        # one user: a decode step of a small dense model from its captured graph
        dict(name="decode dense 1 sequence", kind="decode", model="qwen3-1.7b-shape", sequences=1, context=333, ragged=False),
        # a rollout batch of a small dense model whose sequences are at different lengths
        dict(name="decode dense ragged", kind="decode", model="qwen2-1.5b-shape", sequences=250, context=8192, ragged=True),
        # the headline workload: a rollout batch of the mixture-of-experts model, one of eight pipeline stages
        dict(name="decode moe 512 x 2048", kind="decode", model="qwen3-30b-a3b-shape", sequences=512, context=2048, ragged=False),
        # a rollout batch of the latent-attention model
        dict(name="decode mla 64 x 4096", kind="decode", model="moonlight-16b-a3b-shape", sequences=64, context=4096, ragged=False),
        # one chunk of a long prompt
        dict(name="prefill dense chunk", kind="prefill", model="qwen2-1.5b-shape", prompts=1, tokens=2048, past=2048),
        # fresh prompts packed under the scheduler's token budget
        dict(name="prefill moe 3 prompts", kind="prefill", model="qwen3-30b-a3b-shape", prompts=3, tokens=2048, past=0),
        dict(name="prefill mla 4 prompts", kind="prefill", model="moonlight-16b-a3b-shape", prompts=4, tokens=3001, past=0),
        # a hybrid decoder (state space and latent attention) on fresh prompts
        dict(name="prefill hybrid 3 prompts", kind="hybrid", prompts=3, tokens=4096, decode=False),
        # the trainer's side of a rollout: attention over packed sequences, forward and backward
        dict(name="train attention 4 x 2048", kind="train_attention", model="qwen3-30b-a3b-shape", sequences=4, tokens=8192),
        # one mixture-of-experts layer, forward and backward
        dict(name="train experts 4096 tokens", kind="train_experts", model="qwen3-30b-a3b-shape", tokens=4096, stacked=False),
        # per-token log-probabilities of the trainer's logits, forward and backward
        dict(name="train logprob 2000 rows", kind="train_logprob", rows=2000, vocab=151936, dtype="bf16"),
    ]


def draw(rng: random.Random):
    def log(lo, hi):
        return max(lo, min(hi, round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))

    kind = rng.choice(["suite", "decode", "decode", "decode", "prefill", "prefill", "hybrid", "train_attention",
                       "train_experts", "train_logprob"])
    if kind == "suite":
        return dict(kind=kind, rows=log(1, 256))
    if kind == "decode":
        model = rng.choice(sorted(STAGE_LAYERS))
        sequences = log(1, 64 if "moonlight" in model else 512)
        most = {"moonlight-16b-a3b-shape": 4096 * 64, "qwen3-1.7b-shape": 2048 * 64}.get(model, 2048 * 512)
        context = log(64, min(8192, most // sequences))
        return dict(kind=kind, model=model, sequences=sequences, context=context, ragged=rng.random() < 0.5)
    if kind == "prefill":
        tokens = log(17, 3001)
        return dict(kind=kind, model=rng.choice(sorted(STAGE_LAYERS)), prompts=rng.randint(1, min(4, tokens)), tokens=tokens,
                    past=rng.choice([0, log(16, 2048)]))
    if kind == "hybrid":
        decode = rng.random() < 0.4
        tokens = log(1, 256) if decode else log(40, 4096)
        return dict(kind=kind, prompts=tokens if decode else rng.randint(1, 4), tokens=tokens, decode=decode)
    if kind == "train_attention":
        tokens = log(64, 8192)
        return dict(kind=kind, model=rng.choice(sorted(HEADS)), sequences=rng.randint(1, min(8, tokens)), tokens=tokens)
    if kind == "train_experts":
        return dict(kind=kind, model=rng.choice(["qwen3-30b-a3b-shape", "moonlight-16b-a3b-shape"]), tokens=log(16, 4096),
                    stacked=rng.random() < 0.5)
    return dict(kind=kind, rows=log(1, 2000), vocab=rng.choice([151936, 163840, 32768]), dtype=rng.choice(["bf16", "fp32"]))


# ------------------------------------------------------------------ shapes and lengths
def shape_of(case):
    return dataclasses.replace(inf.PRESETS[case["model"]], num_layers=STAGE_LAYERS[case["model"]])


def parts(total: int, n: int) -> list:
    """`total` tokens over n sequences, unequal, each at least one; the same every time."""
    r = random.Random(total * 131 + n)
    w = [r.uniform(0.4, 1.6) for _ in range(n)]
    lens = [max(1, int(total * x / sum(w))) for x in w]
    while sum(lens) > total:
        lens[lens.index(max(lens))] -= 1
    lens[-1] += total - sum(lens)
    return lens


def lengths(case) -> list:
    """(new, total) tokens of every sequence of a model step."""
    if case["kind"] == "decode":
        S, ctx = case["sequences"], case["context"]
        if not case["ragged"]:
            return [(1, ctx)] * S
        r = random.Random(ctx * 131 + S)
        return [(1, r.randint(max(1, ctx // 32), ctx)) for _ in range(S)]
    if case["kind"] == "hybrid":
        return [(1, 1024)] * case["tokens"] if case["decode"] else [(n, n) for n in parts(case["tokens"], case["prompts"])]
    return [(n, n + case["past"]) for n in parts(case["tokens"], case["prompts"])]


def generator(seed: int) -> torch.Generator:
    return torch.Generator(device="cuda").manual_seed(1000 + seed)


def normal(gen, shape, std=1.0, dtype=BF):
    return torch.empty(shape, device="cuda", dtype=dtype).normal_(0.0, std, generator=gen)


def step_tensors(lens, page: int, vocab: int, gen):
    """Token ids and paged-cache metadata of a packed step; pages are dealt in random order."""
    pages = [(t + page - 1) // page for _, t in lens]
    order = torch.randperm(sum(pages), device="cuda", generator=gen).to(torch.int32)
    table = torch.zeros((len(lens), max(pages)), dtype=torch.int32, device="cuda")
    col = torch.arange(max(pages), device="cuda")
    table[col[None, :] < torch.tensor(pages, device="cuda")[:, None]] = order
    new = torch.tensor([n for n, _ in lens], device="cuda")
    total = torch.tensor([t for _, t in lens], device="cuda")
    T = sum(n for n, _ in lens)
    cu = torch.zeros(len(lens) + 1, dtype=torch.int32, device="cuda")
    cu[1:] = new.cumsum(0)
    seq = torch.repeat_interleave(torch.arange(len(lens), device="cuda"), new)
    pos = torch.arange(T, device="cuda") - cu[seq].long() + (total - new)[seq]
    slots = (table[seq, pos // page].long() * page + pos % page).to(torch.int32)
    ids = torch.randint(0, vocab, (T,), device="cuda", generator=gen)
    return NS(ids=ids, positions=pos, slots=slots, cu=cu, lens=total.to(torch.int32), table=table, blocks=sum(pages),
              max_q=max(n for n, _ in lens))


# ------------------------------------------------------------------ the served models
def stage_tensors(case, seed):
    s, gen = shape_of(case), generator(seed)
    H, D, hq, hkv = s.hidden, s.head_dim, s.num_q_heads, s.num_kv_heads

    def norm(n):
        return (1 + normal(gen, (n,), 0.02, torch.float32)).to(BF)

    def linear(*dims):
        return normal(gen, dims, 0.02)

    layers = []
    for i in range(s.num_layers):
        w = dict(input_norm=norm(H), post_norm=norm(H), qkv_bias=None, q_norm=None, k_norm=None)
        if s.mla:
            a = s.mla
            w.update(qkv=linear(hq * (a.qk_nope + a.qk_rope), H), o=linear(H, hq * a.v_head), kv_a_norm=norm(a.kv_lora_rank),
                     kv_a=linear(a.kv_lora_rank + a.qk_rope, H), kv_b=linear(hq * (a.qk_nope + a.v_head), a.kv_lora_rank))
        else:
            w.update(qkv=linear(s.qkv_out, H), o=linear(H, hq * D))
            if s.qkv_bias:
                w.update(qkv_bias=linear(s.qkv_out))
            if s.qk_norm:
                w.update(q_norm=norm(D), k_norm=norm(D))
        if s.layer_is_moe(i):
            m = s.moe
            w.update(router=linear(m.num_experts, H), experts_gate_up=linear(m.num_experts, 2 * m.intermediate, H),
                     experts_down=linear(m.num_experts, H, m.intermediate))
            if m.scoring == "sigmoid_group":
                w.update(router_bias=normal(gen, (m.num_experts,), 0.02, torch.float32))
            if m.n_shared_experts:
                n = m.intermediate * m.n_shared_experts
                w.update(shared_gate_up=linear(2 * n, H), shared_down=linear(H, n))
        else:
            w.update(gate_up=linear(2 * s.ffn, H), down=linear(H, s.ffn))
        layers.append(w)
    # rows of norm 1 per column: as in a trained model, the residual outweighs what a layer adds to it
    top = dict(embed=normal(gen, (s.vocab, H)), final_norm=norm(H), lm_head=linear(s.vocab, H))
    step = step_tensors(lengths(case), PAGE, s.vocab, gen)
    kc = [normal(gen, (step.blocks, PAGE, hkv, s.k_dim)) for _ in range(s.num_layers)]
    vc = [normal(gen, (step.blocks, PAGE, hkv, s.v_dim)) for _ in range(s.num_layers)]
    rd = s.mla.qk_rope if s.mla else D
    inv_freq = 1.0 / (s.rope_theta ** (torch.arange(0, rd, 2, device="cuda").float() / rd))
    return s, layers, top, step, kc, vc, inv_freq


def prepare_stage(case, seed):
    s, layers, top, st, kc, vc, inv_freq = stage_tensors(case, seed)
    weights = inf.StageWeights(s, 0, s.num_layers, [inf.LayerWeights(**w) for w in layers], inv_freq=inv_freq, **top)
    runner = inf.StageRunner(weights, dict(enumerate(kc)), dict(enumerate(vc)))
    step = inf.StepInputs(st.ids, None, st.positions, st.slots, st.cu, st.lens, st.table, st.max_q)
    runner.prepare(st.ids.numel())
    state = NS(case=case, runner=runner, step=step, caches=[kc, vc], graph=None)
    if case["kind"] == "decode":
        state.graph, state.out = runner.capture(step)
    return state


def run_stage(state):
    if state.graph is not None:      # decode steps are replayed, steps with prompt tokens run eagerly
        state.graph.replay()
        out = state.out
    else:
        out = state.runner.step(state.step)
    return dict(tokens=out[0], logprobs=out[1], logits=out[2], keys=state.caches[0], values=state.caches[1])


def d(t):
    return t.double()


def rms(x, w, eps):
    return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + eps) * d(w)


def turn_halves(x, pos, inv_freq):
    a = (pos.double()[:, None] * d(inv_freq))[:, None, :]
    u, v = x.chunk(2, -1)
    return torch.cat([u * a.cos() - v * a.sin(), v * a.cos() + u * a.sin()], -1)


def swiglu(x, gate_up, down):
    g, u = (x @ d(gate_up).T).chunk(2, -1)
    return (torch.nn.functional.silu(g) * u) @ d(down).T


def exact_mixture(x, w, m):
    logits = x @ d(w["router"]).T
    if m.scoring == "softmax":
        p, sel = torch.softmax(logits, -1).topk(m.top_k, -1)
        p = p / p.sum(-1, keepdim=True)
    else:
        score = torch.sigmoid(logits)
        sel = (score + d(w["router_bias"])).topk(m.top_k, -1).indices
        p = score.gather(1, sel)
        p = p / p.sum(-1, keepdim=True) * m.routed_scaling_factor
    out = torch.zeros_like(x)
    for e in range(m.num_experts):
        tok, k = (sel == e).nonzero(as_tuple=True)
        if tok.numel():
            out.index_add_(0, tok, swiglu(x[tok], w["experts_gate_up"][e], w["experts_down"][e]) * p[tok, k, None])
    if "shared_gate_up" in w:
        out += swiglu(x, w["shared_gate_up"], w["shared_down"])
    return out


def exact_attention(q, kc, vc, table, lens, scale):
    """Causal attention of every sequence's new tokens over its pages; q [T, heads, d] and pages in 64 bits or less."""
    out = q.new_empty(q.shape[:2] + (vc.shape[-1],))
    hkv, group = kc.shape[2], q.shape[1] // kc.shape[2]
    at, i = 0, 0
    while i < len(lens):
        n, total = lens[i]
        j = i + 1
        if n == 1:                       # decode: several sequences at once
            while j < len(lens) and j - i < 32:
                j += 1
            total = max(t for _, t in lens[i:j])
        rows = table[i:j, :(total + kc.shape[1] - 1) // kc.shape[1]].long()
        k = d(kc[rows].flatten(1, 2)[:, :total]).permute(0, 2, 3, 1)
        v = d(vc[rows].flatten(1, 2)[:, :total]).permute(0, 2, 1, 3)
        B = j - i
        qs = q[at:at + B * n].view(B, n, hkv, group, -1).permute(0, 2, 3, 1, 4)
        sees = torch.tensor([t for _, t in lens[i:j]], device="cuda")[:, None] - n + torch.arange(n, device="cuda")
        hide = torch.arange(total, device="cuda") > sees[..., None]
        for h in range(hkv):
            sc = (qs[:, h].reshape(B, group * n, -1) @ k[:, h] * scale).view(B, group, n, total)
            p = torch.softmax(sc.masked_fill_(hide[:, None], -math.inf), -1).view(B, group * n, total)
            o = (p @ v[:, h]).view(B, group, n, -1).permute(0, 2, 1, 3)
            out[at:at + B * n, h * group:(h + 1) * group] = o.reshape(B * n, group, -1)
        at, i = at + B * n, j
    return out


def exact_stage(case, seed):
    s, layers, top, st, kc, vc, inv_freq = stage_tensors(case, seed)
    lens, T, hq, hkv = lengths(case), st.ids.numel(), s.num_q_heads, s.num_kv_heads
    h = d(top["embed"][st.ids])
    slots = st.slots.long()
    keys, values = [], []
    for i, w in enumerate(layers):
        x = rms(h, w["input_norm"], s.rms_eps)
        q = x @ d(w["qkv"]).T
        if s.mla:
            a = s.mla
            q = q.view(T, hq, -1)

            def pairs(t):      # the pairs (2i, 2i + 1), laid out as halves, turned
                return turn_halves(torch.cat([t[..., 0::2], t[..., 1::2]], -1), st.positions, inv_freq)

            q = torch.cat([q[..., :a.qk_nope], pairs(q[..., a.qk_nope:])], -1)
            lat, rot = (x @ d(w["kv_a"]).T).split([a.kv_lora_rank, a.qk_rope], -1)
            kvb = (rms(lat, w["kv_a_norm"], s.rms_eps) @ d(w["kv_b"]).T).view(T, hq, -1)
            k = torch.cat([kvb[..., :a.qk_nope], pairs(rot[:, None]).expand(T, hq, a.qk_rope)], -1)
            v = kvb[..., a.qk_nope:]
        else:
            if w["qkv_bias"] is not None:
                q = q + d(w["qkv_bias"])
            q, k, v = q.view(T, -1, s.head_dim).split([hq, hkv, hkv], 1)
            if s.qk_norm:
                q, k = rms(q, w["q_norm"], s.rms_eps), rms(k, w["k_norm"], s.rms_eps)
            q, k = turn_halves(q, st.positions, inv_freq), turn_halves(k, st.positions, inv_freq)
        # what is cached before the step is bf16; the step's own rows stand in 64 bits
        kd, vd = d(kc[i]), d(vc[i])
        kd.flatten(0, 1)[slots], vd.flatten(0, 1)[slots] = k, v
        att = exact_attention(q, kd, vd, st.table, lens, s.k_dim ** -0.5)
        keys.append(kd)
        values.append(vd)
        h = h + att.reshape(T, -1) @ d(w["o"]).T
        x = rms(h, w["post_norm"], s.rms_eps)
        h = h + (exact_mixture(x, w, s.moe) if "router" in w else swiglu(x, w["gate_up"], w["down"]))
    logits = rms(h[st.cu[1:].long() - 1], top["final_norm"], s.rms_eps) @ d(top["lm_head"]).T
    tokens = logits.argmax(-1)
    logprobs = torch.log_softmax(logits, -1).gather(1, tokens[:, None])[:, 0]
    return dict(tokens=tokens, logprobs=logprobs, logits=logits, keys=keys, values=values)


def work_stage(case):
    s, lens = shape_of(case), lengths(case)
    T = sum(n for n, _ in lens)
    keys = sum(n * t - n * (n - 1) // 2 for n, t in lens)
    params, macs = 0, 0.0
    for i in range(s.num_layers):
        o = s.hidden * s.num_q_heads * s.v_dim
        if s.mla:
            a = s.mla
            o += s.hidden * (s.num_q_heads * s.k_dim + a.kv_lora_rank + a.qk_rope)
            o += s.num_q_heads * (a.qk_nope + a.v_head) * a.kv_lora_rank
        else:
            o += s.hidden * s.qkv_out
        dense = s.ffn
        if s.layer_is_moe(i):
            m = s.moe
            expert = 3 * m.intermediate * s.hidden
            params += round(m.num_experts * (1 - (1 - m.top_k / m.num_experts) ** T)) * expert
            macs += T * m.top_k * expert
            o += m.num_experts * s.hidden
            dense = m.intermediate * m.n_shared_experts
        o += 3 * dense * s.hidden
        params += o
        macs += T * o + keys * s.num_q_heads * (s.k_dim + s.v_dim)
    params += s.vocab * s.hidden
    macs += len(lens) * s.vocab * s.hidden
    cache = s.num_layers * s.num_kv_heads * (s.k_dim + s.v_dim) * sum(t for _, t in lens)
    return dict(bytes=2 * (params + cache + T * s.hidden + len(lens) * s.vocab), flops=2 * macs)


# ------------------------------------------------------------------ a hybrid decoder
def hybrid_shape():
    from vexact_b200.hybrid import DenseSpec, HybridLayer, HybridShape, LatentSpec, SSMSpec

    c = NS(**HYBRID)
    spec = dict(ssm=SSMSpec(c.heads, c.p, c.state, c.groups, c.taps, c.groups),
                latent=LatentSpec(c.lat_heads, c.dim, c.rot, c.vdim, c.rank, (c.dim + c.rot) ** -0.5, c.base, c.rot))
    layers = tuple(HybridLayer(spec[k], DenseSpec(c.ff), i) for i, k in enumerate(c.kinds))
    return HybridShape("hybrid", layers, c.width, c.vocab, c.streams, c.mult, c.eps)


def hybrid_tensors(case, seed):
    """Checkpoint tensors, the packed step, and what the caches hold before it."""
    c, gen, w = NS(**HYBRID), generator(seed), {}
    W, inner = c.width, c.heads * c.p
    channels = inner + 2 * c.groups * c.state

    def linear(name, out, width):
        w[name] = normal(gen, (out, width), width ** -0.5)

    def vector(name, n, mean, std):
        w[name] = (mean + normal(gen, (n,), std, torch.float32)).to(BF)

    for i, kind in enumerate(c.kinds):
        p = f"l{i}."
        if kind == "ssm":
            linear(p + "mix.in", inner + channels + c.heads, W)
            w[p + "mix.conv"] = normal(gen, (channels, c.taps), c.taps ** -0.5)
            vector(p + "mix.conv.b", channels, 0, 0.1)
            vector(p + "mix.dt_bias", c.heads, -2, 1)
            vector(p + "mix.A_log", c.heads, 0, 0.5)
            vector(p + "mix.D", c.heads, 0, 1)
            vector(p + "mix.norm", inner, 1, 0.1)
            linear(p + "mix.o", W, inner)
        else:
            linear(p + "mix.q", c.lat_heads * (c.dim + c.rot), W)
            linear(p + "mix.dkv", c.rank + c.rot, W)
            vector(p + "mix.dkv.norm", c.rank, 1, 0.1)
            linear(p + "mix.uk", c.lat_heads * c.dim, c.rank)
            linear(p + "mix.uv", c.lat_heads * c.vdim, c.rank)
            linear(p + "mix.g", c.lat_heads * c.vdim, W)
            linear(p + "mix.o", W, c.lat_heads * c.vdim)
        linear(p + "mlp.up", c.ff, W)
        vector(p + "mlp.up.b", c.ff, 0, 0.1)
        linear(p + "mlp.down", W, c.ff)
        vector(p + "mlp.down.b", W, 0, 0.1)
        for q in (1, 2):
            vector(p + f"norm{q}", W, 0, 0.1)
            vector(p + f"hc{q}.in", c.streams, 1 / c.streams, 0.2)
            vector(p + f"hc{q}.out", c.streams, 1 / c.streams, 0.2)
            mix = 0.8 * torch.eye(c.streams, device="cuda") + 0.2 / c.streams
            w[p + f"hc{q}.mix"] = (mix + normal(gen, (c.streams, c.streams), 0.05, torch.float32)).to(BF)
    w["embed"] = normal(gen, (c.vocab, W))
    vector("final.norm", W, 0, 0.1)
    linear("head", c.vocab, W)
    step = step_tensors(lengths(case), HYBRID_PAGE, c.vocab, gen)
    S = len(lengths(case))
    before = {}
    for i, kind in enumerate(c.kinds):
        if kind == "ssm":
            before[i] = (normal(gen, (S, c.taps - 1, channels)), normal(gen, (S, c.heads, c.state, c.p), 1, torch.float32))
        else:
            before[i] = (normal(gen, (step.blocks, HYBRID_PAGE, c.rank + c.rot)),)
    return w, step, before


def prepare_hybrid(case, seed):
    from vexact_b200.config import CacheConfig
    from vexact_b200.hybrid import HybridModel, HybridWeights

    w, st, before = hybrid_tensors(case, seed)
    model = HybridModel(HybridWeights.from_tensors(hybrid_shape(), w, BF, "cuda"))
    S = len(lengths(case))
    store = model.make_cache_store(CacheConfig(HYBRID_PAGE, st.blocks), S, "cuda")
    for i, t in before.items():
        if len(t) == 2:
            store.conv_state[i].copy_(t[0])
            store.ssm_state[i].copy_(t[1])
        else:
            store.key_cache[i].copy_(t[0])
    state = NS(case=case, model=model, store=store, step=st, graph=None, slots=torch.arange(S, dtype=torch.int32, device="cuda"),
               lens=lengths(case))
    if case["decode"]:
        side = torch.cuda.Stream()
        with torch.cuda.stream(side):
            hybrid_step(state)
        torch.cuda.synchronize()
        state.graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(state.graph):
            state.out = hybrid_step(state)
        for i, t in before.items():      # the warm-up moved the state on
            if len(t) == 2:
                store.conv_state[i].copy_(t[0])
                store.ssm_state[i].copy_(t[1])
    return state


def hybrid_step(state):
    st = state.step
    vb.set_kv_cache_context(is_paged_attn=True, key_cache=state.store.key_cache, value_cache=state.store.value_cache,
                            block_tables=st.table, context_lens=st.lens, slot_mapping=st.slots, query_start_loc=st.cu,
                            max_seqlen_q=st.max_q, cache_store=state.store, state_slots=state.slots,
                            seq_lens=None if state.case["decode"] else list(state.lens))
    return state.model(input_ids=st.ids[None], position_ids=st.positions[None]).last_logits


def run_hybrid(state):
    if state.graph is not None:
        state.graph.replay()
        logits = state.out
    else:
        logits = hybrid_step(state)
    st = state.store
    return dict(logits=logits, latents=list(st.key_cache.values()), conv=list(st.conv_state.values()),
                state=list(st.ssm_state.values()))


def unit(x, eps):
    return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + eps)


def exact_hybrid(case, seed):
    w, st, before = hybrid_tensors(case, seed)
    c, lens, S, T = NS(**HYBRID), lengths(case), len(lengths(case)), st.ids.numel()
    inner, GN = c.heads * c.p, c.groups * c.state
    w = {k: d(v) for k, v in w.items()}
    starts = st.cu.tolist()
    latents, conv, states = [], [], []

    def ssm(x, p, i):
        z, xbc, dt = (x @ w[p + "in"].T).split([inner, inner + 2 * GN, c.heads], -1)
        old, S0 = (d(t) for t in before[i])
        if not case["decode"]:           # a sequence that starts here starts from zeros
            old, S0 = torch.zeros_like(old), torch.zeros_like(S0)
        taps, mixed = w[p + "conv"], []
        for q in range(S):
            padded = torch.cat([old[q], xbc[starts[q]:starts[q + 1]]])
            n = starts[q + 1] - starts[q]
            mixed.append(sum(padded[k:k + n] * taps[:, k] for k in range(c.taps)) + w[p + "conv.b"])
            old[q] = padded[-(c.taps - 1):]
        xs, B, C = torch.nn.functional.silu(torch.cat(mixed)).split([inner, GN, GN], -1)
        dt = torch.nn.functional.softplus(dt + w[p + "dt_bias"])
        decay = torch.exp(-torch.exp(w[p + "A_log"]) * dt)
        xs = xs.view(T, c.heads, c.p)
        B, C = (t.view(T, c.groups, c.state).repeat_interleave(c.heads // c.groups, 1) for t in (B, C))
        y = torch.empty_like(xs)
        order = sorted(range(S), key=lambda q: -lens[q][0])
        at = torch.tensor(starts, device="cuda")
        for t in range(lens[order[0]][0]):
            live = torch.tensor([q for q in order if lens[q][0] > t], device="cuda")
            r = at[live] + t
            new = decay[r][..., None, None] * S0[live] + (dt[r][..., None] * B[r])[..., None] * xs[r][:, :, None]
            S0[live] = new
            y[r] = (new * C[r][..., None]).sum(2)
        y = (y + w[p + "D"][:, None] * xs).reshape(T, inner) * torch.nn.functional.silu(z)
        conv.append(old)
        states.append(S0)
        return (unit(y.view(T, c.groups, -1), c.eps).reshape(T, inner) * w[p + "norm"]) @ w[p + "o"].T

    def latent(x, p, i):
        def pairs(t):
            f = c.base ** (-torch.arange(0, c.rot, 2, device="cuda", dtype=torch.float64) / c.rot)
            a = (st.positions.double()[:, None] * f)[:, None, :]
            u, v = t[..., 0::2], t[..., 1::2]
            return torch.stack([u * a.cos() - v * a.sin(), v * a.cos() + u * a.sin()], -1).flatten(-2)

        q = (x @ w[p + "q"].T).view(T, c.lat_heads, -1)
        q = torch.cat([q[..., :c.dim], pairs(q[..., c.dim:])], -1)
        lat, rot = (x @ w[p + "dkv"].T).split([c.rank, c.rot], -1)
        rows = d(before[i][0])
        rows.flatten(0, 1)[st.slots.long()] = torch.cat([unit(lat, c.eps) * w[p + "dkv.norm"], pairs(rot[:, None])[:, 0]], -1)
        latents.append(rows)
        up = rows.unsqueeze(2)
        # absorbed into the queries: a key is a latent row, the value its first `rank` columns
        qa = torch.einsum("thd,hdr->thr", q[..., :c.dim], w[p + "uk"].view(c.lat_heads, c.dim, c.rank))
        o = exact_attention(torch.cat([qa, q[..., c.dim:]], -1), up, up[..., :c.rank], st.table, lens, (c.dim + c.rot) ** -0.5)
        o = torch.einsum("thr,hvr->thv", o, w[p + "uv"].view(c.lat_heads, c.vdim, c.rank)).reshape(T, -1)
        return (o * torch.sigmoid(x @ w[p + "g"].T)) @ w[p + "o"].T

    streams = w["embed"][st.ids].expand(c.streams, T, c.width).clone()
    for i, kind in enumerate(c.kinds):
        for q in (1, 2):
            p = f"l{i}."
            x = torch.einsum("s,stw->tw", w[p + f"hc{q}.in"], streams)
            x = unit(x, c.eps) * (1 + w[p + f"norm{q}"])
            if q == 1:
                y = (ssm if kind == "ssm" else latent)(x, p + "mix.", i)
            else:
                y = torch.nn.functional.gelu(x @ w[p + "mlp.up"].T + w[p + "mlp.up.b"], approximate="tanh")
                y = y @ w[p + "mlp.down"].T + w[p + "mlp.down.b"]
            streams = torch.einsum("st,snw->tnw", w[p + f"hc{q}.mix"], streams) + c.mult * w[p + f"hc{q}.out"][:, None, None] * y
    last = streams.sum(0)[st.cu[1:].long() - 1]
    logits = (unit(last, c.eps) * (1 + w["final.norm"])) @ w["head"].T
    return dict(logits=logits, latents=latents, conv=conv, state=states)


def work_hybrid(case):
    c, lens = NS(**HYBRID), lengths(case)
    S, T = len(lens), sum(n for n, _ in lens)
    keys = sum(n * t - n * (n - 1) // 2 for n, t in lens)
    inner = c.heads * c.p
    channels = inner + 2 * c.groups * c.state
    params, macs, moved = c.vocab * c.width, S * c.vocab * c.width, 2 * (T * c.width + 2 * S * c.vocab)
    for kind in c.kinds:
        n = 2 * c.width * c.ff
        if kind == "ssm":
            n += c.width * (inner + channels + c.heads) + c.width * inner
            macs += T * (2 * inner * c.state + c.taps * channels)
            moved += S * (4 * inner * c.state + 2 * (c.taps - 1) * channels) * (2 if case["decode"] else 1)
        else:
            n += c.width * (c.lat_heads * (c.dim + c.rot + 2 * c.vdim) + c.rank + c.rot) + c.lat_heads * (c.dim + c.vdim) * c.rank
            macs += keys * c.lat_heads * (c.dim + c.rot + c.vdim)
            moved += 2 * (c.rank + c.rot) * sum(t for _, t in lens)
        params += n
        macs += T * n
    return dict(bytes=2 * params + moved, flops=2 * macs)


# ------------------------------------------------------------------ the trainer's operators
def prepare_train_attention(case, seed):
    gen, (hq, hkv, dk, dv), T = generator(seed), HEADS[case["model"]], case["tokens"]
    lens = parts(T, case["sequences"]) if case["tokens"] % case["sequences"] else [T // case["sequences"]] * case["sequences"]
    cu = torch.zeros(len(lens) + 1, dtype=torch.int32, device="cuda")
    cu[1:] = torch.tensor(lens, device="cuda").cumsum(0)
    q, k, v = (normal(gen, (T, h, n)).requires_grad_(True) for h, n in ((hq, dk), (hkv, dk), (hkv, dv)))
    return NS(case=case, q=q, k=k, v=v, cu=cu, lens=lens, grad=normal(gen, (T, hq, dv)))


def run_train_attention(state):
    n = max(state.lens)
    out, _ = vb.flash_attn_varlen_func(state.q, state.k, state.v, state.cu, state.cu, max_seqlen_q=n, max_seqlen_k=n, causal=True)
    return (out, *torch.autograd.grad(out, (state.q, state.k, state.v), state.grad))


def exact_train_attention(case, seed):
    s = prepare_train_attention(case, seed)
    hq, hkv = s.q.shape[1], s.k.shape[1]
    out, grads = [], [torch.empty(t.shape, dtype=torch.float64, device="cuda") for t in (s.q, s.k, s.v)]
    at = 0
    for n in s.lens:
        sl = slice(at, at + n)
        o = torch.empty((n, hq, s.v.shape[-1]), dtype=torch.float64, device="cuda")
        hide = torch.ones((n, n), dtype=torch.bool, device="cuda").triu(1)
        for h in range(hkv):
            hs = slice(h * hq // hkv, (h + 1) * hq // hkv)
            q, k, v = (d(t.detach()).requires_grad_(True) for t in (s.q[sl, hs], s.k[sl, h], s.v[sl, h]))
            sc = torch.einsum("qhd,kd->hqk", q, k) * q.shape[-1] ** -0.5
            y = torch.einsum("hqk,kd->qhd", torch.softmax(sc.masked_fill(hide, -math.inf), -1), v)
            for g, t, to in zip(torch.autograd.grad(y, (q, k, v), d(s.grad[sl, hs])), grads, (hs, h, h)):
                t[sl, to] = g
            o[:, hs] = y.detach()
        out.append(o)
        at += n
    return (torch.cat(out), *grads)


def work_train_attention(case):
    hq, hkv, dk, dv = HEADS[case["model"]]
    T, S = case["tokens"], case["sequences"]
    lens = parts(T, S) if T % S else [T // S] * S
    pairs = sum(n * (n + 1) // 2 for n in lens)
    # scores and values forward; scores again, two products each for values' and scores' gradients, backward
    return dict(bytes=2 * T * (hq * (2 * dk + 3 * dv) + 2 * hkv * (dk + dv)), flops=2 * pairs * hq * (4 * dk + 3 * dv))


def prepare_train_experts(case, seed):
    s, gen, T = inf.PRESETS[case["model"]], generator(seed), case["tokens"]
    m, H = s.moe, s.hidden
    x = normal(gen, (T, H)).requires_grad_(True)
    w1, w2 = (normal(gen, (m.num_experts, m.intermediate, H), 0.02) for _ in range(2))
    w3 = normal(gen, (m.num_experts, H, m.intermediate), 0.02).requires_grad_(True)
    w = [torch.cat([w1, w2], 1).requires_grad_(True)] if case["stacked"] else [w1.requires_grad_(True), w2.requires_grad_(True)]
    p, sel = torch.softmax(normal(gen, (T, m.num_experts), 1, torch.float32), -1).topk(m.top_k, -1)
    p = (p / p.sum(-1, keepdim=True)).to(BF).requires_grad_(True)
    return NS(case=case, experts=m.num_experts, x=x, w=w, w3=w3, p=p, sel=sel, grad=normal(gen, (T, H)))


def run_train_experts(s):
    if s.case["stacked"]:
        out = vb.fused_moe_forward(s.experts, s.p, s.sel, s.x, fc2_weight=s.w3, fc1_1_2_weight=s.w[0])
    else:
        out = vb.fused_moe_forward(s.experts, s.p, s.sel, s.x, s.w[0], s.w[1], s.w3)
    return (out, *torch.autograd.grad(out, (s.x, s.p, s.w3, *s.w), s.grad))


def exact_train_experts(case, seed):
    s = prepare_train_experts(case, seed)
    x, p, grad = d(s.x.detach()), d(s.p.detach()), d(s.grad)
    out, gx, gp = torch.zeros_like(x), torch.zeros_like(x), torch.zeros_like(p)
    gw3 = torch.zeros(s.w3.shape, dtype=torch.float64, device="cuda")
    gw = [torch.zeros(t.shape, dtype=torch.float64, device="cuda") for t in s.w]
    for e in range(s.experts):
        tok, k = (s.sel == e).nonzero(as_tuple=True)
        if not tok.numel():
            continue
        w = [d(t[e].detach()).requires_grad_(True) for t in s.w]
        xe, pe, w3 = (t.requires_grad_(True) for t in (x[tok], p[tok, k], d(s.w3[e].detach())))
        g, u = (xe @ w[0].T).chunk(2, -1) if case["stacked"] else (xe @ w[0].T, xe @ w[1].T)
        y = (torch.nn.functional.silu(g) * u * pe[:, None]) @ w3.T
        got = torch.autograd.grad(y, (xe, pe, w3, *w), grad[tok])
        out.index_add_(0, tok, y.detach())
        gx.index_add_(0, tok, got[0])
        gp[tok, k] = got[1]
        gw3[e] = got[2]
        for to, t in zip(gw, got[3:]):
            to[e] = t
    return (out, gx, gp, gw3, *gw)


def work_train_experts(case):
    s, T = inf.PRESETS[case["model"]], case["tokens"]
    m, H = s.moe, s.hidden
    weights = 3 * m.num_experts * m.intermediate * H
    hit = 1 - (1 - m.top_k / m.num_experts) ** T
    return dict(bytes=2 * (round(weights * hit) + weights + T * (4 * H + 2 * m.top_k)) + 8 * T * m.top_k,
                flops=18 * T * m.top_k * m.intermediate * H)


def prepare_train_logprob(case, seed):
    gen, n, V = generator(seed), case["rows"], case["vocab"]
    logits = normal(gen, (n, V), 2.0, BF if case["dtype"] == "bf16" else torch.float32).requires_grad_(True)
    return NS(case=case, logits=logits, labels=torch.randint(0, V, (n,), device="cuda", generator=gen),
              grad=normal(gen, (n,), 1.0, torch.float32))


def run_train_logprob(s):
    out = vb.logprobs_from_logits_flash_attn(s.logits, s.labels)
    return (out, *torch.autograd.grad(out, s.logits, s.grad))


def exact_train_logprob(case, seed):
    s = prepare_train_logprob(case, seed)
    out = torch.empty(case["rows"], dtype=torch.float64, device="cuda")
    dx = torch.empty(s.logits.shape, dtype=torch.float64, device="cuda")
    for a in range(0, case["rows"], 256):
        lp = torch.log_softmax(d(s.logits.detach()[a:a + 256]), -1)
        lab = s.labels[a:a + 256, None]
        out[a:a + 256] = lp.gather(1, lab)[:, 0]
        dx[a:a + 256] = -lp.exp_()
        dx[a:a + 256].scatter_add_(1, lab, torch.ones(lab.shape, dtype=torch.float64, device="cuda"))
    return out, dx.mul_(d(s.grad)[:, None])


def work_train_logprob(case):
    n = case["rows"] * case["vocab"]
    return dict(bytes=2 * n * (2 if case["dtype"] == "bf16" else 4) + 16 * case["rows"], flops=4 * n)


# ------------------------------------------------------------------ the operator suite
def prepare_suite(case, seed):
    gen, n = generator(seed), case["rows"]
    return NS(case=case, x=normal(gen, (n, PROJ_K)), w=normal(gen, (PROJ_N, PROJ_K), 0.02),
              norm=(1 + normal(gen, (PROJ_K,), 0.02, torch.float32)).to(BF),
              logits=normal(gen, (n, VOCAB), 4.0, torch.float32),
              labels=torch.randint(0, VOCAB, (n,), device="cuda", generator=gen))


def run_suite(s):
    return dict(matmul=vb.matmul_persistent(s.x, s.w.t()), norm=vb.batch_invariant_rms_norm(s.x, s.norm, 1e-6),
                log_softmax=vb.log_softmax(s.logits, -1), logprob=vb.logprobs_from_logits_flash_attn(s.logits, s.labels))


def exact_suite(case, seed):
    s = prepare_suite(case, seed)
    lp = torch.log_softmax(d(s.logits), -1)
    return dict(matmul=d(s.x) @ d(s.w).T, norm=rms(d(s.x), s.norm, 1e-6), log_softmax=lp,
                logprob=lp.gather(1, s.labels[:, None])[:, 0])


def work_suite(case):
    n = case["rows"]
    return dict(bytes=2 * (n * (3 * PROJ_K + PROJ_N) + PROJ_N * PROJ_K) + 8 * n * VOCAB, flops=2 * n * PROJ_N * PROJ_K)


# ------------------------------------------------------------------ entry points
FAMILY = {"suite": "suite", "decode": "stage", "prefill": "stage", "hybrid": "hybrid", "train_attention": "train_attention",
          "train_experts": "train_experts", "train_logprob": "train_logprob"}


def _of(what, case):
    return globals()[f"{what}_{FAMILY[case['kind']]}"]


def prepare(case, seed):
    return _of("prepare", case)(case, seed)


def run(state):
    return _of("run", state.case)(state)


def work(case):
    return _of("work", case)(case)


def exact(case, seed):
    return _of("exact", case)(case, seed)


def tolerance(case):
    kind = case["kind"]
    if kind in ("decode", "prefill"):
        # bf16 activations over a stage's layers; a mixture's router adds experts that swap places at near-ties
        return dict(rel=0.03, max=0.9, differ=0.01)
    return dict(suite=dict(rel=0.01), hybrid=dict(rel=0.03, max=0.9), train_attention=dict(rel=0.02, max=0.5),
                train_experts=dict(rel=0.02, max=0.5), train_logprob=dict(rel=0.01))[kind]
