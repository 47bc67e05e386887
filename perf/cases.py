"""Cases of the decoder paths, for measuring: what a user's program has the framework do, over its range of sizes.

Kinds
  chat    a session's greedy or sampled continuation of prompts (Session.generate): prompt, then decode steps
  prompt  the logits behind prompts (Session.forward)
  follow  prompts, then given tokens one by one (Session.forward): scoring a text, routed experts
  serve   a paged session with prompt portions beside single tokens (PagedSession.feed), any model family
  eager   a decoder layer built from the rew.nn forwards (norms, attention with a KvCache, feed-forward)

Models have the widths of the configurations in rew_b200 (about a quarter of their layers and of their vocabulary, so that the
output head keeps its share of a step) or generic ones; weights are those of CausalLM.init_random for the seed.  A chat's
output head has a bias that makes one token certain: a greedy choice among the near ties of random weights would differ between
any two correct implementations, and every logit behind it.
"""
import math
from dataclasses import replace

import numpy as np
import torch

from rew_b200 import _lib, api, girulorn, kugirax, musavik, weights as W

CERTAIN = 30.0           # bias of the certain token
STD = 0.02               # of random weights

# width: (heads, kv heads, head size, feed-forward) of grouped-query decoders; 4096 is the 8B Llama shape
LLAMA = {4096: (32, 8, 128, 14336), 2048: (16, 4, 128, 5632), 1024: (16, 4, 64, 2816)}
FAMILIES = {"girulorn": girulorn.moe_lite, "kugirax": kugirax.dense_8b, "musavik": musavik.dense_8b}
VOCAB = {"llama": 24064, "moe": 25600, "girulorn": 25600, "kugirax": 32064, "musavik": 32064}


def listed():
    return [
        # a busy chat server: 32 conversations, short prompts, greedy
        dict(name="chat_b32", kind="chat", model="llama", width=4096, layers=6, batch=32, prompt=64, new=48, sampling="greedy", nf4=False),
        # one user waiting for sampled tokens: latency
        dict(name="chat_b1_top_k", kind="chat", model="llama", width=4096, layers=6, batch=1, prompt=31, new=32, sampling="top_k", nf4=False),
        # a few users of a model held as 4-bit codes
        dict(name="chat_b4_nf4", kind="chat", model="llama", width=4096, layers=6, batch=4, prompt=19, new=32, sampling="greedy", nf4=True),
        # the smallest call: the tiny f32 model of the parity tests
        dict(name="chat_tiny_f32", kind="chat", model="tiny", width=256, layers=2, batch=1, prompt=12, new=16, sampling="greedy", nf4=False),
        # long documents read in one go: the largest call
        dict(name="prompt_b8_s2048", kind="prompt", model="llama", width=4096, layers=6, batch=8, prompt=2048),
        # time to the first token of one ordinary prompt, odd length
        dict(name="prompt_b1_s333", kind="prompt", model="llama", width=4096, layers=6, batch=1, prompt=333),
        # a mixture-of-experts model (64 experts, 6 a token): prompts and following tokens of 64 sequences
        dict(name="follow_moe_b64", kind="follow", model="moe", layers=3, batch=64, prompt=96, steps=8),
        # continuous batching: a long prompt arrives in portions while other lanes decode
        dict(name="serve_llama", kind="serve", model="llama", width=4096, layers=6, lanes=12, prompt=150, steps=6, portion=100),
        # the same for recurrent, latent and mixed-head families
        dict(name="serve_girulorn", kind="serve", model="girulorn", layers=6, lanes=16, prompt=120, steps=8, portion=61),
        dict(name="serve_kugirax", kind="serve", model="kugirax", layers=8, lanes=8, prompt=300, steps=8, portion=128),
        dict(name="serve_musavik", kind="serve", model="musavik", layers=8, lanes=8, prompt=700, steps=8, portion=150),
        # a model written against the rew.nn forwards: one layer, prompt and single tokens
        dict(name="eager_b8", kind="eager", width=2048, batch=8, prompt=100, steps=8),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["chat", "chat", "prompt", "prompt", "follow", "serve", "serve", "eager"])
    width = rng.choice([4096, 2048, 1024])
    layers = rng.randint(2, 6)
    if kind == "chat":
        if rng.random() < 0.2:
            return dict(kind=kind, model="tiny", width=rng.choice([256, 512, 768]), layers=rng.randint(2, 4), batch=_log(rng, 1, 8), prompt=_log(rng, 3, 60),
                        new=_log(rng, 8, 32), sampling="greedy", nf4=False)
        nf4 = rng.random() < 0.25
        return dict(kind=kind, model="llama", width=width, layers=layers, batch=_log(rng, 1, 16 if nf4 else 96), prompt=_log(rng, 8, 200),
                    new=_log(rng, 12, 48), sampling=rng.choice(["greedy", "greedy", "top_k", "top_p"]), nf4=nf4)
    if kind == "prompt":
        batch = _log(rng, 1, 8)
        return dict(kind=kind, model="llama", width=width, layers=layers, batch=batch, prompt=_log(rng, 20, 2048))
    if kind == "follow":
        return dict(kind=kind, model="moe", layers=rng.randint(2, 3), batch=_log(rng, 1, 64), prompt=_log(rng, 10, 150), steps=rng.randint(2, 10))
    if kind == "serve":
        model = rng.choice(["llama", "girulorn", "kugirax", "musavik"])
        c = dict(kind=kind, model=model, layers=2 * rng.randint(1, 4), lanes=_log(rng, 2, 24), prompt=_log(rng, 20, 800),
                 steps=rng.randint(3, 10), portion=_log(rng, 5, 200))
        return dict(c, width=width) if model == "llama" else c
    return dict(kind=kind, width=rng.choice([2048, 1024]), batch=_log(rng, 1, 48), prompt=_log(rng, 8, 300), steps=rng.randint(2, 10))


# ---- what a program has in hand

def _lengths(case):
    """Prompt lengths of the lanes of a serve case: ragged around `prompt`; the last lane's arrives in portions."""
    n, p = case["lanes"], case["prompt"]
    return [max(1, p - p // 3 + (i * 2 * (p // 3)) // max(1, n - 1)) for i in range(n - 1)] + [case["portion"] * case["steps"]]


def _config(case):
    model = case["model"]
    if model == "tiny":
        heads = case["width"] // 32
        return replace(W.tiny_llama(mask_kind=1), d_model=case["width"], n_layers=case["layers"], n_heads=heads, n_kv_heads=heads // 4,
                       ffn=688 * case["width"] // 256 // 8 * 8)
    if model == "moe":
        return replace(W.deepseek_v2_lite(), n_layers=case["layers"], vocab=VOCAB[model])
    if model == "llama":
        heads, kv, hd, ffn = LLAMA[case["width"]]
        return replace(W.llama3_8b(), vocab=VOCAB[model], d_model=case["width"], n_layers=case["layers"], n_heads=heads, n_kv_heads=kv, head_dim=hd, ffn=ffn,
                       max_seq=2304, weight_quant=int(case.get("nf4", False)))
    layers = FAMILIES[model]().layers[:case["layers"]]
    if model == "girulorn":  # experts are follow's: normed on the way back, one near tie of a router moves a token's logits by a tenth
        layers = [replace(l, ff="dense", ffn=10944, experts=0, top_k=0, router_bias=False, shared_ffn=0) for l in layers]
    return FAMILIES[model](layers=layers, vocab=VOCAB[model], max_seq=2304)


def _certain(seed, vocab):
    return (seed * 7919 + 13) % vocab


def _model(case, cfg, seed):
    m = api.CausalLM(cfg)
    if case["kind"] != "chat":
        return m.init_random(seed, STD)
    bias = np.zeros(cfg.vocab, np.float32)
    bias[_certain(seed, cfg.vocab)] = CERTAIN
    _lib.check(_lib.lib().rewb200_model_init_random(m._h, seed, STD))
    _lib.check(_lib.lib().rewb200_model_set_tensor(m._h, len(W.tensor_specs(cfg)) - 1, bias.ctypes.data_as(_lib.F32P), bias.size))
    _lib.check(_lib.lib().rewb200_model_finalize(m._h))
    return m


def _tokens(seed, vocab, *shape):
    return np.random.default_rng(seed + 1000).integers(0, vocab, size=shape).astype(np.int32)


def _eager_inputs(case, seed):
    """bf16-valued weights and inputs of an eager layer on the GPU, in f32."""
    d = case["width"]
    heads, kv, hd, ffn = LLAMA[d]
    g = torch.Generator("cuda").manual_seed(seed)
    t = lambda *s, std=STD: (torch.randn(*s, generator=g, device="cuda") * std).bfloat16().float()
    w = dict(q=t(d, heads * hd), k=t(d, kv * hd), v=t(d, kv * hd), o=t(heads * hd, d), gate=t(d, ffn), up=t(d, ffn), down=t(ffn, d))
    w = {n: (a, torch.randn(a.shape[1], generator=g, device="cuda") * 0.01) for n, a in w.items()}
    return w, t(case["batch"], case["prompt"], d, std=1.0), [t(case["batch"], 1, d, std=1.0) for _ in range(case["steps"])]


def prepare(case, seed):
    if case["kind"] == "eager":
        heads, kv, hd, ffn = LLAMA[case["width"]]
        w, x, xs = _eager_inputs(case, seed)
        up = lambda a: api.Tensor.from_host(a.cpu().numpy(), dtype=_lib.BF16)
        lin = {n: api.Linear(up(a), api.Tensor.from_host(b.cpu().numpy())) for n, (a, b) in w.items()}
        total = case["prompt"] + case["steps"]
        return dict(kind="eager", gamma=api.Tensor.from_host(np.ones(case["width"], np.float32)),
                    attention=api.GroupedQueryAttention(lin["q"], lin["k"], lin["v"], lin["o"], api.RotaryPositionEncoding(hd, total, 10000.0), mask_kind=1),
                    ff=api.GatedFeedForward(lin["gate"], lin["up"], lin["down"]), cache=api.KvCache(case["batch"], kv, hd, total, dtype=_lib.BF16),
                    x=[up(a) for a in [x] + xs])
    cfg = _config(case)
    model = _model(case, cfg, seed)
    s = dict(kind=case["kind"], model=model)
    if case["kind"] == "serve":
        n = _lengths(case)
        total = max(v + case["steps"] for v in n)
        s["session"] = model.paged_session(case["lanes"], total, 2 + sum((v + case["steps"] + 63) // 64 for v in n))
        ids = _tokens(seed, cfg.vocab, case["lanes"], total)
        s["opening"] = [(i, ids[i, :n[i]]) for i in range(case["lanes"] - 1)]
        last = case["lanes"] - 1
        s["steps"] = [[(i, ids[i, n[i] + j:n[i] + j + 1]) for i in range(last)] + [(last, ids[last, j * case["portion"]:(j + 1) * case["portion"]])]
                      for j in range(case["steps"])]
        return s
    new = case.get("new", case.get("steps", 0))
    s["session"] = model.session(case["batch"], case["prompt"] + new)
    s["ids"] = _tokens(seed, cfg.vocab, case["batch"], case["prompt"] + case.get("steps", 0))
    s["prompt"], s["new"] = case["prompt"], new
    if case.get("sampling", "greedy") != "greedy":
        how = dict(top_k=50, top_p=1.0) if case["sampling"] == "top_k" else dict(top_k=0, top_p=0.9)
        s["session"].set_sampling(temperature=0.8, seeds=np.arange(case["batch"]) + seed, **how)
    return s


# ---- one pass

def _eager_layer(s, x):
    B, S, d = x.shape
    y = api.dispatch("add", [x, s["attention"].forward(api.rmsNorm(x, s["gamma"]), s["cache"])])[0]
    flat = api.reshape(api.rmsNorm(y, s["gamma"]), (B * S, d))
    return api.dispatch("add", [y, api.reshape(s["ff"].forward(flat), (B, S, d))])[0]


def run(s):
    if s["kind"] == "eager":
        s["cache"].reset()
        return [y.to_host() for y in [_eager_layer(s, x) for x in s["x"]]]
    sess = s["session"]
    if s["kind"] == "chat":
        ids, logits = sess.generate(s["ids"], s["new"], want_logits=True)
        return dict(ids=ids, logits=logits)
    sess.reset()
    if s["kind"] == "serve":
        sess.feed(s["opening"], sample=True)
        for portions in s["steps"][:-1]:
            sess.feed(portions, sample=True)
        ends = np.cumsum([len(t) for _, t in s["steps"][-1]]) - 1
        return sess.feed(s["steps"][-1], want=ends)[0]
    first = sess.forward(s["ids"][:, :s["prompt"]], want_logits=True)[1]
    if s["kind"] == "prompt":
        return first
    for j in range(s["prompt"], s["prompt"] + s["new"] - 1):
        sess.forward(s["ids"][:, j:j + 1])
    return dict(first=first, last=sess.forward(s["ids"][:, -1:], want_logits=True)[1])


# ---- what a pass cannot do without

def _layer_sizes(case):
    """[(elements of the matrices of a layer that every token uses, elements of one expert, experts, experts a token uses, elements
    a cached token has, elements of the products of a query with one key and its value)] per layer."""
    model = case["model"]
    if model in ("llama", "tiny", "moe"):
        c = _config(case)
        nq, nkv = c.n_heads * c.head_dim, c.n_kv_heads * c.head_dim
        att = c.d_model * (2 * nq + 2 * nkv)
        out = []
        for l in range(c.n_layers):
            if c.layer_is_moe(l):
                out.append((att + c.d_model * (c.n_routed + 3 * c.n_shared * c.moe_ffn), 3 * c.d_model * c.moe_ffn, c.n_routed, c.top_k, 2 * nkv, 2 * nq))
            else:
                out.append((att + 3 * c.d_model * (c.first_dense or c.ffn), 0, 0, 0, 2 * nkv, 2 * nq))
        return out
    out = []
    for l in _config(case).layers:
        d = 2048 if model == "girulorn" else 4096
        hk, hv = l.heads * l.dim, l.heads * l.vdim
        kv, pair = 0, 0
        if l.mixer == "attention":
            own = l.kv_heads * (l.dim + (0 if l.values_from_keys else l.vdim))
            mat = d * (hk + own + hv + (hv if l.out_gate == "element" else 0))
            kv, pair = l.kv_heads * (l.dim + l.vdim), hk + hv
        elif l.mixer == "latent":
            mat = d * (l.q_rank + (0 if l.kv_from >= 0 else l.kv_rank) + hv) + l.q_rank * hk + l.kv_rank * (hk + hv)
            kv, pair = l.kv_rank, hk + hv
        elif l.mixer == "gla":
            mat = d * (2 * hk + 3 * hv)
        else:
            mat = d * 3 * hk + 2 * l.heads * l.dim * l.dim
        if l.beside:
            b = l.beside
            mat += d * (2 * b.kv_heads * b.dim + 3 * b.heads * b.vdim)
        if l.ff == "dense":
            out.append((mat + (2 if l.ff_act == "gelu_tanh" else 3) * d * l.ffn, 0, 0, 0, kv, pair))
        else:
            out.append((mat + d * (l.experts + 3 * l.shared_ffn), 3 * d * l.ffn, l.experts, l.top_k, kv, pair))
    return out


def _steps(case):
    """[(rows of the step, keys its queries see in all, keys read, rows of the output head)]"""
    if case["kind"] == "serve":
        n = _lengths(case)
        steps = [(sum(n[:-1]), sum(v * (v + 1) // 2 for v in n[:-1]), sum(n[:-1]), case["lanes"] - 1)]
        for j in range(case["steps"]):
            p = case["portion"]
            single = sum(v + j + 1 for v in n[:-1])
            steps.append((case["lanes"] - 1 + p, single + p * (p * j + (p + 1) // 2), single + p * (j + 1), case["lanes"]))
        return steps
    B, p = case["batch"], case["prompt"]
    more = case.get("new", 1) - 1 if case["kind"] == "chat" else case.get("steps", 0)
    return [(B * p, B * p * (p + 1) // 2, B * p, B)] + [(B, B * (p + j + 1), B * (p + j + 1), B) for j in range(more)]


def work(case):
    total = {"bytes": 0.0, "flops": 0.0}
    if case["kind"] == "eager":
        d = case["width"]
        heads, kv, hd, ffn = LLAMA[d]
        layers, head, es, wb = [(d * (2 * heads + 2 * kv) * hd + 3 * d * ffn, 0, 0, 0, 2 * kv * hd, 2 * heads * hd)], 0, 2, 2
    else:
        cfg = _config(case)
        es = 4 if case["model"] == "tiny" else 2
        wb = 0.594 if case.get("nf4") else es
        layers, head = _layer_sizes(case), cfg.d_model * cfg.vocab
    for rows, seen, read, outs in _steps(case):
        total["bytes"] += head * es + outs * (head and cfg.vocab) * 4
        total["flops"] += 2 * outs * head
        for mat, one, experts, top, kv, pair in layers:
            total["bytes"] += mat * wb + min(experts, rows * top) * one * wb + read * kv * es
            total["flops"] += 2 * rows * (mat + top * one) + 2 * seen * pair
    return total


def tolerance(case):
    if case.get("model") == "tiny":
        return {"rel": 2e-6, "max": 5e-5, "differ": 0.0}
    # measured against exact(): eager 0.004, musavik 0.006, the others 0.008 to 0.02 at six layers (bf16 operands, random weights)
    rel = 0.015 if case["kind"] == "eager" else 0.024 if case["model"] == "musavik" else 0.03
    return {"rel": rel, "max": 0.9, "differ": 0.0}


# ---- the same in 64 bits

def _mix(x):
    """splitmix64 on int64 tensors."""
    shift = lambda v, n: (v >> n) & ((1 << (64 - n)) - 1)
    wrap = lambda v: v - (1 << 64) if v >= 1 << 63 else v
    x = x + wrap(0x9E3779B97F4A7C15)
    x = (x ^ shift(x, 30)) * wrap(0xBF58476D1CE4E5B9)
    x = (x ^ shift(x, 27)) * wrap(0x94D049BB133111EB)
    return x ^ shift(x, 31)


def _normal(seed, shape, dtype, std=STD):
    """The random weights of seed: Box-Muller on two hashed uniforms per pair of elements, in `dtype`."""
    n = math.prod(shape)
    out = torch.empty((n + 1) // 2 * 2, dtype=dtype, device="cuda")
    seed &= (1 << 64) - 1
    seed = seed - (1 << 64) if seed >= 1 << 63 else seed
    for at in range(0, (n + 1) // 2, 1 << 25):
        p = torch.arange(at, min(at + (1 << 25), (n + 1) // 2), device="cuda")
        h = _mix(_mix(p) ^ seed)
        u1 = (((h >> 40) & 0xFFFFFF) + 1).float() * np.float32(1.0 / 16777217.0)
        a = ((h >> 8) & 0xFFFFFF).double() * (2.0 * math.pi / 16777216.0)
        r = torch.sqrt(-2.0 * torch.log(u1.double())) * float(np.float32(std))
        out[2 * at:2 * at + 2 * len(p)] = torch.stack([r * torch.cos(a), r * torch.sin(a)], 1).float().to(dtype).reshape(-1)
    return out[:n].view(shape)


def _halves(w):
    """Gate and up of columns interleaved in groups of eight."""
    v = w.view(*w.shape[:-1], -1, 2, 8)
    return v[..., 0, :].flatten(-2), v[..., 1, :].flatten(-2)


NF4 = (-1.0, -0.6961928009986877, -0.5250730514526367, -0.39491748809814453, -0.28444138169288635, -0.18477343022823334, -0.09105003625154495, 0.0,
       0.07958029955625534, 0.16093020141124725, 0.24611230194568634, 0.33791524171829224, 0.44070982933044434, 0.5626170039176941, 0.7229568362236023, 1.0)


def _nf4(w):
    """What the 4-bit codes of w [in, out] stand for: a scale for 64 neighbouring outputs, nearest level."""
    levels = torch.tensor(NF4, device="cuda", dtype=torch.float64)
    out = torch.empty_like(w, dtype=torch.float32)
    for i in range(0, len(w), 256):
        v = w[i:i + 256].double().view(-1, w.shape[1] // 64, 64)
        scale = v.abs().amax(-1, keepdim=True).clamp_min(1e-10)
        at = torch.bucketize(v / scale, (levels[1:] + levels[:-1]) / 2)
        out[i:i + 256] = (levels[at] * scale).view(-1, w.shape[1]).float()
    return out


def _mm(x, w):
    return x @ w.double()


def _rms(x, eps):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + eps)


def _rotate(x, cos, sin):
    """x [.., T, heads, dim]: neighbouring pairs turned by the angles of their position."""
    u, v = x[..., 0::2], x[..., 1::2]
    return torch.stack([u * cos - v * sin, v * cos + u * sin], -1).flatten(-2)


def _angles(T, dim, base):
    a = torch.outer(torch.arange(T, device="cuda", dtype=torch.float64), base ** (-torch.arange(0, dim, 2, device="cuda", dtype=torch.float64) / dim))
    return a.cos()[:, None], a.sin()[:, None]


def _attend(q, k, v, scale, visible, bias=None, sink=False, mix=None):
    """q [T, H, K], k [T, G, K], v [T, G, V] -> [T, H, V]; bias [H, T, T]; sink: one in the denominator; mix [H, H]: of the weights."""
    H, G = q.shape[1], k.shape[1]
    out = torch.empty(q.shape[0], H, v.shape[2], dtype=torch.float64, device="cuda")
    group = H if mix is not None else max(1, min(H, (1 << 27) // q.shape[0] ** 2))
    for a in range(0, H, group):
        at = torch.arange(a, min(a + group, H), device="cuda")
        s = torch.einsum("thk,shk->hts", q[:, at], k[:, at // (H // G)]) * scale
        if bias is not None:
            s += bias[at]
        s.masked_fill_(~visible, -math.inf)
        if sink:
            s = torch.cat([s, torch.zeros_like(s[..., :1])], -1)
        p = s.softmax(-1)[..., :q.shape[0]]
        if mix is not None:
            p = torch.einsum("hg,gts->hts", mix, p)
        out[:, at] = torch.einsum("hts,shv->thv", p, v[:, at // (H // G)])
    return out


def _visible(T, window=0, first=0):
    back = torch.arange(T, device="cuda")[:, None] - torch.arange(T, device="cuda")[None]
    see = back >= 0
    return see & ((back < window) | (torch.arange(T, device="cuda")[None] < first)) if window else see


def _conv(u, w):
    """Causal convolution over time: u [T, C], w [taps, C], the last tap on the current token."""
    y = torch.zeros_like(u)
    for j, back in enumerate(range(len(w) - 1, -1, -1)):
        y[back:] += u[:max(0, len(u) - back)] * w[j]
    return y


def _experts(x, router, gu, down, shared, top):
    z = _mm(x, router)
    val, at = z.topk(top, dim=-1)
    wt = val.softmax(-1)
    y = torch.zeros_like(x)
    for e in range(gu.shape[0]):
        row, j = (at == e).nonzero(as_tuple=True)
        if len(row):
            y.index_add_(0, row, _gated(x[row], gu[e], down[e]) * wt[row, j, None])
    return y + _gated(x, *shared)


def _gated(x, gu, down):
    gate, up = _halves(gu)
    return _mm(torch.nn.functional.silu(_mm(x, gate)) * _mm(x, up), down)


def _llama64(case, cfg, seed, texts):
    """Logits behind the last token, and those of every earlier place listed, of sequences: [(ids, places)]."""
    dt = torch.float32 if cfg.dtype == _lib.F32 else torch.bfloat16
    k = [seed * 1000003]

    def fill(*shape):
        k[0] += 1
        return _normal(k[0], shape, dt)

    hd, nq, nkv = cfg.head_dim, cfg.n_heads * cfg.head_dim, cfg.n_kv_heads * cfg.head_dim
    xs = []
    embed = fill(cfg.vocab, cfg.d_model)
    for ids, _ in texts:
        xs.append(embed[torch.from_numpy(ids.astype(np.int64)).cuda()].double())
    T = max(len(x) for x in xs)
    inv = 1.0 / (cfg.theta ** (torch.arange(0, hd, 2, device="cuda", dtype=torch.float64) / hd)).float()
    angle = (torch.arange(T, device="cuda", dtype=torch.float32)[:, None] * inv).double()
    cos, sin = angle.cos()[:, None], angle.sin()[:, None]
    for l in range(cfg.n_layers):
        moe = cfg.layer_is_moe(l)
        width = cfg.n_shared * cfg.moe_ffn if moe else cfg.first_dense or cfg.ffn
        qkv, o, gu, down = fill(cfg.d_model, nq + 2 * nkv), fill(nq, cfg.d_model), fill(cfg.d_model, 2 * width), fill(width, cfg.d_model)
        if cfg.weight_quant:
            gate, up = _halves(gu)
            qkv, o, down = _nf4(qkv), _nf4(o), _nf4(down)
            gu = torch.stack([_nf4(gate.contiguous()).view(cfg.d_model, -1, 8), _nf4(up.contiguous()).view(cfg.d_model, -1, 8)], 2).flatten(1)
        elif dt == torch.float32:  # gate and up side by side
            v = gu.view(cfg.d_model, 2, -1, 8)
            gu = v.transpose(1, 2).flatten(1)
        if moe:
            r = seed * 1000003 + 500000 + l
            ke = ((r * 31 + 7) & ((1 << 64) - 1)) ^ (1 << 40)
            router = _normal(r, (cfg.d_model, cfg.n_routed), dt)
            egu = _normal(ke + 1, (cfg.n_routed, cfg.d_model, 2 * cfg.moe_ffn), dt)
            edown = _normal(ke + 2, (cfg.n_routed, cfg.moe_ffn, cfg.d_model), dt)
        for i, x in enumerate(xs):
            n = len(x)
            q, kk, v = _mm(_rms(x, cfg.eps), qkv).split([nq, nkv, nkv], -1)
            q, kk = (_rotate(t.view(n, -1, hd), cos[:n], sin[:n]) for t in (q, kk))
            x = x + _mm(_attend(q, kk, v.view(n, -1, hd), hd ** -0.5, _visible(n)).flatten(1), o)
            h = _rms(x, cfg.eps)
            xs[i] = x + (_experts(h, router, egu, edown, (gu, down), cfg.top_k) if moe else _gated(h, gu, down))
    head = fill(cfg.d_model, cfg.vocab)
    return [_mm(_rms(x[places], cfg.eps), head) for x, (_, places) in zip(xs, texts)]


def _bias_table(l, T, table):
    """[heads, T, T] from numbers by distance; the last one stands for all longer ones."""
    back = (torch.arange(T, device="cuda")[:, None] - torch.arange(T, device="cuda")[None]).clamp(0, table.shape[1] - 1)
    return table.double()[:, back]


def _bias_distances(l):
    h, n = l.bias_rows // 2, 0
    bucket = lambda v: v if v < h else min(l.bias_rows - 1, h + math.floor(math.log(v / h) / math.log(l.bias_max / h) * (l.bias_rows - h) + 1e-9))
    while bucket(n) < l.bias_rows - 1:
        n += 1
    return n + 1


def _layered64(case, cfg, seed, texts):
    k = [seed * 1000003]
    d, eps, pad = cfg.d_model, cfg.eps, lambda n: (n + 7) // 8 * 8

    def fill(*shape, std=STD, dtype=torch.bfloat16):
        k[0] += 1
        return _normal(k[0], shape, dtype, std)

    f32 = lambda *shape, std: fill(*shape, std=std, dtype=torch.float32).double()
    silu, sig = torch.nn.functional.silu, torch.sigmoid
    gelu = lambda z: torch.nn.functional.gelu(z, approximate="tanh")
    embed, head = fill(cfg.vocab, d), fill(d, cfg.vocab)
    big = fill(cfg.bigram[0] + 1, d) if cfg.bigram else None
    xs = []
    for ids, _ in texts:
        t = torch.from_numpy(ids.astype(np.int64)).cuda()
        x = embed[t].double() * getattr(cfg, "embed_scale", 1.0)
        if big is not None:
            row = torch.cat([torch.tensor([cfg.bigram[0]], device="cuda"), (t[:-1] * cfg.bigram[1] + t[1:] * cfg.bigram[2]) % cfg.bigram[0]])
            x = x + big[row].double()
        xs.append(x)
    lat = [dict() for _ in xs]

    def delta(l, w, h, proj):
        T, H, K, V = len(h), l.heads, l.dim, l.vdim
        ch = 2 * l.kv_heads * K + H * V
        u = silu(_conv(proj[:, :ch], w))
        unit = lambda t: t / torch.sqrt(t.square().sum(-1, keepdim=True) + 1e-6)
        q, kk, v = u.split([l.kv_heads * K, l.kv_heads * K, H * V], -1)
        r = H // l.kv_heads
        q, kk = (unit(t.reshape(T, -1, K)).repeat_interleave(r, 1) for t in (q, kk))
        q, v = q * K ** -0.5, v.reshape(T, H, V)
        gate, b, a = proj[:, ch:ch + H * V], sig(proj[:, ch + H * V:ch + H * V + H]), proj[:, ch + H * V + H:ch + H * V + 2 * H]
        g = torch.exp(-float(np.float32(0.05)) * torch.nn.functional.softplus(a))
        S, o = torch.zeros(H, K, V, dtype=torch.float64, device="cuda"), torch.empty(T, H, V, dtype=torch.float64, device="cuda")
        for i in range(T):
            S = g[i][:, None, None] * S
            e = b[i][:, None] * (v[i] - torch.matmul(kk[i][:, None], S)[:, 0])
            S = S + kk[i][:, :, None] * e[:, None]
            o[i] = torch.matmul(q[i][:, None], S)[:, 0]
        return _rms(o, eps).flatten(1) * silu(gate) * l.mix_scale

    for li, l in enumerate(cfg.layers):
        H, K, V = l.heads, l.dim, l.vdim
        b = l.beside
        dw = f32(b.conv_taps, 2 * b.kv_heads * b.dim + b.heads * b.vdim, std=0.5) if b else None
        if l.mixer == "lru":
            cw, gates, cols = f32(l.conv_taps, H * K, std=0.5), None, 2 * H * K
            gates = fill(H, K, 2 * K)
        elif l.mixer == "attention":
            own = l.kv_heads * (K + (0 if l.values_from_keys else V))
            cw = f32(l.conv_taps, H * K + l.kv_heads * K, std=0.5) if l.conv_taps else None
            table = f32(H, _bias_distances(l), std=1.0) if l.bias_rows else None
            talk = f32(H, H, std=0.3) if l.head_mix else None
            gate_cols = H * V if l.out_gate == "element" else H if l.out_gate else 0
            cols = H * K + own + gate_cols
        elif l.mixer == "gla":
            a2 = f32(l.decay_rank, H * K, std=STD)
            cols = 2 * H * K + 2 * H * V + l.decay_rank
        else:
            mine = l.kv_from < 0
            cols = l.q_rank + (l.kv_rank if mine else 0)
        more = 2 * b.kv_heads * b.dim + 2 * b.heads * b.vdim + 2 * b.heads if b else 0
        win = fill(d, pad(cols) + pad(more))
        if l.mixer == "latent":
            uq, ukv = fill(l.q_rank, H * K), fill(l.kv_rank, H * (K + V))
        wo = fill(H * V + (b.heads * b.vdim if b else 0), d)
        if l.ff == "dense":
            gu, down = fill(d, l.ffn if l.ff_act == "gelu_tanh" else 2 * l.ffn), fill(l.ffn, d)
        else:
            sgu, sdown = fill(d, 2 * l.shared_ffn), fill(l.shared_ffn, d)
            router, egu, edown = fill(d, l.experts), fill(l.experts, d, 2 * l.ffn), fill(l.experts, l.ffn, d)
        for i, x in enumerate(xs):
            T = len(x)
            h = x if cfg.block == "output_norm" else _rms(x, eps)
            p = _mm(h, win)
            if l.mixer == "lru":
                u = _conv(p[:, H * K:2 * H * K], cw)
                ri = sig(torch.einsum("tbi,bio->tbo", u.view(T, H, K), gates.double()))
                r, ig = ri[..., :K].flatten(1), ri[..., K:].flatten(1)
                a = torch.exp(float(np.float32(-0.1)) * r)
                add = torch.sqrt(1 - a * a) * ig * u
                S, o = torch.zeros_like(u[0]), torch.empty_like(u)
                for t in range(T):
                    S = a[t] * S + add[t]
                    o[t] = S
                y = o * gelu(p[:, :H * K])
            elif l.mixer == "attention":
                G = l.kv_heads
                q, kk = p[:, :H * K], p[:, H * K:(H + G) * K]
                if cw is not None:
                    q, kk = _conv(q, cw[:, :H * K]), _conv(kk, cw[:, H * K:])
                q, kk = q.reshape(T, H, K), kk.reshape(T, G, K)
                v = kk if l.values_from_keys else p[:, (H + G) * K:(H + G) * K + G * V].reshape(T, G, V)
                if l.qk_norm:
                    q, kk = _rms(q, eps), _rms(kk, eps)
                if l.temp_every:
                    q = q * (1 + l.temp_coef * torch.log((torch.arange(T, device="cuda", dtype=torch.float64) + 1).div(l.temp_every).floor() + 1))[:, None, None]
                if l.v_norm:
                    v = _rms(v, eps)
                if l.rope_dims:
                    cos, sin = _angles(T, K, l.rope_base)
                    turn = (lambda t: _rotate(t, cos, sin)) if l.rope_pairs else \
                        (lambda t: torch.cat([t[..., :K // 2] * cos - t[..., K // 2:] * sin, t[..., K // 2:] * cos + t[..., :K // 2] * sin], -1))
                    q, kk = turn(q), turn(kk)
                y = _attend(q, kk, v, l.scale, _visible(T, l.window, l.keep_first), None if table is None else _bias_table(l, T, table), bool(l.sink), talk)
                if gate_cols:
                    g = sig(p[:, H * K + own:H * K + own + gate_cols])
                    y = y * (g.view(T, H, V) if l.out_gate == "element" else g[..., None])
                y = y.flatten(1) * l.mix_scale
            elif l.mixer == "gla":
                q, kk, v, g, f = p[:, :cols].split([H * K, H * K, H * V, H * V, l.decay_rank], -1)
                alpha = torch.exp(torch.nn.functional.logsigmoid(f @ a2 + 2.0) / l.tau).view(T, H, K)
                q, kk, v = q.reshape(T, H, K) * K ** -0.5, kk.reshape(T, H, K), v.reshape(T, H, V)
                S, o = torch.zeros(H, K, V, dtype=torch.float64, device="cuda"), torch.empty(T, H, V, dtype=torch.float64, device="cuda")
                for t in range(T):
                    S = alpha[t][:, :, None] * S + kk[t][:, :, None] * v[t][:, None]
                    o[t] = torch.matmul(q[t][:, None], S)[:, 0]
                y = _rms(o, eps).flatten(1) * silu(g)
            else:
                if mine:
                    lat[i][li] = _rms(p[:, l.q_rank:l.q_rank + l.kv_rank], eps)
                c = lat[i][li if mine else l.kv_from]
                q = _mm(_rms(p[:, :l.q_rank], eps), uq).view(T, H, K)
                kv = _mm(c, ukv)
                y = _attend(q, kv[:, :H * K].reshape(T, H, K), kv[:, H * K:].reshape(T, H, V), l.scale, _visible(T, l.window), None, bool(l.sink)).flatten(1)
            if b:
                y = torch.cat([y, delta(b, dw, h, p[:, pad(cols):])], -1)
            y = _mm(y, wo)

            def ff(h):
                if l.ff != "dense":
                    return _experts(h, router, egu, edown, (sgu, sdown), l.top_k)
                return _mm(gelu(_mm(h, gu)), down) if l.ff_act == "gelu_tanh" else _gated(h, gu, down)

            if cfg.block == "parallel_one_norm":
                xs[i] = x + y + ff(h)
            elif cfg.block == "output_norm":
                x = x + _rms(y, eps)
                xs[i] = x + _rms(ff(x), eps)
            else:
                x = x + _rms(y, eps)
                xs[i] = x + _rms(ff(_rms(x, eps)), eps)
    out = [_mm(_rms(x[places], eps), head) for x, (_, places) in zip(xs, texts)]
    cap = cfg.logit_softcap
    return [cap * torch.tanh(z / cap) for z in out] if cap else out


def _eager64(case, seed):
    d = case["width"]
    heads, kv, hd, _ = LLAMA[d]
    w, x, xs = _eager_inputs(case, seed)
    w = {n: (a.double(), b.double()) for n, (a, b) in w.items()}
    x = torch.cat([x] + xs, 1).double()
    lin = lambda n, v: v @ w[n][0] + w[n][1]
    B, T, _ = x.shape
    inv = 1.0 / (10000.0 ** (torch.arange(0, hd, 2, device="cuda", dtype=torch.float64) / hd))
    angle = torch.arange(T, device="cuda", dtype=torch.float64)[:, None] * inv
    cos, sin = angle.cos()[:, None], angle.sin()[:, None]
    out = torch.empty_like(x)
    for i in range(B):
        h = _rms(x[i], 1e-5)
        q, k = _rotate(lin("q", h).view(T, heads, hd), cos, sin), _rotate(lin("k", h).view(T, kv, hd), cos, sin)
        y = x[i] + lin("o", _attend(q, k, lin("v", h).view(T, kv, hd), hd ** -0.5, _visible(T)).flatten(1))
        h = _rms(y, 1e-5)
        out[i] = y + lin("down", torch.nn.functional.silu(lin("gate", h)) * lin("up", h))
    return [out[:, :case["prompt"]]] + [out[:, case["prompt"] + j:case["prompt"] + j + 1] for j in range(case["steps"])]


def exact(case, seed):
    if case["kind"] == "eager":
        return [t.cpu().numpy() for t in _eager64(case, seed)]
    cfg = _config(case)
    forward = _llama64 if case["model"] in ("llama", "tiny", "moe") else _layered64
    rows = lambda z: torch.stack(z).cpu().numpy()
    if case["kind"] == "serve":
        n = _lengths(case)
        ids = _tokens(seed, cfg.vocab, case["lanes"], max(v + case["steps"] for v in n))
        texts = [(ids[i, :n[i] + (case["steps"] if i < case["lanes"] - 1 else 0)], [-1]) for i in range(case["lanes"])]
        return rows([z[0] for z in forward(case, cfg, seed, texts)])
    ids = _tokens(seed, cfg.vocab, case["batch"], case["prompt"] + case.get("steps", 0))
    if case["kind"] == "chat":
        sure = _certain(seed, cfg.vocab)
        texts = [(np.concatenate([ids[i], np.full(case["new"] - 1, sure, np.int32)]), [-1]) for i in range(case["batch"])]
        logits = rows([z[0] for z in forward(case, cfg, seed, texts)])
        logits[:, sure] += CERTAIN
        return dict(ids=np.full((case["batch"], case["new"]), sure, np.int32), logits=logits)
    z = forward(case, cfg, seed, [(t, [case["prompt"] - 1, -1]) for t in ids])
    first = rows([v[0] for v in z])
    return first if case["kind"] == "prompt" else dict(first=first, last=rows([v[1] for v in z]))
