"""Continuous batching over paged KV blocks (PagedKvCache, src/rew/infer/generate.nim:63-88) on the GPU:
requests of different lengths join and leave lanes between decode steps, sharing a small pool of blocks;
every request must produce exactly what the oracle's batch-1 generate() produces for it alone."""
import numpy as np
import pytest

from rew_b200 import weights as W

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def rb():
    from rew_b200 import _lib, api
    _lib.init()
    return api


def _requests(cfg, n, seed):
    rng = np.random.default_rng(seed)
    out = []
    for i in range(n):
        plen = int(rng.integers(3, 70))
        out.append(dict(id=i, prompt=rng.integers(0, cfg.vocab, size=plen).astype(np.int32), n_new=int(rng.integers(4, 40)),
                        seed=1000 + i))
    return out


def _serve(sess, reqs, lanes, step_sizes):
    """A minimal scheduler: fill idle lanes from the queue, decode a few steps, retire finished requests."""
    pending, active, done, it = list(reqs), {}, {}, 0
    while pending or active:
        for lane in range(lanes):
            if lane not in active and pending:
                r = pending.pop(0)
                r["out"] = [sess.admit(lane, r["prompt"], seed=r["seed"])]
                active[lane] = r
        k = step_sizes[it % len(step_sizes)]
        it += 1
        out = sess.step(k)
        for lane in range(lanes):
            if lane not in active:
                assert np.all(out[lane] == -1)
                continue
            r = active[lane]
            assert sess.lane_length(lane) == len(r["prompt"]) + len(r["out"]) - 1 + k
            r["out"] += out[lane].tolist()
            if len(r["out"]) >= r["n_new"]:
                done[r["id"]] = r["out"][:r["n_new"]]
                sess.release(lane)
                del active[lane]
    return done


@pytest.mark.parametrize("mask_kind", [1, 0])
def test_continuous_batching_matches_per_request_generate(rb, orc, mask_kind):
    cfg = W.tiny_llama(norm_kind=1, mask_kind=mask_kind)
    t = W.init_weights(cfg, seed=21, trivial_affine=False)
    reqs = _requests(cfg, 7, seed=3)
    lanes, blocks = 3, 8                       # 7 usable blocks of 64 tokens for 3 lanes of up to 109 tokens
    sess = rb.CausalLM(cfg).load(t).paged_session(lanes, 112, blocks)
    assert sess.free_blocks() == blocks - 1
    done = _serve(sess, reqs, lanes, step_sizes=[1, 3, 2])
    assert sess.free_blocks() == blocks - 1    # every block came back
    for r in reqs:
        want, _ = orc.generate_greedy(cfg, t, r["prompt"][None, :], r["n_new"])
        assert done[r["id"]] == want[0].tolist(), r["id"]


def test_continuous_batching_with_sampling_matches_oracle(rb, orc):
    cfg = W.tiny_llama(norm_kind=0, mask_kind=1)
    t = W.init_weights(cfg, seed=22)
    reqs = _requests(cfg, 5, seed=4)
    kw = dict(temperature=1.2, top_k=0, top_p=0.9, repetition_penalty=1.15)
    sess = rb.CausalLM(cfg).load(t).paged_session(2, 112, 6)
    sess.set_sampling(**kw)
    done = _serve(sess, reqs, 2, step_sizes=[2, 1])
    for r in reqs:
        want, _ = orc.generate_sampled(cfg, t, r["prompt"][None, :], r["n_new"], seeds=[r["seed"]], **kw)
        assert done[r["id"]] == want[0].tolist(), r["id"]


def test_pool_exhaustion_and_lane_errors(rb):
    cfg = W.tiny_llama(mask_kind=1)
    sess = rb.CausalLM(cfg).load(W.init_weights(cfg, seed=0)).paged_session(2, 128, 3)   # two usable blocks
    p = np.arange(60, dtype=np.int32)
    sess.admit(0, p)
    sess.admit(1, p)
    assert sess.free_blocks() == 0
    with pytest.raises(RuntimeError, match="busy"):
        sess.admit(0, p)
    sess.step(4)                                # 64 tokens each: still one block per lane
    with pytest.raises(RuntimeError, match="out of free blocks"):
        sess.step(1)                            # both lanes would need a second block
    assert sess.lane_length(0) == 64 and sess.lane_length(1) == 64   # nothing moved
    sess.release(1)
    sess.release(1)                             # idempotent
    assert sess.free_blocks() == 1 and sess.lane_length(1) == -1
    out = sess.step(2)                          # lane 0 takes the freed block
    assert np.all(out[1] == -1) and np.all(out[0] >= 0)
    with pytest.raises(RuntimeError, match="out of free blocks"):
        sess.admit(1, p)
    with pytest.raises(RuntimeError, match="out of range"):
        sess.admit(5, p)
    with pytest.raises(RuntimeError, match="paged"):
        sess.generate(p[None, :].repeat(2, 0), 4)
    with pytest.raises(RuntimeError):
        rb.CausalLM(cfg).load(W.init_weights(cfg, seed=0)).paged_session(2, 128, 1)


@pytest.mark.parametrize("dtype,hd,mask,tol", [("f32", 32, 0, 1e-5), ("f32", 32, 1, 1e-5), ("bf16", 64, 1, 2e-2), ("bf16", 128, 1, 2e-2), ("bf16", 128, 0, 2e-2)])
def test_feed_of_unequal_portions_in_any_order(rb, orc, dtype, hd, mask, tol):
    """Every kind of portion (one token, below 64, 64 and more) in one step, several of each, in scrambled order and on lanes
    whose contexts differ: wanted rows equal the oracle's forward of each lane's whole text.  A conventional mask only lets
    later portions see earlier ones; the mask as written is checked on first portions, where it needs no context."""
    from rew_b200 import _lib
    bf = dtype == "bf16"
    cfg = W.ModelConfig(vocab=128, d_model=128, n_layers=2, n_heads=4, n_kv_heads=2, head_dim=hd, ffn=192, max_seq=512, theta=10000.0,
                        dtype=_lib.BF16 if bf else _lib.F32, mask_kind=mask)
    t = [orc.bf16_round(a) if bf and a.ndim == 2 else a for a in W.init_weights(cfg, seed=3, std=0.08, trivial_affine=False)]
    model = rb.CausalLM(cfg).load(t)
    lanes, rng = 7, np.random.default_rng(hd + mask)
    sess = model.paged_session(lanes, 400, 60)
    texts = [np.zeros(0, np.int32) for _ in range(lanes)]
    steps = [[(3, 130), (0, 1), (5, 2), (6, 300), (1, 127), (2, 128)]]
    if mask == 1:
        steps += [[(0, 129), (6, 1), (4, 64), (1, 1), (2, 65), (5, 128)], [(4, 1), (0, 1), (1, 1), (3, 1), (5, 1), (2, 2), (6, 1)]]
    for portions in steps:
        fed = [(l, rng.integers(0, cfg.vocab, n).astype(np.int32)) for l, n in portions]
        start = [len(texts[l]) for l, _ in fed]
        for l, ids in fed:
            texts[l] = np.concatenate([texts[l], ids])
        total = sum(n for _, n in portions)
        want = sorted(set(rng.integers(0, total, 40).tolist()) | set(np.cumsum([n for _, n in portions]) - 1))
        logits, nxt = sess.feed(fed, want=want, sample=[i % 2 == 0 for i in range(len(fed))])
        whole = [orc.model_forward(cfg, t, texts[l][None], 0, True)[0] for l, _ in fed]
        rows = np.concatenate([w[s:] for w, s in zip(whole, start)])
        exp = rows[want]
        err = np.linalg.norm(logits - exp, axis=1) / np.linalg.norm(exp, axis=1)
        assert err.max() <= (1.5 * tol if bf else tol), (portions, err.argmax(), err.max())
        ends = np.cumsum([n for _, n in portions]) - 1
        for i, (l, _) in enumerate(fed):
            assert sess.lane_length(l) == len(texts[l])
            if i % 2:
                assert nxt[i] == -1
            else:
                assert nxt[i] == int(np.argmax(logits[want.index(ends[i])]))
    sess.reset()
    assert sess.free_blocks() == 59 and all(sess.lane_length(l) == -1 for l in range(lanes))


def test_routing_of_a_step_of_portions_in_the_callers_order(rb):
    """The recorded expert choices of a step whose rows were put in the order of their portions' kinds come back in the order the
    tokens were given in: those of every portion fed alone."""
    cfg = W.ModelConfig(vocab=64, d_model=64, n_layers=2, n_heads=2, n_kv_heads=1, head_dim=32, ffn=64, max_seq=256, theta=10000.0, mask_kind=1,
                        n_routed=8, n_shared=1, top_k=2, moe_ffn=32)
    rb.set_option("record_routing", "1")
    try:
        model = rb.CausalLM(cfg).load(W.init_weights(cfg, seed=2, std=0.3))
        rng = np.random.default_rng(4)
        portions = [(l, rng.integers(0, cfg.vocab, n).astype(np.int32)) for l, n in ((1, 1), (3, 40), (0, 130), (2, 1))]
        sess = model.paged_session(4, 200, 20)
        sess.feed(portions)
        rows = sum(len(t) for _, t in portions)
        got = [sess.routing(layer, rows) for layer in range(2)]
        alone = [[], []]
        for l, t in portions:
            sess.reset()
            sess.feed([(l, t)])
            for layer in range(2):
                alone[layer].append(sess.routing(layer, len(t)))
        for layer in range(2):
            assert np.array_equal(got[layer], np.concatenate(alone[layer]))
    finally:
        rb.set_option("record_routing", "0")


def test_short_portions_keep_f32_sums_beside_long_ones(rb, orc):
    """The outputs of o and down reach the residual unrounded for every portion of up to 256 tokens, also when its neighbours bring the
    step above that.  A model made to tell: embeddings of +-64, zero queries, keys and feed-forward, values that pass the
    normed token on and an output matrix of -64 on its diagonal, so that a first token's residual is only what the small rest of
    that matrix adds: multiples of 2^-6 below 2, exact in f32, lost to a bf16 spacing of 2^-2 at 64."""
    from rew_b200 import _lib
    d = 128
    cfg = W.ModelConfig(vocab=64, d_model=d, n_layers=1, n_heads=2, n_kv_heads=2, head_dim=64, ffn=64, max_seq=512, dtype=_lib.BF16, mask_kind=1)
    rng = np.random.default_rng(0)
    sign = lambda *s: np.where(rng.random(s) < 0.5, -1.0, 1.0).astype(np.float32)
    zero, layer = np.zeros((d, d), np.float32), "model.layers.0."
    off = (1 - np.eye(d, dtype=np.float32)) * sign(d, d)
    made = {"model.embedTokens.weight": 64 * sign(cfg.vocab, d), layer + "mlp.downProj.weight": np.zeros((cfg.ffn, d), np.float32),
            layer + "selfAttn.qProj.weight": zero, layer + "selfAttn.kProj.weight": zero, layer + "selfAttn.vProj.weight": np.eye(d, dtype=np.float32),
            layer + "selfAttn.outProj.weight": off / 64 - 64 * np.eye(d, dtype=np.float32)}
    t = [made.pop(name, a) for (name, _), a in zip(W.tensor_specs(cfg), W.init_weights(cfg, seed=1, std=0.1))]
    assert not made
    t = [orc.bf16_round(a) if a.ndim == 2 else a for a in t]
    sess = rb.CausalLM(cfg).load(t).paged_session(5, 400, 40)
    portions = [(l, rng.integers(0, cfg.vocab, n).astype(np.int32)) for l, n in ((2, 1), (0, 300), (4, 1), (1, 1), (3, 257))]
    ends = np.cumsum([len(ids) for _, ids in portions]) - 1
    singles = [i for i, (_, ids) in enumerate(portions) if len(ids) == 1]
    logits, _ = sess.feed(portions, want=[int(ends[i]) for i in singles])
    for got, i in zip(logits, singles):
        want = orc.model_forward(cfg, t, portions[i][1][None], 0, True)[0, -1]
        assert np.linalg.norm(got - want) <= 2e-2 * np.linalg.norm(want)


@pytest.mark.parametrize("S", [1, 20, 64, 300])
def test_feed_of_one_portion_costs_what_a_plain_step_does(rb, S):
    """A step of one portion on a grouped-query model: the bits and the launches of a plain session's step of the same tokens, besides the
    lane tables ahead of it and behind it and the row gathered for the lm_head; then the same for one more token."""
    from rew_b200 import _lib
    cfg = W.ModelConfig(vocab=128, d_model=256, n_layers=5, n_heads=4, n_kv_heads=2, head_dim=64, ffn=512, max_seq=512, dtype=_lib.BF16, mask_kind=1)
    model = rb.CausalLM(cfg).load(W.init_weights(cfg, seed=5, std=0.08))
    plain, paged = model.session(1, 400), model.paged_session(9, 400, 20)
    launches = lambda: _lib.lib().rewb200_launch_count(0)
    paged.feed([(l, np.arange(3, dtype=np.int32)) for l in (2, 8)])
    for ids in (np.random.default_rng(S).integers(0, cfg.vocab, S).astype(np.int32), np.array([7], np.int32)):
        n0 = launches()
        nxt, want = plain.forward(ids[None], want_logits=True)
        n1 = launches()
        logits, got = paged.feed([(5, ids)], want=[len(ids) - 1], sample=True)
        n2 = launches()
        assert np.array_equal(logits, want) and got[0] == nxt[0]
        assert n2 - n1 <= n1 - n0 + 3


def test_feed_with_sampling_and_seeds_in_any_order(rb, orc):
    """Portions on a grouped-query model, sorted by kind inside the step, each lane with a seed of its own: the tokens of the oracle's
    sampled generation of every lane alone, whatever order the lanes are given in and however a prompt is cut."""
    cfg = W.tiny_llama(norm_kind=0, mask_kind=1)
    t = W.init_weights(cfg, seed=23)
    kw = dict(temperature=1.1, top_k=0, top_p=0.9, repetition_penalty=1.1)
    rng = np.random.default_rng(6)
    prompts = [rng.integers(0, cfg.vocab, n).astype(np.int32) for n in (40, 1, 65, 9)]
    seeds = [900, 31, 7, 4000]
    sess = rb.CausalLM(cfg).load(t).paged_session(4, 112, 12)
    sess.set_sampling(**kw)
    n_new, out = 8, [[] for _ in prompts]
    # the first step: lanes 2, 1, 3 and 0, of which lane 0 brings only a part of its prompt and lane 3 only its first token
    first = [(2, prompts[2]), (1, prompts[1]), (3, prompts[3][:1]), (0, prompts[0][:30])]
    _, nxt = sess.feed(first, sample=[True, True, False, False], seeds=[seeds[l] for l, _ in first])
    assert nxt[2] == -1 and nxt[3] == -1
    out[2].append(int(nxt[0])), out[1].append(int(nxt[1]))
    step = 0
    while any(len(o) < n_new for o in out):
        portions = [(l, np.array([out[l][-1]], np.int32) if out[l] else (prompts[0][30:] if l == 0 else prompts[3][1:]))
                    for l in rng.permutation(4) if len(out[l]) < n_new]
        _, nxt = sess.feed(portions, sample=True, seeds=[55 + step] * len(portions))   # seeds count only for a lane's first portion
        for (l, _), tok in zip(portions, nxt):
            out[l].append(int(tok))
        step += 1
    for l, p in enumerate(prompts):
        want, _ = orc.generate_sampled(cfg, t, p[None], n_new, seeds=[seeds[l]], **kw)
        assert out[l] == want[0].tolist(), l


@pytest.mark.parametrize("first", [0, 64, 130])
def test_feed_of_portions_on_either_side_of_64_queries(rb, orc, first):
    """Head size 128: portions of 3 to 63 tokens attend on mma.sync, those of 64 and more on tcgen05, one launch a layer for all of a kind,
    behind nothing, a whole page and pages and a half.  Every row of the step against the oracle."""
    from rew_b200 import _lib
    cfg = W.ModelConfig(vocab=128, d_model=256, n_layers=2, n_heads=4, n_kv_heads=2, head_dim=128, ffn=192, max_seq=512, theta=10000.0,
                        dtype=_lib.BF16, mask_kind=1)
    t = [orc.bf16_round(a) if a.ndim == 2 else a for a in W.init_weights(cfg, seed=3, std=0.08, trivial_affine=False)]
    rng = np.random.default_rng(first)
    sizes = {5: 64, 1: 3, 0: 63, 6: 1, 2: 40, 4: 65, 3: 127}
    texts = {l: rng.integers(0, cfg.vocab, first + l + n).astype(np.int32) for l, n in sizes.items()}   # contexts of unequal length
    at = {l: len(texts[l]) - n for l, n in sizes.items()}
    sess = rb.CausalLM(cfg).load(t).paged_session(7, 300, 40)
    before_it = [(l, texts[l][:at[l]]) for l in sizes if at[l]]
    if before_it:
        sess.feed(before_it)
    count = lambda: [_lib.lib().rewb200_kernel_launches(k.encode()) for k in ("attention_tc", "attention_tc2")]
    before = count()
    logits, _ = sess.feed([(l, texts[l][at[l]:]) for l in sizes], want=range(sum(sizes.values())))
    assert [a - b for a, b in zip(count(), before)] == [cfg.n_layers, 0]
    row = 0
    for l, n in sizes.items():
        want = orc.model_forward(cfg, t, texts[l][None], 0, True)[0, at[l]:]
        err = np.linalg.norm(logits[row:row + n] - want, axis=1) / np.linalg.norm(want, axis=1)
        assert err.max() <= 3e-2, (l, n, err.argmax(), err.max())     # as the test above: rows one by one
        row += n
    # without a portion of 64 or more nothing runs on tcgen05
    sess.reset()
    before = count()
    sess.feed([(l, texts[l][:n]) for l, n in ((0, 63), (1, 3), (2, 40), (6, 1))])
    assert count() == before


def test_feed_of_long_portions_with_two_query_tiles_a_cta(rb):
    """Portions of unequal length through the attention kernel of two query tiles a CTA (one to three tiles of 256, full and ragged):
    the bits of the kernel with one, in one step and on top of contexts of different lengths."""
    from rew_b200 import _lib
    cfg = W.ModelConfig(vocab=128, d_model=256, n_layers=2, n_heads=4, n_kv_heads=2, head_dim=128, ffn=256, max_seq=1024, theta=10000.0,
                        dtype=_lib.BF16, mask_kind=1)
    model = rb.CausalLM(cfg).load(W.init_weights(cfg, seed=3, std=0.08))
    rng = np.random.default_rng(12)
    steps = [[(l, rng.integers(0, cfg.vocab, n).astype(np.int32)) for l, n in step]
             for step in (((2, 600), (0, 128), (3, 257), (1, 1), (4, 512)), ((1, 300), (3, 129), (4, 2), (0, 256)))]
    runs = {}
    for how, kernel in (("tc1", "attention_tc"), ("tc2", "attention_tc2")):
        rb.set_option("attention", how)
        try:
            sess = model.paged_session(5, 1000, 60)
            before = _lib.lib().rewb200_kernel_launches(kernel.encode())
            runs[how] = [sess.feed(p, want=range(0, sum(len(ids) for _, ids in p), 7), sample=True) for p in steps]
            assert _lib.lib().rewb200_kernel_launches(kernel.encode()) - before == 2 * cfg.n_layers
        finally:
            rb.set_option("attention", "tc")
    for (a, x), (b, y) in zip(runs["tc1"], runs["tc2"]):
        assert np.isfinite(a).all() and np.array_equal(a, b) and np.array_equal(x, y)
