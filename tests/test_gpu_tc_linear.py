"""The tcgen05 / tensor-memory Linear against the oracle and against the mma.sync Linear,
through the C ABI (option "linear" = "tc")."""
import numpy as np
import pytest

from conftest import rel_l2
from rew_b200 import weights as W

pytestmark = pytest.mark.gpu


@pytest.fixture()
def rb_tc():
    from rew_b200 import _lib, api
    _lib.init()
    api.set_option("linear", "tc")
    yield api
    api.set_option("linear", "tc")  # the default


@pytest.mark.parametrize("M,K,N", [(1, 64, 8), (32, 64, 128), (32, 4096, 1024), (7, 688, 256), (32, 256, 1376),
                                   (33, 128, 136), (64, 512, 256), (100, 320, 264), (128, 1024, 384),
                                   (200, 320, 264), (256, 2048, 512), (300, 576, 640)])
def test_tc_linear_shapes(rb_tc, orc, M, K, N):
    from rew_b200 import _lib
    rng = np.random.default_rng(M * 1000 + N)
    x = orc.bf16_round(rng.normal(size=(M, K)))
    w = orc.bf16_round(rng.normal(0, 0.05, size=(K, N)))
    b = rng.normal(0, 0.1, size=(N,)).astype(np.float32)
    want = orc.linear(x, w, b)
    T = rb_tc.Tensor.from_host
    got = rb_tc.Linear(T(w, _lib.BF16), T(b)).forward(T(x, _lib.BF16)).to_host()
    assert got.shape == (M, N)
    assert rel_l2(got, want) < 5e-3


def test_tc_model_matches_oracle_and_mma_path(rb_tc, orc):
    """Whole bf16 model on the tcgen05 Linear: split-K partial, SwiGLU and f32-logit epilogues."""
    from rew_b200 import _lib
    cfg = W.ModelConfig(vocab=512, d_model=256, n_layers=2, n_heads=4, n_kv_heads=2, head_dim=64, ffn=688, max_seq=256,
                        theta=500000.0, dtype=_lib.BF16, mask_kind=1)
    t = [orc.bf16_round(a) if a.ndim == 2 else a for a in W.init_weights(cfg, seed=4, std=0.05, trivial_affine=False)]
    for B, S in ((3, 70), (32, 16), (2, 150)):
        prompt = np.random.default_rng(B).integers(0, cfg.vocab, size=(B, S)).astype(np.int32)
        sess = rb_tc.CausalLM(cfg).load(t).session(B, S + 8)
        nxt, logits = sess.forward(prompt, want_logits=True)
        want = orc.model_forward(cfg, t, prompt, 0, True)[:, -1]
        assert rel_l2(logits, want) <= 2e-2
        ids, last = sess.decode(3, want_logits=True)
        seq = np.concatenate([prompt, nxt[:, None], ids[:, :2]], 1)
        want = orc.model_forward(cfg, t, seq, 0, True)[:, -1]
        assert rel_l2(last, want) <= 2e-2
        rb_tc.set_option("linear", "mma")
        sess2 = rb_tc.CausalLM(cfg).load(t).session(B, S + 8)
        _, logits_mma = sess2.forward(prompt, want_logits=True)
        rb_tc.set_option("linear", "tc")
        assert rel_l2(logits, logits_mma) <= 1e-2


@pytest.mark.parametrize("M", [65, 80, 81, 129, 160, 161, 257, 300, 321, 513])
@pytest.mark.parametrize("K,N", [(200, 18968), (1032, 264)])
def test_linear_tiles_of_the_steps_own_size(rb_tc, M, K, N):
    """Tiles of 16-token steps around their edges: more tiles than SMs (two CTAs an SM up to 160 tokens, persistent above) and
    fewer (persistent), a last feature tile that is only partly there, K that is no multiple of a block.  bf16 operands are
    exact in f32, so the only roundings are K + 1 of f32 sums and the bf16 output's half ulp."""
    from rew_b200 import _lib
    rng = np.random.default_rng(M + N)
    x, w = W.bf16_round(rng.normal(size=(M, K))), W.bf16_round(rng.normal(size=(K, N)))
    b = rng.normal(size=N).astype(np.float32)
    T = rb_tc.Tensor.from_host
    lin = rb_tc.Linear(T(w, _lib.BF16), T(b))
    got = lin.forward(T(x, _lib.BF16)).to_host()
    want = x.astype(np.float64) @ w + b
    bound = (K + 1) * 2.0 ** -24 * (np.abs(x).astype(np.float64) @ np.abs(w) + np.abs(b)) + 2.0 ** -8 * np.abs(want)
    assert np.all(np.abs(got - want) <= bound)


@pytest.mark.parametrize("linear", ["tc", "mma"])
@pytest.mark.parametrize("M", [1, 33, 64, 100, 300])
@pytest.mark.parametrize("N", [264, 18968, 37888])
def test_weights_that_the_launch_before_writes(rb_tc, M, N, linear):
    """x @ (A @ B): the weights of a Linear are the output of the Linear just before it, on both sides of one feature tile an SM.
    The same bits as with the weights brought from the host: no launch may request them before they are written."""
    from rew_b200 import _lib
    K, r = 520, 48
    rng = np.random.default_rng(M + N)
    bf = lambda *s: rb_tc.Tensor.from_host(W.bf16_round(rng.normal(size=s).astype(np.float32)), _lib.BF16)
    lin = lambda w: rb_tc.Linear(w, None)
    rb_tc.set_option("linear", linear)
    x = bf(M, K)
    for _ in range(3):
        a, b = bf(r, K), bf(r, N)   # other weights every time: what an early request would find are the last ones
        w = lin(b).forward(rb_tc.Tensor.from_host(np.ascontiguousarray(a.to_host().T), _lib.BF16))
        got = lin(w).forward(x).to_host()
        want = lin(rb_tc.Tensor.from_host(w.to_host(), _lib.BF16)).forward(x).to_host()
        assert np.array_equal(got, want)


@pytest.mark.parametrize("B,S", [(13, 5), (2, 80), (1, 250)])
def test_split_steps_match_the_oracle(rb_tc, orc, B, S):
    """Steps of 65 to 256 rows whose Linears are cut along K into the count of slabs that costs least (here 2 to 4 of 18 blocks)."""
    from rew_b200 import _lib
    cfg = W.ModelConfig(vocab=256, d_model=1152, n_layers=1, n_heads=9, n_kv_heads=3, head_dim=128, ffn=1536, max_seq=256,
                        theta=500000.0, dtype=_lib.BF16, mask_kind=1)
    t = [orc.bf16_round(a) if a.ndim == 2 else a for a in W.init_weights(cfg, seed=6, std=0.03, trivial_affine=False)]
    prompt = np.random.default_rng(S).integers(0, cfg.vocab, size=(B, S)).astype(np.int32)
    _, logits = rb_tc.CausalLM(cfg).load(t).session(B, S).forward(prompt, want_logits=True)
    assert rel_l2(logits, orc.model_forward(cfg, t, prompt, 0, True)[:, -1]) <= 2e-2


def test_persistent_prefill_linear_matches_oracle(rb_tc, orc):
    """Enough 256-token tiles (17 x 20 >= 2 per SM) for the persistent kernel with the double-buffered
    accumulator; a ragged last token tile and a last feature tile that is only half there."""
    from rew_b200 import _lib
    M, K, N = 4100, 320, 2496
    rng = np.random.default_rng(11)
    x = orc.bf16_round(rng.normal(size=(M, K)))
    w = orc.bf16_round(rng.normal(0, 0.05, size=(K, N)))
    b = rng.normal(0, 0.1, size=(N,)).astype(np.float32)
    want = orc.linear(x, w, b)
    T = rb_tc.Tensor.from_host
    lin = rb_tc.Linear(T(w, _lib.BF16), T(b))
    got = lin.forward(T(x, _lib.BF16)).to_host()
    assert rel_l2(got, want) < 5e-3
    rb_tc.set_option("prefill", "tile")
    try:
        again = lin.forward(T(x, _lib.BF16)).to_host()
    finally:
        rb_tc.set_option("prefill", "pair")
    assert np.array_equal(got, again)   # same MMA order, same rounding: the two kernels agree bit for bit


def _launches():
    from rew_b200 import _lib
    return {k: _lib.lib().rewb200_kernel_launches(("linear_" + k).encode()) for k in ("tile", "persistent", "pair")}


@pytest.mark.parametrize("M,K,N,epi_bias,pair", [(4100, 320, 2560, True, False), (8192, 1024, 1024, False, False), (5000, 64, 512, True, False),
                                                 (1025, 200, 15360, True, True), (4100, 320, 4608, True, True), (8200, 320, 2560, True, True), (8449, 64, 2304, True, True), (9000, 1024, 2304, False, True)])
def test_pair_prefill_linear_matches_oracle_and_the_one_cta_kernels(rb_tc, orc, M, K, N, epi_bias, pair):
    """Large launches of widths that are multiples of 256 run on pairs of CTAs
    (tcgen05 cta_group::2, 256 x 256 tiles, each CTA staging half of either operand).  Ragged last token tile
    (8 rows and one), a single 64-row k block, more tiles than pairs: against the oracle, and bit for bit against the one-CTA
    persistent kernel and the one-tile kernel (the same k order and the same rounding).  Smaller launches the same way,
    on the kernel that they run on."""
    from rew_b200 import _lib
    rng = np.random.default_rng(M + N)
    x = orc.bf16_round(rng.normal(size=(M, K)))
    w = orc.bf16_round(rng.normal(0, 0.05, size=(K, N)))
    b = rng.normal(0, 0.1, size=(N,)).astype(np.float32) if epi_bias else np.zeros(N, np.float32)
    want = orc.linear(x, w, b)
    T = rb_tc.Tensor.from_host
    lin = rb_tc.Linear(T(w, _lib.BF16), T(b))
    before = _launches()
    got = lin.forward(T(x, _lib.BF16)).to_host()
    assert _launches()["pair"] - before["pair"] == pair
    assert rel_l2(got, want) < 5e-3
    assert max(rel_l2(got[r], want[r]) for r in (0, 127, 128, 255, 256, M // 2, M - 1)) < 2e-2
    others = {}
    for how in ("persistent", "tile"):
        rb_tc.set_option("prefill", how)
        try:
            before = _launches()
            others[how] = lin.forward(T(x, _lib.BF16)).to_host()
            assert _launches()[how] == before[how] + 1
        finally:
            rb_tc.set_option("prefill", "pair")
    assert np.array_equal(others["persistent"], others["tile"])
    assert np.array_equal(got, others["persistent"])


@pytest.mark.parametrize("M,K,N,pair", [(96, 64, 256, True), (193, 64, 1024, True), (257, 200, 1024, True), (449, 64, 4096, True), (161, 200, 28672, True),
                                        (333, 1024, 28672, True), (385, 200, 28672, True), (511, 136, 18944, True), (900, 200, 6144, True),
                                        (300, 200, 1152, False), (65, 64, 2048, False)])
def test_pairs_with_tiles_of_the_steps_own_size(rb_tc, M, K, N, pair):
    """Pair tiles of 64 to 256 tokens in steps of 32: a last tile of one token, more tiles than pairs, K that is no multiple of a
    block, weights narrower than a wave; a width that pairs cannot take, a step that one CTA a tile suits better.  bf16
    operands are exact in f32, so the only roundings are K + 1 of f32 sums and the bf16 output's half ulp; and the same bits
    as the one-CTA kernels, whose products run in the same order."""
    from rew_b200 import _lib
    rng = np.random.default_rng(M + N)
    x, w = W.bf16_round(rng.normal(size=(M, K))), W.bf16_round(rng.normal(size=(K, N)))
    b = rng.normal(size=N).astype(np.float32)
    T = rb_tc.Tensor.from_host
    lin, xs = rb_tc.Linear(T(w, _lib.BF16), T(b)), T(x, _lib.BF16)
    before = _launches()
    got = lin.forward(xs).to_host()
    assert _launches()["pair"] - before["pair"] == pair
    want = x.astype(np.float64) @ w + b
    bound = (K + 1) * 2.0 ** -24 * (np.abs(x).astype(np.float64) @ np.abs(w) + np.abs(b)) + 2.0 ** -8 * np.abs(want)
    assert np.all(np.abs(got - want) <= bound)
    for how in ("persistent", "tile"):
        rb_tc.set_option("prefill", how)
        try:
            assert np.array_equal(lin.forward(xs).to_host(), got)
        finally:
            rb_tc.set_option("prefill", "pair")


@pytest.mark.parametrize("M,N,kernel", [(96, 28672, "tile"), (112, 28672, "tile"), (128, 28672, "tile"), (272, 11264, "tile"), (360, 11264, "tile"), (833, 5120, "tile"),
                                        (300, 21888, "tile"), (640, 21888, "persistent"), (700, 21888, "persistent"), (800, 21888, "persistent"),
                                        (192, 28672, "pair"), (128, 11264, "pair")])
def test_near_ties_of_the_tile_rule_go_to_the_faster_kernel(rb_tc, M, N, kernel):
    """Steps whose estimates lie within a few per cent of one another, by the kernel that is faster there (the rule's comment has the times);
    bound of the test above."""
    from rew_b200 import _lib
    K, rng = 64, np.random.default_rng(M + N)
    x, w = W.bf16_round(rng.normal(size=(M, K))), W.bf16_round(rng.normal(size=(K, N)))
    T = rb_tc.Tensor.from_host
    lin, xs = rb_tc.Linear(T(w, _lib.BF16), T(np.zeros(N, np.float32))), T(x, _lib.BF16)
    before = _launches()
    got = lin.forward(xs).to_host()
    after = _launches()
    assert {k: after[k] - before[k] for k in after} == {k: int(k == kernel) for k in after}
    bound = (K + 1) * 2.0 ** -24 * (np.abs(x) @ np.abs(w)).astype(np.float64) + 2.0 ** -8 * np.abs(x.astype(np.float64) @ w)
    assert np.all(np.abs(got - x.astype(np.float64) @ w) <= bound)


def test_persistent_prefill_model_equals_tile_kernel(rb_tc):
    """A 20 480-token prefill puts the decoder Linears (f32 partial and bf16 epilogues) on the persistent kernel and gate and up
    (SwiGLU) on the pair kernel; the logits must equal those of the one-tile-per-CTA kernel exactly."""
    from rew_b200 import _lib
    cfg = W.ModelConfig(vocab=512, d_model=512, n_layers=2, n_heads=8, n_kv_heads=2, head_dim=64, ffn=1408, max_seq=640,
                        theta=500000.0, dtype=_lib.BF16, mask_kind=1)
    model = rb_tc.CausalLM(cfg).init_random(seed=3, std=0.05)
    B, S = 40, 512
    prompt = np.random.default_rng(1).integers(0, cfg.vocab, size=(B, S)).astype(np.int32)
    sess = model.session(B, S + 8)
    before = _launches()
    _, a = sess.forward(prompt, want_logits=True)
    ran = {k: n - before[k] for k, n in _launches().items()}
    assert ran["persistent"] == 3 * cfg.n_layers and ran["pair"] == cfg.n_layers, ran
    rb_tc.set_option("prefill", "tile")
    try:
        sess.reset()
        _, b = sess.forward(prompt, want_logits=True)
    finally:
        rb_tc.set_option("prefill", "pair")
    assert np.isfinite(a).all() and np.array_equal(a, b)
