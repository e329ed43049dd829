"""Layer-stack models (Matulorn design) on the GPU against the plain numpy restatement in tests/stack_oracle.py: every
mixer alone, whole prompts against token-by-token decoding, portions down to two tokens, contexts that are cleared and used
again, window edges and far keys with sharpened attention, the soft-max sink, long decoding through the replayed graph,
odd sizes (vector and scalar load paths, grouped key heads, one norm group, partial rotation, no YaRN), bfloat16, and greedy
generation through the bridge's job loop. Small random models written to a temporary folder; float32 is the sharp
comparison."""
import copy
import ctypes as C
import os

import numpy as np
import pytest

import stack_oracle as so
from booster_b200 import _lib, engine

pytestmark = pytest.mark.gpu

TOL32 = 2e-4


def err(got, want):
    """root mean square of the difference with its mean taken off, over the root mean square of the expected row; worst row"""
    got, want = np.asarray(got, np.float64), np.asarray(want, np.float64)
    d = got - want
    d = d - d.mean(-1, keepdims=True)
    w = want - want.mean(-1, keepdims=True)
    return float((np.sqrt((d * d).mean(-1)) / (np.sqrt((w * w).mean(-1)) + 1e-30)).max())


def mingru(width=40, mlp=None):
    return {"type": "mingru", "mixer": {"width": width}, "mlp": mlp}


def latent(heads=3, dim=8, rot_dim=4, vdim=12, kv_rank=20, window=7, scaling=True, dims=None, mlp=None, scale=0.3):
    rot = {"base": 10000.0, "dims": dims if dims is not None else rot_dim}
    if scaling:
        rot["scaling"] = {"factor": 4.0, "fast": 32.0, "slow": 1.0, "original": 16}
    mx = {"heads": heads, "dim": dim, "rot_dim": rot_dim, "vdim": vdim, "kv_rank": kv_rank, "scale": scale, "rot": rot}
    if window:
        mx["mask"] = {"size": window}
    return {"type": "latent_attention", "mixer": mx, "mlp": mlp}


def delta(heads=4, kv_heads=2, dim=8, vdim=6, conv=3, mlp=None):
    return {"type": "delta", "mixer": {"heads": heads, "kv_heads": kv_heads, "dim": dim, "vdim": vdim, "conv": conv}, "mlp": mlp}


def ff(n=56, limit=1.5):
    return {"ff": n, "kind": "dense", "limit": limit}


def config(layers, width=48, vocab=61, groups=3, eps=1e-5):
    return {"architecture": "Matulorn", "layers": layers, "norm": {"eps": eps, "groups": groups}, "vocab": vocab, "width": width}


class Pair:
    """the same random model in the framework and in the oracle"""

    def __init__(self, tmp_path, cfg, seed=0, dtype="float32", n_ctx=512, edit=None):
        self.cfg = cfg
        self.w = so.random_model(cfg, seed)
        if edit:
            edit(self.w)
        d = so.write_model(str(tmp_path / f"m{seed}_{dtype}_{abs(hash(str(cfg))) % 10**8}"), cfg, self.w)
        self.oracle = so.Oracle(cfg, {k: np.asarray(v, np.float64) for k, v in self.w.items()})
        self.model = engine.Model(d, dtype=dtype)
        self.ctx = engine.Context(self.model, n_ctx)
        self.dir = d

    def close(self):
        self.ctx.close()
        self.model.close()

    def tokens(self, n, seed=1):
        return np.random.default_rng(seed).integers(0, self.cfg["vocab"], size=n).tolist()

    def expected(self, toks):
        self.oracle.reset()
        return self.oracle.forward(toks)

    def run(self, toks, cuts=None, ctx=None):
        """logits of every position, the token stream cut into steps of the given sizes (None: one step)"""
        ctx = ctx or self.ctx
        ctx.kv_clear()
        out, pos = [], 0
        cuts = list(cuts) if cuts else [len(toks)]
        i = 0
        while pos < len(toks):
            n = min(cuts[i % len(cuts)], len(toks) - pos)
            out.append(ctx.decode_rows(toks[pos:pos + n], pos, list(range(n))))
            pos += n
            i += 1
        return np.concatenate(out)


@pytest.mark.parametrize("layer", [mingru(), mingru(mlp=ff()), latent(), latent(window=0, mlp=ff()), delta(), delta(heads=3, kv_heads=3, dim=5, vdim=7, conv=4)],
                         ids=["mingru", "mingru+ff", "latent", "latent-unmasked+ff", "delta-grouped", "delta-odd"])
def test_each_mixer_alone_with_layer_taps(tmp_path, layer):
    p = Pair(tmp_path, config([layer]))
    toks = p.tokens(23)
    p.oracle.reset()
    lay = []
    want = p.oracle.forward(toks, lay)
    p.ctx.set_taps(True)
    got = p.ctx.decode_rows(toks, 0, list(range(len(toks))))
    taps = p.ctx.layer_taps(len(toks))
    p.ctx.set_taps(False)
    assert np.abs(taps[0] - lay[0]).max() < 1e-4 * max(1.0, np.abs(lay[0]).max())
    assert err(got, want) < TOL32
    p.close()


FULL = [mingru(), latent(mlp=ff()), delta(), mingru(width=24, mlp=ff(40, 0.75)), latent(heads=2, dim=12, rot_dim=8, vdim=4, kv_rank=16, window=5, dims=4),
        delta(heads=2, kv_heads=1, dim=16, vdim=8, conv=2, mlp=ff(32, 2.0))]


def test_whole_prompt_token_by_token_and_portions_agree(tmp_path):
    p = Pair(tmp_path, config(FULL))
    toks = p.tokens(75)
    want = p.expected(toks)
    whole = p.run(toks)
    assert err(whole, want) < TOL32
    single = p.run(toks, [1])                         # every token through the replayed one-token graph
    assert err(single, want) < TOL32
    for cuts in ([2], [3, 2, 7, 1, 5], [37, 2, 2, 30], [6, 1, 1, 11]):
        assert err(p.run(toks, cuts), want) < TOL32, cuts
    assert err(single, whole) < TOL32
    p.close()


def test_only_wanted_rows_are_returned_in_order(tmp_path):
    p = Pair(tmp_path, config(FULL[:3]))
    toks = p.tokens(19)
    want = p.expected(toks)
    p.ctx.kv_clear()
    a = p.ctx.decode_rows(toks[:11], 0, [0, 4, 10])
    b = p.ctx.decode_rows(toks[11:], 11, [])
    c = p.ctx.decode(toks[:1], 19)                    # b200_decode: the last row
    assert a.shape == (3, p.cfg["vocab"]) and b.shape[0] == 0 and c.shape == (p.cfg["vocab"],)
    assert err(a, want[[0, 4, 10]]) < TOL32
    with pytest.raises(_lib.B200Error):               # recurrent state cannot rewind: a step must continue the sequence
        p.ctx.decode_rows(toks[:2], 3, [0])
    with pytest.raises(_lib.B200Error):
        p.ctx.decode_rows([p.cfg["vocab"]], 20, [0])
    p.close()


def test_cleared_context_is_as_good_as_new(tmp_path):
    p = Pair(tmp_path, config(FULL))
    a, b = p.tokens(40, seed=3), p.tokens(29, seed=4)
    fresh = engine.Context(p.model, 512)
    ref_b = p.run(b, [5, 1, 1, 9], ctx=fresh)
    p.run(a, [7, 1])                                  # fills cache rows, recurrent state and convolution history
    again = p.run(b, [5, 1, 1, 9])                    # run() clears first: the same context, used again
    assert np.array_equal(again, ref_b)
    assert err(again, p.expected(b)) < TOL32
    # several contexts of one model do not disturb each other
    p.ctx.kv_clear(); fresh.kv_clear()
    x1 = p.ctx.decode_rows(a[:9], 0, [8]); y1 = fresh.decode_rows(b[:9], 0, [8])
    x2 = p.ctx.decode_rows(a[9:10], 9, [0]); y2 = fresh.decode_rows(b[9:10], 9, [0])
    assert err(np.concatenate([x1, x2]), p.expected(a[:10])[[8, 9]]) < TOL32
    assert err(np.concatenate([y1, y2]), p.expected(b[:10])[[8, 9]]) < TOL32
    fresh.close()
    p.close()


def sharpen(w):
    """make the soft-max peaky, so that one key more or less in the window moves the logits visibly"""
    for k in list(w):
        if k.endswith("mix.q"):
            w[k] = so.round_bf16(w[k] * 6.0)


@pytest.mark.parametrize("window", [1, 2, 9, 33])
def test_window_edges_in_prompts_and_in_decoding(tmp_path, window):
    cfg = config([latent(window=window, heads=2, kv_rank=12), mingru(width=16)], width=32, groups=2)
    p = Pair(tmp_path, cfg, seed=window, edit=sharpen)
    toks = p.tokens(3 * window + 20, seed=window)
    want = p.expected(toks)
    # the oracle itself tells windows apart by far more than the tolerance: a window one token off would show
    for off in (-1, 1):
        c2 = copy.deepcopy(cfg)
        if window + off >= 1:
            c2["layers"][0]["mixer"]["mask"]["size"] = window + off
            o2 = so.Oracle(c2, p.oracle.w)
            assert err(o2.forward(toks)[window + 1:], want[window + 1:]) > 50 * TOL32
    assert err(p.run(toks), want) < TOL32
    assert err(p.run(toks, [window + 1, 1]), want) < TOL32            # the window passes over decoded tokens
    assert err(p.run(toks, [max(window - 1, 1), 2, 1]), want) < TOL32 # portions that start and end inside a window
    p.close()


def test_far_keys_and_first_tokens_without_a_mask(tmp_path):
    cfg = config([latent(window=0, heads=2, kv_rank=12, scale=1.0), delta(heads=2, kv_heads=2, dim=8, vdim=8, conv=4)], width=32, groups=4)
    p = Pair(tmp_path, cfg, seed=5, edit=sharpen, n_ctx=400)
    toks = p.tokens(330, seed=9)
    want = p.expected(toks)
    got = p.run(toks, [300, 1])
    assert err(got, want) < TOL32
    assert err(got[:4], want[:4]) < TOL32             # the first tokens of a sequence: empty history, zero state
    assert err(p.run(toks[:40], [1]), want[:40]) < TOL32
    p.close()


def test_sink_counts_once_in_the_denominator(tmp_path):
    cfg = config([latent(window=6)])

    def big_sink(w):
        w["l0.mix.sink"] = so.round_bf16(np.array([2.5, -1.0, 0.75], np.float32))
    p = Pair(tmp_path, cfg, seed=7, edit=big_sink)
    toks = p.tokens(20)
    want = p.expected(toks)
    no_sink = dict(p.oracle.w); no_sink["l0.mix.sink"] = np.full(3, -1e30)
    assert err(so.Oracle(cfg, no_sink).forward(toks), want) > 50 * TOL32
    assert err(p.run(toks, [9, 1]), want) < TOL32
    p.close()


def test_long_decoding_through_the_graph(tmp_path):
    p = Pair(tmp_path, config(FULL[:3] + [delta(heads=2, kv_heads=2, dim=40, vdim=33, conv=3)]))
    toks = p.tokens(260, seed=11)
    want = p.expected(toks)
    got = p.run(toks, [4, 1])
    assert err(got, want) < 2 * TOL32
    assert err(got[-1:], want[-1:]) < 2 * TOL32
    p.close()


@pytest.mark.parametrize("width,groups,vocab", [(36, 1, 50), (40, 5, 77), (64, 8, 130)], ids=["scalar-loads", "five-groups", "vector-loads"])
def test_other_sizes(tmp_path, width, groups, vocab):
    layers = [delta(heads=6, kv_heads=2, dim=9, vdim=5, conv=1, mlp=ff(20, 0.5)), latent(heads=1, dim=6, rot_dim=6, vdim=3, kv_rank=9, window=4, scaling=False, dims=2),
              mingru(width=7), latent(heads=4, dim=16, rot_dim=8, vdim=16, kv_rank=32, window=50, dims=8), delta(heads=1, kv_heads=1, dim=64, vdim=40, conv=5)]
    p = Pair(tmp_path, config(layers, width=width, vocab=vocab, groups=groups, eps=1e-6), seed=width)
    toks = p.tokens(70, seed=width)
    want = p.expected(toks)
    assert err(p.run(toks), want) < TOL32
    assert err(p.run(toks, [13, 2, 1]), want) < TOL32
    p.close()


def random_config(rng):
    """a random arrangement of the three mixers with random sizes: nothing may rest on one model's values"""
    pick = lambda values: int(rng.choice(values))
    groups = pick([1, 2, 3, 4, 5, 8])
    layers = []
    for _ in range(pick([2, 3, 4, 5])):
        mlp = ff(pick([24, 64, 100, 136]), float(rng.choice([0.5, 1.0, 7.0]))) if rng.random() < 0.5 else None
        kind = pick([0, 1, 2])
        if kind == 0:
            layers.append(mingru(pick([8, 24, 56, 130]), mlp))
        elif kind == 1:
            rot_dim = pick([2, 4, 8, 16, 32])
            L = latent(heads=pick([1, 2, 3, 5, 6, 12]), dim=pick([4, 8, 24, 64]), rot_dim=rot_dim, vdim=pick([4, 16, 40, 64]), kv_rank=pick([8, 24, 64, 96, 192]),
                       window=pick([0, 1, 3, 17, 64, 100, 300]), scaling=bool(rng.random() < 0.7), dims=rot_dim if rng.random() < 0.6 else pick([d for d in (2, 4, 8, 16) if d <= rot_dim]),
                       mlp=mlp, scale=float(rng.choice([0.1, 0.2, 0.35])))
            if "scaling" in L["mixer"]["rot"]:
                L["mixer"]["rot"]["scaling"] = {"factor": float(rng.choice([2.0, 8.0, 40.0])), "fast": float(rng.choice([32.0, 16.0])), "slow": float(rng.choice([1.0, 2.0])),
                                                "original": pick([16, 64, 4096])}
                L["mixer"]["rot"]["base"] = float(rng.choice([10000.0, 500000.0]))
            layers.append(L)
        else:
            kv = pick([1, 2, 3])
            layers.append(delta(heads=kv * pick([1, 2, 4]), kv_heads=kv, dim=pick([4, 16, 32, 128]), vdim=pick([4, 8, 48, 128]), conv=pick([1, 2, 3, 5]), mlp=mlp))
    return config(layers, width=groups * pick([8, 12, 24, 40, 72]), vocab=pick([37, 100, 257, 513]), groups=groups, eps=float(rng.choice([1e-6, 1e-5])))


@pytest.mark.parametrize("seed", range(8))
def test_random_configurations(tmp_path, seed):
    rng = np.random.default_rng(500 + seed)
    cfg = random_config(rng)
    n = int(rng.choice([70, 150, 330]))
    p = Pair(tmp_path, cfg, seed=seed, n_ctx=n + 4)
    toks = p.tokens(n, seed=seed)
    want = p.expected(toks)
    assert err(p.run(toks), want) < 2 * TOL32, cfg
    assert err(p.run(toks, [n - 20] + [1] * 20), want) < 2 * TOL32, cfg
    assert err(p.run(toks, [2, 67, 3, 129, 1, 5]), want) < 2 * TOL32, cfg
    p.close()


def test_large_heads_and_ranks(tmp_path):
    """more heads than one attention block takes, a latent wider than one sweep of the weighted sum, a row that is no whole number
    of 16-byte chunks, and a delta-rule key size that takes the widest recurrence kernel"""
    layers = [latent(heads=20, dim=16, rot_dim=32, vdim=24, kv_rank=640, window=70), latent(heads=7, dim=20, rot_dim=6, vdim=10, kv_rank=37, window=129, dims=6),
              delta(heads=2, kv_heads=1, dim=192, vdim=80, conv=2)]
    p = Pair(tmp_path, config(layers, width=128, vocab=90, groups=2), seed=2, n_ctx=208)
    toks = p.tokens(200, seed=8)
    want = p.expected(toks)
    assert err(p.run(toks), want) < TOL32
    assert err(p.run(toks, [170] + [1] * 30), want) < TOL32
    assert err(p.run(toks, [2, 67, 3]), want) < TOL32
    p.close()


def test_a_step_longer_than_one_pass(tmp_path):
    """a 700-token step runs as two passes of the layers: the window, the convolution's inputs and the recurrent state cross the pass's edge"""
    layers = [latent(heads=3, dim=8, rot_dim=4, vdim=8, kv_rank=16, window=40), delta(heads=2, kv_heads=1, dim=8, vdim=8, conv=4), mingru(24, ff(40)),
              latent(heads=2, dim=8, rot_dim=8, vdim=4, kv_rank=24, window=0)]
    p = Pair(tmp_path, config(layers), n_ctx=704)
    toks = p.tokens(700, seed=5)
    want = p.expected(toks)
    assert err(p.run(toks), want) < 2 * TOL32
    assert err(p.run(toks, [509, 2, 3, 186]), want) < 2 * TOL32
    p.close()


@pytest.mark.parametrize("taps", [2, 8, 9])
def test_convolution_of_portions_at_the_edges_of_its_tiles(tmp_path, taps):
    """eight tokens of a channel to a thread up to eight taps, a token a thread above; the heads' vectors of every length a block holds in registers and one that it does not"""
    p = Pair(tmp_path, config([delta(heads=2, kv_heads=1, dim=33, vdim=128, conv=taps), delta(heads=3, kv_heads=3, dim=43, vdim=130, conv=taps)]), seed=taps)
    toks = p.tokens(60, seed=taps)
    want = p.expected(toks)
    for cuts in (None, [7, 8, 9, 16, 17], [2, 3, 1]):
        assert err(p.run(toks, cuts), want) < TOL32
    p.close()


@pytest.mark.parametrize("heads,tokens", [(16, 7), (32, 3), (32, 4), (32, 7)])
def test_few_tokens_a_step_in_the_longest_contexts(tmp_path, heads, tokens):
    """an unmasked latent layer in a context whose score rows only fit a block in many key slices: every slice counts, the newest keys' among them, from one key to a slice to several"""
    p = Pair(tmp_path, config([latent(heads=heads, dim=8, rot_dim=8, vdim=8, kv_rank=32, window=0)]), n_ctx=131072)
    toks = p.tokens(50 + 20 * tokens)
    assert err(p.run(toks, [50] + [tokens] * 20), p.expected(toks)) < TOL32
    p.close()


def row_errs(got, want):
    got, want = np.asarray(got, np.float64), np.asarray(want, np.float64)
    d = got - want
    d = d - d.mean(-1, keepdims=True)
    w = want - want.mean(-1, keepdims=True)
    return np.sqrt((d * d).mean(-1)) / (np.sqrt((w * w).mean(-1)) + 1e-30)


def test_bfloat16_prompt_kernels_and_decode(tmp_path):
    cfg = config(FULL, width=64, groups=4, vocab=96)
    p = Pair(tmp_path, cfg, dtype="bfloat16")
    toks = p.tokens(150, seed=2)
    want = p.expected(toks)
    # token by token: mat-vec kernels with float32 activations on the stored bfloat16 weights — nothing is rounded that the
    # oracle does not round, so this path is as sharp as float32
    assert err(p.run(toks[:60], [1]), want[:60]) < TOL32
    assert err(p.run(toks[:60], [3, 4, 2]), want[:60]) < TOL32         # portions of up to 4 tokens take the same kernels
    # longer portions: tensor-core products round the activation operand to bfloat16 (2^-9 relative per product input)
    for cuts in (None, [140, 1], [5, 17, 33]):
        e = row_errs(p.run(toks, cuts), want)
        assert np.median(e) < 3e-2 and e.max() < 0.25, (cuts, float(np.median(e)), float(e.max()))
    p.close()


def test_greedy_generation_through_the_bridge(tmp_path, monkeypatch):
    """initContext / doInference on a folder model: decimal-id prompt, standard chain at temperature 0 (arg-max on the device),
    prompt through the prompt kernels, generation through the one-token graph — the ids the oracle generates greedily"""
    monkeypatch.setenv("BOOSTER_B200_DTYPE", "float32")
    p = Pair(tmp_path, config(FULL[:4]))
    prompt, n_gen = p.tokens(21, seed=6), 10
    p.oracle.reset()
    lg = p.oracle.forward(prompt)[-1]
    ids = []
    for _ in range(n_gen):
        ids.append(int(np.argmax(lg)))
        srt = np.sort(lg)
        assert srt[-1] - srt[-2] > 1e-3               # no near-tie: float32 must pick the same id
        lg = p.oracle.forward([ids[-1]])[-1]
    L = _lib.lib()
    L.init(b"", b"")
    ctx = L.initContext(5, p.dir.encode(), 1, 0, 100, 0, 0, 0, 64, n_gen, 0, 0.0, 0.0, 0.0, 1, 1.0, 1.0, 1.0, 0, 0, 200, 1.0, 1.0, 1.0, 42, b"")
    assert ctx, _lib.last_error()
    n = L.doInference(5, ctx, b"stack-job", b"", " ".join(map(str, prompt)).encode())
    out = [int(x) for x in L.status(b"stack-job").decode().split()]
    assert out[:len(prompt)] == prompt and out[len(prompt):] == ids
    assert n == len(prompt) + n_gen - 1 and L.getPromptTokenCount(b"stack-job") == len(prompt)
    # the device-resident loop of the token-level interface gives the same ids
    p.ctx.kv_clear()
    first = int(np.argmax(p.ctx.decode(prompt, 0)))
    dev = p.ctx.generate_greedy(first, len(prompt), n_gen - 1).tolist()
    assert [first] + dev == ids
    # the burst left cache, state and position where a host-driven step continues them
    after = p.ctx.decode([ids[-1]], len(prompt) + n_gen - 1)
    assert err(after[None], lg[None]) < TOL32
    assert p.ctx.L.b200_kernel_launches(p.ctx.h) > 0
    p.close()


def test_bad_models_fail_loudly(tmp_path):
    cfg = config([mingru()])
    w = so.random_model(cfg)
    d = so.write_model(str(tmp_path / "ok"), cfg, w)
    bad = dict(cfg); bad["architecture"] = "Nonesuch"
    with pytest.raises(_lib.B200Error, match="unsupported architecture"):
        engine.Model(so.write_model(str(tmp_path / "arch"), bad, w))
    w2 = dict(w); del w2["l0.mix.o"]
    with pytest.raises(_lib.B200Error, match="missing tensor"):
        engine.Model(so.write_model(str(tmp_path / "missing"), cfg, w2))
    w3 = dict(w); w3["l0.mix.z.b"] = w["l0.mix.z.b"][:-1]
    with pytest.raises(_lib.B200Error, match="shape"):
        engine.Model(so.write_model(str(tmp_path / "shape"), cfg, w3))
    c3 = copy.deepcopy(cfg); c3["layers"][0]["type"] = "lstm"
    with pytest.raises(_lib.B200Error, match="unknown mixer"):
        engine.Model(so.write_model(str(tmp_path / "mixer"), c3, w))
    with pytest.raises(_lib.B200Error, match="dtype"):
        engine.Model(d, dtype="float16")
    m = engine.Model(d)                               # bfloat16 by default
    assert m.n_vocab == cfg["vocab"] and m.n_embd == cfg["width"] and m.n_layer == 1
    c = engine.Context(m, 16)
    with pytest.raises(_lib.B200Error, match="exceeds the context"):
        c.decode_rows([1] * 17, 0, [16])
    with pytest.raises(_lib.B200Error, match="not available"):
        c.kv_seq_rm(0, 1)
    c.close(); m.close()


@pytest.mark.parametrize("dtype,T,N,K,glu", [
    ("bfloat16", 1, 70, 48, False), ("bfloat16", 4, 66, 36, True),            # mat-vec: vector and scalar loads
    ("bfloat16", 37, 100, 64, False), ("bfloat16", 21, 64, 40, True),         # mma.sync
    ("bfloat16", 200, 300, 136, False), ("bfloat16", 130, 512, 64, True),     # tcgen05 + TMEM: ragged and whole tiles
    ("bfloat16", 513, 258, 1032, False),                                      # more K steps than pipeline stages, several token tiles
    ("bfloat16", 70, 130, 35, False),                                         # odd K: CUDA cores
    ("bfloat16", 512, 168, 2048, False), ("bfloat16", 100, 131, 584, False),  # few output tiles: K in parts, rows of whole and of ragged 16-byte chunks
    ("bfloat16", 200, 600, 4104, False),
    ("bfloat16", 1, 37, 2048, False), ("bfloat16", 3, 160, 4096, False), ("float32", 2, 20, 1028, False),      # few long rows: eight warps each
    ("float32", 4, 11, 1031, False),
    ("float32", 50, 70, 33, True), ("float32", 3, 9, 7, False)], ids=str)
def test_products_pick_their_kernel_and_agree_with_numpy(dtype, T, N, K, glu):
    rng = np.random.default_rng(T * 1000 + N)
    x = rng.standard_normal((T, K)).astype(np.float32)
    w = so.round_bf16(rng.standard_normal((N, K)).astype(np.float32) / np.sqrt(K))
    b = so.round_bf16(rng.standard_normal(N).astype(np.float32))
    limit = 0.8
    y = np.zeros((T, N // 2 if glu else N), np.float32)
    f32p = C.POINTER(C.c_float)
    L = _lib.lib()
    rc = L.b200_stack_linear(0, 0 if dtype == "bfloat16" else 1, T, N, K, x.ctypes.data_as(f32p), w.ctypes.data_as(f32p), b.ctypes.data_as(f32p),
                             int(glu), limit, y.ctypes.data_as(f32p))
    assert rc == 0, _lib.last_error()
    # the tensor-core paths round the activations to bfloat16; everything else keeps them in float32
    tensor = dtype == "bfloat16" and T > 4 and K % 8 == 0
    xe = so.round_bf16(x) if tensor else x
    ref = xe.astype(np.float64) @ w.astype(np.float64).T + b
    if glu:
        g, u = np.minimum(ref[:, 0::2], limit), np.clip(ref[:, 1::2], -limit, limit)
        ref = g * so.sigmoid(1.702 * g) * (u + 1.0)
    assert np.abs(y - ref).max() < 2e-5 * max(1.0, np.abs(ref).max()) * np.sqrt(K)


@pytest.mark.parametrize("dtype", ["bfloat16", "float32"])
@pytest.mark.parametrize("T,N,K,glu", [
    (1, 513, 1024, False), (1, 1001, 2056, False), (1, 2048, 4096, True), (1, 600, 8192, False), (1, 530, 16384, False), (1, 514, 1032, True), (1, 512, 1024, False),
    (1, 1001, 2040, False), (1, 1001, 4088, False), (1, 530, 8184, False), (1, 514, 2040, True), (1, 518, 4088, True), (1, 1030, 8192, True),
    (64, 128, 64, False), (65, 257, 72, False), (130, 300, 4096, False), (200, 2056, 1000, False), (129, 514, 264, True), (300, 130, 2064, False)])
def test_products_where_their_rules_change(dtype, T, N, K, glu):
    """one token: eight rows a block and each number of chunks per lane, rows and K that end inside a block or fill too little of one; portions: TMA tiles that end inside T, N and K,
    and float32 products in K parts. Bound: a sum of K float32 products in any order is off by at most (K + 8) 2^-24 sum |x w|."""
    rng = np.random.default_rng(T * 7 + N + K)
    x = rng.standard_normal((T, K)).astype(np.float32)
    w = so.round_bf16((rng.standard_normal((N, K)) / np.sqrt(K)).astype(np.float32))
    b = rng.standard_normal(N).astype(np.float32)
    y = np.zeros((T, N // 2 if glu else N), np.float32)
    f32p = C.POINTER(C.c_float)
    L = _lib.lib()
    rc = L.b200_stack_linear(0, 0 if dtype == "bfloat16" else 1, T, N, K, x.ctypes.data_as(f32p), w.ctypes.data_as(f32p), b.ctypes.data_as(f32p), int(glu), 7.0, y.ctypes.data_as(f32p))
    assert rc == 0, _lib.last_error()
    xe = (so.round_bf16(x) if dtype == "bfloat16" and T > 4 else x).astype(np.float64)
    we = w.astype(np.float64)
    ref = xe @ we.T + b
    off = (K + 8) * 2.0 ** -24 * (np.abs(xe) @ np.abs(we).T + np.abs(b))
    if glu:      # y = g sigmoid(1.702 g) (u + 1): slopes below 1.13 in g (times |u + 1|) and below |g| + 1 in u, both clamped at 7; 1e-5 for the exponential
        g, u = np.minimum(ref[:, 0::2], 7.0), np.clip(ref[:, 1::2], -7.0, 7.0)
        ref = g * so.sigmoid(1.702 * g) * (u + 1.0)
        off = 1.13 * np.abs(u + 1.0) * off[:, 0::2] + (np.abs(g) + 1.0) * off[:, 1::2] + 1e-5 * (1.0 + np.abs(ref))
    assert (np.abs(y - ref) <= off).all(), np.max(np.abs(y - ref) / off)


@pytest.mark.parametrize("dtype", ["bfloat16", "float32"])
@pytest.mark.parametrize("N,K,glu", [
    (1, 8, False), (13, 256, False), (300, 264, True), (147, 504, False), (2, 520, True), (149, 1024, False), (1184, 1032, True), (297, 2040, False), (38000, 2048, False),
    (40002, 64, True), (130, 2056, False), (606, 4096, True), (7, 4104, False), (301, 8192, False), (34, 8184, True), (301, 8200, False), (60, 1031, False)])
def test_one_token_products_in_a_pass(dtype, N, K, glu):
    """the ring kernel at the edges of its teams of warps and pieces per lane, with fewer and more rows than SMs and stages, in one round and several, behind itself; and what it leaves
    to the kernels of products by themselves. Bound: test_products_where_their_rules_change"""
    rng = np.random.default_rng(N + K)
    x = rng.standard_normal((1, K)).astype(np.float32)
    w = so.round_bf16((rng.standard_normal((N, K)) / np.sqrt(K)).astype(np.float32))
    b = so.round_bf16(rng.standard_normal(N).astype(np.float32))
    y = np.full(N // 2 if glu else N, np.nan, np.float32)
    f32p = C.POINTER(C.c_float)
    rc = _lib.lib().b200_stack_linear_in_pass(0, 0 if dtype == "bfloat16" else 1, 1, N, K, x.ctypes.data_as(f32p), w.ctypes.data_as(f32p), b.ctypes.data_as(f32p), int(glu), 7.0, y.ctypes.data_as(f32p))
    assert rc == 0, _lib.last_error()
    ref = (x.astype(np.float64) @ w.astype(np.float64).T + b)[0]
    off = (K + 8) * 2.0 ** -24 * ((np.abs(x.astype(np.float64)) @ np.abs(w.astype(np.float64)).T)[0] + np.abs(b))
    if glu:
        g, u = np.minimum(ref[0::2], 7.0), np.clip(ref[1::2], -7.0, 7.0)
        ref = g * so.sigmoid(1.702 * g) * (u + 1.0)
        off = 1.13 * np.abs(u + 1.0) * off[0::2] + (np.abs(g) + 1.0) * off[1::2] + 1e-5 * (1.0 + np.abs(ref))
    assert (np.abs(y - ref) <= off).all(), np.nanmax(np.abs(y - ref) / off)


@pytest.mark.parametrize("dtype", ["bfloat16", "float32"])
@pytest.mark.parametrize("T,N,K,glu", [(2, 1, 8, False), (3, 149, 520, False), (4, 302, 1032, True), (2, 16001, 2048, False), (3, 16001, 2048, False), (2, 5000, 2048, True), (4, 150, 8192, False), (3, 40002, 64, True), (4, 37, 8200, False)])
def test_products_of_few_tokens_in_a_pass(dtype, T, N, K, glu):
    """the ring kernel with a token to each layer of its grid: fewer rows than blocks, several rounds, odd tokens; and rows that it leaves alone. Bound: test_products_where_their_rules_change"""
    rng = np.random.default_rng(T + N + K)
    x = rng.standard_normal((T, K)).astype(np.float32)
    w = so.round_bf16((rng.standard_normal((N, K)) / np.sqrt(K)).astype(np.float32))
    b = so.round_bf16(rng.standard_normal(N).astype(np.float32))
    y = np.full((T, N // 2 if glu else N), np.nan, np.float32)
    f32p = C.POINTER(C.c_float)
    rc = _lib.lib().b200_stack_linear_in_pass(0, 0 if dtype == "bfloat16" else 1, T, N, K, x.ctypes.data_as(f32p), w.ctypes.data_as(f32p), b.ctypes.data_as(f32p), int(glu), 7.0, y.ctypes.data_as(f32p))
    assert rc == 0, _lib.last_error()
    xe, we = x.astype(np.float64), w.astype(np.float64)
    ref = xe @ we.T + b
    off = (K + 8) * 2.0 ** -24 * (np.abs(xe) @ np.abs(we).T + np.abs(b))
    if glu:
        g, u = np.minimum(ref[:, 0::2], 7.0), np.clip(ref[:, 1::2], -7.0, 7.0)
        ref = g * so.sigmoid(1.702 * g) * (u + 1.0)
        off = 1.13 * np.abs(u + 1.0) * off[:, 0::2] + (np.abs(g) + 1.0) * off[:, 1::2] + 1e-5 * (1.0 + np.abs(ref))
    assert (np.abs(y - ref) <= off).all(), np.nanmax(np.abs(y - ref) / off)


@pytest.mark.parametrize("T,N,K,glu", [
    (5, 128, 64, False), (31, 130, 72, True), (33, 256, 1032, False), (63, 1000, 2048, False), (96, 258, 128, True), (257, 600, 64, False), (256, 514, 200, True), (300, 3000, 520, False),
    (513, 2056, 264, True), (600, 256, 4096, False), (1100, 140, 96, False), (7, 20000, 64, True),
    (5, 256, 192, False), (31, 386, 200, True), (7, 20000, 192, True)])
def test_bfloat16_products_on_pairs_of_sms(T, N, K, glu):
    """few tokens and many, tiles that end inside T, N and K, one accumulator and two, K parts, more tiles than pairs. Bound: test_products_where_their_rules_change; the tensor cores
    add without rounding to nearest, which at worst doubles it"""
    rng = np.random.default_rng(T + N + K)
    x = rng.standard_normal((T, K)).astype(np.float32)
    w = so.round_bf16((rng.standard_normal((N, K)) / np.sqrt(K)).astype(np.float32))
    b = so.round_bf16(rng.standard_normal(N).astype(np.float32))
    y = np.full((T, N // 2 if glu else N), np.nan, np.float32)
    f32p = C.POINTER(C.c_float)
    rc = _lib.lib().b200_stack_linear(0, 0, T, N, K, x.ctypes.data_as(f32p), w.ctypes.data_as(f32p), b.ctypes.data_as(f32p), int(glu), 7.0, y.ctypes.data_as(f32p))
    assert rc == 0, _lib.last_error()
    xe, we = so.round_bf16(x).astype(np.float64), w.astype(np.float64)
    ref = xe @ we.T + b
    off = 2 * (K + 8) * 2.0 ** -24 * (np.abs(xe) @ np.abs(we).T + np.abs(b))
    if glu:
        g, u = np.minimum(ref[:, 0::2], 7.0), np.clip(ref[:, 1::2], -7.0, 7.0)
        ref = g * so.sigmoid(1.702 * g) * (u + 1.0)
        off = 1.13 * np.abs(u + 1.0) * off[:, 0::2] + (np.abs(g) + 1.0) * off[:, 1::2] + 1e-5 * (1.0 + np.abs(ref))
    assert (np.abs(y - ref) <= off).all(), np.nanmax(np.abs(y - ref) / off)


def run_products(x, w, seg=None, glu=0, limit=0.0, rounded=False):
    """b200_stack_products: bfloat16 products of heads (x [batch][T][K]) or of rows sorted by matrix (x [T][K], seg)"""
    i32p, f32p = C.POINTER(C.c_int32), C.POINTER(C.c_float)
    batch, N, K = w.shape
    T = x.shape[-2]
    y = np.zeros(x.shape[:-1] + (N // 2 if glu else N,), np.float32)
    s = None if seg is None else np.ascontiguousarray(seg, np.int32)
    rc = _lib.lib().b200_stack_products(0, 0, T, N, K, batch, None if s is None else s.ctypes.data_as(i32p), x.ctypes.data_as(f32p), w.ctypes.data_as(f32p), glu, limit, int(rounded), y.ctypes.data_as(f32p))
    assert rc == 0, _lib.last_error()
    return y


def test_launches_are_counted_as_they_are_made(tmp_path):
    """a portion of one minGRU layer whose norm leaves rounded rows: embedding, input product (nothing to round) and gates, rounding, output product, end of the layer, last norm, head;
    and a K-part sum where the plan has one"""
    p = Pair(tmp_path, config([mingru(width=512)], width=256, groups=4, vocab=160), dtype="bfloat16")
    def parts(N, K):
        out = (C.c_int32 * 8)()
        assert _lib.lib().b200_stack_product_plan(0, 64, N, K, 1, 0, 0, 148, out) == 0 and out[0] == 8
        return 1 + (out[4] > 1)
    before = p.ctx.kernel_launches()
    p.ctx.decode_rows(p.tokens(64), 0, [63])
    assert p.ctx.kernel_launches() - before == 1 + parts(1536, 256) + 1 + 1 + parts(256, 512) + 1 + 1 + 1
    p.close()


def sorted_rows(counts):
    return np.concatenate([[0], np.cumsum(counts)])


@pytest.mark.parametrize("counts,N,K", [
    ([0, 300, 7, 0, 33, 0], 512, 128), ([1, 2, 600], 258, 264), ([257, 0, 0, 256], 130, 64), ([3, 1, 1], 300, 200), ([2] * 511 + [40], 256, 192),      # pairs of SMs: 512 experts at most
    ([1] * 100 + [0] * 400 + [3] * 13, 128, 64), ([0] * 512 + [300], 136, 72),                                                                      # more: a block per tile
    ([4, 0, 9], 140, 192), ([30, 1, 0, 25], 600, 72)], ids=lambda v: f"{len(v)}x{max(v)}" if isinstance(v, list) else str(v))      # mma.sync
def test_rows_sorted_by_expert(counts, N, K):
    """every row on its own expert's matrix: experts without rows beside full ones, several tiles of tokens to an expert, rows of no expert left alone. Bound:
    test_bfloat16_products_on_pairs_of_sms"""
    rng = np.random.default_rng(sum(counts) + N + K)
    T, extra = sum(counts), 3
    x = rng.standard_normal((T + extra, K)).astype(np.float32)
    w = so.round_bf16((rng.standard_normal((len(counts), N, K)) / np.sqrt(K)).astype(np.float32))
    seg = sorted_rows(counts)
    y = run_products(x, w, seg)
    assert np.isnan(y[T:]).all()
    xe = so.round_bf16(x).astype(np.float64)
    for z in range(len(counts)):
        rows = slice(seg[z], seg[z + 1])
        off = 2 * (K + 8) * 2.0 ** -24 * (np.abs(xe[rows]) @ np.abs(w[z].astype(np.float64)).T)
        assert (np.abs(y[rows] - xe[rows] @ w[z].astype(np.float64).T) <= off).all(), z


@pytest.mark.parametrize("batch,T,N,K", [(3, 64, 128, 64), (2, 129, 257, 328), (5, 70, 1030, 72), (4, 300, 140, 1032), (1, 64, 127, 64), (3, 33, 300, 200)])
def test_products_of_heads(batch, T, N, K):
    """k_gemm_bf16_umma, and mma.sync for few tokens: tiles that end inside T, N and K, more slices than stages. Bound: test_bfloat16_products_on_pairs_of_sms"""
    rng = np.random.default_rng(batch + T + N + K)
    x = rng.standard_normal((batch, T, K)).astype(np.float32)
    w = so.round_bf16((rng.standard_normal((batch, N, K)) / np.sqrt(K)).astype(np.float32))
    xe, we = so.round_bf16(x).astype(np.float64), w.astype(np.float64).transpose(0, 2, 1)
    off = 2 * (K + 8) * 2.0 ** -24 * (np.abs(xe) @ np.abs(we))
    assert (np.abs(run_products(x, w) - xe @ we) <= off).all()


@pytest.mark.parametrize("counts,N,K,glu,limit", [
    ([5], 256, 192, 1, 7.0), ([300], 514, 136, 1, np.inf), ([600], 1030, 520, 1, 3.0), ([70], 300, 2048, 2, 0.0),              # one matrix: few columns, one accumulator and two
    ([0, 300, 7, 0, 33, 0], 512, 128, 1, np.inf), ([1, 2, 600], 258, 264, 1, 7.0), ([40, 0, 20], 320, 208, 2, 0.0)], ids=str)      # experts: empty ones, a second tile of tokens
def test_gated_units_handed_on_are_the_units_rounded(counts, N, K, glu, limit):
    """gates of every size, far beyond the clamps: what the product behind reads is the float32 unit of the same sums, rounded to bfloat16 once"""
    rng = np.random.default_rng(sum(counts) + N + K)
    x = (rng.standard_normal((sum(counts), K)) * rng.choice([0.05, 1.0, 40.0], size=(sum(counts), 1))).astype(np.float32)
    w = so.round_bf16((rng.standard_normal((len(counts), N, K)) / np.sqrt(K)).astype(np.float32))
    seg = sorted_rows(counts) if len(counts) > 1 else None
    xs = x if seg is not None else x[None]
    whole = run_products(xs, w, seg, glu, limit)
    assert np.isfinite(whole).all()
    assert np.array_equal(run_products(xs, w, seg, glu, limit, rounded=True), so.round_bf16(whole))


@pytest.mark.parametrize("cuts", [None, [5, 33, 262], [64, 1, 235]], ids=str)
def test_bfloat16_portions_hand_rounded_rows_on(tmp_path, cuts):
    """a model wide enough for pairs of SMs: norms and gated units leave their rows rounded for the products behind them, in portions of few tokens and many"""
    cfg = config([mingru(width=136, mlp=ff(192)), delta(heads=4, kv_heads=2, dim=32, vdim=32, mlp=ff(200)), latent(heads=4, dim=32, rot_dim=16, vdim=32, kv_rank=64, window=40, mlp=ff(128))], width=128, groups=4, vocab=160)
    p = Pair(tmp_path, cfg, dtype="bfloat16")
    toks = p.tokens(300, seed=2)
    e = row_errs(p.run(toks, cuts), p.expected(toks))
    assert np.median(e) < 3e-2 and e.max() < 0.25, (float(np.median(e)), float(e.max()))      # 2^-9 relative per product input, as test_bfloat16_prompt_kernels_and_decode
    p.close()


def test_float32_contexts_hold_no_room_for_products_they_never_run(tmp_path):
    """a float32 context has room for the K parts of its own model's products and no more (19 MB would hold any): sixteen small contexts stay well below what
    that alone would take, and a portion that is cut into parts decodes the oracle's rows"""
    torch = pytest.importorskip("torch")
    p = Pair(tmp_path, config([mingru(width=200)], width=1056), n_ctx=160)      # 600 x 1056: four K parts
    free = torch.cuda.mem_get_info()[0]
    more = [engine.Context(p.model, 160) for _ in range(16)]
    used = free - torch.cuda.mem_get_info()[0]
    assert used < 16 * 16 << 20, used
    toks = np.random.default_rng(3).integers(0, 61, size=128).tolist()
    a, b = (c.decode_rows(toks, 0, [5, 127]) for c in more[:2])
    assert np.array_equal(a, b)
    assert err(a, p.expected(toks)[[5, 127]]) < TOL32
    for c in more:
        c.close()
    p.close()


@pytest.mark.parametrize("T,N,K,glu", [(64, 64, 64, False), (65, 66, 68, False), (127, 130, 132, True), (128, 128, 256, False), (129, 257, 196, False), (300, 1030, 4096, False),
                                       (600, 300, 1024, True)])
def test_float32_products_on_the_tensor_cores(T, N, K, glu):
    """k_gemm_f32_umma at the edges of its tiles and slices, whole and in K parts, on numbers of 24 bits and of many magnitudes. Bound: a slice of 64 k is an accumulator added to 24
    times, cut short each time (2^-23 of sum |x w|), the slices' sums are added in float32, and the products that are left out are below 2^-25. Rows with an infinity or a
    NaN are what fmaf gives, their neighbours untouched."""
    rng = np.random.default_rng(T + N + K)
    x = (rng.standard_normal((T, K)) * np.exp(2.0 * rng.standard_normal((T, K)))).astype(np.float32)
    w = (rng.standard_normal((N, K)) / np.sqrt(K)).astype(np.float32)
    y, z = (np.zeros((T, N // 2 if glu else N), np.float32) for _ in range(2))
    f32p = C.POINTER(C.c_float)
    L = _lib.lib()

    def product(x, y):
        rc = L.b200_stack_linear(0, 1, T, N, K, x.ctypes.data_as(f32p), w.ctypes.data_as(f32p), None, int(glu), 7.0, y.ctypes.data_as(f32p))
        assert rc == 0, _lib.last_error()
    product(x, y)
    xe, we = x.astype(np.float64), w.astype(np.float64)
    ref, off = xe @ we.T, (K / 64 + 48 + 2) * 2.0 ** -24 * (np.abs(xe) @ np.abs(we).T)
    if glu:      # slopes as in the test above
        g, u = np.minimum(ref[:, 0::2], 7.0), np.clip(ref[:, 1::2], -7.0, 7.0)
        ref = g * so.sigmoid(1.702 * g) * (u + 1.0)
        off = 1.13 * off[:, 0::2] * (np.abs(u) + 1.0) + off[:, 1::2] * (np.abs(g) + 1.0) + 1e-5 * np.abs(ref) + 1e-30
    assert (np.abs(y - ref) <= off + 1e-30).all(), float((np.abs(y - ref) / (off + 1e-30)).max())
    x[5, 3], x[9, 0] = np.inf, np.nan
    product(x, z)
    if not glu:  # (the unit's clamps take them in)
        assert np.isnan(z[9]).all() and np.isinf(z[5]).all() and np.array_equal(np.sign(z[5]), np.sign(w[:, 3]))
    assert np.abs(np.delete(z, [5, 9], 0) - np.delete(ref, [5, 9], 0)).max() <= (K + 8) * 2.0 ** -22 * np.abs(ref).max() + off.max()


@pytest.mark.parametrize("T,N,K", [(65, 66, 68), (129, 257, 196), (300, 1030, 4096)])
def test_float32_products_leave_rows_beside_odd_ones_alone(T, N, K):
    """k_gemm_f32_umma, whole and in K parts: rows and columns with an infinity or a NaN are what fmaf gives, rows of nothing but numbers around 2^-113 lose what three bfloat16 parts
    cannot hold of them, and every other output has the bits it has without them. Bound: (K + 8) 2^-24 sum |x w|; a part below 2^-133 is gone from each x (times |w|) and each w
    (times |x|), and each of six products and sums can end below the smallest float32 number, 2^-149."""
    rng = np.random.default_rng(T + N + K)
    x, w = rng.standard_normal((T, K)).astype(np.float32), (rng.standard_normal((N, K)) / np.sqrt(K)).astype(np.float32)
    f32p = C.POINTER(C.c_float)

    def product(x, w):
        y = np.zeros((T, N), np.float32)
        rc = _lib.lib().b200_stack_linear(0, 1, T, N, K, x.ctypes.data_as(f32p), w.ctypes.data_as(f32p), None, 0, 7.0, y.ctypes.data_as(f32p))
        assert rc == 0, _lib.last_error()
        return y
    y = product(x, w)
    x[3, K // 2], x[40, 1] = np.inf, np.nan
    x[64] *= np.float32(2.0 ** -113)
    w[7, K - 1] = np.nan
    w[33] *= np.float32(2.0 ** -111)
    z = product(x, w)
    rows, cols = np.setdiff1d(np.arange(T), [3, 40, 64]), np.setdiff1d(np.arange(N), [7, 33])
    assert np.array_equal(z[np.ix_(rows, cols)], y[np.ix_(rows, cols)])
    assert np.isnan(z[40]).all() and np.isnan(z[:, 7]).all() and not np.isfinite(z[3]).any()
    tiny = np.ones((T, N), bool)
    tiny[[3, 40]], tiny[:, 7] = False, False
    tiny[np.ix_(rows, cols)] = False
    xe, we = np.nan_to_num(x.astype(np.float64), posinf=0.0), np.nan_to_num(w.astype(np.float64))
    off = (K + 8) * (2.0 ** -24 * (np.abs(xe) @ np.abs(we).T) + 6 * 2.0 ** -149) + 2.0 ** -133 * (np.abs(we).sum(1)[None, :] + np.abs(xe).sum(1)[:, None])
    assert (np.abs(z - xe @ we.T) <= off)[tiny].all()


@pytest.mark.parametrize("dtype", ["bfloat16", "float32"])
def test_attention_tiles_do_not_depend_on_rows_past_the_last_token(tmp_path, dtype):
    """the last tile of 16 tokens has rows that no token of the portion fills. They hold an earlier pass's queries, here infinite ones of a token whose queries overflow (its cached
    rows do not), and the portion's logits are those of a context that never saw it, bit for bit"""
    def edit(w):
        w["embed"][:, 0] = 0.0
        w["embed"][60, 0] = 1.0
        w["l0.mix.q"][:, 0] = 3e38
        w["l0.mix.dkv"][:, 0] = 0.0
    p = Pair(tmp_path, config([latent(heads=8, dim=8, rot_dim=16, vdim=8, kv_rank=64, window=0)]), dtype=dtype, n_ctx=96, edit=edit)
    toks = [t % 60 for t in p.tokens(70)]
    want = p.run(toks)
    other = engine.Context(p.model, 96)
    other.decode_rows(toks[:66] + [60] * 14, 0, [0])
    got = p.run(toks, ctx=other)
    assert np.isfinite(want).all() and np.array_equal(got, want)
    other.close()
    p.close()
