"""Whole models whose heads are 128 wide, or whose cached latent is a multiple of 64, so that their prompts and single tokens reach
the kernels that the other designs' small test models do not: attention with options, with a distance table, without
softmax, over one cached row, over a latent, differential.  Prompts of changing length in one padded shape, single tokens, and
portions beside single tokens, each shape run kernel by kernel, captured and replayed with another batch; every token's
logits against the plain implementation."""
import importlib

import numpy as np
import pytest

from helpers import bf16_noise, random_tokens

gpu = pytest.mark.gpu


def designs(P):
    if P.__name__ == "plain_tagulix":
        return P.make_config(vocab=96, width=64, mult=0.6, layers=[
            P.attention_layer(4, 2, 128, 128, window=70, rot=(16, 10000.0)),
            P.parallel_layer(4, 2, 128, 128, bias_max=100, lin_heads=2, lin_dim=32, lin_vdim=64, decay=[0.7, 0.99], temp=(0.3, 33))])
    if P.__name__ == "plain_gamanex":
        return P.make_config(vocab=96, width=64, layers=[
            P.attention_layer(4, 2, 128, 128, scale=0.1, temp=(0.25, 64), mlp=P.dense(96)),
            P.attention_layer(2, 2, 128, 128, scale=0.1, kv_from=0)])
    if P.__name__ == "plain_losalorn":
        return P.make_config(vocab=96, width=64, emb_scale=2.0, cap=20.0, loop=(0, 1, 2), layers=[
            P.attention_layer(4, 2, 128, window=90, rot=16, base=10000.0, scale=0.1, mlp=P.dense(96, 1.0)),
            P.attention_layer(4, 1, 128, rot=64, base=500.0, scale=0.1)])
    if P.__name__ == "plain_pirerax":
        return P.make_config(vocab=96, width=64, layers=[
            P.attention_layer(4, 2, 128, 128, 0.1, temp=(0.4, 24)),
            P.latent_layer(4, 32, 64, 32, 128, 0.1, base=500.0)])
    return P.make_config(vocab=96, width=128, scale=0.8, layers=[
        P.attention_layer(4, 2, 64, 128, chunk=100, softcap=30.0, diff=0.2, ff=96, limit=1.0),
        P.gla_layer(2, 32, 64, tau=12.0)])


REACHED = {"tagulix": ("attn_prompt_kind", "attn_single_kind"), "gamanex": ("attn_prompt_kind", "attn_single_kind"),
           "losalorn": ("attn_prompt_kind", "attn_single_kind"), "pirerax": ("attn_prompt_kind", "attn_single_kind", "latent_prefill_tc"),
           "vedizen": ("diff_prefill_tc",)}


@pytest.fixture(scope="module")
def models(tmp_path_factory):
    made = {}

    def model(name):
        if name not in made:
            P = importlib.import_module("plain_" + name)
            cfg = designs(P)
            W = P.random_weights(cfg, seed=3)
            made[name] = importlib.import_module("test_" + name), cfg, W, P.write_folder(str(tmp_path_factory.mktemp("m")), cfg, W)
        return made[name]

    return model


def spied(monkeypatch, names):
    """Counts the calls of these wrappers that took their work."""
    from airun_b200.kernels import fast
    took = {n: 0 for n in names}

    def spy(name, real):
        def call(*a, **k):
            got = real(*a, **k)
            took[name] += bool(got)
            return got
        return call

    for n in names:
        monkeypatch.setattr(fast, n, spy(n, getattr(fast, n)))
    return took


def check(T, cfg, W, got, seqs, what):
    """The noise of a row is how far rounding alone moves it (helpers.bf16_noise).  A few rows of these designs lie where a
    normed difference is nearly nothing and rounding moves them several times further from one kernel to the next (three
    noises, the mma.sync kernels alike), so a row is held to six of them and a sequence as a whole to its noise; rows that
    ran over another tile, page or request are off by the size of the logits, tens of noises."""
    first = lambda r: (r[0] if isinstance(r, tuple) else r).numpy()
    for i, s in enumerate(seqs):
        exact, rounded = first(T.P.plain_forward(cfg, W, s)), first(T.P.plain_forward(cfg, W, s, rnd=T.P.to_bf16_and_back))
        noise = bf16_noise(rounded, exact)
        bound = 6.0 * np.maximum(noise, 0.25 * np.median(noise)) + 1e-3
        err = np.abs(got[i] - rounded)
        assert np.isfinite(got[i]).all() and (err <= bound).all(), (what, i, float((err / bound).max()), int((err / bound).max(axis=1).argmax()))
        assert np.sqrt((err ** 2).mean()) <= np.sqrt((noise ** 2).mean()) + 1e-4, (what, i)


@gpu
@pytest.mark.parametrize("name", list(REACHED))
def test_prompts_single_tokens_and_both_from_graphs(models, name, monkeypatch):
    T, cfg, W, folder = models(name)
    took = spied(monkeypatch, REACHED[name])
    eng = T.engine(folder, "bfloat16", 16, tokens=2048, batch=512, reqs=6)
    schedule = [[(0, 260)], [(1, 290)], [(2, 333)]]                                    # prompts: eager, captured, replayed
    schedule += [[(0, 1), (1, 1), (2, 1)] for _ in range(3)]                           # single tokens
    schedule += [[(0, 1), (3, 300), (1, 1)], [(2, 1), (4, 257), (0, 1)], [(1, 1), (2, 1), (5, 350)]]      # portions beside them
    schedule += [[(5, 1), (4, 1), (3, 1), (2, 1)], [(3, 200), (4, 190)], [(0, 1), (1, 1), (5, 1)]]
    lens = {}
    for step in schedule:
        for i, n in step:
            lens[i] = lens.get(i, 0) + n
    seqs = [random_tokens(lens[i], cfg["vocab"], 70 + i) for i in sorted(lens)]
    got = T.run_schedule(eng, seqs, schedule)
    assert eng.runner.graph_launches > 0 and all(took.values()), took
    check(T, cfg, W, got, seqs, name)


@gpu
@pytest.mark.parametrize("name", ["pirerax", "tagulix"])
def test_many_prompts_of_a_new_shape_behind_another_prompt(models, name, monkeypatch):
    """29 requests' prompts in one step, whose list of tiles is new, right behind a prompt whose list lies where it goes."""
    T, cfg, W, folder = models(name)
    took = spied(monkeypatch, [n for n in REACHED[name] if n != "attn_single_kind"])
    eng = T.engine(folder, "bfloat16", 16, tokens=8192, batch=1024, reqs=32)
    one = [[(0, 500)], [(1, 480)]]
    waves = [[(2 + 29 * w + i, 3 + (7 * i + 11 * w) % 50) for i in range(29)] for w in range(3)]
    schedule = [one[0], waves[0], one[1], waves[1], waves[2]]
    lens = {i: n for step in schedule for i, n in step}
    seqs = [random_tokens(lens[i], cfg["vocab"], 700 + i) for i in sorted(lens)]
    got = T.run_schedule(eng, seqs, schedule)
    assert all(took.values()), took
    check(T, cfg, W, got, seqs, name)
