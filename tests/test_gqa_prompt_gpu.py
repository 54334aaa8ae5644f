"""Prompt attention of grouped-query layers on the tensor cores at the edges of its tiles: 128 queries, 64 keys, head sizes of 65 to 128."""
import copy
import re

import numpy as np
import pytest

import datasun_util as du
import densecore_b200 as dc
import gomuzen_util as gu
import vepitar_util as vu
from oracle import layers_ref as R
from stack_util import rel, write_model

pytestmark = pytest.mark.gpu

CASES = {
    "sink": (du, lambda w: du.config([du.attention(heads=4, kv_heads=2, dim=96, window=w)], ff=48)),
    "sigmoid": (vu, lambda w: vu.config([vu.attention(heads=8, kv_heads=2, dim=128, vdim=72, window=w)], [vu.dense(48)])),
    "kept": (gu, lambda w: gu.config([gu.kept(heads=4, kv_heads=1, dim=72, vdim=128, window=w, keep=3)], gu.moe())),
    # odd numbers of query heads a key head: the mma.sync kernel, which serves these head sizes too
    "sink_own_128": (du, lambda w: du.config([du.attention(heads=2, kv_heads=2, dim=128, window=w)], ff=48)),
    "kept_odd_64_128": (gu, lambda w: gu.config([gu.kept(heads=3, kv_heads=1, dim=56, vdim=128, window=w, keep=3)])),
    "kept_odd_128": (gu, lambda w: gu.config([gu.kept(heads=3, kv_heads=1, dim=128, vdim=128, window=w, keep=3)])),
    "sigmoid_odd_96": (vu, lambda w: vu.config([vu.attention(heads=3, kv_heads=1, dim=96, vdim=80, window=w)], [vu.dense(48)])),
    "sigmoid_odd_128": (vu, lambda w: vu.config([vu.attention(heads=3, kv_heads=1, dim=128, vdim=128, window=w)], [vu.dense(48)])),
}


@pytest.mark.parametrize("window", [1, 64, 200, 1000])
@pytest.mark.parametrize("name", list(CASES))
def test_prompt_attention_at_tile_edges(ctx, tmp_path, name, window):
    """Whole prompts and portions that end beside, on and past the tiles; several runs of one prompt agree bit for bit."""
    util, make = CASES[name]
    cfg = make(window)
    t = util.make_tensors(cfg, 5)
    rng = np.random.default_rng(window)
    tokens = rng.integers(0, cfg["vocab"], size=390)
    if util in (gu, vu):
        tokens, _ = util.settled_tokens(cfg, t, tokens, rng)
    want = R.Stepper(cfg, t).step(tokens)
    m = dc.Model.from_dir(ctx, write_model(tmp_path, cfg, t), "bfloat16", max_seqs=2, max_ctx=512)
    m.finalize()
    first = None
    for cuts in ((390,), (390,), (17, 111, 129, 133), (128, 65, 197), (127, 64, 199)):
        s, at, got = m.seq_alloc(), 0, []
        for n in cuts:
            got.append(m.forward_batch([(s, tokens[at:at + n])], np.arange(n)))
            at += n
        m.seq_free(s)
        got = np.concatenate(got)
        r = rel(got, want[:len(got)])
        assert np.median(r) < 2.5e-2 and r.max() < 0.12, (cuts, np.median(r), r.max())
        if len(cuts) == 1:
            assert first is None or np.array_equal(got, first)
            first = got
    m.close()


def with_own_key_heads(cfg, t):
    """The same model with a key head for every query head: copies of the key and value rows that it shares.  Such layers keep k_gqa_prompt."""
    cfg, t = copy.deepcopy(cfg), dict(t)
    for i, ly in enumerate(cfg["layers"]):
        m = ly["mixer"]
        for n in [n for n in t if re.fullmatch(rf"l{i}\.mix\.[kv](\.\w+)?", n)]:
            t[n] = np.repeat(t[n].reshape(m["kv_heads"], -1, *t[n].shape[1:]), m["heads"] // m["kv_heads"], axis=0).reshape(-1, *t[n].shape[1:])
        m["kv_heads"] = m["heads"]
    return cfg, t


def logits_in_steps(ctx, path, cfg, t, steps):
    """Logits of all tokens of all steps; a step: (sequence, tokens) pairs."""
    m = dc.Model.from_dir(ctx, write_model(path, cfg, t), "bfloat16", max_seqs=8, max_ctx=512)
    m.finalize()
    seqs = [m.seq_alloc() for _ in range(8)]
    out = [m.forward_batch([(seqs[i], tok) for i, tok in step], np.arange(sum(len(tok) for _, tok in step))) for step in steps]
    m.close()
    return np.concatenate(out)


def several_prompts(rng, vocab):
    """Steps of several entries: whole prompts, their next portions, single tokens among them."""
    lengths = ([300, 5, 130, 64, 1], [90, 123, 1, 65, 127], [1, 130, 129, 1, 17])
    return [[(i, rng.integers(0, vocab, size=n)) for i, n in enumerate(step)] for step in lengths]


BOTH = {
    "softmax": (gu, lambda w: gu.config([gu.kept(heads=4, kv_heads=1, dim=72, vdim=128, softcap=None, window=w, keep=3)])),
    "capped": (gu, lambda w: gu.config([gu.kept(heads=4, kv_heads=2, dim=128, vdim=96, window=w, keep=70)])),
    "sigmoid": (vu, lambda w: vu.config([vu.attention(heads=8, kv_heads=2, dim=128, vdim=72, window=w)], [vu.dense(48)])),
}


@pytest.mark.parametrize("window", [1, 40, 1000])
@pytest.mark.parametrize("name", list(BOTH))
def test_both_prompt_kernels_agree_bit_for_bit(ctx, tmp_path, name, window):
    """Shared key heads (tcgen05) against copies of them (mma.sync): the same products, weights and sums in the same order."""
    util, make = BOTH[name]
    cfg = make(window)
    t = util.make_tensors(cfg, 6)
    steps = several_prompts(np.random.default_rng(window), cfg["vocab"])
    shared = logits_in_steps(ctx, tmp_path / "shared", cfg, t, steps)
    own = logits_in_steps(ctx, tmp_path / "own", *with_own_key_heads(cfg, t), steps)
    assert np.isfinite(shared).all() and np.array_equal(shared, own)


@pytest.mark.parametrize("window", [1, 40, 1000])
@pytest.mark.parametrize("name", list(BOTH))
def test_infinite_values_stay_where_they_are_seen(ctx, tmp_path, name, window):
    """Token 0 has an infinite value row, which weights of zero turn into NaN: only queries that share its tile with keys that they see may meet it, in either kernel."""
    util, make = BOTH[name]
    cfg = make(window)
    t = util.make_tensors(cfg, 6)
    rng = np.random.default_rng(window)
    t["embed"][:, :2] = 0
    t["embed"][0, :2] = 4
    for n in t:
        if re.fullmatch(r"l0\.mix\.[qkg]", n):
            t[n][:, :2] = 0
    t["l0.mix.v"][:, :2] = 2.0 ** 127
    steps = [[(i, 1 + tok % (cfg["vocab"] - 1)) for i, tok in step] for step in several_prompts(rng, cfg["vocab"])]
    bad = {(0, 0): 250, (0, 2): 3, (1, 1): 100, (2, 2): 128}      # (step, entry): place of token 0
    for (i, j), at in bad.items():
        steps[i][j][1][at] = 0
    shared = logits_in_steps(ctx, tmp_path / "shared", cfg, t, steps)
    own = logits_in_steps(ctx, tmp_path / "own", *with_own_key_heads(cfg, t), steps)
    assert np.array_equal(shared, own, equal_nan=True)
    assert not np.isfinite(shared[250]).all() and np.isfinite(shared[:250 - 64 - 16]).all() and (window > 1 or np.isfinite(shared[256:300]).all())
