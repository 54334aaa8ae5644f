"""Prompt attention of grouped-query layers on the tensor cores at the edges of its tiles: 128 queries, 64 keys, head sizes of 65 to 128."""
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
