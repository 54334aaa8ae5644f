"""Decode kernels at the sizes where they can go wrong: K-quant rows on the integer tensor instructions (ragged tiles, rows of every
number of super-blocks that splits differently over warps, every class of token counts), expert rows, the cluster attention kernel
against the split kernels and the oracle, and the fused decode step against the chunk path."""
import numpy as np
import pytest

import densecore_b200 as dc
from densecore_b200 import blocks as B

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = dc.Context(0)
    yield c
    c.close()


@pytest.fixture(scope="module")
def oracle():
    from oracle import oracle as o
    o.set_threads(min(8, o.max_threads()))
    return o


@pytest.mark.parametrize("t", [B.GGML_TYPE_Q4_K, B.GGML_TYPE_Q6_K])
@pytest.mark.parametrize("N,K", [(1, 256), (15, 512), (16, 768), (17, 1280), (333, 2048), (2050, 1024), (130, 4352), (33, 8448), (16, 16384), (9000, 256)])
def test_rows_are_the_cpu_kernels_bit_for_bit(ctx, oracle, t, N, K):
    """Sums of exact integers and the CPU kernels' float order: equality, for every class of token counts and its edges."""
    rng = np.random.default_rng(N * 7 + K + t)
    w = B.random_weight(rng, t, N, K)
    W = ctx.upload_weight(t, w, K, N)
    x = rng.normal(size=(16, K)).astype(np.float32)
    x[3, :256] = 0.0                                    # a block whose scale is zero
    want = oracle.mul_mat(t, w, N, K, x)
    for M in (1, 2, 3, 4, 5, 8, 9, 15, 16):
        assert np.array_equal(ctx.mul_mat(W, x[:M]), want[:M]), M
    W.free()


@pytest.mark.parametrize("E,F,H,k,down", [(3, 256, 512, 2, B.GGML_TYPE_Q6_K), (128, 768, 512, 8, B.GGML_TYPE_Q6_K), (200, 256, 1280, 16, B.GGML_TYPE_Q4_K)])
def test_expert_rows_match_rows_of_single_tokens(ctx, E, F, H, k, down):
    """A token's result does not depend on the tokens beside it, up to the order in which its experts' outputs are added (routing order
    for few tokens, ascending experts for more): sums of at most sixteen f32 terms, 16 x 2^-24 of the largest."""
    rng = np.random.default_rng(E + F)
    up = lambda t, n, kk: ctx.upload_weight(t, B.random_weight(rng, t, E * n, kk), kk, n, E)      # noqa: E731
    W = [ctx.upload_weight(B.GGML_TYPE_F32, rng.normal(size=(E, H)).astype(np.float32) * 0.05, H, E), up(B.GGML_TYPE_Q4_K, F, H), up(B.GGML_TYPE_Q4_K, F, H), up(down, H, F)]
    x = rng.normal(size=(16, H)).astype(np.float32)
    x[9] = x[2]                                         # two tokens with the same experts
    one = [ctx.mul_mat_id(*W, x[i:i + 1], k) for i in range(16)]
    for T in (2, 3, 4, 5, 8, 11, 16):
        y, ids, wt = ctx.mul_mat_id(*W, x[:T], k)
        assert np.array_equal(ids, np.concatenate([o[1] for o in one[:T]])), T
        want = np.concatenate([o[0] for o in one[:T]])
        assert np.abs(y - want).max() <= 16 * 2.0 ** -24 * np.abs(want).max() * k, T
    for w in W:
        w.free()


@pytest.mark.parametrize("n_head,n_kv,blocks", [(32, 4, 176), (16, 8, 130), (12, 2, 512), (64, 16, 256)])
def test_cluster_attention_against_split_kernels_and_oracle(ctx, oracle, n_head, n_kv, blocks):
    """The same keys in a cache short enough for the cluster kernel and in one that is not; lengths at which a CTA of the cluster gets
    no block, one key, or a full share.  Gate 1e-5 as for the split kernels: f32 sums in another order."""
    rng = np.random.default_rng(n_head)
    scale = float(128 ** -0.5)
    small, large = ctx.kv_cache(1, n_kv, 128, blocks, 1, blocks), ctx.kv_cache(1, n_kv, 128, 600, 1, 600)
    a, b = small.seq_alloc(), large.seq_alloc()
    n = blocks * 16
    k, v = (rng.normal(size=(n, n_kv, 128)).astype(np.float32) for _ in range(2))
    k *= np.linspace(0.2, 1.5, n)[:, None, None].astype(np.float32)      # the running maximum keeps moving
    at = [0, 1, 15, 16, 17, 127, 128, 129, 255, 256, 640, 2047, 2048, 2049, n - 1] if blocks == 176 else [0, 16, 255, 1500, n - 1]
    rk, rv = np.zeros((n, n_kv, 128), np.uint16), np.zeros((n, n_kv, 128), np.uint16)
    done = 0
    for pos in at:
        for i in range(done, pos, 16):                  # fill the cache up to pos
            m = min(16, pos - i)
            q0 = np.zeros((m, n_head, 128), np.float32)
            for c, s in ((small, a), (large, b)):
                c.flash_attn_decode(0, q0, k[i:i + m], v[i:i + m], [s] * m, list(range(i, i + m)), scale)
        q = rng.normal(size=(1, n_head, 128)).astype(np.float32)
        got, split = (c.flash_attn_decode(0, q, k[pos:pos + 1], v[pos:pos + 1], [s], [pos], scale) for c, s in ((small, a), (large, b)))
        rk[done:pos + 1], rv[done:pos + 1] = k[done:pos + 1].astype(np.float16).view(np.uint16), v[done:pos + 1].astype(np.float16).view(np.uint16)
        done = pos + 1
        want = oracle.paged_attention(q[0], rk, rv, np.arange(blocks, dtype=np.int32), pos, n_head, n_kv, 128, scale, "blockwise")
        top = np.abs(want).max()
        assert np.abs(got[0] - want).max() < 1e-5 * top, pos
        assert np.abs(got - split).max() < 1e-5 * top, pos
    small.close()
    large.close()


@pytest.mark.parametrize("moe", [True, False])
def test_decode_steps_are_the_chunk_path_bit_for_bit(ctx, moe):
    """Tokens one at a time and in two sequences (norm, rotation and cache write inside the attention kernel) and as chunks of one
    sequence (kernels of their own): the same arithmetic, hence the same logits."""
    kw = dict(n_expert=16, n_expert_used=4, expert_ffn=256) if moe else dict(ffn=1024)
    m = dc.Model(ctx, dc.Config(n_layer=3, hidden=512, n_head=8, n_kv_head=2, vocab=1000, max_seqs=4, max_ctx=256, **kw))
    m.init_synthetic(5, 0.05)
    m.finalize()
    m.set_option("persistent", 0)
    rng = np.random.default_rng(8)
    prompt, toks = rng.integers(0, 1000, size=37), rng.integers(0, 1000, size=(4, 2))
    s = [m.seq_alloc() for _ in range(4)]
    for q in s:
        m.prefill(q, prompt)
    chunk = m.forward_chunk(s[0], toks[:, 0]), m.forward_chunk(s[1], toks[:, 1])
    steps = [m.decode_step(s[2:], t, want_logits=True)[1] for t in toks]
    for i in range(4):
        for j in range(2):
            assert np.array_equal(chunk[j][i], steps[i][j]), (i, j)
    m.seq_truncate(s[0], 37)
    for i in range(4):
        assert np.array_equal(m.decode_step(s[:1], [toks[i, 0]], want_logits=True)[1][0], chunk[0][i]), i
    m.close()
