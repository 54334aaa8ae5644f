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


@pytest.mark.parametrize("t", [B.GGML_TYPE_Q4_K, B.GGML_TYPE_Q6_K])
def test_block_sums_of_every_instance(ctx, oracle, t):
    """The exact integer sums of the instances that serve 1, 2, 3-4, 5-8 and 9-16 tokens, in groups of warps and alone."""
    for N, K in ((37, 1280), (9000, 256)):
        rng = np.random.default_rng(N + t)
        w = B.random_weight(rng, t, N, K)
        W = ctx.upload_weight(t, w, K, N)
        x = rng.normal(size=(16, K)).astype(np.float32)
        q8 = ctx.quantize_q8k(x).reshape(16, -1)
        rows = np.unique(np.concatenate([np.arange(min(N, 37)), rng.integers(N, size=20), [N - 1]]))
        want = [[oracle.block_sums(t, w.reshape(N, -1)[n], q8[m], K) for n in rows] for m in range(16)]
        for M in (1, 2, 3, 4, 5, 8, 9, 16):
            I, Mn = ctx.mul_mat_block_sums(W, x[:M])
            for m in range(M):
                assert np.array_equal(I[m][rows], np.stack([r[0] for r in want[m]])), (N, M, m)
                if t == B.GGML_TYPE_Q4_K:
                    assert np.array_equal(Mn[m][rows], np.stack([r[1] for r in want[m]])), (N, M, m)
        W.free()


@pytest.mark.parametrize("noalloc", [False, True])
@pytest.mark.parametrize("t,n,M", [(B.GGML_TYPE_Q4_K, 512, 12), (B.GGML_TYPE_Q6_K, 1024, 6), (B.GGML_TYPE_Q4_K, 6144, 1), (B.GGML_TYPE_Q4_K, 1024, 7)])
def test_product_in_place(ctx, t, n, M, noalloc):
    """Results stored over the rows themselves, and over their end: few rows (24 blocks or fewer, which the product would else quantise
    itself while others already store) and one block more."""
    rng = np.random.default_rng(n + M)
    W = ctx.upload_weight(t, B.random_weight(rng, t, n, n), n, n)
    x = rng.normal(size=(M, n)).astype(np.float32)
    want = ctx.mul_mat(W, x)
    buf = ctx.alloc(3 * x.nbytes)
    for shift in (0, x.nbytes - 4096, 4096 - x.nbytes) if M > 1 else (0, 1024, -1024):
        ctx.to_device(buf + x.nbytes, x)
        ctx.mul_mat_dev(W, buf + x.nbytes, M, buf + x.nbytes + shift, noalloc=noalloc)
        ctx.synchronize()
        assert np.array_equal(ctx.from_device(buf + x.nbytes + shift, np.empty((M, n), np.float32)), want), shift
    ctx.free(buf)
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


@pytest.mark.parametrize("E,k", [(1, 1), (2, 2), (16, 16), (31, 5), (32, 8), (33, 16), (100, 8), (128, 8), (255, 16), (256, 8)])
def test_routing_takes_the_best_experts_in_order(ctx, E, k):
    """Larger logit first, then lower id, NaN last: ties, both zeros, infinities and NaN at the edges of a warp's lanes.  Weights: a softmax
    over the picks, k terms of f32 exponentials (2 ulp each) and one division; equal shares where a pick is not finite."""
    rng = np.random.default_rng(E)
    for T in (1, 3, 8, 9, 16):
        lg = rng.integers(-3, 4, size=(T, E)).astype(np.float32) * np.float32(0.5)      # many ties
        lg[lg == 0] *= rng.choice([-1, 1])
        if T > 1:
            lg[1] = rng.normal(size=E)
            lg[1, rng.integers(E, size=3)] = np.nan
        if T > 2:
            lg[2] = rng.permutation(E)
            lg[2, [0, -1]] = np.inf, -np.inf
        ids, w = ctx.moe_route(lg, k)
        key = np.where(np.isnan(lg), -np.inf, lg).astype(np.float64)
        order = np.lexsort((np.broadcast_to(np.arange(E), lg.shape), -key, np.isnan(lg)), axis=-1)[:, :k]
        assert np.array_equal(ids.reshape(T, k), order), T
        v = np.take_along_axis(lg, order, 1).astype(np.float64)
        with np.errstate(invalid="ignore"):
            x = np.exp(v - v.max(1, keepdims=True))
            want = np.where(np.isfinite(v).all(1, keepdims=True), x / x.sum(1, keepdims=True), 1.0 / k)
        assert np.abs(w.reshape(T, k) - want).max() <= (k + 6) * 2.0 ** -24, T


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


@pytest.mark.parametrize("n_head,n_kv,T", [(32, 4, 2), (16, 2, 4), (16, 2, 16), (12, 2, 5), (32, 8, 4), (8, 4, 1)])
def test_cluster_attention_is_the_split_kernels_bit_for_bit(ctx, oracle, n_head, n_kv, T):
    """A table short enough for clusters of eight or sixteen CTAs, and one that takes the split kernels (more than 64 blocks a run would
    take the third form): the same runs, the same order of every sum, hence equal outputs.  Tokens of several sequences of unequal length,
    and neighbours in one sequence, whose rows the call itself writes."""
    rng = np.random.default_rng(n_head + T)
    scale, blocks = float(128 ** -0.5), 160
    small, large = (ctx.kv_cache(1, n_kv, 128, 17 * b, 17, b) for b in (blocks, 1024))
    lens = [int(x) for x in np.linspace(2300, 1, T)]
    seqs = [[c.seq_alloc() for _ in range(T + 1)] for c in (small, large)]
    for i, n in enumerate(lens + [1500]):
        k, v = (rng.normal(size=(n, n_kv, 128)).astype(np.float32) for _ in range(2))
        k *= np.linspace(0.2, 1.5, n)[:, None, None].astype(np.float32)      # the running maximum keeps moving
        for p in range(0, n, 16):
            m = min(16, n - p)
            for c, s in zip((small, large), seqs):
                c.flash_attn_decode(0, np.zeros((m, n_head, 128), np.float32), k[p:p + m], v[p:p + m], [s[i]] * m, list(range(p, p + m)), scale)
    q, k, v = (rng.normal(size=(T, h, 128)).astype(np.float32) for h in (n_head, n_kv, n_kv))
    for step in range(2):
        got, want = (c.flash_attn_decode(0, q, k, v, s[:T], [n + step for n in lens], scale) for c, s in zip((small, large), seqs))
        assert np.abs(got).max() > 0 and np.array_equal(got, want), step
    got, want = (c.flash_attn_decode(0, q, k, v, [s[T]] * T, list(range(1500, 1500 + T)), scale) for c, s in zip((small, large), seqs))
    assert np.abs(got).max() > 0 and np.array_equal(got, want)
    small.close()
    large.close()


def _prefilled(ctx, cfg, lens, seed=11):
    m = dc.Model(ctx, cfg)
    m.init_synthetic(5, 0.05)
    m.finalize()
    rng = np.random.default_rng(seed)
    seqs = [m.seq_alloc() for _ in lens]
    for s, n in zip(seqs, lens):
        m.prefill(s, rng.integers(0, cfg.vocab, size=n))
    return m, seqs


@pytest.mark.parametrize("n_head,n_kv,streams", [(32, 8, 4), (32, 8, 1), (16, 8, 3), (64, 8, 2)])
def test_fused_decode_steps_do_not_depend_on_the_table(ctx, n_head, n_kv, streams):
    """Steps of streams of unequal length, several blocks a CTA, with norm, rotation and cache write inside the attention kernel (table of
    3072 positions) and with the split kernels (16384 positions; 37 runs in both): equal logits, also for a chunk of one sequence."""
    lens = [1900, 1130, 517, 64][:streams]
    kw = dict(n_layer=2, hidden=512, n_head=n_head, n_kv_head=n_kv, vocab=1000, ffn=1024, max_seqs=4)
    toks = np.random.default_rng(3).integers(0, 1000, size=(3, 4))
    out = []
    for max_ctx in (3072, 16384):
        m, seqs = _prefilled(ctx, dc.Config(max_ctx=max_ctx, **kw), lens)
        lg = [m.decode_step(seqs, t[:streams], want_logits=True)[1] for t in toks]
        lg.append(m.forward_chunk(seqs[0], toks[0]))
        out.append((np.concatenate(lg), m.step_stats()[0]))
        m.close()
    assert np.array_equal(out[0][0], out[1][0])


@pytest.mark.parametrize("softmax", [0, 1])
@pytest.mark.parametrize("hidden,n_head,n_kv", [(2048, 32, 4), (512, 8, 2), (1024, 16, 8)])
def test_one_stream_has_the_persistent_kernels_results(ctx, hidden, n_head, n_kv, softmax):
    """By default one stream of a mixture-of-experts model runs as separate kernels, which form their sums (router logits, attention runs)
    as the persistent kernel does: the same logits bit for bit, whichever serves the step."""
    cfg = dc.Config(n_layer=2, hidden=hidden, n_head=n_head, n_kv_head=n_kv, vocab=1000, n_expert=24, n_expert_used=4, expert_ffn=512, max_seqs=2, max_ctx=2200)
    m, seqs = _prefilled(ctx, cfg, [2040, 70])
    m.set_option("route_mode", softmax)
    toks = np.random.default_rng(4).integers(0, 1000, size=(4, 2))
    res = {}
    for mode in (1, 2):
        m.set_option("persistent", mode)
        lg = [m.decode_step([s], [t[i]], want_logits=True)[1] for i, s in enumerate(seqs) for t in toks]
        res[mode] = (np.concatenate(lg), m.step_stats()[0])
        for s, n in zip(seqs, (2040, 70)):
            m.seq_truncate(s, n)
    assert res[2][1] == 1 < res[1][1], "the two runs must have taken different paths"
    assert np.array_equal(res[1][0], res[2][0])
    m.close()


@pytest.mark.parametrize("n_head,n_kv,max_ctx,streams,cluster", [(32, 16, 640, 1, True), (32, 16, 640, 4, False), (32, 16, 4096, 2, False), (16, 8, 4096, 4, False),
                                                                 (16, 8, 2112, 4, True), (16, 8, 2112, 16, True), (16, 8, 640, 16, False), (32, 4, 4096, 1, True)])
def test_attention_form_of_a_step(ctx, n_head, n_kv, max_ctx, streams, cluster):
    """The one-kernel form serves the steps for which it is the faster one, by streams, heads and length of the block table: a layer then has
    two launches less than with a table that only the split kernels take."""
    launches = []
    for n in (max_ctx, 32768):
        m, seqs = _prefilled(ctx, dc.Config(n_layer=2, hidden=512, n_head=n_head, n_kv_head=n_kv, vocab=1000, ffn=1024, max_seqs=16, max_ctx=n), [20] * streams)
        m.decode_step(seqs, [1] * streams)
        launches.append(m.step_stats()[0])
        m.close()
    assert launches[1] - launches[0] == (4 if cluster else 0)
