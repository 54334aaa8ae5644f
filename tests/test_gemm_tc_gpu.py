"""The prompt-sized products of K-quant matrices at the edges of their tiles, and where their sums are largest."""
import numpy as np
import pytest

import densecore_b200 as dc
from densecore_b200 import blocks as B

pytestmark = pytest.mark.gpu

Q4, Q6 = B.GGML_TYPE_Q4_K, B.GGML_TYPE_Q6_K


def check(got, want, t):
    if t == Q4:
        assert np.array_equal(got, want)
    else:       # equal integers, one float term per block where the oracle keeps eight partials: a few roundings of 2^-24 for each of up to eight blocks
        assert np.abs(got - want).max() <= 2e-6 * np.abs(want).max()


@pytest.mark.parametrize("t", [Q4, Q6])
@pytest.mark.parametrize("N,K", [(1, 256), (127, 768), (129, 512), (300, 1280)])
def test_edges_of_rows_tokens_and_blocks(ctx, oracle, t, N, K):
    """Lone and paired token tiles, full, ragged and empty at the end; rows on either side of the 128-row tile; even and odd numbers of blocks."""
    rng = np.random.default_rng(N + K)
    w = B.random_weight(rng, t, N, K)
    W = ctx.upload_weight(t, w, K, N)
    for M in (32, 33, 64, 65, 127, 128, 129, 193, 257):
        x = rng.normal(size=(M, K)).astype(np.float32)
        check(ctx.mul_mat(W, x), oracle.mul_mat(t, w, N, K, x), t)
    W.free()


@pytest.mark.parametrize("t", [Q4, Q6])
def test_largest_sums(ctx, oracle, t):
    """Codes, scales and minima at the ends of their ranges with activations that are all one value: block sums beyond 2^24."""
    N, K, M = 130, 512, 70
    rng = np.random.default_rng(7)
    nb = K // 256
    if t == Q4:
        blk = B.random_q4k(rng, N, K).reshape(N, nb, 144)
        hi = rng.integers(60, 64, size=(N, nb, 8), dtype=np.uint8)
        blk[:, :, 4:16] = B.pack_q4k_scales(hi, hi)
        blk[:, :, 16:] = rng.choice(np.array([0xFF, 0xFE, 0xEF], np.uint8), size=(N, nb, 128))
    else:
        blk = B.random_q6k(rng, N, K).reshape(N, nb, 210)
        blk[:, :, :192] = rng.choice(np.array([0x00, 0xFF], np.uint8), size=(N, nb, 1))      # every code -32 or every code 31
        blk[:, :, 192:208] = rng.choice(np.array([-128, -127, 127], np.int8), size=(N, nb, 1)).view(np.uint8)
    w = blk.reshape(N, -1)
    x = np.where(rng.random((M, K)) < 0.002, 0.5, 1.0).astype(np.float32) * rng.choice([-1.0, 1.0], size=(M, 1)).astype(np.float32)
    W = ctx.upload_weight(t, w, K, N)
    check(ctx.mul_mat(W, x), oracle.mul_mat(t, w, N, K, x), t)
    W.free()


@pytest.mark.parametrize("M", [70, 128, 200])
def test_q6k_block_sums_round_once(ctx, oracle, M):
    """Codes of 0, 1 and few others: a block's sum is small beside its parts (lower and upper bits), which pass 2^24.  The whole result, step by step:
    the sum as an integer, rounded once, times d yd, added in block order; to the bit."""
    N, K = 150, 768
    rng = np.random.default_rng(M)
    nb = K // 256
    blk = np.zeros((N, nb, 210), np.uint8)
    codes = rng.choice(np.array([32, 33, 34, 47, 31, 63]), p=[0.5, 0.4, 0.06, 0.02, 0.01, 0.01], size=(N, nb, 256))
    codes[N // 2:] = np.maximum(codes[N // 2:] - 32 * (rng.random((N - N // 2, nb, 1)) < 0.5), 0)        # and sums beyond 2^26
    q = codes.reshape(N, nb, 2, 4, 32)       # a half block's quadrants: lower bits of 0 and 2, 1 and 3 share bytes, upper bits of all four
    low, up = q & 15, q >> 4
    blk[:, :, :128] = np.stack([low[:, :, :, 0] | low[:, :, :, 2] << 4, low[:, :, :, 1] | low[:, :, :, 3] << 4], 3).reshape(N, nb, 128)
    blk[:, :, 128:192] = (up[:, :, :, 0] | up[:, :, :, 1] << 2 | up[:, :, :, 2] << 4 | up[:, :, :, 3] << 6).reshape(N, nb, 64)
    scale = rng.choice(np.array([127, 126, 125, -128], np.int8), p=[0.5, 0.3, 0.1, 0.1], size=(N, nb, 16))
    blk[:, :, 192:208] = scale.view(np.uint8)
    d = np.abs(rng.normal(0.0, 0.01, size=(N, nb))).astype(np.float16)
    blk[:, :, 208:] = d[:, :, None].view(np.uint8)
    x = np.abs(rng.normal(1.0, 0.1, size=(M, K))).astype(np.float32)
    yd, y, _ = oracle.q8k_fields(oracle.quantize_q8k(x))
    sums = np.einsum("nbv,mbv->nmb", ((codes - 32).reshape(N, nb, 16, 16) * scale[:, :, :, None].astype(np.int64)).reshape(N, nb, 256), y.astype(np.int64))
    lower = np.einsum("nbv,mbv->nmb", (((codes & 15) - 8).reshape(N, nb, 16, 16) * scale[:, :, :, None].astype(np.int64)).reshape(N, nb, 256), y.astype(np.int64))
    assert (np.abs(lower) > 1 << 24).mean() > 0.2 and (np.abs(sums) > 1 << 26).any() and (np.abs(sums) < 1 << 24).any()
    want = np.zeros((N, M), np.float32)
    for b in range(nb):
        want += d[:, None, b].astype(np.float32) * yd[None, :, b] * sums[:, :, b].astype(np.float32)
    W = ctx.upload_weight(Q6, blk.reshape(N, -1), K, N)
    got = ctx.mul_mat(W, x)
    W.free()
    assert np.array_equal(got, want.T)


@pytest.mark.parametrize("t", [Q4, Q6])
def test_unused_slots_may_hold_anything(ctx, oracle, t):
    """The last token tile's slots beyond the rows are not written: with the scratch full of NaN patterns (of f32 and of fp16) the results are the same bits."""
    N, K = 200, 512
    rng = np.random.default_rng(3)
    w = B.random_weight(rng, t, N, K)
    W = ctx.upload_weight(t, w, K, N)
    for M in (33, 65, 190):
        x = rng.normal(size=(M, K)).astype(np.float32)
        first = ctx.mul_mat(W, x)
        ctx.mul_mat(W, np.full((1024, K), 0xFFFFFFFF, np.uint32).view(np.float32))      # its inputs lie where the next call's activations will
        again = ctx.mul_mat(W, x)
        check(again, oracle.mul_mat(t, w, N, K, x), t)
        assert np.array_equal(again, first)
    W.free()


def test_unused_expert_slots_may_hold_anything(ctx):
    """A prompt through a mixture of experts whose buffers come out of memory full of NaN patterns, and out of zeros."""
    cfg = dc.Config(max_seqs=1, max_ctx=512, n_layer=2, hidden=512, n_head=4, n_kv_head=2, vocab=1000, n_expert=8, n_expert_used=2, expert_ffn=256)
    prompt = np.random.default_rng(5).integers(0, cfg.vocab, size=300)
    out = []
    for fill in (0, 0xFFFFFFFF):
        m = dc.Model(ctx, cfg)
        m.init_synthetic(11, 0.05)
        m.finalize()
        pattern = np.full(1 << 24, fill, np.uint32)
        blocks = [ctx.alloc(pattern.nbytes) for _ in range(16)]      # 1 GB, given back ahead of the prompt's buffers
        for b in blocks:
            ctx.to_device(b, pattern)
        for b in blocks:
            ctx.free(b)
        out.append(m.prefill(m.seq_alloc(), prompt, want_logits=True)[1].copy())
        m.close()
    assert np.isfinite(out[0]).all() and np.array_equal(out[0], out[1])
