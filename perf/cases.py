"""The work that programs have this library do, as cases that can be timed and compared.

  product  MUL_MAT of a Q4_K or Q6_K matrix: one row (decode), a few rows (streams, verify), a prompt's rows
  experts  one mixture-of-experts feed-forward layer on up to sixteen tokens
  decode   steps of a decoder on one or several sequences that already hold a prompt, the caller choosing the tokens
  prompt   a prompt on a fresh sequence of a decoder, up to the logits of its last token

Decoders: the quantized mixture-of-experts and dense ones, and the layer-list ones (Garilix, Datasun, Gomuzen, Vepitar).
"""
import math

import numpy as np
import torch

import densecore_b200 as dc

GPU = torch.device("cuda")
F8 = torch.float64
BLOCK = {"q4_k": (dc.GGML_TYPE_Q4_K, 144), "q6_k": (dc.GGML_TYPE_Q6_K, 210)}
HIDDEN, EXPERTS, TOP, EXPERT_FF, VOCAB = 2048, 128, 8, 768, 151936      # of the mixture-of-experts decoder
LISTED_LAYERS = 12      # of a layer-list decoder
STEPS = 8               # of a decode case
EXACT_LAYERS = 12       # deepest quantized decoder whose logits rounding leaves near those of 64 bits


# ------------------------------------------------------------------------------------------------- the cases
def listed():
    return [
        # the projection of one token: the smallest call, where latency counts
        {"name": "row_q4k", "kind": "product", "type": "q4_k", "N": 6144, "K": 2048, "M": 1},
        # the output matrix for five tokens: what verifying four drafted tokens ends with
        {"name": "verify_head_q6k", "kind": "product", "type": "q6_k", "N": VOCAB, "K": 2048, "M": 5},
        # a projection of a prompt whose length is no multiple of anything
        {"name": "prompt_rows_q4k", "kind": "product", "type": "q4_k", "N": 4096, "K": 2048, "M": 1531},
        # the expert layer of a step with several streams or drafted tokens
        {"name": "experts_t12", "kind": "experts", "T": 12},
        # the headline workload: greedy or sampled generation after a long prompt, one request
        {"name": "moe_decode_1", "kind": "decode", "model": "moe", "layers": 48, "context": 2048, "seqs": 1},
        # the same with four concurrent requests
        {"name": "moe_decode_4", "kind": "decode", "model": "moe", "layers": 48, "context": 2048, "seqs": 4},
        # time to first token of that decoder
        {"name": "moe_prompt", "kind": "prompt", "model": "moe", "layers": 48, "tokens": 2011},
        # the small dense decoder, alone or as a draft model
        {"name": "dense_decode_1", "kind": "decode", "model": "dense", "layers": 28, "context": 512, "seqs": 1},
        # one architecture of the layer-list decoders each, prompts and decoding in turn
        {"name": "garilix_decode_1", "kind": "decode", "model": "garilix", "width": 2048, "context": 1500, "seqs": 1},
        {"name": "datasun_prompt", "kind": "prompt", "model": "datasun", "width": 2048, "tokens": 2048},
        {"name": "gomuzen_decode_4", "kind": "decode", "model": "gomuzen", "width": 2048, "context": 1024, "seqs": 4},
        {"name": "vepitar_prompt", "kind": "prompt", "model": "vepitar", "width": 2048, "tokens": 1357},
    ]


def spread(rng, lo, hi):
    """A whole number from lo to hi, even over the logarithm."""
    return min(hi, max(lo, round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def draw(rng):
    kind = rng.choice(["product", "product", "product", "experts", "decode", "decode", "decode", "prompt", "prompt"])
    if kind == "product":
        t = rng.choice(["q4_k", "q6_k"])
        if rng.random() < 0.65:         # a step's rows
            return {"kind": kind, "type": t, "N": spread(rng, 512, VOCAB), "K": 256 * spread(rng, 3, 16), "M": spread(rng, 1, 16)}
        return {"kind": kind, "type": t, "N": spread(rng, 512, 8192), "K": 256 * spread(rng, 3, 16), "M": spread(rng, 17, 2048)}
    if kind == "experts":
        return {"kind": kind, "T": rng.randint(1, 16)}
    model = rng.choice(["moe", "moe", "dense", "dense", "garilix", "datasun", "gomuzen", "vepitar"])
    case = {"kind": kind, "model": model}
    if model == "moe":
        case["layers"] = rng.randint(4, 16)
    elif model == "dense":
        case["layers"] = 28
    else:
        case["width"] = rng.choice([1024, 1536, 2048])
    if kind == "decode":
        case.update(context=spread(rng, 64, 2048), seqs=rng.choice([1, 1, 2, 3, 4, 4]))
    else:
        case["tokens"] = spread(rng, 48, 2048)
    return case


# -------------------------------------------------------------------------------------------- seeded values
class Values:
    """Random values on the GPU; every name has a stream of its own."""

    def __init__(self, seed):
        self.seed = seed

    def of(self, name):
        h = 2166136261
        for b in ("%d/%s" % (self.seed, name)).encode():
            h = (h ^ b) * 16777619 % (1 << 32)
        return torch.Generator(GPU).manual_seed(h)

    def normal(self, name, *shape):
        return torch.randn(*shape, generator=self.of(name), device=GPU)

    def below(self, name, hi, *shape):
        return torch.randint(0, hi, shape, generator=self.of(name), device=GPU)

    def blocks(self, name, kind, rows, K):
        """Rows of random super-blocks: codes and scales over their whole range, fp16 block scales |N(0, 0.01)|."""
        n = rows * (K // 256)
        b = self.below(name, 256, n, BLOCK[kind][1]).to(torch.uint8)
        half = (0.01 * self.normal(name + ".d", n, 2)).abs().half().view(torch.uint8).reshape(n, 4)
        if kind == "q4_k":
            b[:, :4] = half
        else:
            b[:, 192:208] = self.below(name + ".s", 64, n, 16).sub(32).to(torch.int8).view(torch.uint8)
            b[:, 208:] = half[:, :2]
        return b.reshape(rows, -1)


# ---------------------------------------------------------------------------------------- K-quants in 64 bits
def halves(b):
    return b.contiguous().view(torch.float16).to(F8)


def dequantize(kind, blocks, K):
    """Super-blocks [rows, bytes] -> values [rows, K]."""
    b = blocks.reshape(-1, BLOCK[kind][1])
    n = b.shape[0]
    if kind == "q4_k":
        d, m, s = halves(b[:, 0:2]), halves(b[:, 2:4]), b[:, 4:16].int()
        lo, mid, hi = s[:, 0:4], s[:, 4:8], s[:, 8:12]
        scale = torch.cat([lo & 63, (hi & 15) | ((lo >> 6) << 4)], 1).to(F8) * d
        least = torch.cat([mid & 63, (hi >> 4) | ((mid >> 6) << 4)], 1).to(F8) * m
        q = b[:, 16:].reshape(n, 4, 1, 32)
        q = torch.cat([q & 15, q >> 4], 2).reshape(n, 8, 32).to(F8)
        return (q * scale[:, :, None] - least[:, :, None]).reshape(-1, K)
    ql, qh = b[:, :128].reshape(n, 2, 2, 32).int(), b[:, 128:192].reshape(n, 2, 32).int()
    q = torch.stack([(ql[:, :, 0] & 15) | ((qh & 3) << 4), (ql[:, :, 1] & 15) | ((qh >> 2 & 3) << 4),
                     (ql[:, :, 0] >> 4) | ((qh >> 4 & 3) << 4), (ql[:, :, 1] >> 4) | ((qh >> 6) << 4)], 2) - 32
    scale = b[:, 192:208].contiguous().view(torch.int8).to(F8) * halves(b[:, 208:210])
    return (q.to(F8).reshape(n, 16, 16) * scale[:, :, None]).reshape(-1, K)


def silu(z):
    return z * torch.sigmoid(z)


def rms(x, w, eps):
    return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + eps) * w


def swiglu_experts(x, logits, top, gate, up, down):
    """x [T, H]; gate(e), up(e), down(e) give an expert's matrices; weights are the softmax over the chosen experts' logits."""
    z, ids = logits.topk(top, dim=1)
    w, y = torch.softmax(z, 1), torch.zeros_like(x)
    for e in ids.unique().tolist():
        t, k = (ids == e).nonzero(as_tuple=True)
        h = silu(x[t] @ gate(e).T) * (x[t] @ up(e).T)
        y.index_add_(0, t, w[t, k][:, None] * (h @ down(e).T))
    return y


# ------------------------------------------------------------------------------------------ single operations
def product_inputs(case, seed):
    v = Values(seed)
    return v.blocks("w", case["type"], case["N"], case["K"]), v.normal("x", case["M"], case["K"])


def experts_inputs(case, seed):
    v = Values(seed)
    return {"router": 0.02 * v.normal("router", EXPERTS, HIDDEN), "gate": v.blocks("gate", "q4_k", EXPERTS * EXPERT_FF, HIDDEN),
            "up": v.blocks("up", "q4_k", EXPERTS * EXPERT_FF, HIDDEN), "down": v.blocks("down", "q6_k", EXPERTS * HIDDEN, EXPERT_FF)}, v.normal("x", case["T"], HIDDEN)


class Product:
    """A matrix on the GPU, rows in and rows out in the caller's device memory."""

    def __init__(self, case, seed):
        self.ctx = dc.Context(0)
        blocks, self.x = product_inputs(case, seed)
        self.w = self.ctx.upload_weight(BLOCK[case["type"]][0], blocks.cpu().numpy(), case["K"], case["N"])
        self.y = torch.empty(case["M"], case["N"], device=GPU)
        torch.cuda.synchronize()

    def run(self):
        self.ctx.mul_mat_dev(self.w, self.x.data_ptr(), self.x.shape[0], self.y.data_ptr())
        return self.y

    def __del__(self):
        self.w.free()
        self.ctx.close()


class Experts:
    def __init__(self, case, seed):
        self.ctx = dc.Context(0)
        t, self.x = experts_inputs(case, seed)
        q4, q6 = dc.GGML_TYPE_Q4_K, dc.GGML_TYPE_Q6_K
        self.w = [self.ctx.upload_weight(dc.GGML_TYPE_F32, t["router"].cpu().numpy(), HIDDEN, EXPERTS),
                  self.ctx.upload_weight(q4, t["gate"].cpu().numpy(), HIDDEN, EXPERT_FF, EXPERTS),
                  self.ctx.upload_weight(q4, t["up"].cpu().numpy(), HIDDEN, EXPERT_FF, EXPERTS),
                  self.ctx.upload_weight(q6, t["down"].cpu().numpy(), EXPERT_FF, HIDDEN, EXPERTS)]
        self.y = torch.empty_like(self.x)
        self.ids = torch.empty(case["T"], TOP, dtype=torch.int32, device=GPU)
        torch.cuda.synchronize()

    def run(self):
        self.ctx.mul_mat_id_dev(*self.w, self.x.data_ptr(), self.x.shape[0], TOP, self.y.data_ptr(), ids_dev=self.ids.data_ptr())
        return {"y": self.y, "ids": self.ids}

    def __del__(self):
        for w in self.w:
            w.free()
        self.ctx.close()


# ------------------------------------------------------------------------------------------- layer-list models
def family_config(name, width):
    """(config, shapes that it leaves open) of a decoder with the layer sizes of a real one of this width."""
    h, g = width // 128, max(1, width // 512)
    rot = {"base": 10000.0, "dims": 64}
    yarn = dict(rot, scaling={"factor": 2.0, "original": 2048, "fast": 32.0, "slow": 1.0})
    c = {"architecture": name.capitalize(), "vocab": 32768, "width": width, "norm": {"eps": 1e-5}}
    shapes = {}
    if name == "garilix":
        latent = {"heads": h, "dim": 128, "rot_dim": 64, "vdim": 128, "kv_rank": 512, "scale": 192 ** -0.5, "mask": {"size": 1024}, "rot": rot}
        kinds = [("channel_delta", {"heads": h, "kv_heads": h, "dim": 128, "vdim": 128, "conv": 4}), ("latent_attention", latent),
                 ("mamba2", {"heads": 2 * width // 64, "vdim": 64, "state": 128, "groups": 8, "norm_groups": 8, "conv": 4})]
        mlp = {"kind": "dense", "ff": 3 * width}
    elif name == "datasun":
        light = ("lightning", {"heads": h, "dim": 128, "vdim": 128, "decay": [math.exp(-8.0 * 0.5 ** (i * 10.0 / h)) for i in range(h)]})
        kinds = [light, light, ("attention", {"heads": h, "kv_heads": g, "dim": 128, "vdim": 128, "scale": 128 ** -0.5, "mask": {"size": 1024}, "rot": yarn})]
        mlp = {"kind": "dense", "ff": 3 * width, "limit": 7.0}
        c["embedding"] = {"scale": 1.0}
    elif name == "gomuzen":
        kept = ("attention_2", {"heads": h, "kv_heads": g, "dim": 128, "vdim": 128, "scale": 128 ** -0.5, "softcap": 50.0,
                                "mask": {"size": 1024, "keep_first": 4}, "rot": yarn})
        kinds = [("latent_attention", {"heads": h, "dim": 128, "rot_dim": 64, "vdim": 128, "kv_rank": 512, "scale": 192 ** -0.5, "rot": rot}),
                 ("attention", {"heads": h, "kv_heads": g, "dim": 64, "vdim": 128, "diff": 0.5, "scale": 0.125, "softcap": 30.0, "rot": rot}), kept, kept]
        mlp = {"kind": "moe", "expert": {"ff": 3 * width // 8, "limit": 7.0},
               "router": {"experts": 64, "top": 8, "scale": 2.0, "groups": {"count": 8, "keep": 4}}}
        c["loop"] = {"start": 0, "stop": 4, "times": 2}
    else:
        rec = ("general_delta", {"heads": width // 64, "dim": 64})
        kinds = [rec, rec, ("attention", {"heads": h, "kv_heads": g, "dim": 128, "vdim": 128, "conv": 4, "scale": 128 ** -0.5, "mask": {"size": 1024}})]
        mlp = {"kind": "moe", "expert": {"ff": 9 * width // 16}, "router": {"experts": 64, "top": 8}}
        c.update(streams=4, residual_mult=0.5)
    n = LISTED_LAYERS - (4 if "loop" in c else 0)
    c["layers"] = [{"type": kinds[i % len(kinds)][0], "mixer": dict(kinds[i % len(kinds)][1]), "mlp": mlp} for i in range(n)]
    if name == "vepitar":
        c["layers"][0]["mlp"] = {"kind": "dense", "ff": 3 * width}
    for i, ly in enumerate(c["layers"]):
        if ly["type"] == "channel_delta":
            shapes["l%d.mix.a1" % i] = shapes["l%d.mix.g1" % i] = [128, width]
        if ly["type"] == "general_delta":
            shapes["l%d.mix.w1" % i] = [max(32, width // 32), width]
        if name == "garilix" and i % 6 == 4:        # every second attention layer reads the cache of the one before
            ly["mixer"]["kv_from"] = i - 3
    return c, shapes


class Tensors:
    """The decoder's bf16 tensors by name, made when asked for.  Where there are experts, the last dimensions of the residual hold a
    code of the token that sublayers leave alone and that routers read, so that choices have margins, as trained ones have."""

    def __init__(self, name, width, seed):
        self.c, self.shapes = family_config(name, width)
        self.v, self.W = Values(seed), width
        self.codes = max(ly["mlp"]["router"]["experts"] if ly["mlp"]["kind"] == "moe" else 0 for ly in self.c["layers"])
        self.made = {}
        self.vec("final.norm", width, 0.0 if name == "vepitar" else 1.0)
        e = self.v.normal("embed", self.c["vocab"], width)
        if self.codes:
            order = torch.rand(self.c["vocab"], self.codes, generator=self.v.of("codes"), device=GPU).argsort(1)
            e[:, width - self.codes:] = torch.linspace(-2.0, 2.0, self.codes, device=GPU)[order]
        self.put("embed", e)
        if name in ("garilix", "gomuzen"):
            self.mat("head", self.c["vocab"], width)
        if "loop" in self.c:
            s = 0.7 * self.v.normal("loop.step", self.c["loop"]["times"], width)
            s[:, width - self.codes:] *= 0.1
            self.put("loop.step", s)
        for i, ly in enumerate(self.c["layers"]):
            p = "l%d." % i
            self.vec(p + "norm1", width, 0.0 if name == "vepitar" else 1.0, 0.1)
            getattr(self, ly["type"])(p + "mix.", ly["mixer"], i)
            if name != "datasun":
                self.vec(p + "norm2", width, 0.0 if name == "vepitar" else 1.0, 0.1)
            if name == "vepitar":
                self.streams(p + "hc1.")
                self.streams(p + "hc2.")
            self.feed_forward(p + "mlp.", ly["mlp"], gated=name == "gomuzen")

    def put(self, name, x):
        self.made[name] = x.to(torch.bfloat16)

    def mat(self, name, n, k, gain=1.0, to_residual=False):
        x = self.v.normal(name, n, k) * (gain / math.sqrt(k))
        if to_residual and self.codes:
            x[n - self.codes:] = 0
        self.put(name, x)

    def vec(self, name, n, mean=1.0, dev=0.2):
        self.put(name, mean + dev * self.v.normal(name, n))

    def taps(self, name, n, k):
        x = 0.4 * self.v.normal(name, n, k)
        x[:, -1] += 1.0
        self.put(name, x)

    def streams(self, p):
        n = self.c["streams"]
        self.vec(p + "in", n, 1.0 / n, 0.3 / n)
        self.vec(p + "out", n, 1.0, 0.5)
        self.put(p + "mix", 0.75 * torch.eye(n, device=GPU) + 0.25 / n + 0.1 / n * self.v.normal(p + "mix", n, n))

    def feed_forward(self, p, mlp, gated):
        if mlp["kind"] == "dense":
            self.mat(p + "gate", mlp["ff"], self.W, 1.5)
            self.mat(p + "up", mlp["ff"], self.W, 1.5)
            self.mat(p + "down", self.W, mlp["ff"], 1.0, True)
            return
        E, ff = mlp["router"]["experts"], mlp["expert"]["ff"]
        r = 0.02 * self.v.normal(p + "router", E, self.W) / math.sqrt(self.W)
        r[:, self.W - E:] += 1.5 * torch.eye(E, device=GPU)[torch.randperm(E, generator=self.v.of(p + "order"), device=GPU)]
        self.put(p + "router", r)
        if gated:
            self.vec(p + "correction", E, 0.0, 0.15)
        for e in range(E):
            for n in ("gate", "up") if gated else ("up",):
                self.mat("%se%d.%s" % (p, e, n), ff, self.W, 1.5)
            self.mat("%se%d.down" % (p, e), self.W, ff, 0.5, True)

    def channel_delta(self, p, m, i):
        Q, U, W, R = m["kv_heads"] * m["dim"], m["heads"] * m["vdim"], self.W, self.shapes["l%d.mix.a1" % i][0]
        for n, k in (("q", Q), ("k", Q), ("v", U)):
            self.mat(p + n, k, W)
            self.taps(p + n + ".conv", k, m["conv"])
        self.mat(p + "b", m["heads"], W)
        self.vec(p + "A_log", m["heads"], -0.5, 0.8)
        self.vec(p + "norm", m["vdim"])
        self.mat(p + "a1", R, W)
        self.mat(p + "a2", m["heads"] * m["dim"], R)
        self.vec(p + "dt_bias", m["heads"] * m["dim"], -3.0, 1.0)
        self.mat(p + "g1", R, W)
        self.mat(p + "g2", U, R)
        self.mat(p + "o", W, U)

    def mamba2(self, p, m, i):
        inner = m["heads"] * m["vdim"]
        C = inner + 2 * m["groups"] * m["state"]
        self.mat(p + "in", inner + C + m["heads"], self.W)
        self.taps(p + "conv", C, m["conv"])
        self.vec(p + "conv.b", C, 0.0)
        self.vec(p + "dt_bias", m["heads"], -1.0, 1.0)
        self.vec(p + "A_log", m["heads"], -1.0, 1.0)
        self.vec(p + "D", m["heads"])
        self.vec(p + "norm", inner)
        self.mat(p + "o", self.W, inner)

    def latent_attention(self, p, m, i):
        self.mat(p + "q", m["heads"] * (m["dim"] + m["rot_dim"]), self.W)
        if "kv_from" not in m:
            self.mat(p + "dkv", m["kv_rank"] + m["rot_dim"], self.W)
            self.vec(p + "dkv.norm", m["kv_rank"])
        self.mat(p + "uk", m["heads"] * m["dim"], m["kv_rank"])
        self.mat(p + "uv", m["heads"] * m["vdim"], m["kv_rank"])
        if self.c["architecture"] == "Gomuzen":
            self.mat(p + "g", m["heads"], self.W, 2.0)
        self.mat(p + "o", self.W, m["heads"] * m["vdim"], 1.0, True)

    def lightning(self, p, m, i):
        Q, V = m["heads"] * m["dim"], m["heads"] * m["vdim"]
        for n, k in (("q", Q), ("k", Q), ("v", V), ("g", V)):
            self.mat(p + n, k, self.W)
        self.vec(p + "norm", V)
        self.mat(p + "o", self.W, V)

    def general_delta(self, p, m, i):
        Q, R = m["heads"] * m["dim"], self.shapes["l%d.mix.w1" % i][0]
        for n in "rkvga":
            self.mat(p + n, Q, self.W)
        self.vec(p + "a.b", Q, 0.0, 0.5)
        self.mat(p + "w1", R, self.W)
        self.mat(p + "w2", Q, R)
        self.vec(p + "w0", Q, -1.0, 1.0)
        self.vec(p + "norm", Q)
        self.mat(p + "o", self.W, Q, 1.0, True)

    def attention(self, p, m, i):
        a, Q, K, V = self.c["architecture"], m["heads"] * m["dim"], m["kv_heads"] * m["dim"], m["kv_heads"] * m["vdim"]
        if a == "Gomuzen":
            Q, K = 2 * Q, 2 * K
        self.mat(p + "q", Q, self.W)
        self.mat(p + "k", K, self.W)
        if a != "Datasun":
            self.mat(p + "v", V, self.W)
        if a == "Datasun":
            for n, k in (("q", Q), ("k", K)):
                self.vec(p + n + ".b", k, 0.0, 0.5)
                self.vec(p + n + ".norm", k)
            self.vec(p + "o.b", self.W, 0.0, 0.3)
        elif a == "Gomuzen":
            self.vec(p + "q.norm", m["dim"])
            self.vec(p + "k.norm", m["dim"])
            for n in ("lq1", "lk1", "lq2", "lk2"):
                self.vec(p + n, m["dim"], 0.0, 0.3)
        else:
            for n, k in (("q", Q), ("k", K), ("v", V)):
                self.taps(p + n + ".conv", k, m["conv"])
            self.vec(p + "pb", m["heads"], -2.0, 0.5)
            self.mat(p + "g", m["heads"], self.W)
        self.mat(p + "o", self.W, m["heads"] * m["vdim"], 1.0, True)

    def attention_2(self, p, m, i):
        for n, k in (("q", m["heads"] * m["dim"]), ("k", m["kv_heads"] * m["dim"]), ("v", m["kv_heads"] * m["vdim"])):
            self.mat(p + n, k, self.W)
            self.vec(p + n + ".b", k, 0.0, 0.5)
        self.mat(p + "o", self.W, m["heads"] * m["vdim"], 1.0, True)


# ---------------------------------------------------------------------------------------------------- decoders
def quantized_config(case, seqs, ctx):
    if case["model"] == "moe":
        return dc.Config(n_layer=case["layers"], hidden=HIDDEN, n_head=32, n_kv_head=4, vocab=VOCAB, n_expert=EXPERTS, n_expert_used=TOP,
                         expert_ffn=EXPERT_FF, max_seqs=seqs, max_ctx=ctx)
    return dc.dense_0p8b(max_seqs=seqs, max_ctx=ctx)


def quantized(case):
    return case["model"] in ("moe", "dense")


def build(case, seed, ctx, seqs, max_ctx):
    if quantized(case):
        m = dc.Model(ctx, quantized_config(case, seqs, max_ctx))
        m.init_synthetic(seed, 0.02)
    else:
        t = Tensors(case["model"], case["width"], seed)
        m = dc.Model.from_config(ctx, t.c, t.shapes, max_seqs=seqs, max_ctx=max_ctx)
        for name, x in t.made.items():
            m.set_tensor(name, 30, x.view(torch.int16).cpu().numpy(), x.shape[-1], x.shape[0] if x.dim() == 2 else 1)
    m.finalize()
    return m


def contexts(case):
    """Lengths of a decode case's sequences: requests that run together are never equally far."""
    return [case["context"] - (case["context"] // 7) * i for i in range(case["seqs"])]


def token_ids(case, seed):
    """Token ids of every sequence: its prompt, then what the steps of a decode case are given."""
    vocab = VOCAB if quantized(case) else 32768
    lengths = [n + STEPS for n in contexts(case)] if case["kind"] == "decode" else [case["tokens"]]
    return [Values(seed).below("tokens%d" % i, vocab, n).cpu().numpy().astype(np.int32) for i, n in enumerate(lengths)]


class Decode:
    """Sequences that hold their prompts.  A pass runs STEPS steps on given tokens (sampled elsewhere, or forced), takes the last
    step's logits, and goes back to the prompts."""

    def __init__(self, case, seed):
        self.ctx = dc.Context(0)
        self.back = quantized(case)     # a recurrent state cannot go back: such sequences are forked
        n = case["seqs"]
        self.model = build(case, seed, self.ctx, n if self.back else 2 * n, case["context"] + 64)
        ids = token_ids(case, seed)
        self.held = contexts(case)
        self.seqs = [self.model.seq_alloc() for _ in ids]
        for s, t, k in zip(self.seqs, ids, self.held):
            self.model.prefill(s, t[:k])
        self.steps = np.stack([t[k:] for t, k in zip(ids, self.held)], axis=1)

    def run(self):
        m = self.model
        seqs = self.seqs if self.back else [m.seq_fork(s) for s in self.seqs]
        for tokens in self.steps[:-1]:
            m.decode_step(seqs, tokens)
        _, logits = m.decode_step(seqs, self.steps[-1], want_logits=True)
        for s, k in zip(seqs, self.held):
            if self.back:
                m.seq_truncate(s, k)
            else:
                m.seq_free(s)
        return logits

    def __del__(self):
        self.model.close()
        self.ctx.close()


class Prompt:
    def __init__(self, case, seed):
        self.ctx = dc.Context(0)
        self.model = build(case, seed, self.ctx, 2, case["tokens"] + 64)
        self.tokens = token_ids(case, seed)[0]

    def run(self):
        s = self.model.seq_alloc()
        _, logits = self.model.prefill(s, self.tokens, want_logits=True)
        self.model.seq_free(s)
        return logits

    def __del__(self):
        self.model.close()
        self.ctx.close()


def prepare(case, seed):
    return {"product": Product, "experts": Experts, "decode": Decode, "prompt": Prompt}[case["kind"]](case, seed)


def run(state):
    return state.run()


# ---------------------------------------------------------------------------------- the decoders in 64 bits
def attend(q, k, v, scale, cap=None, window=None, keep=0, sink=None, bias=None):
    """Causal attention of a whole sequence: q [T, H, d], k [T, G, d], v [T, G, e].  bias: sigmoid weights instead of a softmax."""
    T, H, _ = q.shape
    i = torch.arange(T, device=GPU)
    seen = i[:, None] >= i[None]
    if window:
        seen &= (i[:, None] - i[None] < window) | (i[None] < keep)
    out = torch.empty(T, H, v.shape[2], dtype=F8, device=GPU)
    for h in range(H):
        g = h // (H // k.shape[1])
        s = q[:, h] @ k[:, g].T * scale
        if cap:
            s = cap * torch.tanh(s / cap)
        if bias is not None:
            w = torch.sigmoid(s + bias[h]) * seen
        else:
            s = s.masked_fill(~seen, -math.inf)
            if sink is not None:
                s = torch.cat([s, torch.full((T, 1), sink, dtype=F8, device=GPU)], 1)
            w = torch.softmax(s, 1)[:, :T]
        out[:, h] = w @ v[:, g]
    return out


def frequencies(dims, base, scaling=None):
    f = base ** (-torch.arange(0, dims, 2, dtype=F8, device=GPU) / dims)
    if not scaling:
        return f, 1.0
    place = lambda turns: dims * math.log(scaling["original"] / (2 * math.pi * turns)) / (2 * math.log(base))  # noqa: E731
    lo, hi = max(math.floor(place(scaling["fast"])), 0), min(math.ceil(place(scaling["slow"])), dims - 1)
    ramp = ((torch.arange(dims // 2, dtype=F8, device=GPU) - lo) / max(hi - lo, 0.001)).clamp(0, 1)
    return f * (1 - ramp) + f / scaling["factor"] * ramp, 0.1 * math.log(scaling["factor"]) + 1.0


def rotate(x, freq, mul=1.0, halves_apart=False):
    """x [T, H, D]: pairs of the first 2 len(freq) dimensions, neighbours or half of them apart, turned by the position."""
    n = len(freq)
    a = torch.arange(x.shape[0], dtype=F8, device=GPU)[:, None, None] * freq
    c, s = mul * torch.cos(a), mul * torch.sin(a)
    out = x.clone()
    even, odd = (slice(0, n), slice(n, 2 * n)) if halves_apart else (slice(0, 2 * n, 2), slice(1, 2 * n, 2))
    u, v = x[:, :, even], x[:, :, odd]
    out[:, :, even], out[:, :, odd] = u * c - v * s, v * c + u * s
    return out


class Device:
    """What torch needs to see memory of the library as a tensor."""

    def __init__(self, address, nbytes):
        self.__cuda_array_interface__ = {"shape": (nbytes,), "typestr": "|u1", "data": (address, False), "version": 2}


def quantized_logits(case, m, tokens):
    """Logits of the last token of a sequence; m: the library's model, whose tensors are read as bytes."""
    c = m.cfg

    def raw(name):
        t, ne, address, nbytes = m.get_tensor_info(name)
        return {dc.GGML_TYPE_Q4_K: "q4_k", dc.GGML_TYPE_Q6_K: "q6_k"}.get(t), ne, torch.as_tensor(Device(address, nbytes), device=GPU)

    def vector(name):
        return raw(name)[2].view(torch.float32).to(F8)

    def matrix(name, rows=None):
        kind, (K, N, E, _), b = raw(name)
        b = b.reshape(N * E, -1)
        return dequantize(kind, b if rows is None else b[rows], K)

    T, freq = len(tokens), frequencies(128, c.rope_theta)[0]
    x = matrix("token_embd.weight", torch.from_numpy(tokens).long().to(GPU))
    for i in range(c.n_layer):
        p = "blk.%d." % i
        h = rms(x, vector(p + "attn_norm.weight"), c.rms_eps)
        q, k, v = ((h @ matrix(p + "attn_%s.weight" % n).T).reshape(T, -1, 128) for n in "qkv")
        q = rotate(rms(q, vector(p + "attn_q_norm.weight"), c.rms_eps), freq)
        k = rotate(rms(k, vector(p + "attn_k_norm.weight"), c.rms_eps), freq)
        x = x + attend(q, k, v, 128 ** -0.5).reshape(T, -1) @ matrix(p + "attn_output.weight").T
        h = rms(x, vector(p + "ffn_norm.weight"), c.rms_eps)
        if c.n_expert:
            expert = lambda n, rows: lambda e: matrix(p + "ffn_%s_exps.weight" % n, slice(e * rows, (e + 1) * rows))  # noqa: E731
            x = x + swiglu_experts(h, h @ vector(p + "ffn_gate_inp.weight").reshape(c.n_expert, -1).T, c.n_expert_used,
                                   expert("gate", c.expert_ffn), expert("up", c.expert_ffn), expert("down", c.hidden))
        else:
            x = x + (silu(h @ matrix(p + "ffn_gate.weight").T) * (h @ matrix(p + "ffn_up.weight").T)) @ matrix(p + "ffn_down.weight").T
    h = rms(x[-1], vector("output_norm.weight"), c.rms_eps)
    return matrix("token_embd.weight" if c.tie_embeddings else "output.weight") @ h


class Exact:
    """A layer-list decoder on one whole sequence."""

    def __init__(self, name, width, seed):
        self.t = Tensors(name, width, seed)
        self.c, self.eps = self.t.c, self.t.c["norm"]["eps"]

    def w(self, name):
        return self.t.made[name].to(F8)

    def conv(self, x, name, bias=0.0):
        w = self.w(name)
        xx = torch.cat([torch.zeros(w.shape[1] - 1, x.shape[1], dtype=F8, device=GPU), x])
        return sum(xx[j:j + x.shape[0]] * w[:, j] for j in range(w.shape[1])) + bias

    def logits(self, tokens):
        c, hyper = self.c, "streams" in self.c
        x = self.w("embed")[torch.from_numpy(tokens).long().to(GPU)]
        if hyper:
            x = torch.stack([x] * c["streams"])
        order = [(i, None) for i in range(len(c["layers"]))]
        if "loop" in c:
            a, b = c["loop"]["start"], c["loop"]["stop"]
            order = order[:a] + [(i, t if i == a else None) for t in range(c["loop"]["times"]) for i in range(a, b)] + order[b:]
        self.cache = {}
        for i, step in order:
            ly, p = c["layers"][i], "l%d." % i
            mixer = getattr(self, ly["type"])
            if step is not None:
                x = x + self.w("loop.step")[step]
            if c["architecture"] == "Garilix":
                x = x + rms(mixer(x, p + "mix.", ly["mixer"], i), self.w(p + "norm1"), self.eps)
                x = x + rms(self.feed_forward(x, p + "mlp.", ly["mlp"]), self.w(p + "norm2"), self.eps)
            elif c["architecture"] == "Datasun":
                h = rms(x, self.w(p + "norm1"), self.eps)
                x = x + mixer(h, p + "mix.", ly["mixer"], i) + self.feed_forward(h, p + "mlp.", ly["mlp"])
            elif c["architecture"] == "Gomuzen":
                x = x + mixer(rms(x, self.w(p + "norm1"), self.eps), p + "mix.", ly["mixer"], i)
                x = x + self.feed_forward(rms(x, self.w(p + "norm2"), self.eps), p + "mlp.", ly["mlp"])
            else:
                for hc, norm, part in (("hc1.", "norm1", lambda h: mixer(h, p + "mix.", ly["mixer"], i)),
                                       ("hc2.", "norm2", lambda h: self.feed_forward(h, p + "mlp.", ly["mlp"]))):
                    y = part(rms(torch.einsum("s,stw->tw", self.w(p + hc + "in"), x), 1.0 + self.w(p + norm), self.eps))
                    x = torch.einsum("st,snw->tnw", self.w(p + hc + "mix"), x) + c["residual_mult"] * self.w(p + hc + "out")[:, None, None] * y
        if hyper:
            x = x.sum(0)
        return self.w("head" if "head" in self.t.made else "embed") @ rms(x[-1], self.w("final.norm") + (1.0 if hyper else 0.0), self.eps)

    def feed_forward(self, h, p, mlp):
        if mlp["kind"] == "dense":
            g, u, d = (self.w(p + n) for n in ("gate", "up", "down"))
            return self.gated(h, g, u, d, mlp.get("limit"))
        r = mlp["router"]
        z = h @ self.w(p + "router").T
        if "groups" in r:
            s = torch.sigmoid(z)
            choice = s + self.w(p + "correction")
            per = choice.reshape(len(h), r["groups"]["count"], -1)
            best = per.topk(2, dim=2)[0].sum(2).topk(r["groups"]["keep"], dim=1)[1]
            open_ = torch.zeros(per.shape[:2], dtype=torch.bool, device=GPU).scatter_(1, best, True)
            ids = per.masked_fill(~open_[:, :, None], -math.inf).flatten(1).topk(r["top"], dim=1)[1]
            w = s.gather(1, ids) * r["scale"]
        else:
            s, ids = torch.softmax(z, 1).topk(r["top"], dim=1)
            w = s / (s.sum(1, keepdim=True) + 1e-20)
        y = torch.zeros_like(h)
        for e in ids.unique().tolist():
            t, k = (ids == e).nonzero(as_tuple=True)
            q = "%se%d." % (p, e)
            if "groups" in r:
                o = self.gated(h[t], self.w(q + "gate"), self.w(q + "up"), self.w(q + "down"), mlp["expert"]["limit"])
            else:
                o = (h[t] @ self.w(q + "up").T).clamp(min=0) ** 2 @ self.w(q + "down").T
            y.index_add_(0, t, w[t, k][:, None] * o)
        return y

    def gated(self, h, gate, up, down, limit):
        g, u = h @ gate.T, h @ up.T
        if limit:
            g, u = g.clamp(max=limit), u.clamp(-limit, limit)
            return (g * torch.sigmoid(1.702 * g) * (u + 1)) @ down.T
        if self.c["architecture"] == "Garilix":
            return (torch.nn.functional.gelu(g, approximate="tanh") * u) @ down.T
        return (silu(g) * u) @ down.T

    def channel_delta(self, h, p, m, i):
        T, H, d, e = len(h), m["heads"], m["dim"], m["vdim"]
        q, k, v = (silu(self.conv(h @ self.w(p + n).T, p + n + ".conv")).reshape(T, H, -1) for n in "qkv")
        q, k = (y * torch.rsqrt((y * y).sum(2, keepdim=True) + 1e-6) for y in (q, k))
        q = q * d ** -0.5
        beta = torch.sigmoid(h @ self.w(p + "b").T)
        raw = (h @ self.w(p + "a1").T @ self.w(p + "a2").T + self.w(p + "dt_bias")).reshape(T, H, d)
        g = torch.exp(-torch.exp(self.w(p + "A_log"))[:, None] * torch.nn.functional.softplus(raw))
        S, o = torch.zeros(H, d, e, dtype=F8, device=GPU), torch.empty(T, H, e, dtype=F8, device=GPU)
        for t in range(T):
            S = g[t][:, :, None] * S
            u = beta[t][:, None] * (v[t] - (k[t][:, None] @ S)[:, 0])
            S = S + k[t][:, :, None] * u[:, None]
            o[t] = (q[t][:, None] @ S)[:, 0]
        o = rms(o, self.w(p + "norm"), self.eps) * torch.sigmoid(h @ self.w(p + "g1").T @ self.w(p + "g2").T).reshape(T, H, e)
        return o.reshape(T, -1) @ self.w(p + "o").T

    def mamba2(self, h, p, m, i):
        T, H, e, N, G = len(h), m["heads"], m["vdim"], m["state"], m["groups"]
        inner = H * e
        z, xbc, dt = (h @ self.w(p + "in").T).split([inner, inner + 2 * G * N, H], 1)
        x, B, C = silu(self.conv(xbc, p + "conv", self.w(p + "conv.b"))).split([inner, G * N, G * N], 1)
        x, B, C = x.reshape(T, H, e), *(y.reshape(T, G, N).repeat_interleave(H // G, 1) for y in (B, C))
        dt = torch.nn.functional.softplus(dt + self.w(p + "dt_bias"))
        a = torch.exp(-torch.exp(self.w(p + "A_log")) * dt)
        S, y = torch.zeros(H, N, e, dtype=F8, device=GPU), torch.empty(T, H, e, dtype=F8, device=GPU)
        for t in range(T):
            S = a[t][:, None, None] * S + (dt[t][:, None] * B[t])[:, :, None] * x[t][:, None]
            y[t] = (C[t][:, None] @ S)[:, 0]
        y = (y + self.w(p + "D")[:, None] * x).reshape(T, inner) * silu(z)
        y = rms(y.reshape(T, m["norm_groups"], -1), 1.0, self.eps).reshape(T, inner) * self.w(p + "norm")
        return y @ self.w(p + "o").T

    def latent_attention(self, h, p, m, i):
        T, H, d = len(h), m["heads"], m["dim"]
        freq = frequencies(m["rot"]["dims"], m["rot"]["base"])[0]
        if "kv_from" not in m:
            c, r = (h @ self.w(p + "dkv").T).split([m["kv_rank"], m["rot_dim"]], 1)
            self.cache[i] = rms(c, self.w(p + "dkv.norm"), self.eps), rotate(r[:, None], freq)
        c, r = self.cache[m.get("kv_from", i)]
        q = (h @ self.w(p + "q").T).reshape(T, H, -1)
        q = torch.cat([q[:, :, :d], rotate(q[:, :, d:], freq)], 2)
        k = torch.cat([(c @ self.w(p + "uk").T).reshape(T, H, d), r.expand(T, H, -1)], 2)
        o = attend(q, k, (c @ self.w(p + "uv").T).reshape(T, H, -1), m["scale"], window=(m.get("mask") or {}).get("size"))
        if p + "g" in self.t.made:
            o = o * torch.sigmoid(h @ self.w(p + "g").T)[:, :, None]
        return o.reshape(T, -1) @ self.w(p + "o").T

    def lightning(self, h, p, m, i):
        T, H = len(h), m["heads"]
        q, k, v = (silu(h @ self.w(p + n).T).reshape(T, H, -1) for n in "qkv")
        decay = torch.tensor(m["decay"], dtype=F8, device=GPU)[:, None, None]
        S, o = torch.zeros(H, m["dim"], m["vdim"], dtype=F8, device=GPU), torch.empty(T, H, m["vdim"], dtype=F8, device=GPU)
        for t in range(T):
            S = decay * S + k[t][:, :, None] * v[t][:, None]
            o[t] = (q[t][:, None] @ S)[:, 0]
        return (rms(o.reshape(T, -1), self.w(p + "norm"), self.eps) * torch.sigmoid(h @ self.w(p + "g").T)) @ self.w(p + "o").T

    def general_delta(self, h, p, m, i):
        T, H, d = len(h), m["heads"], m["dim"]
        r, k, v = ((h @ self.w(p + n).T).reshape(T, H, d) for n in "rkv")
        w = torch.exp(-math.exp(-0.5) * torch.sigmoid(torch.tanh(h @ self.w(p + "w1").T) @ self.w(p + "w2").T + self.w(p + "w0"))).reshape(T, H, d)
        a = torch.sigmoid(h @ self.w(p + "a").T + self.w(p + "a.b")).reshape(T, H, d)
        u = k * torch.rsqrt((k * k).sum(2, keepdim=True) + 1e-6)
        S, o = torch.zeros(H, d, d, dtype=F8, device=GPU), torch.empty(T, H, d, dtype=F8, device=GPU)
        for t in range(T):
            S = w[t][:, :, None] * S - (a[t] * u[t])[:, :, None] * (u[t][:, None] @ S) + k[t][:, :, None] * v[t][:, None]
            o[t] = (r[t][:, None] @ S)[:, 0]
        o = rms(o, 1.0, self.eps).reshape(T, -1) * self.w(p + "norm")
        return (o * torch.sigmoid(h @ self.w(p + "g").T)) @ self.w(p + "o").T

    def attention(self, h, p, m, i):
        T, H, G, a, window = len(h), m["heads"], m["kv_heads"], self.c["architecture"], (m.get("mask") or {}).get("size")
        if a == "Datasun":          # values are the raw keys; a sink of score 0
            freq, mul = frequencies(m["rot"]["dims"], m["rot"]["base"], m["rot"].get("scaling"))
            q, v = (h @ self.w(p + n).T + self.w(p + n + ".b") for n in "qk")
            k = rotate(rms(v, self.w(p + "k.norm"), self.eps).reshape(T, G, -1), freq, mul)
            q = rotate(rms(q, self.w(p + "q.norm"), self.eps).reshape(T, H, -1), freq, mul)
            return attend(q, k, v.reshape(T, G, -1), m["scale"], window=window, sink=0.0).reshape(T, -1) @ self.w(p + "o").T + self.w(p + "o.b")
        if a == "Gomuzen":          # two maps over the same values, one taken off the other
            freq, mul = frequencies(m["rot"]["dims"], m["rot"]["base"], m["rot"].get("scaling"))
            q, k = (rotate(rms((h @ self.w(p + n).T).reshape(T, -1, m["dim"]), self.w(p + n + ".norm"), self.eps), freq, mul, True) for n in "qk")
            v = (h @ self.w(p + "v").T).reshape(T, G, -1)
            one, two = (attend(q[:, j::2], k[:, j::2], v, m["scale"], m["softcap"], window) for j in range(2))
            lam = torch.exp((self.w(p + "lq1") * self.w(p + "lk1")).sum()) - torch.exp((self.w(p + "lq2") * self.w(p + "lk2")).sum()) + m["diff"]
            return (rms(one - lam * two, 1.0, self.eps) * (1.0 - m["diff"])).reshape(T, -1) @ self.w(p + "o").T
        q, k, v = (rms(self.conv(h @ self.w(p + n).T, p + n + ".conv").reshape(T, -1, s), 1.0, self.eps) for n, s in (("q", m["dim"]), ("k", m["dim"]), ("v", m["vdim"])))
        o = attend(q, k, v, m["scale"], window=window, bias=self.w(p + "pb")) * torch.sigmoid(h @ self.w(p + "g").T)[:, :, None]
        return o.reshape(T, -1) @ self.w(p + "o").T

    def attention_2(self, h, p, m, i):
        T, H, G = len(h), m["heads"], m["kv_heads"]
        freq, mul = frequencies(m["rot"]["dims"], m["rot"]["base"], m["rot"].get("scaling"))
        q, k, v = ((h @ self.w(p + n).T + self.w(p + n + ".b")).reshape(T, x, -1) for n, x in (("q", H), ("k", G), ("v", G)))
        o = attend(rotate(q, freq, mul, True), rotate(k, freq, mul, True), v, m["scale"], m["softcap"], m["mask"]["size"], m["mask"]["keep_first"])
        return o.reshape(T, -1) @ self.w(p + "o").T


def exact(case, seed):
    if case["kind"] == "product":
        blocks, x = product_inputs(case, seed)
        rows = max(1, (1 << 27) // case["K"])       # a gigabyte of 64-bit values at a time
        return torch.cat([x.to(F8) @ dequantize(case["type"], b, case["K"]).T for b in blocks.split(rows)], 1)
    if case["kind"] == "experts":
        t, x = experts_inputs(case, seed)
        x = x.to(F8)
        part = lambda n, kind, rows, K: lambda e: dequantize(kind, t[n][e * rows:(e + 1) * rows], K)  # noqa: E731
        y = swiglu_experts(x, x @ t["router"].to(F8).T, TOP, part("gate", "q4_k", EXPERT_FF, HIDDEN), part("up", "q4_k", EXPERT_FF, HIDDEN),
                           part("down", "q6_k", HIDDEN, EXPERT_FF))
        return {"y": y, "ids": None}
    ids = token_ids(case, seed)
    if quantized(case):
        if case["layers"] > EXACT_LAYERS and case["model"] == "moe":
            return None
        ctx = dc.Context(0)
        m = dc.Model(ctx, quantized_config(case, 1, 64))
        m.init_synthetic(seed, 0.02)
        out = [quantized_logits(case, m, t) for t in ids]
        m.close()
        ctx.close()
    else:
        model = Exact(case["model"], case["width"], seed)
        out = [model.logits(t) for t in ids]
    return torch.stack(out) if case["kind"] == "decode" else out[0]


# ------------------------------------------------------------------------------------- work and tolerances
def distinct(n, experts, top):
    """Experts that n tokens are expected to meet."""
    return experts * (1.0 - (1.0 - top / experts) ** n)


def quantized_work(case, tokens, keys, rows):
    """tokens in one pass over the weights, keys that they see in all, rows of logits."""
    c = quantized_config(case, 1, 64)
    Q, K = c.n_head * 128, c.n_kv_head * 128
    q4, q6 = 144 / 256, 210 / 256
    mid = (q4 + q6) / 2         # half of the down projections are Q6_K
    att = c.hidden * ((Q + K) * q4 + K * q6) + Q * c.hidden * q4
    params = c.hidden * (2 * Q + 2 * K)
    if c.n_expert:
        one = 3 * c.hidden * c.expert_ffn
        ffn = 4 * c.hidden * c.n_expert + distinct(tokens, c.n_expert, c.n_expert_used) * one * (2 * q4 + mid) / 3
        used = c.hidden * c.n_expert + one * c.n_expert_used
    else:
        used = 3 * c.hidden * c.ffn
        ffn = used * (2 * q4 + mid) / 3
    head = c.vocab * c.hidden
    n_bytes = c.n_layer * (att + ffn + (tokens + keys) * 2 * K * 2) + head * q6 + 4 * rows * c.vocab
    return n_bytes, 2.0 * (c.n_layer * (tokens * (params + used) + keys * 2 * Q) + rows * head)


def family_params(c):
    """(weights of every layer run that any token reads, of one expert, experts, experts of a token, layer runs)."""
    W = c["width"]
    runs = c["layers"] + (c["layers"][c["loop"]["start"]:c["loop"]["stop"]] * (c["loop"]["times"] - 1) if "loop" in c else [])
    dense, expert, met = 0, 0, (0, 0)
    n_moe = 0
    for ly in runs:
        m, f = ly["mixer"], ly["mlp"]
        inner = m["heads"] * (m["vdim"] if "vdim" in m else m["dim"])
        Q = m["heads"] * m.get("dim", 0)
        if ly["type"] == "channel_delta":
            dense += W * (2 * m["kv_heads"] * m["dim"] + 2 * inner + m["heads"] + 256) + 128 * (Q + inner)
        elif ly["type"] == "mamba2":
            dense += W * (3 * inner + 2 * m["groups"] * m["state"] + m["heads"])
        elif ly["type"] == "latent_attention":
            dense += W * (m["heads"] * (m["dim"] + m["rot_dim"]) + (0 if "kv_from" in m else m["kv_rank"] + m["rot_dim"]) + inner) + m["kv_rank"] * (Q + inner)
        elif ly["type"] == "lightning":
            dense += W * (2 * Q + 3 * inner)
        elif ly["type"] == "general_delta":
            dense += W * 6 * Q + max(32, W // 32) * (W + Q)
        else:
            maps = 2 if "diff" in m else 1
            dense += W * (maps * (Q + m["kv_heads"] * m["dim"]) + m["kv_heads"] * m["vdim"] + inner)
        if f["kind"] == "dense":
            dense += 3 * W * f["ff"]
        else:
            n_moe += 1
            dense += W * f["router"]["experts"]
            expert = (3 if "limit" in f["expert"] else 2) * W * f["expert"]["ff"]
            met = f["router"]["experts"], f["router"]["top"]
    return dense, expert, met, n_moe


def family_work(case, tokens, keys, rows):
    c, _ = family_config(case["model"], case["width"])
    dense, expert, (experts, top), n_moe = family_params(c)
    head = c["vocab"] * c["width"]
    read = dense + n_moe * expert * (distinct(tokens, experts, top) if experts else 0)
    attention = sum("attention" in ly["type"] for ly in c["layers"])
    return 2 * (read + head) + 4 * rows * c["vocab"], 2.0 * (tokens * (dense + n_moe * top * expert) + keys * attention * 2 * c["width"] + rows * head)


def work(case):
    if case["kind"] == "product":
        b = BLOCK[case["type"]][1] * case["K"] // 256
        return {"bytes": case["N"] * b + 4 * case["M"] * (case["K"] + case["N"]), "flops": 2.0 * case["M"] * case["N"] * case["K"]}
    if case["kind"] == "experts":
        one = 2 * EXPERT_FF * (HIDDEN // 256) * 144 + HIDDEN * (EXPERT_FF // 256) * 210
        return {"bytes": 4 * EXPERTS * HIDDEN + distinct(case["T"], EXPERTS, TOP) * one + 8 * case["T"] * HIDDEN,
                "flops": 2.0 * case["T"] * HIDDEN * (EXPERTS + 3 * TOP * EXPERT_FF)}
    f = quantized_work if quantized(case) else family_work
    if case["kind"] == "prompt":
        n = case["tokens"]
        b, o = f(case, n, 0, 1)
        return {"bytes": b, "flops": o + f(case, 0, n * (n + 1) // 2, 0)[1]}
    n = case["seqs"]
    b, o = f(case, n, sum(contexts(case)), n)
    return {"bytes": STEPS * b, "flops": STEPS * o}


def tolerance(case):
    if case["kind"] == "product":
        return {"rel": 1e-5}            # sums of 32-bit terms in another order
    if case["kind"] == "experts":
        return {"rel": 2e-3, "max": 0.05, "differ": 0.0}    # hidden values are rounded to eight bits: a sum in another order turns some of them over
    return {"rel": 0.03, "max": 0.3}    # the same in every layer, of values or of bf16 products
