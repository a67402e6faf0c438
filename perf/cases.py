"""The work that a user of this library has it do, as cases that can be timed and whose outputs can be compared.

A case is a dict of plain values; `kind` names one of six uses:

  pass     a recorded decode pass over resident matrices (Pass): every projection of `layers` layers and, where `vocab` is
           set, the output head with its top-k, for `nb` activation columns (1: plain decode, 2..8: the columns of a
           speculative verify step or of a small batch)
  matvec   matrices called directly, one call each, from fp32 activations (gemv_f32): a host that keeps its own step loop
  actq8    the same with the per-32 activations of the drop-in header (quantize_act_q8, then gemv_act_q8 per matrix)
  prefill  the GEMMs of one layer for a chunk of `tokens` tokens, with the SwiGLU between gate / up and down
  sample   residual add + norm, output head and top-k called directly: what follows the last layer of a decode step
  dequant  rows of a matrix written out as dense values (embedding rows, or a library GEMM's operand)

In `pass` every layer takes its input from the host's buffer (the residual stream and the norm between the layers are
the host's own kernels), so that outputs of two correct builds can be compared: each step rounds its activations to 8
bits, and in an unbroken chain of layers one activation that rounds the other way grows into percents of the result.
"""
import math

import torch

from qwengine_b200 import Context, Pass, formats as F

OUT_KIND = {"f32": 0, "f16": 1, "bf16": 2}

# formats by role: attention-side projections, gate / up, down, output head
MIXES = {
    "iq3": ("Q4_K", "IQ3_XXS", "IQ4_XS", "Q6_K"),        # the 27B-shaped benchmark pass
    "q4": ("Q4_K", "Q4_K", "Q6_K", "Q6_K"),              # the benchmark's FFN block; the usual 4-bit K-quant file
    "q5": ("Q5_K", "Q5_K", "Q6_K", "Q6_K"),
    "q8": ("Q8_0", "Q8_0", "Q8_0", "Q8_0"),
    "iq4": ("IQ4_XS", "IQ4_XS", "IQ4_XS", "Q6_K"),
    "iq3s": ("IQ3_S", "IQ3_S", "IQ4_XS", "Q6_K"),
    "iq2": ("Q4_K", "IQ2_XXS", "IQ2_S", "Q6_K"),         # the reference's own 27B file is mostly 2-bit blocks
    "iq2xs": ("IQ3_XXS", "IQ2_XS", "Q2_K", "Q6_K"),
    "iq1": ("Q2_K", "IQ1_S", "IQ1_M", "Q6_K"),
}
ATTN, FFN, DOWN, HEAD = 0, 1, 2, 3

# byte offsets of a block's fp16 scales, and the root mean square of its weights for a scale of |N(0,1)| x 1
FP16_AT = {"Q8_0": (0,), "Q4_K": (0, 2), "Q5_K": (0, 2), "Q6_K": (208,), "IQ3_XXS": (0,), "IQ3_S": (0,), "IQ4_XS": (0,),
           "Q2_K": (80, 82), "IQ2_XXS": (0,), "IQ2_XS": (0,), "IQ2_S": (0,), "IQ1_S": (0,), "IQ1_M": ()}
RMS_AT_ONE = {"IQ3_XXS": 145.0, "IQ3_S": 144.0, "IQ4_XS": 1295.0, "Q4_K": 258.0, "Q5_K": 529.0, "Q6_K": 1365.0, "Q8_0": 75.0,
              "IQ2_XXS": 53.0, "IQ2_XS": 54.0, "IQ2_S": 53.0, "IQ1_S": 7.7, "IQ1_M": 7.0, "Q2_K": 15.5}
MIN_PER_SCALE = {"Q4_K": 7.5, "Q5_K": 15.5, "Q2_K": 1.5}      # the minimum that makes the mean of uniform quants zero


def listed():
    b27 = dict(hidden=5120, ff=17408, inner=6144, proj=16384)
    return [
        # one token of the 27B-shaped model: the headline workload, 12.5 GB of blocks
        dict(name="decode_27b", kind="pass", layers=64, vocab=248320, mix="iq3", nb=1, **b27),
        # the same step verifying seven drafted tokens
        dict(name="verify7_27b", kind="pass", layers=64, vocab=248320, mix="iq3", nb=7, **b27),
        # a short draft (two columns) on a model in 4-bit K-quants of the same width
        dict(name="verify2_q4", kind="pass", layers=8, vocab=0, mix="q4", nb=2, **b27),
        # one token of a smaller model in 2-bit blocks, row lengths that are no multiple of 1024, odd row counts
        dict(name="decode_small_iq2", kind="pass", layers=12, vocab=32003, mix="iq2", nb=1, hidden=2816, ff=9728, inner=2816, proj=6156),
        # four sequences stepped together on 2-bit and 3-bit blocks
        dict(name="batch4_iq2", kind="pass", layers=6, vocab=0, mix="iq2xs", nb=4, **b27),
        # the smallest call: a key projection straight from the host's step loop
        dict(name="call_k_proj", kind="matvec", fmt="Q4_K", M=1024, K=5120, nb=1, mats=1),
        # the drop-in header verifying four columns: gate and up of three layers
        dict(name="dropin_verify4", kind="actq8", fmt="IQ3_XXS", M=17408, K=5120, nb=4, mats=6),
        # a full prompt chunk of one layer, bf16
        dict(name="prefill_1024", kind="prefill", tokens=1024, mix="iq3", dtype="bf16", **b27),
        # the ragged tail of a prompt through the fp16 operands of the drop-in header
        dict(name="prefill_tail_77", kind="prefill", tokens=77, mix="q4", dtype="f16", **b27),
        # a long prompt of a smaller model
        dict(name="prefill_2500_small", kind="prefill", tokens=2500, mix="q5", dtype="bf16", hidden=4096, ff=11008, inner=4096, proj=6144),
        # after the last layer: norm, head, top-k for one column
        dict(name="sample_27b", kind="sample", fmt="Q6_K", hidden=5120, vocab=248320, nb=1, k=32),
        # a matrix written out in fp16 for a library GEMM
        dict(name="dequant_iq3", kind="dequant", fmt="IQ3_XXS", M=17408, K=5120, out="f16"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _k256(rng, lo, hi):
    """A row length: a multiple of 256, more often than not no multiple of 1024."""
    return 256 * _log(rng, lo // 256, hi // 256)


def draw(rng):
    kind = rng.choice(["pass"] * 4 + ["prefill"] * 3 + ["matvec", "actq8", "sample", "dequant"])
    fmts = sorted(F.ALL_FORMATS)
    if kind == "pass":
        hidden = _k256(rng, 1024, 8192)
        inner = _k256(rng, 1024, 6144)
        return dict(kind=kind, layers=_log(rng, 2, 16), vocab=rng.choice([0, _log(rng, 32000, 248320)]), mix=rng.choice(sorted(MIXES)),
                    nb=rng.choice([1, 1, 1, 2, 3, 4, 5, 6, 7, 8]), hidden=hidden, ff=_k256(rng, 2048, 17408), inner=inner, proj=inner + 4 * _log(rng, 64, 2560))
    if kind == "prefill":
        hidden = _k256(rng, 1024, 6144)
        inner = _k256(rng, 1024, 6144)
        return dict(kind=kind, tokens=_log(rng, 9, 2500), mix=rng.choice(sorted(MIXES)), dtype=rng.choice(["bf16", "bf16", "f16"]), hidden=hidden,
                    ff=_k256(rng, 2048, 17408), inner=inner, proj=inner + 4 * _log(rng, 64, 2560))
    if kind in ("matvec", "actq8"):
        return dict(kind=kind, fmt=rng.choice(fmts), M=_log(rng, 128, 17408), K=_k256(rng, 512, 17408), nb=rng.choice([1, 1, 2, 3, 4, 7, 8]),
                    mats=rng.randint(1, 8))
    if kind == "sample":
        return dict(kind=kind, fmt=rng.choice(["Q4_K", "Q6_K", "Q8_0"]), hidden=_k256(rng, 1024, 8192), vocab=_log(rng, 32000, 248320),
                    nb=rng.randint(1, 8), k=rng.choice([1, 8, 32, 40, 64]))
    return dict(kind=kind, fmt=rng.choice(fmts), M=_log(rng, 16, 17408), K=_k256(rng, 1024, 17408), out=rng.choice(["f32", "f16", "bf16"]))


# ---------------------------------------------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------------------------------------------
_CTX = None


def _context():
    """One per process and GPU, as a program keeps it."""
    global _CTX
    if _CTX is None:
        _CTX = Context(0)
    return _CTX


def _weights(fmt, M, K, gen):
    """Random valid blocks on the device: uniform quant bytes, fp16 scales |N(0,1)| of a size that gives a matvec unit gain."""
    f = F.get(fmt)
    nblk = K // f.block_elems
    w = torch.randint(0, 1 << 62, ((M * nblk * f.block_bytes + 7) // 8,), dtype=torch.int64, device="cuda", generator=gen).view(torch.uint8)
    w ^= w.roll(3)                                       # the top bits of the 64-bit words are not drawn
    w = w[: M * nblk * f.block_bytes].view(M, nblk, f.block_bytes)
    d = (torch.randn((M, nblk), device="cuda", generator=gen).abs() / (RMS_AT_ONE[f.name] * math.sqrt(K))).to(torch.float16)
    for i, at in enumerate(FP16_AT[f.name]):
        v = d if i == 0 else (d.float() * MIN_PER_SCALE[f.name]).to(torch.float16)
        w[:, :, at:at + 2] = v.view(torch.uint8).view(M, nblk, 2)
    if f.name == "IQ1_M":                                # its scale lies in the top nibbles of four 16-bit words
        bits = d.view(torch.int16).to(torch.int32)
        for k in range(4):
            hi = w[:, :, 49 + 2 * k]
            w[:, :, 49 + 2 * k] = (hi & 0x0F) | (((bits >> (4 * k)) & 0xF) << 4).to(torch.uint8)
    return w.view(M, nblk * f.block_bytes)


def _shapes(c):
    """(role, M, K) of a layer's matrices in execution order."""
    return [(ATTN, c["proj"], c["hidden"]), (ATTN, c["hidden"], c["inner"]), (FFN, c["ff"], c["hidden"]), (FFN, c["ff"], c["hidden"]),
            (DOWN, c["hidden"], c["ff"])]


class _Step:
    """A recorded pass and the buffers it reads and writes; the pass goes with it."""

    def __init__(self, c, gen):
        mix, L, nb = MIXES[c["mix"]], c["layers"], c["nb"]
        hidden, ff, inner, proj, vocab = c["hidden"], c["ff"], c["inner"], c["proj"], c["vocab"]
        self.nb, self.vocab, self.k = nb, vocab, 32
        self.ps = ps = Pass(_context(), max_nb=nb)
        xin = ps.buffer_f32((L + 1) * hidden)            # each layer's input, and the head's, as the host leaves them
        out = ps.buffer_f32(L * hidden)                  # each layer's attention-side output
        ffn = ps.buffer_f32(L * hidden)                  # and its FFN output
        big, gu = ps.buffer_f32(proj), ps.buffer_f32(2 * ff)
        xq, iq, hq = ps.buffer_q8k(hidden), ps.buffer_q8k(inner), ps.buffer_q8k(ff)
        for il in range(L):
            m = [ps.matrix_device(mix[role], _weights(mix[role], M, K, gen), K) for role, M, K in _shapes(c)]
            ps.quantize(xin, il * hidden, hidden, xq)
            ps.gemv(m[0], xq, big, 0)
            ps.quantize(big, 0, inner, iq)
            ps.gemv(m[1], iq, out, il * hidden)
            ps.quantize(out, il * hidden, hidden, xq)
            ps.gemv(m[2], xq, gu, 0)
            ps.gemv(m[3], xq, gu, ff)
            ps.swiglu(gu, 0, gu, ff, ff, hq)
            ps.gemv(m[4], hq, ffn, il * hidden)
        self.bufs = [out, ffn]
        if vocab:
            logits, best = ps.buffer_f32(vocab), ps.buffer_f32(2 * self.k)
            w = ps.matrix_device(mix[HEAD], _weights(mix[HEAD], vocab, hidden, gen), hidden)
            ps.quantize(xin, L * hidden, hidden, xq)
            ps.gemv(w, xq, logits, 0)
            ps.topk(logits, 0, vocab, self.k, best)
            self.bufs += [logits, best]
        ps.buffer_tensor(xin).copy_(torch.randn((nb, (L + 1) * hidden), device="cuda", generator=gen))
        ps.run(nb)                                       # the first run records the graph: part of loading the model

    def outputs(self):
        """The pass's own buffers; they are gone with the pass, so each view holds on to it."""
        views = [self.ps.buffer_tensor(b) for b in self.bufs]
        if self.vocab:
            best = views.pop()
            views += [best[:, :self.k], best[:, self.k:].view(torch.int32)]
        for v in views:
            v.step = self
        return views

    def __del__(self):
        ps = getattr(self, "ps", None)
        if ps is not None:
            torch.cuda.synchronize()
            ps.close()


def prepare(case, seed):
    c, gen = case, torch.Generator(device="cuda").manual_seed(int(seed))
    s = dict(case=c, ctx=_context())

    def normal(*shape):
        return torch.randn(shape, device="cuda", generator=gen)

    if c["kind"] == "pass":
        s["step"] = _Step(c, gen)
    elif c["kind"] in ("matvec", "actq8"):
        s["W"] = [_weights(c["fmt"], c["M"], c["K"], gen) for _ in range(c["mats"])]
        s["x"] = normal(c["nb"], c["K"])
        s["y"] = [torch.empty((c["nb"], c["M"]), device="cuda") for _ in range(c["mats"])]
        s["scratch"] = torch.empty(c["nb"] * (c["K"] // 256) * F.Q8K_BLOCK_BYTES, dtype=torch.uint8, device="cuda")
    elif c["kind"] == "prefill":
        dt = torch.bfloat16 if c["dtype"] == "bf16" else torch.float16
        mix, B = MIXES[c["mix"]], c["tokens"]
        s["fmts"] = [mix[role] for role, _, _ in _shapes(c)]
        s["W"] = [_weights(mix[role], M, K, gen) for role, M, K in _shapes(c)]
        s["X"] = [normal(B, k).to(dt) for k in (c["hidden"], c["inner"], c["hidden"])]   # before attention, after it, before the FFN
        s["Y"] = [torch.empty((B, M), device="cuda") for _, M, _ in _shapes(c)]
        s["dt"] = dt
    elif c["kind"] == "sample":
        s["W"] = _weights(c["fmt"], c["vocab"], c["hidden"], gen)
        s["x"], s["w"] = normal(c["nb"], c["hidden"]), 1.0 + 0.1 * normal(c["hidden"])
        s["y"] = torch.empty((c["nb"], c["vocab"]), device="cuda")
    else:
        s["W"] = _weights(c["fmt"], c["M"], c["K"], gen)
    return s


# ---------------------------------------------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------------------------------------------
def run(s):
    c, ctx = s["case"], s["ctx"]
    if c["kind"] == "pass":
        st = s["step"]
        st.ps.run(st.nb)
        return st.outputs()
    if c["kind"] == "matvec":
        return [ctx.gemv_f32(c["fmt"], W, s["x"], c["K"], scratch=s["scratch"], out=y) for W, y in zip(s["W"], s["y"])]
    if c["kind"] == "actq8":
        q, d, _ = ctx.quantize_act_q8(s["x"])
        return [ctx.gemv_act_q8(c["fmt"], W, q, d, c["K"], out=y) for W, y in zip(s["W"], s["y"])]
    if c["kind"] == "prefill":
        f, W, X, Y, ff = s["fmts"], s["W"], s["X"], s["Y"], c["ff"]
        ctx.gemm_prefill(f[0], W[0], X[0], c["hidden"], out=Y[0])
        ctx.gemm_prefill(f[1], W[1], X[1], c["inner"], out=Y[1])
        ctx.gemm_prefill(f[2], W[2], X[2], c["hidden"], out=Y[2])
        ctx.gemm_prefill(f[3], W[3], X[2], c["hidden"], out=Y[3])
        ctx.swiglu_rows_inplace(Y[2], Y[3], ff, OUT_KIND[c["dtype"]])
        h = Y[2].view(s["dt"])[:, :ff]
        ctx.gemm_prefill(f[4], W[4], h, ff, out=Y[4])
        return [Y[0], Y[1], h, Y[3], Y[4]]
    if c["kind"] == "sample":
        xn, q8 = ctx.add_rmsnorm_q8k(s["x"], s["w"], want_xn=False)
        logits = ctx.gemv(c["fmt"], s["W"], q8, c["hidden"], out=s["y"])
        vals, idx = ctx.topk(logits, c["k"])
        return [logits, vals, idx]
    return ctx.dequant_rows(c["fmt"], s["W"], c["K"], kind=OUT_KIND[c["out"]])


# ---------------------------------------------------------------------------------------------------------------
# what one pass cannot do without, and how exact its results are
# ---------------------------------------------------------------------------------------------------------------
def work(case):
    c = case

    def matrix(fmt, M, K):
        return M * F.get(fmt).row_bytes(K)

    if c["kind"] == "pass":
        mix, nb = MIXES[c["mix"]], c["nb"]
        mats = [(mix[role], M, K) for role, M, K in _shapes(c)] * c["layers"]
        nbytes = 12 * c["layers"] * c["hidden"] * nb     # a layer's input, its two outputs
        if c["vocab"]:
            mats.append((mix[HEAD], c["vocab"], c["hidden"]))
            nbytes += 4 * (c["hidden"] + c["vocab"]) * nb
        return {"bytes": nbytes + sum(matrix(*m) for m in mats), "flops": sum(2.0 * nb * M * K for _, M, K in mats)}
    if c["kind"] in ("matvec", "actq8"):
        nb, n = c["nb"], c["mats"]
        return {"bytes": n * (matrix(c["fmt"], c["M"], c["K"]) + 4 * nb * c["M"]) + 4 * nb * c["K"], "flops": 2.0 * n * nb * c["M"] * c["K"]}
    if c["kind"] == "prefill":
        mix, B = MIXES[c["mix"]], c["tokens"]
        mats = [(mix[role], M, K) for role, M, K in _shapes(c)]
        io = 2 * (c["hidden"] + c["inner"] + c["hidden"]) + 4 * (c["proj"] + c["hidden"] + c["ff"] + c["hidden"]) + 2 * c["ff"]
        return {"bytes": B * io + sum(matrix(*m) for m in mats), "flops": sum(2.0 * B * M * K for _, M, K in mats)}
    if c["kind"] == "sample":
        nb = c["nb"]
        return {"bytes": matrix(c["fmt"], c["vocab"], c["hidden"]) + nb * (4 * c["hidden"] + c["hidden"] // 256 * 292 + 4 * c["vocab"] + 8 * c["k"]) + 4 * c["hidden"],
                "flops": 2.0 * nb * c["vocab"] * c["hidden"]}
    return {"bytes": matrix(c["fmt"], c["M"], c["K"]) + c["M"] * c["K"] * {"f32": 4, "f16": 2, "bf16": 2}[c["out"]], "flops": 2.0 * c["M"] * c["K"]}


def tolerance(case):
    c = case
    if c["kind"] == "pass":
        # 8-bit activations between the steps: one that rounds the other way is 1/127 of its block's largest
        return {"rel": 2e-2, "max": 0.3, "differ": 0.01}
    if c["kind"] in ("matvec", "actq8"):
        return {"rel": 1e-6, "max": 1e-5}                # exact integer sums, fp32 sums of them
    if c["kind"] == "prefill":
        # weights (for the K-quants their scales as well) and the SwiGLU rounded to 8 or 11 bits
        return {"rel": 1e-2, "max": 0.3} if c["dtype"] == "bf16" else {"rel": 2.5e-3, "max": 3e-2}
    if c["kind"] == "sample":
        # as above, behind one 8-bit rounding of the normed row: a value that rounds the other way moves every logit a little
        return {"rel": 1e-3, "max": 1e-2, "differ": 0.01}
    return "exact"
