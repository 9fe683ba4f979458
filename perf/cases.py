"""Timed cases of the conv-attention operators, through the package's public entry points.

Families (the ``op`` of a case):

* ``train``    ``ConvAttentionCUDA`` forward and backward through autograd: what one attention layer adds to a training
               step.  q, k, v are bf16, the filter is an fp32 parameter, the layer's output and its gradient are fp32.
* ``prefill``  the same module without gradients: a prompt is read before decoding starts, or a model is evaluated.
* ``decode``   ``fwd_conv_attn_inference`` over a contiguous key/value cache: one generated token.
* ``paged``    ``kv_append_paged`` then ``forward_inference_paged``: one generated token of a batch of sequences of
               different lengths whose caches live in a shared page pool.
* ``headmix``  ``head_conv_attention`` (all heads mixed by one matrix, no key-query filter), forward and backward.
* ``convmix``  ``conv_headmix_attention`` (filter, then heads mixed within groups), forward and backward.
"""
import math
import os
import sys

import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
if os.getcwd() not in sys.path:
    sys.path.insert(0, os.getcwd())
for _base in (os.getcwd(), _ROOT):
    _pkg = os.path.join(_base, "flash-multi-token-attention_b200")
    if os.path.isdir(_pkg):
        sys.path.insert(0, _pkg)
        break

import fmta_b200 as F  # noqa: E402


def listed():
    return [
        # the smallest training problem of the repository's configurations: a unit-test-sized layer, bound by launches
        dict(name="train_small", op="train", B=1, H=4, N=256, d=64, cq=3, ck=5, causal=True),
        # a short-context layer with a square filter, a quarter of the GPU's worth of heads
        dict(name="train_1k_square", op="train", B=1, H=8, N=1024, d=64, cq=7, ck=7, causal=True),
        # the headline training layer
        dict(name="train_4k", op="train", B=4, H=16, N=4096, d=64, cq=6, ck=11, causal=True),
        # an encoder layer: no causal mask, and a length that is a multiple of nothing
        dict(name="train_full_ragged", op="train", B=3, H=5, N=1537, d=64, cq=5, ck=9, causal=False),
        # the scaling configuration's layer at head dim 128
        dict(name="train_4k_d128", op="train", B=8, H=32, N=4096, d=128, cq=6, ck=11, causal=True),
        # one long prompt of an odd length
        dict(name="prefill_8k_d128", op="prefill", B=1, H=32, N=8191, d=128, cq=6, ck=11, causal=True),
        # a single short request: latency of one token
        dict(name="decode_small", op="decode", B=2, H=2, Nk=4096, d=64, q_len=16, cq=7, ck=7, splits=32, causal=False),
        # the serving configuration: 17 GB of cache read for each token
        dict(name="decode_32k", op="decode", B=32, H=32, Nk=32768, d=128, q_len=6, cq=6, ck=11, splits=4, causal=False),
        # continuous batching: ragged lengths in a page pool, new rows appended, mask as in training
        dict(name="paged_ragged", op="paged", B=16, H=32, Nk=8192, d=128, q_len=6, cq=6, ck=11, splits=4, page=256),
        # the reference's head-mixing operator over 16 heads
        dict(name="headmix_16", op="headmix", B=2, H=16, N=2048, d=64, causal=True),
        # filter and mix at an everyday size, odd length
        dict(name="convmix_1k", op="convmix", B=2, H=8, N=1001, d=64, G=4, cq=6, ck=11, causal=True),
        # the head-mixing training configuration
        dict(name="convmix_8k", op="convmix", B=2, H=32, N=8192, d=128, G=4, cq=6, ck=11, causal=True),
    ]


def _log(rng, lo, hi):
    """An integer spread evenly over the logarithm of [lo, hi]."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _length(rng, lo, hi):
    """A sequence length: half of them as they fall, half rounded to a multiple of 128 (where that is in the range)."""
    n = _log(rng, lo, hi)
    r = max(1, n // 128) * 128
    return r if rng.random() < 0.5 and lo <= r <= hi else n


FILTERS = [(3, 3), (3, 5), (5, 5), (5, 9), (6, 11), (6, 11), (7, 7)]


def draw(rng):
    op = rng.choice(["train", "train", "train", "prefill", "decode", "paged", "headmix", "convmix"])
    while True:
        if op in ("train", "prefill"):
            d = rng.choice([64, 64, 64, 128, 128, 32])
            cq, ck = rng.choice([f for f in FILTERS if f[0] <= 6] if d == 128 else FILTERS)
            c = dict(op=op, B=rng.choice([1, 1, 2, 3, 4, 8]), H=rng.choice([2, 4, 5, 8, 12, 16, 32]), N=_length(rng, 64, 16384), d=d,
                     cq=cq, ck=ck, causal=rng.random() < 0.8)
            limit = 2.75e11
        elif op in ("decode", "paged"):
            d = rng.choice([64, 128])
            cq, ck = rng.choice(FILTERS)
            c = dict(op=op, B=_log(rng, 1, 32), H=rng.choice([2, 4, 8, 16, 32]), Nk=_length(rng, 256, 32768), d=d, q_len=rng.choice([cq, cq, 16, 1]),
                     cq=cq, ck=ck, splits=rng.choice([1, 4, 8, 16, 32]))
            c.update(dict(page=rng.choice([64, 256])) if op == "paged" else dict(causal=rng.random() < 0.5))
            limit = 4.3e9
        elif op == "headmix":
            c = dict(op=op, B=rng.choice([1, 2, 4]), H=rng.choice([16, 16, 32]), N=_length(rng, 64, 4096), d=64, causal=rng.random() < 0.8)
            limit = 5e10
        else:
            G = rng.choice([2, 4, 4, 8])
            cq, ck = rng.choice([f for f in FILTERS if f[0] <= 6])
            c = dict(op=op, B=rng.choice([1, 2]), H=G * rng.choice([1, 2, 4, 8]), N=_length(rng, 128, 4096), d=rng.choice([64, 128]), G=G,
                     cq=cq, ck=ck, causal=rng.random() < 0.8)
            limit = 2.75e11
        # score entries (training) or cache elements (decoding) times the head dim: no more than the largest of the kind
        size = c["B"] * c["H"] * c["d"] * (c["Nk"] if "Nk" in c else c["N"] * c["N"] * (0.5 if c["causal"] else 1.0))
        if size <= limit:
            return c


def _normal(gen, *shape, dtype=torch.bfloat16):
    return torch.randn(*shape, device="cuda", dtype=dtype, generator=gen)


def _filter(gen, H, cq, ck):
    """Identity plus noise, fp32, as a trained filter starts."""
    th = 0.02 * _normal(gen, H, cq, ck, dtype=torch.float32)
    th[:, cq - 1, ck // 2] += 1.0
    return th


def prepare(case, seed):
    c, gen = case, torch.Generator(device="cuda").manual_seed(seed)
    s = dict(case=c, scale=1.0 / math.sqrt(c["d"]))
    op, B, H, d = c["op"], c["B"], c["H"], c["d"]
    if op == "decode":
        s["q"] = _normal(gen, B, H, c["q_len"], d)
        s["k"], s["v"] = (_normal(gen, B, H, c["Nk"], d) for _ in range(2))
        s["theta"] = _filter(gen, H, c["cq"], c["ck"])
        return s
    if op == "paged":
        pages = -(-c["Nk"] // c["page"])
        s["q"] = _normal(gen, B, H, c["q_len"], d)
        s["k"], s["v"] = (_normal(gen, B * pages, H, c["page"], d) for _ in range(2))
        s["k_new"], s["v_new"] = (_normal(gen, B, H, 1, d) for _ in range(2))
        s["table"] = torch.randperm(B * pages, device="cuda", generator=gen).to(torch.int32).view(B, pages).contiguous()
        # the sequences of a batch are anywhere between an eighth of the longest and the longest
        n = torch.randint(max(c["Nk"] // 8, 1), c["Nk"], (B,), device="cuda", generator=gen)
        n[0] = c["Nk"] - 1
        s["before"] = n.to(torch.int32)
        s["after"] = (n + 1).to(torch.int32)
        s["theta"] = _filter(gen, H, c["cq"], c["ck"])
        return s
    shape = (B, H, c["N"], d)
    grads = op != "prefill"
    s["q"], s["k"], s["v"] = (_normal(gen, *shape).requires_grad_(grads) for _ in range(3))
    if op in ("train", "prefill"):
        s["layer"] = F.ConvAttentionCUDA(H, c["cq"], c["ck"], init_random=False).to("cuda")
        with torch.no_grad():
            s["layer"].conv_weight.copy_(_filter(gen, H, c["cq"], c["ck"]))
        s["do"] = _normal(gen, *shape, dtype=torch.float32)
    elif op == "headmix":
        s["w"] = (_normal(gen, H, H, dtype=torch.float32) / math.sqrt(H)).requires_grad_()
        s["do"] = _normal(gen, *shape)
    else:
        G = c["G"]
        w = torch.eye(G, device="cuda").repeat(H // G, 1, 1) + 0.02 * _normal(gen, H // G, G, G, dtype=torch.float32)
        s["w"] = w.requires_grad_()
        s["theta"] = _filter(gen, H, c["cq"], c["ck"]).requires_grad_()
        s["do"] = _normal(gen, *shape, dtype=torch.float32)
    return s


def run(s):
    c, op = s["case"], s["case"]["op"]
    if op == "decode":
        return F.fwd_conv_attn_inference(s["q"], s["k"], s["v"], s["theta"], c["splits"], s["scale"], c["cq"] - 1, (c["ck"] - 1) // 2,
                                         False, offset_causal=c["causal"])
    if op == "paged":
        F.kv_append_paged(s["k"], s["v"], s["table"], s["before"], s["k_new"], s["v_new"])
        return F.forward_inference_paged(s["q"], s["k"], s["v"], s["table"], s["theta"], c["splits"], s["scale"], c["cq"] - 1,
                                         (c["ck"] - 1) // 2, seq_lens=s["after"], max_seq_len=c["Nk"], offset_causal=True)
    if op == "prefill":
        with torch.no_grad():
            return s["layer"](s["q"], s["k"], s["v"], causal=c["causal"])
    if op == "train":
        o = s["layer"](s["q"], s["k"], s["v"], causal=c["causal"])
        wrt = (s["q"], s["k"], s["v"], s["layer"].conv_weight)
    elif op == "headmix":
        o = F.head_conv_attention(s["q"], s["k"], s["v"], s["w"], c["causal"], s["scale"])
        wrt = (s["q"], s["k"], s["v"], s["w"])
    else:
        o = F.conv_headmix_attention(s["q"], s["k"], s["v"], s["theta"], s["w"], c["causal"], s["scale"])
        wrt = (s["q"], s["k"], s["v"], s["theta"], s["w"])
    return (o.detach(),) + torch.autograd.grad(o, wrt, s["do"])


def work(case):
    """Attention products (4d per score entry forward, 10d backward), filter and mix (2 per tap or head forward, 6
    backward); each input read once, each output written once."""
    c, op = case, case["op"]
    B, H, d = c["B"], c["H"], c["d"]
    if op in ("decode", "paged"):
        # of a ragged batch: lengths are spread over [Nk/8, Nk]
        keys = c["Nk"] if op == "decode" else c["Nk"] * (1.0 + (B - 1) * 0.5625) / B
        rows = min(c["q_len"], c["cq"])
        outs = 1 if op == "decode" else c["splits"]
        return dict(bytes=B * H * (2 * keys * d * 2 + c["q_len"] * d * 2 + outs * (d + 2) * 4),
                    flops=B * H * keys * (2 * d * rows + 2 * c["cq"] * c["ck"] + 2 * d))
    n = B * H * c["N"] * d
    E = B * H * (c["N"] * (c["N"] + 1) / 2 if c["causal"] else c["N"] ** 2)
    taps = (c["cq"] * c["ck"] if op != "headmix" else 0) + (0 if op in ("train", "prefill") else c.get("G", H))
    if op == "prefill":
        return dict(bytes=n * (3 * 2 + 4), flops=E * (4 * d + 2 * taps))
    o = 2 if op == "headmix" else 4
    return dict(bytes=n * (3 * 2 + 2 * o + 3 * 2), flops=E * (14 * d + 8 * taps))


def tolerance(case):
    if case["op"] in ("decode", "paged"):
        # bf16 products are exact in the 32-bit sums, and everything after them is 32-bit
        return {"rel": 5e-5}
    # probabilities, gradients of the scores and filtered keys are bf16 operands of the products
    return {"rel": 1e-2}
