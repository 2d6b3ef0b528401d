"""The calls that a user of the package makes, with the sizes and values they come with, for measuring.

``listed()`` and ``draw(rng)`` give cases, ``prepare`` makes what a program holds before the call (on the GPU, from a
seed), ``run`` is one pass through the public entry points, ``work`` what a pass cannot do without, ``tolerance`` how far
two correct implementations at the same precision lie apart.

Six ways in, by the case's ``kind``:

* ``decode``    one token of a serving loop: ``ops.decode_step`` on key / value / gate caches and the decay state.
* ``prefill``   inference over a prompt: the operator's forward, no gradient (8 kv heads, 4 query heads
                each, head_dim 128, keys and queries of standard deviation 0.5).
* ``train``     an attention layer's training step, as the reference's driver runs it: projections -> ``prepare_inputs``
                (unit keys, sigmoid gates) -> ``UniversalAttention`` -> ``SMVecMatMul`` -> a loss -> gradients of the projections.
* ``operator``  the operator's forward and backward under upstream gradients of its own two outputs (the benchmark's step).
* ``stress``    the same with raw normal keys and gates of sigmoid(N(-4, 2)), one query head per kv head.
* ``attention`` the flash-style ``attention(q, k, v, ...)`` call, forward and backward.
"""
import math

import torch

from universal_attention_triton_b200 import SMVecMatMul, UniversalAttention, ops
from universal_attention_triton_b200.input_prep import prepare_inputs
from universal_attention_triton_b200.Universal_Attention.attention_opt import attention

DTYPES = {"bf16": torch.bfloat16, "fp32": torch.float32}


def _case(kind, dtype, batch, kv_heads, rep, length, chunk, head_dim, **more):
    return dict(kind=kind, dtype=dtype, batch=batch, kv_heads=kv_heads, rep=rep, length=length, chunk=chunk, head_dim=head_dim, **more)


def listed():
    named = {
        # the first replies of one conversation: a few hundred cached tokens, where launch and host latency are everything
        "decode_one_short": _case("decode", "bf16", 1, 8, 4, 512, 128, 64, position=300),
        # a batch of long conversations in a serving loop: one read of the caches per token
        "decode_batch_long": _case("decode", "bf16", 16, 8, 4, 8192, 128, 128, position=6150),
        # a short prompt of an odd number of chunks
        "prefill_short": _case("prefill", "bf16", 1, 8, 4, 640, 128, 64),
        # a long prompt at head_dim 128
        "prefill_long": _case("prefill", "bf16", 1, 8, 4, 8192, 128, 128),
        # the fp32 mode in which a model is checked (bench.py configuration c1)
        "train_fp32": _case("train", "fp32", 1, 2, 2, 256, 64, 64),
        # chunks of 64 keys, the other chunk length of the configurations, in the training type
        "train_chunk64": _case("train", "bf16", 2, 8, 4, 768, 64, 64),
        # a training step on one short sequence: as many blocks as half the chip
        "train_small": _case("train", "bf16", 1, 8, 4, 1024, 128, 64),
        # the layer of a 1B model, batch of four sequences of 4096
        "train_layer": _case("train", "bf16", 4, 8, 4, 4096, 128, 64),
        # the same size as bench.py runs it: both outputs have gradients of their own
        "operator_layer": _case("operator", "bf16", 4, 8, 4, 4096, 128, 64),
        # chunks of 256 keys at head_dim 128
        "operator_chunk256": _case("operator", "bf16", 1, 8, 4, 2048, 256, 128),
        # heavy pruning, one query head per kv head
        "stress_pruning": _case("stress", "bf16", 1, 16, 1, 4096, 128, 128),
        # the flash-style call on a head_dim that is padded
        "attention_dim80": _case("attention", "bf16", 2, 8, 2, 1536, 128, 80),
    }
    return [dict(c, name=n) for n, c in named.items()]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """A case of the ranges between the smallest and the largest listed one of its kind; whole chunks, any number of them."""
    while True:
        kind = rng.choice(["decode", "prefill", "train", "train", "operator", "stress", "attention"])
        dtype, chunk, more = "bf16", 128, {}
        batch, kv_heads, rep, head_dim = _log(rng, 1, 4), rng.choice([4, 8, 8, 16]), rng.choice([1, 2, 4, 4]), rng.choice([64, 64, 128])
        if kind == "decode":
            batch, chunks = _log(rng, 1, 16), _log(rng, 2, 64)
            more["position"] = _log(rng, 100, chunks * chunk - 1)
        elif kind == "prefill":
            chunks = _log(rng, 3, 64)
        elif kind == "train":
            way = rng.choice(["fp32", "chunk64", "usual", "usual", "usual"])
            if way == "fp32":
                dtype, batch, kv_heads, chunk, head_dim, chunks = "fp32", rng.choice([1, 2]), rng.choice([1, 2, 4]), rng.choice([64, 128]), 64, _log(rng, 2, 8)
            elif way == "chunk64":
                chunk, chunks, head_dim, batch = 64, _log(rng, 3, 16), 64, rng.choice([1, 2])
            else:
                chunks = _log(rng, 3, 32)
        elif kind == "operator":
            chunk = rng.choice([128, 128, 256])
            chunks = _log(rng, 4, 32) if chunk == 128 else _log(rng, 2, 8)
        elif kind == "stress":
            rep, head_dim, chunks = 1, 128, _log(rng, 4, 32)
        else:
            chunks, head_dim, rep = _log(rng, 2, 16), rng.choice([48, 64, 80, 96, 128]), rng.choice([1, 2, 4])
        case = _case(kind, dtype, batch, kv_heads, rep, chunks * chunk, chunk, head_dim, **more)
        # never above the largest listed case of its kind (for prefill: 2.2e9 values of output)
        most = {"decode": 16 * 8 * 8192 * 128, "prefill": 8 * 4 * 64 * 8192 * 128, "stress": 16 * 4096 * 4096 * 128,
                "attention": 2 * 16 * 2048 * 2048 * 128}.get(kind, 4 * 8 * 4 * 4096 * 4096 * 64)
        size = batch * kv_heads * chunks * chunk * head_dim
        if kind == "prefill":
            size *= rep * chunks
        elif kind != "decode":
            size *= rep * chunks * chunk
        if size <= most:
            return case


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    dt, b, h, r, L, c, d = (DTYPES[case["dtype"]], case["batch"], case["kv_heads"], case["rep"], case["length"], case["chunk"], case["head_dim"])
    n = L // c

    def normal(*shape, std=1.0, mean=0.0, dtype=dt):
        return (torch.randn(*shape, generator=gen, device="cuda", dtype=torch.float32 if dtype == torch.float32 else dtype) * std + mean).to(dtype)

    def unit(*shape):                                       # keys as the layer hands them over: divided by their length
        k = normal(*shape, dtype=torch.float32)
        return (k / (k.norm(dim=-1, keepdim=True) + 1e-6)).to(dt)

    def gate(*shape, mean=0.0, std=1.0):
        return torch.sigmoid(normal(*shape, mean=mean, std=std, dtype=torch.float32)).to(dt)

    s = {"case": case}
    if case["kind"] == "decode":
        t = case["position"]
        # the decay that the cached keys have met so far: nothing at the last one, more the older the key
        age = torch.arange(t - 1, t - 1 - L, -1, device="cuda", dtype=torch.float32).clamp_min(0.0)
        decay = -0.02 * age * torch.rand(b, h, L, generator=gen, device="cuda")
        s.update(t=t, chunk=c, k=unit(b, h, L, d), v=normal(b, h, L, d), src=gate(b, h, L), q=normal(b, h, r, d), dest=gate(b, h), decay=decay)
    elif case["kind"] == "prefill":
        s["inputs"] = (normal(b, h, n, c, d, std=0.5), normal(b, h, n, c, d, std=0.5), normal(b, h, r, L, d, std=0.5), gate(b, h, n, c), gate(b, h, L))
    elif case["kind"] == "train":
        s["inputs"] = (normal(b, L, h * r, d), normal(b, L, h, d), normal(b, L, h, d), normal(b, L, 2 * h))
        s["chunk"] = c
    elif case["kind"] == "attention":
        s["inputs"] = (normal(b, h * r, L, d), unit(b, h, L, d), normal(b, h, L, d), gate(b, h, L), gate(b, h, L))
        s["g"] = normal(b, h * r, L, d)
    else:
        stress = case["kind"] == "stress"
        gates = dict(mean=-4.0, std=2.0) if stress else {}
        keys = normal(b, h, n, c, d) if stress else unit(b, h, n, c, d)
        s["inputs"] = (keys, normal(b, h, n, c, d), normal(b, h, r, L, d), gate(b, h, n, c, **gates), gate(b, h, L, **gates))
        # gradients as a consumer of the two outputs leaves them: in the strides of the outputs
        s["g_out"] = ops.as_reference_out(normal(b, h, n, r, L, d))
        s["g_denom"] = ops.as_reference_denom(normal(b, h, n, r, L))
    if case["kind"] not in ("decode", "prefill"):
        for x in s["inputs"]:
            x.requires_grad_()
    return s


def run(s):
    kind = s["case"]["kind"]
    if kind == "decode":
        out, lse = ops.decode_step(s["t"], s["k"], s["v"], s["src"], s["q"], s["dest"], s["decay"], s["chunk"])
        return {"out": out, "lse": lse, "decay": s["decay"]}
    x = s["inputs"]
    if kind == "prefill":
        with torch.no_grad():
            out, denom = UniversalAttention.apply(*x)
        return {"out": out, "denom": denom}
    if kind == "train":
        out, denom = UniversalAttention.apply(*prepare_inputs(*x, chunk=s["chunk"], normalize_keys=True, sigmoid_gates=True))
        merged = SMVecMatMul.apply(out, denom)
        loss = merged.float().pow(2).sum()
        return {"loss": loss.detach(), "merged": merged.detach(), "grads": torch.autograd.grad(loss, x)}
    if kind == "attention":
        q, k, v, src, dest = x
        o = attention(q, k, v, True, 1.0, src, dest)
        return {"o": o.detach(), "grads": torch.autograd.grad(o, x, s["g"])}
    out, denom = UniversalAttention.apply(*x)
    return {"out": out.detach(), "denom": denom.detach(), "grads": torch.autograd.grad([out, denom], x, [s["g_out"], s["g_denom"]])}


def work(case):
    """Causal products of the path (one of K K^T, and per query head Q K^T and P V, forward; three and five, backward) over the
    blocks of rows that see a chunk; each input read once and each output written once."""
    b, h, r, L, c, d = (case[k] for k in ("batch", "kv_heads", "rep", "length", "chunk", "head_dim"))
    e = 4 if case["dtype"] == "fp32" else 2
    n = L // c
    if case["kind"] == "decode":
        t = case["position"] + 1
        nt = case["position"] // c + 1
        nbytes = b * h * (t * (2 * d * e + e + 8) + r * d * e + e + nt * r * (d * e + 4))
        return {"bytes": nbytes, "flops": 2 * b * h * t * d * (1 + 2 * r)}
    causal = 2 * b * h * L * L * d * (n + 1) / (2 * n)
    inputs = b * h * L * (2 * d + r * d + 2) * e
    outs = b * h * r * n * L * (d + 1) * e
    if case["kind"] == "prefill":
        return {"bytes": inputs + outs, "flops": causal * (1 + 2 * r)}
    flops = causal * (1 + 2 * r + 3 + 5 * r)
    if case["kind"] in ("train", "attention"):         # the per-chunk outputs do not leave the path
        up = b * h * r * L * d * e if case["kind"] == "attention" else 0
        return {"bytes": 2 * inputs + b * h * r * L * d * e + up, "flops": flops}
    return {"bytes": 2 * inputs + 2 * outs, "flops": flops}


def tolerance(case):
    # fp32: sums of a thousand terms behind cbrt / log1p / exp; bf16: probabilities and score gradients are rounded to
    # eight bits before their products, and the decay gradient is a sum along the rows of such values
    return {"rel": 5e-5} if case["dtype"] == "fp32" else {"rel": 1.5e-2}
