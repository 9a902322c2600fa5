"""Performance cases of the framework on one GPU: what a program that uses it has it do, through the public entry points.

A case is a dict of plain values.  ``listed()`` names the fixed ones, ``draw(rng)`` makes another of the same ranges,
``prepare(case, seed)`` builds what a program holds before the call (context, weights, op, inputs), ``run(state)`` is one
pass and returns its outputs, ``work(case)`` the bytes and operations one pass cannot do without and ``tolerance(case)``
how far another correct implementation of the same precision may be off.

Kinds:

``all_scatter``  GEMM + all-scatter of a prepared op (``gemm_all_scatter``): column-parallel projections.
``all_reduce``   GEMM + all-reduce / reduce-scatter of a prepared op (``gemm_all_reduce``, ``gemm_reduce_scatter``):
                 row-parallel projections, from one token to a long prefill.
``gemm``         the one-call product ``gemm(a, bt)``.
``attention``    self-attention over a projection's output (``attention_fwd``).
``decoder``      a forward pass of the decoder stack (``TPDecoder``).
``messages``     a producer / consumer hand-off guarded by flags (``MessagePassing``), both sides on this GPU.
"""
import math

import torch

import iris_b200
from iris_b200.context import Iris
from iris_b200.models.tp_block import TPConfig, TPDecoder
from iris_b200.ops import attention as A
from iris_b200.ops import gemm as G
from iris_b200.ops import p2p

DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32, "int8": torch.int8}
SIZE = {"bf16": 2, "fp16": 2, "fp32": 4, "int8": 1}
HEAD = 128


def listed():
    return [
        # One token through a row-parallel projection: the step of a decode loop, the smallest call there is.
        {"name": "all_reduce_1_token", "kind": "all_reduce", "variant": "auto", "m": 1, "n": 4096, "k": 11008, "dtype": "bf16"},
        # A batch of 128 decoding sequences through the same projection, in half precision.
        {"name": "all_reduce_128_fp16", "kind": "all_reduce", "variant": "auto", "m": 128, "n": 4096, "k": 11008,
         "dtype": "fp16"},
        # A short prefill (or a large decode batch) through it.
        {"name": "all_reduce_1024", "kind": "all_reduce", "variant": "auto", "m": 1024, "n": 4096, "k": 11008, "dtype": "bf16"},
        # The benchmark configuration of bench.py: a long prefill through a column-parallel projection.
        {"name": "all_scatter_8192", "kind": "all_scatter", "m": 8192, "n": 14336, "k": 4096, "dtype": "bf16"},
        # Quantised inference: int8 operands, a projection of the swept list with a long K.
        {"name": "all_scatter_int8", "kind": "all_scatter", "m": 8192, "n": 3584, "k": 14336, "dtype": "int8"},
        # float32 matrices of a medium size (multiplied as tf32).
        {"name": "all_scatter_fp32", "kind": "all_scatter", "m": 2048, "n": 4096, "k": 4096, "dtype": "fp32"},
        # A product of sizes that are no multiples of any tile, made in one call without a prepared op.
        {"name": "gemm_ragged_fp16", "kind": "gemm", "m": 1000, "n": 2504, "k": 1736, "dtype": "fp16"},
        # Attention of a decoder layer in prefill: 16384 tokens, 32 heads.
        {"name": "attention_causal", "kind": "attention", "batch": 8, "seq": 2048, "heads": 32, "causal": True, "dtype": "bf16"},
        # Encoder-style attention of short sequences, with a number of key tiles that is odd.
        {"name": "attention_full_short", "kind": "attention", "batch": 3, "seq": 384, "heads": 5, "causal": False, "dtype": "fp16"},
        # Prefill of 16384 tokens through the four layers of the decoder's default configuration: the largest pass.
        {"name": "decoder_16384", "kind": "decoder", "hidden": 4096, "intermediate": 11008, "layers": 4, "batch": 8, "seq": 2048,
         "variant": "two_shot"},
        # Two short prompts through the same four layers: bound by reading the weights.
        {"name": "decoder_256", "kind": "decoder", "hidden": 4096, "intermediate": 11008, "layers": 4, "batch": 2, "seq": 128,
         "variant": "two_shot"},
        # The message-passing example: eight chunks of 1 MB.
        {"name": "messages_8x1MB", "kind": "messages", "chunks": 8, "chunk_bytes": 1 << 20, "put": True},
    ]


def _log(rng, lo, hi, step=1):
    """A multiple of ``step`` in [lo, hi], spread over the logarithm."""
    v = math.exp(rng.uniform(math.log(lo), math.log(hi + 1)))
    return max(lo, min(hi, int(v) // step * step))


def _draw(rng):
    kind = rng.choice(["all_scatter", "all_scatter", "all_reduce", "all_reduce", "gemm", "gemm", "attention", "attention",
                       "decoder", "messages"])
    if kind == "all_scatter":
        dt = rng.choice(["bf16", "bf16", "fp16", "fp32", "int8"])
        step = 16 // SIZE[dt]   # rows of N and of K elements are multiples of 16 bytes
        return {"kind": kind, "m": _log(rng, 128, 8192), "n": _log(rng, 1024, 14336, step), "k": _log(rng, 1024, 14336, step),
                "dtype": dt}
    if kind == "all_reduce":
        variant = rng.choice(["auto", "auto", "auto", "one_shot", "two_shot", "atomic", "reduce_scatter"])
        m = 128 * _log(rng, 1, 64) if variant == "reduce_scatter" else _log(rng, 1, 8192)
        return {"kind": kind, "variant": variant, "m": m, "n": _log(rng, 1024, 8192, 8), "k": _log(rng, 1024, 14336, 8),
                "dtype": rng.choice(["bf16", "bf16", "fp16"])}
    if kind == "gemm":
        dt = rng.choice(["bf16", "bf16", "fp16", "fp32", "int8"])
        step = 16 // SIZE[dt]
        return {"kind": kind, "m": _log(rng, 1, 4096), "n": _log(rng, 256, 8192, step), "k": _log(rng, 256, 8192, step),
                "dtype": dt}
    if kind == "attention":
        return {"kind": kind, "batch": _log(rng, 1, 8), "seq": 128 * _log(rng, 1, 32), "heads": _log(rng, 1, 32),
                "causal": rng.random() < 0.6, "dtype": rng.choice(["bf16", "bf16", "fp16"])}
    if kind == "decoder":
        heads = rng.choice([4, 8, 16, 32])
        return {"kind": kind, "hidden": heads * HEAD, "intermediate": 8 * (heads * HEAD * 43 // 128), "layers": rng.randint(1, 4),
                "batch": _log(rng, 1, 8), "seq": 128 * _log(rng, 1, 16), "variant": rng.choice(["two_shot", "two_shot", "reduce_scatter"])}
    return {"kind": "messages", "chunks": _log(rng, 1, 64), "chunk_bytes": _log(rng, 4096, 1 << 22, 16), "put": rng.random() < 0.7}


def draw(rng):
    largest = max(_cost(c) for c in listed())
    while True:
        case = _draw(rng)
        if _cost(case) <= largest:
            return case


def _cost(case):
    """Nominal time of a case: what its operations and bytes take at 1.5 PFLOP/s and 6.5 TB/s."""
    w = work(case)
    return max(w["flops"] / 1.5e15, w["bytes"] / 6.5e12)


# ---- contexts -------------------------------------------------------------------------------------------------------
# The outputs of an op may live on its context's heap, which a program keeps while it uses them.  A state that is gone
# leaves its context here, and the next prepare() closes it.
_left = []


class State(dict):
    def __del__(self):
        ctx = self.get("ctx")
        if ctx is not None:
            _left.append(ctx)


def _close_left():
    while _left:
        _left.pop().close()


def _heap(nbytes):
    return (int(nbytes * 1.05) + (160 << 20)) >> 20 << 20


def _operand(shape, dtype, gen, scale=1.0):
    if dtype == "int8":
        return torch.randint(-127, 128, shape, generator=gen, device="cuda", dtype=torch.int8)
    return (torch.randn(shape, generator=gen, device="cuda") * scale).to(DTYPES[dtype])


def prepare(case, seed):
    _close_left()
    gen = torch.Generator(device="cuda").manual_seed(seed)
    kind = case["kind"]
    s = State(case=case)
    if kind in ("all_scatter", "all_reduce", "gemm"):
        m, n, k, dt = case["m"], case["n"], case["k"], case["dtype"]
        a = _operand((m, k), dt, gen)                        # activations
        bt = _operand((n, k), dt, gen, 1.0 / math.sqrt(k))   # weights, K-contiguous
        if kind == "gemm":
            s.update(a=a, bt=bt)
            return s
        rows = -(-m // 256) * 256
        s["ctx"] = iris_b200.iris(_heap(3 * rows * n * SIZE[dt]))   # output and, for the summing variants, two partials
        if kind == "all_scatter":
            s["op"] = G.gemm_all_scatter(s["ctx"], [a], [bt])
        elif case["variant"] == "reduce_scatter":
            s["op"] = G.gemm_reduce_scatter(s["ctx"], [a], [bt])
        else:
            s["op"] = G.gemm_all_reduce(s["ctx"], [a], [bt], variant=case["variant"])
        return s
    if kind == "attention":
        t, w = case["batch"] * case["seq"], case["heads"] * HEAD
        s["qkv"] = _operand((t, 3 * w), case["dtype"], gen)
        s["out"] = torch.empty((t, w), dtype=DTYPES[case["dtype"]], device="cuda")
        return s
    if kind == "decoder":
        cfg = _config(case, seed)
        t, h, i = cfg.tokens, cfg.hidden, cfg.intermediate
        rows = -(-t // 256) * 256
        per_layer = 2 * rows * (2 * h + 3 * h + 2 * i + 6 * h) + 4 * (40 << 20)
        s["ctx"] = iris_b200.iris(_heap(cfg.n_layers * per_layer))
        s["model"] = TPDecoder(s["ctx"], cfg, variant=case["variant"])
        s["x0"] = _operand((t, h), "bf16", gen)   # the embedded tokens of this pass
        s["x"] = torch.empty_like(s["x0"])
        return s
    nbytes = case["chunks"] * case["chunk_bytes"]
    two = Iris.local_world(2, heap_size=_heap(3 * nbytes))
    s["ctx"] = two[0]
    s["producer"], s["consumer"] = [p2p.MessagePassing(c, case["chunks"], case["chunk_bytes"]) for c in two]
    s["producer"].src.copy_(torch.randn(nbytes // 4, generator=gen, device="cuda"))
    return s


def _config(case, seed=0):
    return TPConfig(hidden=case["hidden"], n_heads=case["hidden"] // HEAD, head_dim=HEAD, intermediate=case["intermediate"],
                    n_layers=case["layers"], batch=case["batch"], seq=case["seq"], seed=seed % 100003)


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind in ("all_scatter", "all_reduce"):
        return state["op"]()[0]
    if kind == "gemm":
        return G.gemm(state["a"], state["bt"])
    if kind == "attention":
        return A.attention_fwd(state["qkv"], state["out"], case["batch"], case["seq"], case["heads"], causal=case["causal"])
    if kind == "decoder":
        state["x"].copy_(state["x0"])
        return state["model"].forward([state["x"]])[0]
    state["producer"].run(roles=3, use_put=case["put"])
    return state["consumer"].dst, state["consumer"].out


def work(case):
    kind = case["kind"]
    if kind in ("all_scatter", "all_reduce", "gemm"):
        m, n, k = case["m"], case["n"], case["k"]
        return {"bytes": (m * k + n * k + m * n) * SIZE[case["dtype"]], "flops": 2 * m * n * k}
    if kind == "attention":
        b, q, h = case["batch"], case["seq"], case["heads"]
        pairs = q * (q + 1) // 2 if case["causal"] else q * q
        return {"bytes": 4 * b * q * h * HEAD * 2, "flops": 4 * b * h * pairs * HEAD}
    if kind == "decoder":
        cfg = _config(case)
        t, h, i = cfg.tokens, cfg.hidden, cfg.intermediate
        weights = 4 * h * h + 3 * h * i
        attention = 4 * cfg.batch * h * (cfg.seq * (cfg.seq + 1) // 2)
        return {"bytes": 2 * (cfg.n_layers * weights + 2 * t * h), "flops": cfg.n_layers * (2 * t * weights + attention)}
    return {"bytes": 3 * case["chunks"] * case["chunk_bytes"], "flops": case["chunks"] * case["chunk_bytes"] // 4}


def tolerance(case):
    """About four times the error measured against the same path in 64 bits, which is that of the rounded results (16 bits)
    or operands (tf32) and, where parts of a sum meet as 16-bit values or pass through several layers, of those roundings."""
    kind, dt = case["kind"], case.get("dtype")
    if kind == "messages" or dt == "int8":
        return "exact"   # copies and doubled floats; the low 8 bits of integer sums
    if kind == "decoder":
        return {"rel": 3e-2, "max": 0.3}       # 1.1e-2 .. 1.3e-2, largest 8e-2
    if kind == "attention":
        return {"rel": 9e-3, "max": 0.14} if dt == "bf16" else {"rel": 1.2e-3, "max": 2e-2}   # 2.3e-3, 3.5e-2; 2.8e-4
    if dt == "fp32":
        return {"rel": 3e-3, "max": 1e-2}      # 7.8e-4, 2.3e-3
    if kind == "all_reduce":
        return {"rel": 1.6e-2, "max": 0.1} if dt == "bf16" else {"rel": 2e-3, "max": 1e-2}    # 4.0e-3, 2.3e-2; 3.9e-4
    return {"rel": 7e-3, "max": 1.6e-2} if dt == "bf16" else {"rel": 9e-4, "max": 2e-3}       # 1.7e-3, 3.9e-3; 2.1e-4


# ---- the same results in 64 bits ------------------------------------------------------------------------------------
def exact(case, seed):
    """What ``run`` returns for these inputs, from plain torch in float64 and the definitions of the operations."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    kind = case["kind"]
    if kind in ("all_scatter", "all_reduce", "gemm"):
        a = _operand((case["m"], case["k"]), case["dtype"], gen)
        bt = _operand((case["n"], case["k"]), case["dtype"], gen, 1.0 / math.sqrt(case["k"]))
        c = a.double() @ bt.double().t()
        if case["dtype"] == "int8":   # sums below 2^28, exact in float64; the low 8 bits of each
            c = c.to(torch.int64).to(torch.int8)
        return c
    if kind == "attention":
        t, w = case["batch"] * case["seq"], case["heads"] * HEAD
        return _exact_attention(_operand((t, 3 * w), case["dtype"], gen).double(), case["batch"], case["seq"], case["heads"],
                                case["causal"])
    if kind == "decoder":
        cfg = _config(case, seed)
        return _exact_decoder(_operand((cfg.tokens, cfg.hidden), "bf16", gen).double(), cfg)
    src = torch.randn(case["chunks"] * case["chunk_bytes"] // 4, generator=gen, device="cuda").double()
    return src, 2 * src


def _exact_attention(qkv, batch, seq, heads, causal):
    q, k, v = qkv.view(batch, seq, 3, heads, HEAD).unbind(2)
    out = torch.empty((batch, seq, heads, HEAD), dtype=torch.float64, device=qkv.device)
    later = torch.ones((seq, seq), dtype=torch.bool, device=qkv.device).triu(1)   # keys after the query
    for b in range(batch):
        for h in range(heads):
            s = q[b, :, h] @ k[b, :, h].t() / math.sqrt(HEAD)
            if causal:
                s.masked_fill_(later, -math.inf)
            out[b, :, h] = torch.softmax(s, -1) @ v[b, :, h]
    return out.view(batch * seq, heads * HEAD)


def _exact_decoder(x, cfg):
    h, i = cfg.hidden, cfg.intermediate

    def norm(t):   # the norms' weights are ones
        return t * torch.rsqrt(t.pow(2).mean(-1, keepdim=True) + cfg.eps)
    for layer in range(cfg.n_layers):
        gen = torch.Generator(device="cuda").manual_seed(cfg.seed * 1000 + layer)
        wq, wk, wv, wo, wg, wu, wd = [(torch.randn(s, generator=gen, device="cuda") * cfg.std).to(torch.bfloat16).double()
                                      for s in ((h, h), (h, h), (h, h), (h, h), (i, h), (i, h), (h, i))]
        n = norm(x)
        a = _exact_attention(torch.cat([n @ wq.t(), n @ wk.t(), n @ wv.t()], 1), cfg.batch, cfg.seq, cfg.n_heads, True)
        x = x + a @ wo.t()
        n = norm(x)
        x = x + (torch.nn.functional.silu(n @ wg.t()) * (n @ wu.t())) @ wd.t()
    return x
