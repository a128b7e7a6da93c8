"""The work this framework does for its users, as cases that can be timed: ternary linears, routed-expert (MoE) layers
from one decode token to a 16 384-token step, ternary lookup tables, and the int8 grouped GEMM with the reference
project's own signature.

Values follow the benchmark's synthetic model: trits with P(0) = 0.4 and P(+1) = P(-1) = 0.3, one scale per 128
K-elements ~ lognormal(-4, 0.3) (second stacked term x 0.25), activations and router logits ~ N(0, 1).
"""

import torch

from deepseekternarized_b200.kernels.ternary_b200 import grouped_ternary_gemm
from deepseekternarized_b200.moe import ExpertWeights, MoELayer
from deepseekternarized_b200.ternary.ops import LookupTable, PackedTerm, TernaryLinear
from deepseekternarized_b200.ternary.pack import pack, packed_cols

GROUP = 128
DEV = "cuda"


# ------------------------------------------------------------------------------------------------- the cases
def linear(name, fmt, terms, act, rows, K, N):
    return {"name": name, "kind": "linear", "fmt": fmt, "terms": terms, "act": act, "rows": rows, "K": K, "N": N}


def moe(name, fmt, terms, tokens, experts=384, hidden=4096, inter=2048, top_k=6, flavour="v4", score="softmax", shared=False):
    return {"name": name, "kind": "moe", "fmt": fmt, "terms": terms, "tokens": tokens, "experts": experts, "hidden": hidden,
            "inter": inter, "top_k": top_k, "flavour": flavour, "score": score, "shared": shared}


def listed():
    return [
        # one decode token through one dense projection: the smallest call, latency and launches count
        linear("linear_tq2_1row", "tq2", 1, "bf16", 1, 4096, 4096),
        # a few sequences decoding through a wide projection kept at 1.6 bits per weight (no 2-bit copy: the default)
        linear("linear_tq1_4rows", "tq1", 1, "bf16", 4, 4096, 11008),
        # a short prompt under the default activation mode (per-token int8); the row count fills no tile
        linear("linear_int8_333rows", "tq1", 1, "int8", 333, 4096, 4096),
        # a long prompt through two stacked terms
        linear("linear_k2_2048rows", "tq2", 2, "bf16", 2048, 4096, 11008),
        # MoE layer, one sequence decoding: six experts of two stacked terms
        moe("moe_1tok_k2", "tq2", 2, 1),
        # a small decode batch over 1.6-bit experts, mostly one row per expert
        moe("moe_8tok_tq1", "tq1", 1, 8),
        # a larger decode batch over two stacked terms, router by sqrt(softplus), with the shared expert
        moe("moe_64tok_k2_shared", "tq2", 2, 64, score="sqrtsoftplus", shared=True),
        # prefill of 4096 tokens: about 64 rows per expert
        moe("moe_4096tok_tq1", "tq1", 1, 4096),
        # the benchmark's own step: 16 384 tokens, about 256 rows per expert
        moe("moe_16384tok_tq1", "tq1", 1, 16384),
        # the standard flavour (bf16 intermediates, weights after the experts, top-8 of 64), a ragged prompt
        moe("moe_standard_777tok", "tq2", 1, 777, 64, 2048, 1024, 8, flavour="standard"),
        # 24 looked-up table rows per token of a 16 384-token step, two stacked terms, one record per row
        {"name": "table_rows", "kind": "table", "fmt": "tq1", "terms": 2, "table_rows": 1 << 22, "K": 256, "ids": 24 * 16384},
        # the int8 grouped GEMM as the reference's callers use it: canonical weights, float32 scales, host offsets
        {"name": "grouped_int8_f32", "kind": "grouped", "fmt": "tq2", "experts": 16, "rows": 96, "K": 2048, "N": 2048},
    ]


def _log(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["linear"] * 5 + ["moe"] * 5 + ["table", "grouped"])
    fmt, terms = rng.choice(["tq1", "tq2"]), rng.choice([1, 1, 2])
    if kind == "linear":
        return {"kind": "linear", "fmt": fmt, "terms": terms, "act": rng.choice(["bf16", "bf16", "int8"]), "rows": _log(rng, 1, 4096),
                "K": 128 * _log(rng, 4, 64), "N": _log(rng, 256, 12288)}
    if kind == "moe":
        standard = rng.random() < 0.25
        experts, hidden, inter, top_k = rng.choice([(64, 2048, 1024, 8), (128, 2048, 768, 8), (256, 3072, 1536, 6), (384, 4096, 2048, 6)])
        most = 16384 * 6 * 4096 * 2048 // (top_k * hidden * inter * terms)  # no more multiplications than the largest listed case
        return {"kind": "moe", "fmt": fmt, "terms": terms, "tokens": _log(rng, 1, min(16384, most)), "experts": experts, "hidden": hidden,
                "inter": inter, "top_k": top_k, "flavour": "standard" if standard else "v4",
                "score": "softmax" if standard else rng.choice(["softmax", "sigmoid", "sqrtsoftplus"]),
                "shared": not standard and rng.random() < 0.5}
    if kind == "table":
        return {"kind": "table", "fmt": fmt, "terms": terms, "table_rows": _log(rng, 1 << 16, 1 << 22), "K": rng.choice([128, 256, 512]),
                "ids": _log(rng, 100, 24 * 16384)}
    return {"kind": "grouped", "fmt": fmt, "experts": rng.randint(2, 32), "rows": _log(rng, 4, 256), "K": 32 * _log(rng, 16, 96),
            "N": _log(rng, 256, 3072)}


# ------------------------------------------------------------------------------------------------- inputs
def _trits(gen, rows, K):
    r = torch.randint(0, 10, (rows, K), generator=gen, device=DEV, dtype=torch.int8)
    return (r >= 4).to(torch.int8) - (r >= 7).to(torch.int8) * 2


def _trit_blocks(gen, rows, K):
    """(first row, fresh trits) of consecutive rows, some 64 M weights at a time."""
    step = max(1, (1 << 26) // K)
    for i in range(0, rows, step):
        yield i, _trits(gen, min(step, rows - i), K)


def _packed(gen, E, N, K, fmt):
    """[E, N, packed_cols] of fresh trits."""
    out = torch.empty(E, N, packed_cols(fmt, K), dtype=torch.uint8, device=DEV)
    flat = out.view(E * N, -1)
    for i, t in _trit_blocks(gen, E * N, K):
        flat[i:i + t.size(0)] = pack(t, fmt)
    return out


def _plain(gen, E, N, K):
    """[E, N, K] int8: the trits that _packed draws from the same generator state."""
    out = torch.empty(E * N, K, dtype=torch.int8, device=DEV)
    for i, t in _trit_blocks(gen, E * N, K):
        out[i:i + t.size(0)] = t
    return out.view(E, N, K)


def _scales(gen, term, *shape, dtype=torch.float16):
    s = torch.randn(*shape, generator=gen, device=DEV).mul_(0.3).sub_(4.0).exp_()
    return (s * 0.25 if term else s).to(dtype)


def _experts(gen, E, hidden, inter, fmt, terms):
    w13, s13, w2, s2 = [], [], [], []
    for t in range(terms):
        w13.append(_packed(gen, E, 2 * inter, hidden, fmt))
        s13.append(_scales(gen, t, E, 2 * inter, hidden // GROUP))
        w2.append(_packed(gen, E, hidden, inter, fmt))
        s2.append(_scales(gen, t, E, hidden, inter // GROUP))
    return ExpertWeights(w13, s13, w2, s2, hidden, inter, GROUP, fmt).prepare()


def prepare(case, seed):
    c, gen = case, torch.Generator(device=DEV).manual_seed(seed)
    if c["kind"] == "linear":
        terms = [PackedTerm(_packed(gen, 1, c["N"], c["K"], c["fmt"])[0], _scales(gen, t, c["N"], c["K"] // GROUP)) for t in range(c["terms"])]
        return {"kind": "linear", "layer": TernaryLinear(terms, c["K"], c["fmt"], GROUP, act=c["act"]),
                "x": torch.randn(c["rows"], c["K"], generator=gen, device=DEV).bfloat16()}
    if c["kind"] == "moe":
        w = _experts(gen, c["experts"], c["hidden"], c["inter"], c["fmt"], c["terms"])
        options = {"flavour": c["flavour"]}
        if c["flavour"] == "v4":
            options.update(score_func=c["score"], shared=_experts(gen, 1, c["hidden"], c["inter"], c["fmt"], c["terms"]) if c["shared"] else None)
        return {"kind": "moe", "layer": MoELayer(w, c["top_k"], **options),
                "x": torch.randn(c["tokens"], c["hidden"], generator=gen, device=DEV).bfloat16(),
                "logits": torch.randn(c["tokens"], c["experts"], generator=gen, device=DEV)}
    if c["kind"] == "table":
        terms = [PackedTerm(_packed(gen, 1, c["table_rows"], c["K"], c["fmt"])[0], _scales(gen, t, c["table_rows"], c["K"] // GROUP))
                 for t in range(c["terms"])]
        return {"kind": "table", "table": LookupTable(terms, c["K"], c["fmt"], GROUP),
                "ids": torch.randint(0, c["table_rows"], (c["ids"],), generator=gen, device=DEV)}
    E, T, K, N = c["experts"], c["rows"], c["K"], c["N"]
    ids = torch.randint(0, E, (T,), generator=gen, device=DEV)
    offsets = torch.cat([ids.new_zeros(1), torch.bincount(ids, minlength=E).cumsum(0)])
    return {"kind": "grouped", "fmt": c["fmt"], "K": K, "offsets": offsets.cpu(), "packed": _packed(gen, E, N, K, c["fmt"]),
            "scale": _scales(gen, 0, E, N, -(-K // GROUP), dtype=torch.float32),
            "x": torch.randint(-127, 128, (T, K), generator=gen, device=DEV, dtype=torch.int8),
            "x_scale": torch.rand(T, generator=gen, device=DEV) * 0.02 + 0.01}


def run(state):
    s = state
    if s["kind"] == "linear":
        return s["layer"](s["x"])
    if s["kind"] == "moe":
        return s["layer"](s["x"], s["logits"])
    if s["kind"] == "table":
        return s["table"].rows(s["ids"])
    return grouped_ternary_gemm(s["x"], s["x_scale"], s["offsets"], s["packed"], s["scale"], s["K"], GROUP, s["fmt"])


# ------------------------------------------------------------------------------------------------- the same in 64 bits
def _weight(terms, e, K):
    """[N, K] float64 of matrix e: sum over the stacked terms of trit * group scale."""
    return sum(t[e].double() * s[e].double().repeat_interleave(GROUP, -1)[:, :K] for t, s in terms)


def _plain_experts(gen, E, hidden, inter, terms):
    """(w13, w2) as lists of (trits, scales), drawn in the order of _experts."""
    w13, w2 = [], []
    for t in range(terms):
        w13.append((_plain(gen, E, 2 * inter, hidden), _scales(gen, t, E, 2 * inter, hidden // GROUP)))
        w2.append((_plain(gen, E, hidden, inter), _scales(gen, t, E, hidden, inter // GROUP)))
    return w13, w2


def _expert64(experts, e, x, hidden, inter, row_weight=None):
    gate, up = (x @ _weight(experts[0], e, hidden).T).split(inter, -1)
    h = gate * torch.sigmoid(gate) * up
    return (h if row_weight is None else h * row_weight[:, None]) @ _weight(experts[1], e, inter).T


def exact(case, seed):
    """What run() returns, from the same draws, without any rounding in between (the int8 modes' own quantisation of the
    activations included: it is part of what they compute)."""
    c, gen = case, torch.Generator(device=DEV).manual_seed(seed)
    if c["kind"] == "linear":
        terms = [(_plain(gen, 1, c["N"], c["K"]), _scales(gen, t, c["N"], c["K"] // GROUP)[None]) for t in range(c["terms"])]
        x = torch.randn(c["rows"], c["K"], generator=gen, device=DEV).bfloat16().double()
        if c["act"] == "int8":
            s = x.abs().amax(-1, keepdim=True) / 127
            x = (x / s).round() * s
        return x @ _weight(terms, 0, c["K"]).T
    if c["kind"] == "moe":
        H, I = c["hidden"], c["inter"]
        experts = _plain_experts(gen, c["experts"], H, I, c["terms"])
        shared = _plain_experts(gen, 1, H, I, c["terms"]) if c["flavour"] == "v4" and c["shared"] else None
        x = torch.randn(c["tokens"], H, generator=gen, device=DEV).bfloat16().double()
        logits = torch.randn(c["tokens"], c["experts"], generator=gen, device=DEV).double()
        score = {"softmax": lambda v: v.softmax(-1), "sigmoid": torch.sigmoid,
                 "sqrtsoftplus": lambda v: torch.nn.functional.softplus(v).sqrt()}[c["score"]](logits)
        w, ids = score.topk(c["top_k"], -1)
        w = w / w.sum(-1, keepdim=True)
        y = torch.zeros_like(x)
        for e in range(c["experts"]):
            tok, slot = (ids == e).nonzero(as_tuple=True)
            if tok.numel():
                y.index_add_(0, tok, _expert64(experts, e, x[tok], H, I, w[tok, slot]))
        return y if shared is None else y + _expert64(shared, 0, x, H, I)
    if c["kind"] == "table":
        terms = [(_plain(gen, 1, c["table_rows"], c["K"])[0], _scales(gen, t, c["table_rows"], c["K"] // GROUP)) for t in range(c["terms"])]
        ids = torch.randint(0, c["table_rows"], (c["ids"],), generator=gen, device=DEV)
        return sum(t[ids].double() * s[ids].double().repeat_interleave(GROUP, -1) for t, s in terms)
    E, T, K, N = c["experts"], c["rows"], c["K"], c["N"]
    of = torch.randint(0, E, (T,), generator=gen, device=DEV).sort().values
    terms = [(_plain(gen, E, N, K), _scales(gen, 0, E, N, -(-K // GROUP), dtype=torch.float32))]
    x = torch.randint(-127, 128, (T, K), generator=gen, device=DEV, dtype=torch.int8).double()
    x = x * (torch.rand(T, generator=gen, device=DEV) * 0.02 + 0.01).double()[:, None]
    y = x.new_empty(T, N)
    for e in of.unique().tolist():
        y[of == e] = x[of == e] @ _weight(terms, e, K).T
    return y


# ------------------------------------------------------------------------------------------------- work and tolerance
def _weight_bytes(N, K, fmt, terms, scale_bytes=2):
    return terms * N * (packed_cols(fmt, K) + scale_bytes * -(-K // GROUP))


def work(case):
    c = case
    if c["kind"] == "linear":
        M, K, N = c["rows"], c["K"], c["N"]
        return {"bytes": _weight_bytes(N, K, c["fmt"], c["terms"]) + 2 * M * (K + N), "flops": 2 * M * K * N}
    if c["kind"] == "moe":
        T, E, H, I = c["tokens"], c["experts"], c["hidden"], c["inter"]
        pairs = T * c["top_k"]
        touched = E * (1 - (1 - c["top_k"] / E) ** T)  # experts that the tokens reach, expected for uniform routing
        rows = pairs + (T if c["shared"] else 0)
        per_expert = _weight_bytes(2 * I, H, c["fmt"], c["terms"]) + _weight_bytes(H, I, c["fmt"], c["terms"])
        return {"bytes": int((touched + (1 if c["shared"] else 0)) * per_expert) + 4 * T * E + 4 * T * H, "flops": 6 * rows * H * I}
    if c["kind"] == "table":
        row = c["terms"] * (packed_cols(c["fmt"], c["K"]) + 2 * c["K"] // GROUP)
        return {"bytes": c["ids"] * (8 + row + 2 * c["K"]), "flops": 2 * c["ids"] * c["K"] * c["terms"]}
    T, E, K, N = c["rows"], c["experts"], c["K"], c["N"]
    return {"bytes": int(E * (1 - (1 - 1 / E) ** T)) * _weight_bytes(N, K, c["fmt"], 1, 4) + T * (K + 4) + 4 * T * N, "flops": 2 * T * K * N}


def tolerance(case):
    """Relative 2-norm errors from the rounding of the results, measured against the same path in 64 bits and then
    about four times that: a bf16 output alone is off by 1.7e-3 of its norm (the fp32 sums before it by some 1e-6, by
    7e-5 where activations are held as 15-bit integers); a MoE layer rounds to bf16 after every linear (3.9e-3; 5.8e-3
    in the standard flavour, which rounds every sum, but alike everywhere); the int8 linear quantises its activations,
    which every implementation does alike. Table rows are exact (products with trits, one rounding); the int8 grouped
    GEMM returns float32 sums."""
    if case["kind"] == "table":
        return "exact"
    if case["kind"] == "grouped":
        return {"rel": 1e-5}
    return {"rel": 6e-3 if case["kind"] == "linear" else 1.4e-2}
