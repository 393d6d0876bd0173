"""What is timed when this library's speed is judged: calls through the Python binding of the C ABI, over the sizes,
types and options its users run.  Sizes are the baseline configurations (bench.py, the sweep of run_all_config.sh, the
GPU tests) or generic ones; `draw` gives further cases of the same ranges.
"""
import math
import os
import sys

import torch

_PKG = os.path.join(os.getcwd(), "cutlass-kernels_b200")     # the package folder of the tree that is being timed
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)
import cfk_b200  # noqa: E402

LIB = cfk_b200.load()
CODE = {"fp16": cfk_b200.FP16, "bf16": cfk_b200.BF16, "e4m3": cfk_b200.E4M3, "hybrid": cfk_b200.E4M3, "fp32": cfk_b200.FP32}
TORCH = {"fp16": torch.float16, "bf16": torch.bfloat16, "e4m3": torch.float8_e4m3fn, "fp32": torch.float32}
SIZE = {"fp16": 2, "bf16": 2, "e4m3": 1, "fp32": 4}


def _fmha(name, prec, B, H, Sq, Skv, D, causal, lse=False, of_heads=0, out="fp16"):
    c = {"op": "fmha", "prec": prec, "B": B, "H": H, "Sq": Sq, "Skv": Skv, "D": D, "causal": causal, "lse": lse,
         "of_heads": of_heads or H, "out": out}
    return dict(c, name=name) if name else c


def _gemm(name, prec, m, n, k, l=1, row_major=False, alpha=1.0, beta=0.0):
    c = {"op": "gemm", "prec": prec, "m": m, "n": n, "k": k, "l": l, "row_major": row_major, "alpha": alpha, "beta": beta}
    return dict(c, name=name) if name else c


def _convert(name, src, dst, n):
    c = {"op": "convert", "src": src, "dst": dst, "n": n}
    return dict(c, name=name) if name else c


def listed():
    return [
        # the baseline's first configuration: one tiny call, where latency is all there is
        _fmha("attn tiny", "fp16", 1, 2, 128, 128, 64, False),
        # encoder-style attention with the log-sum-exp a later pass needs (baseline configuration)
        _fmha("attn fp16 4k lse", "fp16", 4, 16, 4096, 4096, 128, False, lse=True),
        # long-context causal prefill, the headline benchmark
        _fmha("attn bf16 causal 8k", "bf16", 2, 32, 8192, 8192, 128, True),
        # quantised attention with per-tensor scales (baseline configuration)
        _fmha("attn e4m3 8k", "e4m3", 4, 16, 8192, 8192, 128, False),
        # the reference sweep's smallest and largest head dimensions at dim 2048
        _fmha("attn bf16 causal d64", "bf16", 4, 32, 4096, 4096, 64, True),
        _fmha("attn fp16 d256", "fp16", 4, 8, 4096, 4096, 256, False),
        # a chunk of queries against a longer cache, lengths that no tile divides, output in the model's type
        _fmha("attn chunk ragged", "bf16", 3, 16, 777, 1300, 128, True, lse=True, out="bf16"),
        # one new token per sequence against its cache
        _fmha("attn decode", "bf16", 4, 32, 1, 6001, 128, True, out="bf16"),
        # the baseline's dense GEMM
        _gemm("gemm fp16 8192", "fp16", 8192, 8192, 8192),
        # a projection of a short batch of tokens: tall reduction, few output tiles
        _gemm("gemm fp16 narrow", "fp16", 2048, 768, 4096),
        # small ragged update with both scalars, D = alpha A B + beta C
        _gemm("gemm bf16 ragged", "bf16", 1000, 776, 264, row_major=True, alpha=0.5, beta=2.0),
        # quantising one operand of the e4m3 configuration
        _convert("quantise e4m3", "fp32", "e4m3", 4 * 16 * 8192 * 128),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.random()
    if kind < 0.42:      # prefill: self-attention, or a chunk of queries against a longer cache
        D = rng.choice([64, 128, 128, 256])
        prec = rng.choice(["fp16", "bf16", "bf16", "e4m3"] + (["hybrid"] if D != 256 else []))
        Sq = _log(rng, 32, 16384)
        if Sq >= 256 and rng.random() < 0.5:
            Sq = Sq // 128 * 128
        Skv = Sq if rng.random() < 0.65 else Sq + _log(rng, 16, 8192)
        causal = rng.random() < 0.6
        B, H = _log(rng, 1, 16), _log(rng, 2, 64)
        # the largest listed case is 2.2e12 operations at the fastest type's rate
        room = 5e11 / (4.0 * Sq * Skv * D)
        if room < 1:
            Sq, Skv, room = 4096, 8192, 5e11 / (4.0 * 4096 * 8192 * D)
        while B * H > room:
            if B > 1:
                B = B // 2
            else:
                H = H // 2
        of_heads = H * rng.choice([1, 1, 1, 2, 8])          # a rank's share addresses its heads of the unsharded tensor
        if B * max(Sq, Skv) * of_heads * D > 1 << 29:
            of_heads = H
        return _fmha(None, prec, B, H, Sq, Skv, D, causal, lse=rng.random() < 0.5, of_heads=of_heads,
                     out="bf16" if prec == "bf16" and rng.random() < 0.5 else "fp16")
    if kind < 0.58:      # decode: one or a few new tokens per sequence against its cache
        D = rng.choice([64, 128, 128, 256])
        prec = rng.choice(["fp16", "bf16", "bf16", "e4m3"])
        Sq = 1 if rng.random() < 0.6 else rng.randint(2, 16)
        Skv = _log(rng, 128, 65536)
        B, H = _log(rng, 1, 64), _log(rng, 2, 64)
        while 2 * B * H * Skv * D * SIZE[prec] > 1 << 30 and B * H > 1:
            if B > 1:
                B = B // 2
            else:
                H = H // 2
        return _fmha(None, prec, B, H, Sq, Skv, D, True, lse=rng.random() < 0.5,
                     out="bf16" if prec == "bf16" else "fp16")
    if kind < 0.9:
        prec = rng.choice(["fp16", "fp16", "bf16", "bf16", "fp32"])
        m, n, k = 8 * _log(rng, 1, 1024), 8 * _log(rng, 8, 2048), 8 * _log(rng, 8, 2048)
        l = 1 if rng.random() < 0.75 else rng.randint(2, 16)
        while m * n * k * l > (5.5e11 if prec != "fp32" else 2.5e11):
            if l > 1:
                l = l // 2
            elif n >= k:
                n = max(8, n // 16 * 8)
            else:
                k = max(8, k // 16 * 8)
        beta = rng.choice([0.0, 0.0, 0.0, 1.0, 0.5])
        return _gemm(None, prec, m, n, k, l, row_major=rng.random() < 0.5, alpha=rng.choice([1.0, 1.0, 0.125]), beta=beta)
    src, dst = rng.choice([("fp32", "e4m3"), ("fp32", "e4m3"), ("fp32", "bf16"), ("fp32", "fp16"), ("bf16", "fp32"),
                           ("fp16", "fp32"), ("e4m3", "fp32")])
    return _convert(None, src, dst, _log(rng, 10000, 4 * 16 * 8192 * 128))


def _normal(g, *shape):
    return torch.randn(*shape, generator=g, device="cuda", dtype=torch.float32)


def _to(x, prec):
    """Values of N(0,1) in the stored type; e4m3 with a per-tensor scale amax/448.  Returns (tensor, de-scale)."""
    if prec != "e4m3":
        return x.to(TORCH[prec]), 1.0
    s = float(x.abs().max()) / 448.0
    return (x / s).to(torch.float8_e4m3fn), s


def prepare(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    if case["op"] == "convert":
        x = _normal(g, case["n"])
        scale = 1.0
        if case["dst"] == "e4m3":
            scale = 448.0 / float(x.abs().max())
        x = x.to(TORCH[case["src"]])
        return {"op": "convert", "src": x, "dst": torch.empty(case["n"], dtype=TORCH[case["dst"]], device="cuda"),
                "scale": scale, "codes": (CODE[case["src"]], CODE[case["dst"]]), "n": case["n"]}
    if case["op"] == "gemm":
        m, n, k, l = case["m"], case["n"], case["k"], case["l"]
        dt = TORCH[case["prec"]]
        uniform = lambda *s: torch.rand(*s, generator=g, device="cuda").mul_(2).sub_(1).to(dt)   # noqa: E731
        shape = (l, m, n) if case["row_major"] else (l, n, m)
        return {"op": "gemm", "a": uniform(l, m, k), "b": uniform(l, n, k), "c": torch.empty(shape, dtype=dt, device="cuda"),
                "kw": {"dtype": CODE[case["prec"]], "m": m, "n": n, "k": k, "l": l, "alpha": case["alpha"],
                       "beta": case["beta"], "c_row_major": case["row_major"],
                       "c_src": uniform(*shape) if case["beta"] else None}}
    B, H, Sq, Skv, D, HT = (case[x] for x in ("B", "H", "Sq", "Skv", "D", "of_heads"))
    low, vt = ("e4m3", "fp16") if case["prec"] == "hybrid" else (case["prec"], case["prec"])
    q, qs = _to(_normal(g, B, Sq, HT, D), low)
    k, ks = _to(_normal(g, B, Skv, HT, D), low)
    v, vs = _to(_normal(g, B, Skv, HT, D), vt)
    o = torch.zeros(B, Sq, HT, D, dtype=TORCH[case["out"]], device="cuda")
    kw = {"dtype": CODE[case["prec"]], "batch": B, "heads": H, "seqlen_q": Sq, "seqlen_kv": Skv, "head_dim": D,
          "softmax_scale": 1.0 / math.sqrt(D), "causal": case["causal"], "out_dtype": CODE[case["out"]],
          "q_descale": qs, "k_descale": ks, "v_descale": vs,
          "lse": torch.zeros(B, H, Sq, dtype=torch.float32, device="cuda") if case["lse"] else None,
          "v_fp16": case["prec"] == "hybrid"}
    at = [q, k, v, o]
    if HT != H:          # a head range of the unsharded tensors: pointer offset and the unsharded strides
        off = (HT - H) // 2 * D
        at = [t.data_ptr() + off * t.element_size() for t in at]
        sq, skv = (Sq * HT * D, HT * D, D), (Skv * HT * D, HT * D, D)
        kw.update(q_stride=sq, k_stride=skv, v_stride=skv, o_stride=sq)
    return {"op": "fmha", "held": (q, k, v), "o": o, "at": at, "kw": kw}


def run(state):
    if state["op"] == "convert":
        LIB.convert(state["src"], state["codes"][0], state["dst"], state["codes"][1], state["n"], scale=state["scale"])
        d = state["dst"]
        return d.view(torch.uint8) if d.element_size() == 1 else d
    if state["op"] == "gemm":
        LIB.gemm(state["a"], state["b"], state["c"], **state["kw"])
        return state["c"]
    LIB.fmha_forward(*state["at"], **state["kw"])
    lse = state["kw"]["lse"]
    return state["o"] if lse is None else (state["o"], lse)


def work(case):
    if case["op"] == "convert":
        return {"bytes": case["n"] * (SIZE[case["src"]] + SIZE[case["dst"]]), "flops": 0}
    if case["op"] == "gemm":
        m, n, k, l, e = case["m"], case["n"], case["k"], case["l"], SIZE[case["prec"]]
        return {"bytes": l * e * (m * k + n * k + m * n * (2 if case["beta"] else 1)), "flops": 2.0 * m * n * k * l}
    B, H, Sq, Skv, D = (case[x] for x in ("B", "H", "Sq", "Skv", "D"))
    e = 1 if case["prec"] in ("e4m3", "hybrid") else 2
    ev = 1 if case["prec"] == "e4m3" else 2
    pairs = Sq * Skv - (Sq * (Sq - 1) // 2 if case["causal"] else 0)       # (query, key) pairs the mask leaves
    return {"bytes": B * H * (D * (Sq * (e + 2) + Skv * (e + ev)) + (4 * Sq if case["lse"] else 0)),
            "flops": 4.0 * B * H * D * pairs}


def tolerance(case):
    """Four times what the library shows against the same computation in 64 bits on the stored operands (fp16 attention
    2.9e-4 / 1.4e-3, bf16 2.3e-3 / 1.2e-2, e4m3 2.6e-2 / 0.26 from the rounding of P; GEMM output rounding 2.1e-4 / 5e-4
    and 1.7e-3 / 3.9e-3), capped for e4m3.  fp32 GEMM: its tf32 products are exact in every implementation that truncates
    the operands alike, so only the 32-bit sums differ."""
    if case["op"] == "convert":
        return "exact"
    if case["op"] == "gemm":
        return {"fp16": {"rel": 8e-4, "max": 2e-3}, "bf16": {"rel": 7e-3, "max": 1.6e-2}, "fp32": {"rel": 2e-5, "max": 2e-4}}[case["prec"]]
    return {"fp16": {"rel": 1.2e-3, "max": 6e-3}, "hybrid": {"rel": 1.2e-3, "max": 6e-3}, "bf16": {"rel": 9e-3, "max": 5e-2},
            "e4m3": {"rel": 2.9e-2, "max": 0.6}}[case["prec"]]
