"""What is timed when the performance of this framework is judged: its operators as a user's program
calls them, over the range of sizes, data types and options that they are used with.

Four kinds of work ("op"):
  attend     flash_attention_v2_cutlass on fp8 tensors that are on the GPU already
  quantise   quantize_e4m3 of one fp16 / bf16 tensor
  pipeline   half-precision Q, K, V in, O out: quantize_e4m3 of each, then attention with the descales
  host       HostRunner: fp8 tensors in pinned host memory in, fp16 O in pinned host memory out
"""
import math

import torch

import attention_cutlass_fp8
from cutlass_flash_atten_fp8_b200 import HostRunner, flash_attention_v2_cutlass, quantize_e4m3

FP8 = {"e4m3": torch.float8_e4m3fn, "e5m2": torch.float8_e5m2}
FP8_MAX = {"e4m3": 448.0, "e5m2": 57344.0}
HALF = {"fp16": torch.float16, "bf16": torch.bfloat16}

# the dearest listed case (flops of one pass, and seconds of it at the rate of a memory-bound pass)
LARGEST_FLOPS = 4.0 * 16 * 32 * 4096 * 4096 * 128
LARGEST_BYTES = 2 ** 30


def _attend(name, B, H, Hk, Sq, Sk, D, causal, v, fmt="e4m3", descale="none", data="randn", lse=False, via="package"):
    return {"name": name, "op": "attend", "B": B, "H": H, "Hk": Hk, "Sq": Sq, "Sk": Sk, "D": D, "causal": causal, "v": v,
            "fmt": fmt, "descale": descale, "data": data, "lse": lse, "via": via}


def listed():
    return [
        # The smallest shape of the repository's workloads ("tiny"): one 128-row tile per head, where a call is launch
        # latency and host work.
        _attend("tiny_h2_s128_d64", 1, 2, 2, 128, 128, 64, False, "transposed"),
        # The reference's own benchmark (batch 1, 16-64 heads, S 1024-4096, causal, D 64 / 128, small clamped inputs,
        # scale 1/sqrt(S)), its first shape through the compiled module that carries the reference's name ...
        _attend("refbench_h16_s1024_d64_causal", 1, 16, 16, 1024, 1024, 64, True, "transposed", data="clamp", via="module"),
        # ... and one from its middle through the package's operator.
        _attend("refbench_h32_s2048_d128_causal", 1, 32, 32, 2048, 2048, 128, True, "transposed", data="clamp"),
        # Batched prefill of short prompts at head_dim 64 (the "prefill_s1024_d64" workload).
        _attend("prefill_b16h32_s1024_d64", 16, 32, 32, 1024, 1024, 64, False, "transposed", descale="tensor"),
        # The headline workload of the benchmark ("mid_s4096_d128"): mid-length, outliers in the data, per-tensor scales.
        _attend("mid_b16h32_s4096_d128", 16, 32, 32, 4096, 4096, 128, False, "transposed", descale="tensor", data="outliers"),
        # One long causal sequence ("long_s16384_d128_causal").
        _attend("long_h32_s16384_d128_causal", 1, 32, 32, 16384, 16384, 128, True, "transposed", descale="tensor"),
        # The widest head dim ("mid_s4096_d256_b2").
        _attend("mid_b2h16_s4096_d256", 2, 16, 16, 4096, 4096, 256, False, "natural", descale="tensor", data="outliers"),
        # Cross-attention over ragged lengths: different query and key counts, no multiple of any tile, a head dim between
        # the kernels' own, V as the projection left it, the other fp8 format.
        _attend("cross_b3h20_q1000_k1777_d96_e5m2", 3, 20, 20, 1000, 1777, 96, False, "natural", fmt="e5m2", descale="tensor"),
        # Decoding one token per sequence against an fp8 key/value cache shared by groups of four query heads.
        _attend("decode_b16h32_hk8_k8192_d128", 16, 32, 8, 1, 8192, 128, False, "natural", descale="head"),
        # What a model's layer does in prefill from bf16 activations: one scale per head, grouped key/value heads, causal,
        # with the log-sum-exp.
        {"name": "layer_bf16_b4h32_hk8_s4096_d128_causal", "op": "pipeline", "B": 4, "H": 32, "Hk": 8, "Sq": 4096, "Sk": 4096, "D": 128,
         "causal": True, "half": "bf16", "per_head": True, "lse": True},
        # Putting a whole fp16 key or value tensor into fp8 with one scale.
        {"name": "quantise_fp16_b16h32_s2048_d128", "op": "quantise", "B": 16, "H": 32, "S": 2048, "D": 128, "half": "fp16", "per_head": False},
        # Host tensors in, host tensor out (uploads, kernel and downloads overlap).
        {"name": "host_b4h16_s2048_d128_causal", "op": "host", "B": 4, "H": 16, "Sq": 2048, "D": 128, "causal": True},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _length(rng, lo, hi, step=1):
    """A length between lo and hi, spread over its logarithm; every third one a power of two, the others whatever comes."""
    n = _log_int(rng, lo, hi)
    if rng.random() < 1 / 3:
        n = 2 ** int(round(math.log2(n)))
    return max(step, min(hi, n) // step * step)


def draw(rng):
    """One more case of the listed ones' ranges, at most as dear as the dearest of them."""
    kind = rng.choice(["attend"] * 6 + ["decode", "decode", "pipeline", "pipeline", "quantise", "host"])
    while True:
        B, H = _log_int(rng, 1, 16), rng.choice([1, 2, 4, 8, 12, 16, 20, 24, 32, 40, 64])
        D = rng.choice([64, 64, 128, 128, 128, 128, 256, 32, 96, 160, 192])
        group = rng.choice([g for g in (1, 1, 2, 4, 8) if H % g == 0])
        if kind == "quantise":
            c = {"op": "quantise", "B": B, "H": H, "S": _length(rng, 64, 16384), "D": D, "half": rng.choice(["fp16", "bf16"]),
                 "per_head": rng.random() < 0.5}
        elif kind == "host":
            c = {"op": "host", "B": min(B, 8), "H": min(H, 32), "Sq": _length(rng, 256, 4096, 16), "D": D, "causal": rng.random() < 0.5}
        elif kind == "pipeline":
            S = _length(rng, 128, 8192)
            c = {"op": "pipeline", "B": B, "H": H, "Hk": H // group, "Sq": S, "Sk": S, "D": D, "causal": rng.random() < 0.7,
                 "half": rng.choice(["fp16", "bf16"]), "per_head": rng.random() < 0.5, "lse": rng.random() < 0.5}
        elif kind == "decode":
            c = _attend("", B, H, H // group, rng.choice([1, 1, 1, 2, 4, 7]), _length(rng, 256, 32768), D, False, "natural",
                        descale=rng.choice(["none", "tensor", "head"]), lse=rng.random() < 0.3)
        else:
            v = rng.choice(["transposed", "natural"])
            Sk = _length(rng, 64, 16384, 16 if v == "transposed" else 1)
            Sq = Sk if rng.random() < 0.7 else _length(rng, 64, 8192)
            causal = Sq == Sk and rng.random() < 0.5
            c = _attend("", B, H, H // group, Sq, Sk, D, causal, v, fmt=rng.choice(["e4m3"] * 4 + ["e5m2"]),
                        descale=rng.choice(["none", "tensor", "tensor", "head"]), data=rng.choice(["randn", "randn", "outliers", "clamp"]),
                        lse=rng.random() < 0.2)
            if v == "transposed" and c["descale"] == "none" and not c["lse"] and rng.random() < 0.3:
                c["via"] = "module"
        c.pop("name", None)
        w = work(c)
        if w["flops"] <= LARGEST_FLOPS and w["bytes"] <= (LARGEST_BYTES // 8 if kind == "host" else LARGEST_BYTES):
            return c


def _visible_pairs(c):
    """Query-key pairs of one slice that are not masked (the causal mask is aligned top-left)."""
    Sq, Sk = c["Sq"], c["Sk"]
    if not c["causal"]:
        return Sq * Sk
    n = min(Sq, Sk)
    return n * (n + 1) // 2 + (Sq - n) * Sk


def work(case):
    if case["op"] == "quantise":
        n = case["B"] * case["H"] * case["S"] * case["D"]
        return {"bytes": 3.0 * n, "flops": 0.0}
    c = dict(case)
    c.setdefault("Hk", c["H"])
    c.setdefault("Sk", c["Sq"])
    n_q, n_kv = c["B"] * c["H"] * c["Sq"] * c["D"], c["B"] * c["Hk"] * c["Sk"] * c["D"]
    size = 2.0 if c["op"] == "pipeline" else 1.0
    lse = 4.0 * c["B"] * c["H"] * c["Sq"] if c.get("lse") else 0.0
    return {"bytes": size * (n_q + 2.0 * n_kv) + 2.0 * n_q + lse, "flops": 4.0 * c["B"] * c["H"] * _visible_pairs(c) * c["D"]}


def tolerance(case):
    """Quantisation gives the same bytes.  Attention rounds its probabilities to fp8 (relative steps of 2^-3, 2^-2 for e5m2), and
    that noise is averaged over a row's keys like the output itself, whatever their number.  Measured over these ranges: against
    attention in 64 bits a relative 0.016-0.032 (e5m2 0.041-0.052), against one that rounds the probabilities relative to the
    row's final maximum instead 0.02-0.048 (e5m2 up to 0.07), single values up to 0.7 (1.07) of the larger of themselves and the
    root mean square; for the small clamped inputs, whose probabilities are nearly equal, 0.004-0.013 and 0.05."""
    if case["op"] == "quantise":
        return "exact"
    return {"rel": 0.02, "max": 0.2} if case.get("data") == "clamp" else {"rel": 0.03, "max": 0.95}


def _values(shape, data, gen, device):
    x = torch.randn(shape, generator=gen, device=device)
    if data == "outliers":          # 0.1 % of the entries at +-8 sigma
        u = torch.rand(shape, generator=gen, device=device)
        x = torch.where(u < 0.001, torch.where(u < 0.0005, -8.0, 8.0), x)
    elif data == "clamp":           # the reference's benchmark inputs
        x = x.clamp_(-0.1, 0.1)
    return x


def _fp8(shape, c, gen, device):
    """(x8, descale or None): plain cast, or scaled to the format's largest value per tensor or per (batch, head)."""
    dtype, descale = FP8[c["fmt"]], c["descale"]
    x8 = torch.empty(shape, dtype=dtype, device=device)
    parts = [_values(shape[1:], c["data"], gen, device) for _ in range(shape[0])]
    if descale == "none":
        for b, x in enumerate(parts):
            x8[b] = x.to(dtype)
        return x8, None
    amax = torch.stack([x.abs().amax(dim=(1, 2)) for x in parts])             # [B, heads]
    if descale == "tensor":
        amax = amax.amax().expand_as(amax)
    top = FP8_MAX[c["fmt"]]
    for b, x in enumerate(parts):
        x8[b] = (x * (top / amax[b]).view(-1, 1, 1)).to(dtype)
    d = amax / top
    return x8, (d[0, 0].reshape(1).clone() if descale == "tensor" else d.reshape(-1).contiguous())


def prepare(case, seed):
    device = torch.device("cuda", torch.cuda.current_device())
    gen = torch.Generator(device=device)
    gen.manual_seed(seed)
    c = dict(case)
    if c["op"] == "quantise":
        x = torch.randn((c["B"], c["H"], c["S"], c["D"]), generator=gen, device=device, dtype=torch.float32)
        return {"case": c, "x": x.to(HALF[c["half"]])}
    if c["op"] == "pipeline":
        q, k, v = (torch.randn((c["B"], h, s, c["D"]), generator=gen, device=device, dtype=torch.float32).to(HALF[c["half"]])
                   for h, s in ((c["H"], c["Sq"]), (c["Hk"], c["Sk"]), (c["Hk"], c["Sk"])))
        return {"case": c, "q": q, "k": k, "v": v, "scale": 1.0 / math.sqrt(c["D"])}
    if c["op"] == "host":
        def pinned(*shape):
            x8 = torch.randn(shape, generator=gen, device=device).to(torch.float8_e4m3fn)
            return torch.empty(shape, dtype=x8.dtype, pin_memory=True).copy_(x8)
        B, H, S, D = c["B"], c["H"], c["Sq"], c["D"]
        return {"case": c, "q": pinned(B, H, S, D), "k": pinned(B, H, S, D), "v": pinned(B, H, D, S), "scale": 1.0 / math.sqrt(D),
                "runner": HostRunner(device)}
    s = {"case": c}
    s["q"], dq = _fp8((c["B"], c["H"], c["Sq"], c["D"]), c, gen, device)
    s["k"], dk = _fp8((c["B"], c["Hk"], c["Sk"], c["D"]), c, gen, device)
    s["v"], dv = _fp8((c["B"], c["Hk"], c["Sk"], c["D"]), c, gen, device)
    if c["v"] == "transposed":
        s["v"] = s["v"].transpose(2, 3).contiguous()
    s["scale"] = 1.0 / math.sqrt(c["Sk"] if c["data"] == "clamp" else c["D"])
    s["kw"] = {"return_lse": True} if c["lse"] else {}
    if dq is not None:
        s["kw"].update(descale_q=dq, descale_k=dk, descale_v=dv)
    return s


def run(state):
    c = state["case"]
    if c["op"] == "quantise":
        return quantize_e4m3(state["x"], per_head=c["per_head"])
    if c["op"] == "pipeline":
        q8, dq = quantize_e4m3(state["q"], per_head=c["per_head"])
        k8, dk = quantize_e4m3(state["k"], per_head=c["per_head"])
        v8, dv = quantize_e4m3(state["v"], per_head=c["per_head"])
        return flash_attention_v2_cutlass(q8, k8, v8, c["causal"], state["scale"], v_layout="natural", return_lse=c["lse"],
                                          descale_q=dq, descale_k=dk, descale_v=dv)
    if c["op"] == "host":
        return state["runner"](state["q"], state["k"], state["v"], c["causal"], state["scale"])
    if c["via"] == "module":
        return attention_cutlass_fp8.flash_attention_v2_cutlass(state["q"], state["k"], state["v"], c["causal"], state["scale"])
    return flash_attention_v2_cutlass(state["q"], state["k"], state["v"], c["causal"], state["scale"], v_layout=c["v"], **state["kw"])


def _attention64(q, k, v, causal, scale, rows_at_once=2 ** 26):
    """Softmax attention of one slice in 64 bits, q [Sq, D], k and v [Sk, D]; returns (O, log-sum-exp)."""
    Sq, Sk = q.shape[0], k.shape[0]
    step = max(1, rows_at_once // Sk)
    o = torch.empty((Sq, v.shape[1]), dtype=torch.float64, device=q.device)
    lse = torch.empty((Sq,), dtype=torch.float64, device=q.device)
    for r in range(0, Sq, step):
        s = (q[r:r + step] @ k.T) * scale
        if causal:
            n = s.shape[0]
            s.masked_fill_(torch.arange(Sk, device=q.device) > torch.arange(r, r + n, device=q.device).unsqueeze(1), -math.inf)
        lse[r:r + step] = torch.logsumexp(s, dim=1)
        s -= lse[r:r + step].unsqueeze(1)
        o[r:r + step] = s.exp_() @ v
    return o, lse


def _quantised(x, per_head):
    """What quantize_e4m3 stands for, in plain torch: x * 448 / max|x| in 32 bits, rounded to e4m3; and the scale."""
    amax = x.abs().amax(dim=(2, 3), keepdim=True).float() if per_head else x.abs().amax().float().reshape(1, 1, 1, 1)
    return (x.float() * (448.0 / amax)).to(torch.float8_e4m3fn), (amax.double() / 448.0).reshape(-1)


def exact(case, seed):
    """The outputs of run() in 64 bits from the same fp8 values; the fp8 bytes of a quantisation have none of their own."""
    c = dict(case)
    s = prepare(c, seed)
    if c["op"] == "quantise":
        return None, _quantised(s["x"], c["per_head"])[1]
    q, k, v = s["q"], s["k"], s["v"]
    scale, transposed = s["scale"], c["op"] == "host" or c.get("v") == "transposed"
    d = [s.get("kw", {}).get("descale_" + n) for n in "qkv"]
    if c["op"] == "pipeline":
        (q, dq), (k, dk), (v, dv) = (_quantised(x, c["per_head"]) for x in (q, k, v))
        d = [dq, dk, dv]
    device = torch.device("cuda", torch.cuda.current_device())
    B, H, Sq, D = q.shape
    Hk = k.shape[1]
    o = torch.empty((B, H, Sq, D), dtype=torch.float64, device="cpu" if c["op"] == "host" else device)
    lse = torch.empty((B, H, Sq), dtype=torch.float64, device=device)
    at = lambda t, i: 1.0 if t is None else (t[0] if t.numel() == 1 else t[i]).double()
    for b in range(B):
        for h in range(H):
            hk = h // (H // Hk)
            q1, k1, v1 = (x.to(device).double() for x in (q[b, h], k[b, hk], v[b, hk]))
            if transposed:
                v1 = v1.T
            o1, lse[b, h] = _attention64(q1 * at(d[0], b * H + h), k1 * at(d[1], b * Hk + hk), v1 * at(d[2], b * Hk + hk), c["causal"], scale)
            o[b, h] = o1
    return [o, lse] if c.get("lse") else [o]
