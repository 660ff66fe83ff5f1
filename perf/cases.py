"""What is timed: the calls a user of this package makes, from the smallest to the headline workload.

Four kinds of call, told apart by a case's "call":
  attention  fp16 Q/K/V in, attention out: `int_flash_attention`, the quantisation prologue and the forward
  op         the forward on tensors that are quantised already (`attention_full_int8`, `attention_int8`), as the
             reference's benchmark calls it: self-attention, a chunk of a prompt against a longer int8 K/V cache, or
             the decode step (one or a few query rows against the cache)
  quantise   the three quantisers in a row (Q and K per token, V per channel or per tensor), as the accuracy script does
"variant" is full (int8 V and P), half (fp16 V and P) or half_fp8 (float8_e5m2 V and P).  Where Nq < Nk the query rows
are the last ones of the sequence (q_offset = Nk - Nq), and H > Hkv is grouped-query attention.
"""
import importlib
import math

import torch

intfa = importlib.import_module("int-flashattention_b200")


def _case(call, variant, B, H, Nq, D, *, Hkv=None, Nk=None, causal=False, scales="fp32", v_scale="channel",
          out="fp16", outlier=False):
    return {"call": call, "variant": variant, "B": B, "H": H, "Hkv": Hkv or H, "Nq": Nq, "Nk": Nk or Nq, "D": D,
            "causal": causal, "scales": scales, "v_scale": v_scale, "out": out, "outlier": outlier}


def listed():
    cases = {
        # the CPU-runnable configuration of the baseline: one call of a few microseconds of arithmetic
        "call_small": _case("attention", "full", 1, 4, 512, 64),
        # the smallest calls: a short prompt of odd length
        "call_tiny_odd": _case("attention", "half", 1, 8, 77, 64, causal=True),
        # first point of the reference's benchmark sweep (B4 H32 d64, N = 1024 ... 16384), scales as it hands them over:
        # fp16, one V scale per (batch, head)
        "sweep_d64": _case("op", "full", 4, 32, 1024, 64, scales="fp16", v_scale="tensor"),
        # the headline workload: the configuration bench.py times
        "headline": _case("attention", "full", 4, 32, 8192, 128),
        # the half-int8 configuration of the baseline, with its activation outliers
        "half_causal": _case("attention", "half", 8, 32, 4096, 128, causal=True, outlier=True),
        # prompt prefill of a grouped-query model at a length that is no multiple of anything
        "gqa_ragged": _case("attention", "full", 2, 32, 3001, 128, Hkv=8, causal=True),
        # the widest head of the reference's operators
        "wide_head": _case("attention", "half", 2, 16, 4096, 256, causal=True),
        # half-int8 with V (and P) in fp8, bf16 output
        "fp8_v": _case("op", "half_fp8", 2, 32, 2048, 128, causal=True, out="bf16"),
        # chunked prefill: 512 new rows of one sequence against a cache of 8192
        "chunk": _case("op", "full", 1, 32, 512, 128, Hkv=8, Nk=8192, causal=True),
        # decode, a batch of sequences of ordinary length
        "decode_batch": _case("op", "full", 16, 32, 1, 128, Hkv=8, Nk=4097, causal=True),
        # decode, one long sequence, V kept in fp16
        "decode_long": _case("op", "half", 1, 32, 1, 128, Hkv=8, Nk=32768, causal=True),
        # the quantisers by themselves
        "quantise": _case("quantise", "full", 4, 32, 2048, 128),
    }
    return [dict(c, name=n) for n, c in cases.items()]


def _log(rng, lo, hi):
    """A whole number between lo and hi, spread evenly over the logarithm."""
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _cost(c):
    """(score pairs weighted by how much one costs, cached or input elements): what the two limits of draw() apply to."""
    pairs = c["B"] * c["H"] * _pairs(c) * {16: 4, 32: 4, 64: 1.5, 128: 1, 256: 2}[c["D"]]
    return pairs, c["B"] * (c["H"] * c["Nq"] + 2 * c["Hkv"] * c["Nk"]) * c["D"]


def draw(rng):
    kind = rng.choice(("attention", "attention", "attention", "op", "chunk", "chunk", "decode", "decode", "decode", "quantise"))
    ratio = rng.choice((1, 1, 4, 8))
    hkv = rng.choice((1, 2, 4, 8, 8, 16))
    variant = rng.choice(("full", "half"))
    causal = rng.random() < 0.6
    scales = rng.choice(("fp32", "fp32", "fp16"))
    v_scale = rng.choice(("channel", "channel", "tensor"))
    out = rng.choice(("fp16", "fp16", "bf16"))
    if kind == "attention":
        c = _case("attention", variant, _log(rng, 1, 16), hkv * ratio, _log(rng, 32, 16384), rng.choice((32, 64, 64, 128, 128, 128, 256)),
                  Hkv=hkv, causal=causal, v_scale=v_scale, out=out, outlier=rng.random() < 0.3)
    elif kind == "op":
        c = _case("op", rng.choice(("full", "half", "half_fp8")), _log(rng, 1, 16), hkv * ratio, _log(rng, 32, 16384),
                  rng.choice((64, 128)), Hkv=hkv, causal=causal, scales=scales, v_scale=v_scale, out=out)
    elif kind == "chunk":
        n = _log(rng, 64, 2048)
        c = _case("op", variant, _log(rng, 1, 4), hkv * ratio, n, rng.choice((64, 128, 128)), Hkv=hkv, Nk=n + _log(rng, 256, 32768),
                  causal=True, scales=scales, v_scale=v_scale, out=out)
    elif kind == "decode":
        n = rng.choice((1, 1, 1, 2, 4, 8))
        c = _case("op", variant, _log(rng, 1, 64), hkv * ratio, n, rng.choice((64, 128, 128)), Hkv=hkv, Nk=n + _log(rng, 128, 65536),
                  causal=True, scales=scales, v_scale=v_scale, out=out)
    else:
        c = _case("quantise", "full", _log(rng, 1, 16), hkv * ratio, _log(rng, 32, 16384), rng.choice((32, 64, 128, 256)),
                  Hkv=hkv, v_scale=v_scale)
    # no drawn case costs more than the headline workload, in arithmetic or in memory
    top = _cost(listed()[3])
    while any(x > y for x, y in zip(_cost(c), top)):
        if c["B"] > 1:
            c["B"] = (c["B"] + 1) // 2
        elif c["Nq"] == c["Nk"]:
            c["Nq"] = c["Nk"] = c["Nk"] * 3 // 4
        else:
            c["Nk"] = c["Nk"] * 3 // 4
    return c


def _pairs(c):
    """Visible (query row, key) pairs of one head."""
    nq, nk = c["Nq"], c["Nk"]
    return nq * nk - nq * (nq - 1) // 2 if c["causal"] else nq * nk


def prepare(case, seed):
    dev = torch.device("cuda", torch.cuda.current_device())
    g = torch.Generator(device=dev).manual_seed(seed)
    B, H, Hkv, D = case["B"], case["H"], case["Hkv"], case["D"]

    def normal(heads, n):
        return torch.randn(B, heads, n, D, device=dev, dtype=torch.float16, generator=g)

    q, k, v = normal(H, case["Nq"]), normal(Hkv, case["Nk"]), normal(Hkv, case["Nk"])
    if case["outlier"]:                        # one channel of Q and K x20: activation outliers
        ch = seed % D
        q[..., ch] *= 20
        k[..., ch] *= 20
    state = {"case": case, "sm_scale": D ** -0.5,
             "out_dtype": torch.bfloat16 if case["out"] == "bf16" else torch.float16}
    if case["call"] != "op":
        return dict(state, q=q, k=k, v=v)
    (q8, qs), (k8, ks) = intfa.quant_pertoken(q), intfa.quant_pertoken(k)
    if case["variant"] == "full":
        v, vs = intfa.quant_perchannel(v) if case["v_scale"] == "channel" else intfa.quant_pertensor(v)
    else:
        vs = None
        if case["variant"] == "half_fp8":
            v = v.to(torch.float8_e5m2)
    if case["scales"] == "fp16":               # the dtype that follows from quantising fp16 tensors with PyTorch
        qs, ks, vs = qs.half(), ks.half(), None if vs is None else vs.half()
    return dict(state, q=q8, k=k8, v=v, qs=qs, ks=ks, vs=vs, q_offset=case["Nk"] - case["Nq"])


def run(state):
    case = state["case"]
    q, k, v = state["q"], state["k"], state["v"]
    if case["call"] == "attention":
        return intfa.int_flash_attention(q, k, v, case["causal"], state["sm_scale"], variant=case["variant"],
                                         v_mode="per_channel" if case["v_scale"] == "channel" else "per_tensor",
                                         out_dtype=state["out_dtype"])
    if case["call"] == "quantise":
        quant_v = intfa.quant_perchannel if case["v_scale"] == "channel" else intfa.quant_pertensor
        return [*intfa.quant_pertoken(q), *intfa.quant_pertoken(k), *quant_v(v)]
    if case["variant"] == "full":
        return intfa.attention_full_int8(q, k, v, state["qs"], state["ks"], state["vs"], case["causal"], state["sm_scale"],
                                         q_offset=state["q_offset"], out_dtype=state["out_dtype"])
    return intfa.attention_int8(q, k, v, state["qs"], state["ks"], case["causal"], state["sm_scale"],
                                q_offset=state["q_offset"], out_dtype=state["out_dtype"])


def work(case):
    B, H, Hkv, Nq, Nk, D = (case[n] for n in ("B", "H", "Hkv", "Nq", "Nk", "D"))
    rows_q, rows_k = B * H * Nq, B * Hkv * Nk
    if case["call"] == "quantise":             # fp16 in, int8 and scales out; the division and rounding are not counted
        return {"bytes": 3 * D * (rows_q + 2 * rows_k) + 4 * (rows_q + rows_k + B * Hkv * (D if case["v_scale"] == "channel" else 1)),
                "flops": 0}
    flops = 4 * B * H * _pairs(case) * D       # Q K^T and P V
    if case["call"] == "attention":
        return {"bytes": 2 * D * (2 * rows_q + 2 * rows_k), "flops": flops}
    s = 2 if case["scales"] == "fp16" else 4
    v_bytes = 2 if case["variant"] == "half" else 1
    v_scales = 0 if case["variant"] != "full" else B * Hkv * (D if case["v_scale"] == "channel" else 1)
    return {"bytes": D * (3 * rows_q + (1 + v_bytes) * rows_k) + s * (rows_q + rows_k + v_scales), "flops": flops}


def tolerance(case):
    if case["call"] == "quantise":
        return "exact"
    # The quantised operands, the running maximum and the rounding of P are part of the operators' definition, so what is
    # left to an implementation is the last bit of fp32 sums and exponentials and the rounding of the output to 16 bits.
    return {"rel": 4e-3 if case["out"] == "bf16" else 1e-3}
