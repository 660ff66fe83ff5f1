"""GPU: a few query rows against a longer K/V cache (the path that packs the heads of a K/V head into one row tile and splits
the keys over the GPU), against the CPU oracle.  Sizes sit at the edges of its tiles: 1 to 16 and more packed rows, key counts
around the 8-, 32-, 64-key steps and the groups of G keys, one split and many, and the last row count the path takes."""
import pytest
import torch

pytestmark = pytest.mark.gpu

CASES = [
    # variant, B, Hkv, ratio, Nq, Nk, D, G, causal, scales
    ("full", 1, 1, 1, 1, 1, 128, 128, True, "fp32"),            # one key
    ("full", 2, 2, 4, 1, 129, 128, 128, True, "fp16"),
    ("full", 1, 2, 8, 1, 1000, 128, 64, True, "fp32"),          # exactly 8 rows
    ("full", 1, 2, 4, 4, 4097, 128, 128, True, "fp16"),         # 16 rows, many splits, odd rows of the scales
    ("full", 1, 1, 8, 5, 777, 128, 128, True, "fp32"),          # 40 rows: three row tiles
    ("full", 1, 3, 1, 32, 65, 64, 64, True, "fp32"),            # one group and one key
    ("full", 1, 2, 1, 3, 2500, 64, 128, False, "fp16"),
    ("full", 1, 1, 1, 2, 20000, 64, 64, True, "fp32"),          # 40 splits of the fewest keys
    ("full", 1, 2, 1, 256, 256, 64, 64, True, "fp32"),          # short prompts: the most rows a head, causal over the whole tile
    ("full", 1, 2, 2, 131, 700, 128, 128, True, "fp16"),
    ("half", 1, 2, 1, 77, 77, 64, 128, True, "fp32"),
    ("half", 1, 1, 2, 200, 1100, 128, 128, False, "fp16"),
    ("half", 1, 1, 1, 1, 1, 64, 128, True, "fp32"),
    ("half", 2, 2, 4, 1, 31, 128, 128, True, "fp16"),
    ("half", 1, 2, 8, 2, 1025, 128, 128, True, "fp32"),
    ("half", 1, 1, 4, 9, 4100, 128, 64, True, "fp16"),          # 36 rows
    ("half", 1, 3, 1, 32, 200, 64, 128, False, "fp32"),
    ("half", 1, 2, 4, 1, 9000, 64, 128, True, "fp32"),
]


@pytest.mark.parametrize("variant,B,Hkv,ratio,Nq,Nk,D,G,causal,scales", CASES)
def test_few_rows_against_a_cache(variant, B, Hkv, ratio, Nq, Nk, D, G, causal, scales, pkg, oracle):
    dev = torch.device("cuda:0")
    g = torch.Generator().manual_seed(Nk + 7 * Nq + D)
    H = Hkv * ratio
    q = torch.randn(B, H, Nq, D, generator=g).half()
    k, v = (torch.randn(B, Hkv, Nk, D, generator=g).half() for _ in range(2))
    k[:, :, Nk // 2:] *= 2                                       # the running maximum moves late as well
    q8, qs = oracle.quant_pertoken(q)
    k8, ks = oracle.quant_pertoken(k)
    sm, off = D ** -0.5, (max(0, Nk - Nq) if causal else 0)
    rep = lambda t: t.repeat_interleave(ratio, dim=1)
    if scales == "fp32":
        qs, ks = qs.float(), ks.float()
    if variant == "full":
        v8, vs = oracle.quant_perchannel(v)
        ref, (m, l, _) = oracle.int8_attention(q8, rep(k8), rep(v8), qs, rep(ks), rep(vs), causal, sm, variant="full", G=G,
                                               q_offset=off, return_state=True)
        args = [t.to(dev) for t in (q8, k8, v8, qs, ks, vs)]
        out, lse = pkg.attention_full_int8(*args, causal, sm, G=G, q_offset=off, return_lse=True)
    else:
        ref, (m, l, _) = oracle.int8_attention(q8, rep(k8), rep(v), qs, rep(ks), None, causal, sm, variant="half", G=G,
                                               q_offset=off, return_state=True)
        args = [t.to(dev) for t in (q8, k8, v, qs, ks)]
        out, lse = pkg.attention_int8(*args, causal, sm, G=G, q_offset=off, return_lse=True)
    pkg.check_status()
    e = oracle.err_metrics(out.cpu(), ref)
    assert e["max_abs"] <= 4e-3 and e["mean_rel"] <= 3e-4, e
    assert (lse.cpu() - oracle.log2_lse(m, l)).abs().max() < 1e-3
    fn = pkg.attention_full_int8 if variant == "full" else pkg.attention_int8
    again = fn(*args, causal, sm, G=G, q_offset=off, out_dtype=torch.bfloat16)
    assert ((again.float() - out.float()).abs() <= out.float().abs() * (2.0 ** -8 + 2.0 ** -11) + 1e-7).all()


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("Nq,Nk", [(1, 77), (77, 77), (2, 4097), (3, 8)])
def test_an_infinity_in_the_last_key_of_v(Nq, Nk, D, pkg, oracle):
    """It reaches its own channel only, as an infinity: the keys that fill up the last step weigh nothing."""
    g = torch.Generator().manual_seed(Nk + D)
    q, k, v = (torch.randn(1, 2, n, D, generator=g).half() for n in (Nq, Nk, Nk))
    v[:, :, -1, 3] = float("inf")
    v[:, :, -1, D - 1] = -float("inf")
    (q8, qs), (k8, ks) = oracle.quant_pertoken(q), oracle.quant_pertoken(k)
    out = pkg.attention_int8(*(t.cuda() for t in (q8, k8, v, qs.float(), ks.float())), False, D ** -0.5).cpu()
    v[:, :, -1, 3] = v[:, :, -1, D - 1] = 0
    ref = oracle.attention_int8(q8, k8, v, qs, ks, False, D ** -0.5, G=128)
    assert (out[..., 3] == float("inf")).all() and (out[..., D - 1] == -float("inf")).all()
    out[..., 3], out[..., D - 1] = ref[..., 3], ref[..., D - 1]
    e = oracle.err_metrics(out, ref)
    assert e["max_abs"] <= 4e-3 and e["mean_rel"] <= 3e-4, e


@pytest.mark.parametrize("sm", [1e-27, 1e-30, 1e-37])
@pytest.mark.parametrize("Nq,Nk,G", [(1, 300, 128), (5, 70, 64), (77, 77, 64)])
def test_masked_keys_weigh_nothing_at_any_softmax_scale(Nq, Nk, G, sm, pkg, oracle):
    g = torch.Generator().manual_seed(Nk)
    q, k, v = (torch.randn(1, 2, n, 64, generator=g).half() for n in (Nq, Nk, Nk))
    (q8, qs), (k8, ks), (v8, vs) = oracle.quant_pertoken(q), oracle.quant_pertoken(k), oracle.quant_perchannel(v)
    off = (Nk - Nq) // 3
    ref = oracle.attention_full_int8(q8, k8, v8, qs, ks, vs, True, sm, G=G, q_offset=off)
    out = pkg.attention_full_int8(*(t.cuda() for t in (q8, k8, v8, qs, ks, vs)), True, sm, G=G, q_offset=off)
    e = oracle.err_metrics(out.cpu(), ref)
    assert e["max_abs"] <= 4e-3 and e["mean_rel"] <= 3e-4, e


@pytest.mark.parametrize("variant,B,Hkv,ratio,Nk,D,G", [
    ("full", 115, 2, 1, 8700, 64, 64),        # one split but for the limit of 8192 keys a CTA: a full one and a short one
    ("full", 115, 2, 1, 8700, 64, 128),
    ("full", 15, 10, 1, 6000, 128, 128),      # 2 to 3 splits of many units a warp
    ("full", 10, 10, 9, 5000, 64, 64),        # ... with 16 rows
    ("half", 20, 5, 1, 6000, 64, 128),
    ("half", 15, 10, 12, 4100, 128, 128),
    ("full", 32, 8, 1, 33000, 64, 64),        # more scores than the scratch holds: two slices of the heads and more
    ("full", 66, 5, 9, 13000, 64, 128),
])
def test_long_caches_of_many_heads(variant, B, Hkv, ratio, Nk, D, G, pkg, oracle):
    dev = torch.device("cuda:0")
    g = torch.Generator(device=dev).manual_seed(Nk)
    H = Hkv * ratio
    rand = lambda h, n: torch.randn(B, h, n, D, device=dev, dtype=torch.float16, generator=g)
    (q8, qs), k, v = pkg.quant_pertoken(rand(H, 1)), rand(Hkv, Nk), rand(Hkv, Nk)
    k[:, :, Nk // 2:] *= 2
    k8, ks = pkg.quant_pertoken(k)
    vs = None
    if variant == "full":
        v, vs = pkg.quant_perchannel(v)
        out, lse = pkg.attention_full_int8(q8, k8, v, qs, ks, vs, True, D ** -0.5, G=G, q_offset=Nk - 1, return_lse=True)
    else:
        out, lse = pkg.attention_int8(q8, k8, v, qs, ks, True, D ** -0.5, G=G, q_offset=Nk - 1, return_lse=True)
    pkg.check_status()
    for b, hk in {(0, 0), (B // 2, Hkv - 1), (B // 2, 0), (B - 1, Hkv - 1)}:
        one = lambda t: t[b:b + 1, hk:hk + 1].cpu()
        of = lambda t: t[b:b + 1, hk * ratio:(hk + 1) * ratio].cpu()
        rep = lambda t: one(t).repeat_interleave(ratio, dim=1)
        ref, (m, l, _) = oracle.int8_attention(of(q8), rep(k8), rep(v), of(qs), rep(ks), rep(vs) if vs is not None else None, True, D ** -0.5,
                                               variant=variant, G=G, q_offset=Nk - 1, return_state=True)
        e = oracle.err_metrics(of(out), ref)
        assert e["max_abs"] <= 4e-3 and e["mean_rel"] <= 3e-4, (b, hk, e)
        assert (of(lse) - oracle.log2_lse(m, l)).abs().max() < 1e-3
