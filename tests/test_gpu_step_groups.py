"""GPU: the softmax groups take KV steps in turn, across work items; so CTAs that run several work items of 1 to 5 steps each
(no multiple of the number of groups), whole and ragged, against the CPU oracle on sampled heads, for every configuration
with its own number of groups, its own hand-over order or its own number of O_j buffers."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("variant,D,G", [("full", 128, 128), ("full", 64, 64), ("full", 32, 32), ("f8", 128, 128), ("half", 128, 128), ("half", 64, 64), ("half", 32, 64), ("half", 128, 64),
                                         ("half", 256, 64), ("f8", 256, 64)])
@pytest.mark.parametrize("N,causal", [(128, False), (257, True), (384, False), (500, False), (640, True)])
def test_step_counts_that_are_no_multiple_of_the_groups(variant, D, G, N, causal, pkg, oracle):
    dev = torch.device("cuda:0")
    B, H = 2, 85                                                 # more work items than SMs
    g = torch.Generator().manual_seed(N + D)
    q, k, v = (torch.randn(B, H, N, D, generator=g).half() for _ in range(3))
    sm = D ** -0.5
    q8, qs = pkg.quant_pertoken(q.to(dev))
    k8, ks = pkg.quant_pertoken(k.to(dev))
    if variant == "full":
        vv, vs = pkg.quant_perchannel(v.to(dev))
        out = pkg.attention_full_int8(q8, k8, vv, qs, ks, vs, causal, sm, G=G)
    else:
        vv = v.to(dev).to(torch.float8_e5m2) if variant == "f8" else v.to(dev)
        out = pkg.attention_int8(q8, k8, vv, qs, ks, causal, sm, G=G)
    pkg.check_status()
    for b, h in ((0, 0), (0, 84), (1, 63)):
        one = lambda t: t[b:b + 1, h:h + 1].cpu()
        if variant == "full":
            ref = oracle.attention_full_int8(one(q8), one(k8), one(vv), one(qs), one(ks), one(vs), causal, sm, G=G)
        else:
            ref = oracle.attention_int8(one(q8), one(k8), one(vv), one(qs), one(ks), causal, sm, G=G)
        e = oracle.err_metrics(one(out), ref)
        assert e["max_abs"] <= 4e-3 and e["mean_rel"] <= 3e-4, (b, h, e)


@pytest.mark.parametrize("variant,D,G", [("full", 128, 128), ("full", 128, 64), ("full", 64, 64), ("full", 32, 32), ("full", 256, 128), ("f8", 128, 128), ("f8", 64, 64),
                                         ("half", 128, 128), ("half", 64, 64), ("half", 256, 64)])
@pytest.mark.parametrize("N", [1280, 1333])
def test_every_step_has_its_own_k_scales(variant, D, G, N, pkg, oracle):
    """Scales that differ from step to step by up to 2^7 (in a period that no ring of slots has), whole and ragged lengths,
    fp32 and fp16: the scales of another step would show."""
    dev = torch.device("cuda:0")
    g = torch.Generator(device=dev).manual_seed(N + D)
    B, H = 1, 31                                                 # several work items a CTA
    i8 = lambda: torch.randint(-127, 128, (B, H, N, D), device=dev, generator=g).to(torch.int8)
    q8, k8 = i8(), i8()
    qs = torch.full((B, H, N), 2.0 ** -7, device=dev)
    step = torch.arange(N, device=dev) // G
    ks = (2.0 ** (-7 - (step * 5 % 11) * 0.7)).half().float().expand(B, H, N).contiguous()
    sm, causal = D ** -0.5, N % 128 != 0
    if variant == "full":
        vv, vs = i8(), torch.rand(B, H, D, device=dev, generator=g) / 64
        run = lambda ks: pkg.attention_full_int8(q8, k8, vv, qs, ks, vs, causal, sm, G=G)
    else:
        vv = torch.randn(B, H, N, D, device=dev, generator=g).half()
        vv = vv.to(torch.float8_e5m2) if variant == "f8" else vv
        run = lambda ks: pkg.attention_int8(q8, k8, vv, qs, ks, causal, sm, G=G)
    out = run(ks)
    assert torch.equal(out, run(ks.half()))
    pkg.check_status()
    for h in (0, 17, 30):
        one = lambda t: t[:, h:h + 1].cpu()
        if variant == "full":
            ref = oracle.attention_full_int8(one(q8), one(k8), one(vv), one(qs), one(ks), one(vs), causal, sm, G=G)
        else:
            ref = oracle.attention_int8(one(q8), one(k8), one(vv), one(qs), one(ks), causal, sm, G=G)
        e = oracle.err_metrics(one(out), ref)
        assert e["max_abs"] <= 4e-3 and e["mean_rel"] <= 3e-4, (h, e)
