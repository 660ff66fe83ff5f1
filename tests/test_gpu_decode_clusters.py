"""GPU: few query rows of full-int8 where the splits of a K/V head are a cluster of CTAs (scores in shared memory, maxima and results
through distributed shared memory): 1 to 8 CTAs, the last one with one key or all of its keys, one and two row halves, many heads, one
wave and several; on a side stream and in a captured graph."""
import ctypes
import importlib

import pytest
import torch

import test_gpu_decode as base

pytestmark = pytest.mark.gpu


def in_one_kernel(B, Hkv, ratio, Nq, Nk, D, G, causal=True):
    """Does the call take the kernel of this file?  (256 bytes of scratch are asked for there, more for the three kernels.)"""
    lib = importlib.import_module("int-flashattention_b200._lib")
    p = lib.IntfaFwdParams()
    p.B, p.H, p.H_kv, p.Nq, p.Nk, p.D, p.G, p.variant, p.causal = B, Hkv * ratio, Hkv, Nq, Nk, D, G, lib.VARIANT_FULL, int(causal)
    p.sm_scale, p.write_o, p.q_offset = D ** -0.5, 1, Nk - Nq if causal else 0
    return lib.load().intfa_fwd_workspace_bytes(ctypes.byref(p)) == 256


CASES = [
    # B, Hkv, ratio, Nq, Nk, D, G, causal, scales
    (1, 1, 1, 1, 7, 128, 128, True, "fp32"),
    (9, 4, 4, 1, 512, 128, 128, True, "fp16"),                # one CTA
    (1, 2, 4, 2, 513, 128, 128, True, "fp32"),                # two, the second with one key
    (1, 1, 8, 1, 1537, 64, 64, True, "fp16"),
    (1, 2, 1, 5, 2500, 128, 64, False, "fp32"),
    (1, 1, 2, 3, 3583, 64, 128, True, "fp32"),                # seven
    (1, 2, 2, 1, 4096, 128, 128, True, "fp16"),               # eight, all full
    (1, 4, 4, 4, 4000, 128, 128, True, "fp32"),               # eight, 16 rows
    (1, 2, 4, 5, 1025, 64, 64, True, "fp32"),                 # 20 rows: two tiles
    (3, 2, 2, 6, 2047, 64, 128, True, "fp16"),
]


@pytest.mark.parametrize("B,Hkv,ratio,Nq,Nk,D,G,causal,scales", CASES)
def test_splits_as_a_cluster(B, Hkv, ratio, Nq, Nk, D, G, causal, scales, pkg, oracle):
    assert in_one_kernel(B, Hkv, ratio, Nq, Nk, D, G, causal)
    base.test_few_rows_against_a_cache("full", B, Hkv, ratio, Nq, Nk, D, G, causal, scales, pkg, oracle)


@pytest.mark.parametrize("B,Hkv,ratio,Nk,D,G", [
    (10, 40, 1, 1920, 64, 64),        # as many keys as a CTA takes, all of them, in one CTA
    (10, 32, 1, 1367, 64, 64),        # shared memory rounded up
    (5, 82, 1, 1761, 128, 128),       # ... and more of it than a kernel has without asking
    (16, 6, 4, 5700, 128, 64),        # four CTAs of as many keys as they take at 128 channels
    (110, 8, 1, 70, 64, 64),          # two waves, one CTA a head
    (64, 8, 4, 4097, 128, 128),       # four waves of clusters of three
])
def test_many_heads(B, Hkv, ratio, Nk, D, G, pkg, oracle):
    assert in_one_kernel(B, Hkv, ratio, 1, Nk, D, G)
    base.test_long_caches_of_many_heads("full", B, Hkv, ratio, Nk, D, G, pkg, oracle)


def test_calls_that_stay_with_three_kernels():
    """Rules of the choice: more than eight CTAs, one that would hold too many keys, few CTAs with a long chain each."""
    for call in ((1, 8, 4, 1, 32768, 128, 128), (1, 1, 4, 1, 512, 128, 128), (30, 8, 1, 8, 2000, 128, 64), (16, 8, 4, 4, 4097, 128, 128)):
        assert not in_one_kernel(*call), call


def test_on_a_side_stream_and_in_a_graph(pkg):
    g = torch.Generator(device="cuda").manual_seed(3)
    rand = lambda h, n: torch.randn(2, h, n, 128, device="cuda", dtype=torch.float16, generator=g)
    (q8, qs), (k8, ks), (v8, vs) = pkg.quant_pertoken(rand(32, 1)), pkg.quant_pertoken(rand(8, 3000)), pkg.quant_perchannel(rand(8, 3000))
    assert in_one_kernel(2, 8, 4, 1, 3000, 128, 128)
    call = lambda: pkg.attention_full_int8(q8, k8, v8, qs, ks, vs, True, 0.09, q_offset=2999)
    want = call()
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        got = [call() for _ in range(3)]
    torch.cuda.current_stream().wait_stream(side)
    assert all(torch.equal(t, want) for t in got)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        outs = [call() for _ in range(3)]
    for t in outs:
        t.zero_()
    graph.replay()
    graph.replay()
    assert all(torch.equal(t, want) for t in outs)
    pkg.check_status()
