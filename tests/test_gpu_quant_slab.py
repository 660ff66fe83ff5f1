"""V quantised in one pass by a cluster of CTAs that keeps it in registers: the edges of the chunks, of the loads a thread makes
and of the lengths that take this path, for every head dim, both scale modes, and V as a view of [B, N, H, D] storage."""
import pytest
import torch

pytestmark = pytest.mark.gpu

# rows that one CTA loads at a time are 2048/D; a cluster of 8 CTAs holds 8 * 16 of those
CASES = [(D, N) for D in (16, 32, 64, 128, 256)
         for N in sorted({1, 2048 // D - 1, 4 * 2048 // D, 4 * 2048 // D + 1, 32 * 2048 // D, 32 * 2048 // D + 1, 64 * 2048 // D + 1, 80 * 2048 // D, 80 * 2048 // D + 1,
                          128 * 2048 // D - 1, 128 * 2048 // D, 128 * 2048 // D + 1}) if N > 0]


@pytest.mark.parametrize("D,N", CASES)
def test_v_in_one_pass(D, N, pkg, oracle):
    g = torch.Generator().manual_seed(N * 1000 + D)
    B, H, dev = 2, 3, torch.device("cuda:0")
    v = torch.randn(B, N, H, D, generator=g).half().transpose(1, 2)          # a view: [B, H, N, D] of [B, N, H, D] storage
    v[:, 1, :, 3] = 0                                                         # an all-zero channel
    v[0, 2] = 0                                                               # an all-zero head
    v[1, 0, N - 1, 5] = 300.0                                                 # the maximum in the last row
    for mode, quant in (("per_channel", oracle.quant_perchannel), ("per_tensor", oracle.quant_pertensor)):
        r8, rs = quant(v)
        zero = (rs == 0)[:, :, None, :] if mode == "per_channel" else (rs == 0)[:, :, None, None]
        r8 = torch.where(zero, torch.zeros_like(r8), r8)                     # (the reference has 0/0 there)
        for t in (v.to(dev), v.contiguous().to(dev)):
            v8, vs = (pkg.quant_perchannel if mode == "per_channel" else pkg.quant_pertensor)(t)
            assert torch.equal(v8.cpu(), r8) and torch.equal(vs.cpu(), rs.float())
        q = torch.randn(B, H, 5, D, generator=g).half().to(dev)
        k = v.contiguous().to(dev)
        q8, qs, k8, ks, v8, vs = pkg.quant_qkv(q, k, v.to(dev), mode)
        assert torch.equal(v8.cpu(), r8) and torch.equal(vs.cpu(), rs.float())
        a8, a_s = pkg.quant_pertoken(k)
        assert torch.equal(k8, a8) and torch.equal(ks, a_s)
        a8, a_s = pkg.quant_pertoken(q)
        assert torch.equal(q8, a8) and torch.equal(qs, a_s)


@pytest.mark.parametrize("B,Hkv,N,D", [
    (5, 64, 65, 64),          # one CTA a head, more of them than fit beside those of Q and K
    (4, 32, 513, 64),         # clusters, the last chunk short
    (4, 32, 1025, 64),        # 5 loads a thread
    (4, 32, 2100, 64),        # 9
    (4, 32, 3001, 64),        # 12
    (2, 40, 512, 128),        # 4
    (2, 32, 257, 256),        # 5
    (2, 20, 1024, 256),       # 16
    (16, 32, 130, 256),       # (two passes: several waves at 256 channels)
    (3, 100, 513, 128),       # (two passes: 5 loads of 8)
])
def test_v_after_q_and_k(B, Hkv, N, D, pkg, oracle):
    """More CTAs than fit at once: Q and K in a launch of their own, V in the next, which reads it before that one has ended."""
    g = torch.Generator(device="cuda").manual_seed(N + D)
    v = torch.randn(B, N, Hkv, D, device="cuda", dtype=torch.float16, generator=g).transpose(1, 2)
    q, k = (torch.randn(B, Hkv, n, D, device="cuda", dtype=torch.float16, generator=g) for n in (max(1, N // 2), N))
    v[:, 1, :, 3] = 0
    v[B - 1, 0, N - 1, 5] = 300.0
    for mode, quant in (("per_channel", oracle.quant_perchannel), ("per_tensor", oracle.quant_pertensor)):
        q8, qs, k8, ks, v8, vs = pkg.quant_qkv(q, k, v, mode)
        a8, a_s = (pkg.quant_perchannel if mode == "per_channel" else pkg.quant_pertensor)(v)
        assert torch.equal(v8, a8) and torch.equal(vs, a_s)
        for b, h in {(0, 1), (B - 1, 0), (B - 1, Hkv - 1), (B // 2, Hkv // 2)}:
            r8, rs = quant(v[b:b + 1, h:h + 1].cpu())
            if mode == "per_channel":
                r8 = torch.where((rs == 0)[:, :, None, :], torch.zeros_like(r8), r8)
            assert torch.equal(v8[b:b + 1, h:h + 1].cpu(), r8) and torch.equal(vs[b:b + 1, h:h + 1].cpu(), rs.float()), (mode, b, h)
        for x, x8, xs in ((q, q8, qs), (k, k8, ks)):
            a8, a_s = pkg.quant_pertoken(x)
            assert torch.equal(x8, a8) and torch.equal(xs, a_s)


@pytest.mark.parametrize("B,H,N,D", [(1, 4, 512, 64), (4, 32, 1025, 64), (2, 40, 700, 128)])       # one launch; two; two
def test_on_a_side_stream_and_in_a_graph(B, H, N, D, pkg):
    g = torch.Generator(device="cuda").manual_seed(N)
    q, k, v = (torch.randn(B, H, N, D, device="cuda", dtype=torch.float16, generator=g) for _ in range(3))
    call = lambda: [*pkg.quant_qkv(q, k, v), *pkg.quant_perchannel(v)]
    want = call()
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        got = [call() for _ in range(2)]
    torch.cuda.current_stream().wait_stream(side)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got += [call() for _ in range(2)]
    for out in got[2:]:
        for t in out:
            t.zero_()
    graph.replay()
    graph.replay()
    for out in got:
        assert all(torch.equal(a, b) for a, b in zip(out, want))
