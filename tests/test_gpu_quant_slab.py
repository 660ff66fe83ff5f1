"""V quantised in one pass by a cluster of CTAs that keeps it in registers: the edges of the chunks, of the loads a thread makes
and of the lengths that take this path, for every head dim, both scale modes, and V as a view of [B, N, H, D] storage."""
import pytest
import torch

pytestmark = pytest.mark.gpu

# rows that one CTA loads at a time are 2048/D; a cluster of 8 CTAs holds 8 * 16 of those
CASES = [(D, N) for D in (16, 32, 64, 128, 256)
         for N in sorted({1, 2048 // D - 1, 4 * 2048 // D, 4 * 2048 // D + 1, 32 * 2048 // D, 32 * 2048 // D + 1, 64 * 2048 // D + 1,
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
