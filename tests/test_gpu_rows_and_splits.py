"""GPU: the per-token quantiser at row counts around its groups of four rows a lane, every scale significand against many
quotients; and the sum of the splits of the few-rows path, from two splits to more than one group of threads takes at once."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D", [16, 32, 64, 128, 256])
@pytest.mark.parametrize("N", [1, 3, 67, 4099])
def test_rows_of_the_quantiser(D, N, pkg, oracle):
    g = torch.Generator().manual_seed(D + N)
    x = torch.randn(2, 3, N, D, generator=g).half()
    x[:, :, ::5] *= torch.rand(2, 3, (N + 4) // 5, 1, generator=g).half() * 2.0 ** -12       # scales below the normal range
    x[0, 0, 0] = 0
    got, want = pkg.quant_pertoken(x.cuda()), oracle.quant_pertoken(x)
    assert torch.equal(got[0].cpu(), want[0]) and torch.equal(got[1].cpu(), want[1].float().nan_to_num())
    y = torch.cat([x, x], dim=3)[..., ::2].transpose(1, 2).contiguous().transpose(1, 2)       # rows that are not contiguous
    got, want = pkg.quant_pertoken(y.cuda()), oracle.quant_pertoken(y)
    assert torch.equal(got[0].cpu(), want[0]) and torch.equal(got[1].cpu(), want[1].float().nan_to_num())


@pytest.mark.parametrize("shift", [-20, -3, 0, 3])
def test_every_significand_of_scale_and_quotient(shift, pkg, oracle):
    """Rows of 256 values below each absmax significand: eight sweeps of X/S over the fp16 significands of both."""
    sig = torch.arange(1024, 2048, dtype=torch.float64)
    amax = (sig * 2.0 ** (shift - 4)).half()                                                  # [1024]
    x = (torch.arange(1024, 2048, dtype=torch.float64).reshape(4, 1, 256) * 2.0 ** (shift - 5)).half().repeat(1, 1024, 1)
    x = torch.cat([x, (x.double() / 2).half()]).clone()                                       # [8, 1024, 256]
    x[..., 0] = amax
    x = x[None]
    for q, ref in ((pkg.quant_pertoken, oracle.quant_pertoken),):
        got, want = q(x.cuda()), ref(x)
        assert torch.equal(got[0].cpu(), want[0]) and torch.equal(got[1].cpu(), want[1].float())
    v = x.transpose(2, 3).reshape(1, 8, 4, 64, 1024).transpose(3, 4).reshape(1, 32, 1024, 64).contiguous()
    got, want = pkg.quant_perchannel(v.cuda()), oracle.quant_perchannel(v)
    assert torch.equal(got[0].cpu(), want[0]) and torch.equal(got[1].cpu().reshape(-1), want[1].float().reshape(-1))


@pytest.mark.parametrize("variant,Nk,D", [("half", 1030, 128), ("half", 1540, 128), ("half", 2500, 64), ("half", 33000, 128),
                                          ("half", 70001, 64), ("full", 2100, 128), ("full", 2600, 64), ("full", 33000, 128),
                                          ("full", 70001, 64)])
def test_sum_of_the_splits(variant, Nk, D, pkg, oracle):
    g = torch.Generator().manual_seed(Nk)
    q, k, v = (torch.randn(1, 1, n, D, generator=g).half() for n in (2, Nk, Nk))
    k[:, :, Nk // 2:] *= 2
    (q8, qs), (k8, ks) = oracle.quant_pertoken(q), oracle.quant_pertoken(k)
    args, vs = [q8, k8, v, qs.float(), ks.float()], None
    if variant == "full":
        args[2], vs = oracle.quant_perchannel(v)
    ref, (m, l, _) = oracle.int8_attention(*args, vs, False, D ** -0.5, variant=variant, G=64, return_state=True)
    op = pkg.attention_full_int8 if variant == "full" else pkg.attention_int8
    dev = [t.cuda() for t in args] + ([vs.cuda()] if variant == "full" else [])
    out, lse = op(*dev, False, D ** -0.5, G=64, return_lse=True)
    pkg.check_status()
    e = oracle.err_metrics(out.cpu(), ref)
    assert e["max_abs"] <= 4e-3 and e["mean_rel"] <= 3e-4, e
    assert (lse.cpu() - oracle.log2_lse(m, l)).abs().max() < 1e-3
