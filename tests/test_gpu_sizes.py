"""GPU: tensors that are too short for the sizes of a call are refused by the host, before anything runs."""
import pytest
import torch

pytestmark = pytest.mark.gpu

B, H, HKV, D = 2, 4, 2, 64


def _tensors(Nq, Nk, variant, v_scale=3, G=64):
    dev = "cuda:0"
    i8 = lambda h, n: torch.zeros(B, h, n, D, dtype=torch.int8, device=dev)
    t = {"q": i8(H, Nq), "k": i8(HKV, Nk), "v": i8(HKV, Nk), "qs": torch.ones(B, H, Nq, device=dev), "ks": torch.ones(B, HKV, Nk, device=dev),
         "vs": torch.ones({2: (B, HKV), 3: (B, HKV, D), 4: (B, HKV, (Nk + G - 1) // G, D)}[v_scale], device=dev)}
    if variant == "half":
        t["v"], t["vs"] = t["v"].half(), None
    return t


def _call(pkg, t, causal=False, **kw):
    if t["vs"] is None:
        return pkg.attention_int8(t["q"], t["k"], t["v"], t["qs"], t["ks"], causal, 0.125, **kw)
    return pkg.attention_full_int8(t["q"], t["k"], t["v"], t["qs"], t["ks"], t["vs"], causal, 0.125, **kw)


def _cut(x, dim):
    return x.narrow(dim, 0, x.shape[dim] - 1).contiguous()


@pytest.mark.parametrize("variant", ["full", "half"])
@pytest.mark.parametrize("Nq,Nk", [(128, 256), (130, 200), (1, 300)])
def test_short_tensors_are_refused(variant, Nq, Nk, pkg):
    t = _tensors(Nq, Nk, variant)
    _call(pkg, t)
    for name, dims in (("k", (0, 1)), ("v", (0, 1, 2)), ("qs", (0, 1, 2)), ("ks", (0, 1, 2)), ("vs", (0, 1, 2))):
        for dim in dims if t[name] is not None else ():
            with pytest.raises(ValueError):
                _call(pkg, dict(t, **{name: _cut(t[name], dim)}))
    pkg.check_status()


@pytest.mark.parametrize("v_scale,dims", [(2, (0, 1)), (4, (0, 1, 2, 3))])
def test_short_v_scales_are_refused(v_scale, dims, pkg):
    t = _tensors(128, 200, "full", v_scale)
    _call(pkg, t, G=64)
    for dim in dims:
        with pytest.raises(ValueError):
            _call(pkg, dict(t, vs=_cut(t["vs"], dim)), G=64)


def test_a_k_scale_of_another_length_on_a_ragged_call_is_refused(pkg):
    t = _tensors(130, 200, "full")
    for n in (199, 201, 256):
        with pytest.raises(ValueError):
            _call(pkg, dict(t, ks=torch.ones(B, HKV, n, device="cuda:0")), G=64)


@pytest.mark.parametrize("variant", ["full", "half"])
@pytest.mark.parametrize("Nq,Nk", [(1, 77), (130, 200)])
def test_one_k_scale_for_all_keys_of_a_ragged_call(variant, Nq, Nk, pkg):
    g = torch.Generator().manual_seed(2)
    t = _tensors(Nq, Nk, variant)
    for n in ("q", "k", "v"):
        t[n] = torch.randint(-127, 128, t[n].shape, generator=g).to(t[n].dtype).cuda()
    one = torch.tensor([[1.0, 2.0], [0.5, 3.0]], device="cuda:0").view(B, HKV, 1) / 500
    for dtype in (torch.float32, torch.float16):
        got = _call(pkg, dict(t, ks=one.to(dtype)), True, q_offset=Nk - Nq)
        assert torch.equal(got, _call(pkg, dict(t, ks=one.to(dtype).expand(B, HKV, Nk).contiguous()), True, q_offset=Nk - Nq))


def test_longer_tensors_are_read_in_part(pkg):
    g = torch.Generator().manual_seed(1)
    t = _tensors(128, 256, "full")
    for n in ("q", "k", "v"):
        t[n] = torch.randint(-127, 128, t[n].shape, generator=g).to(torch.int8).cuda()
    want = _call(pkg, t)
    pad = lambda x, dim: torch.cat([x, x], dim)
    for name, dim in (("k", 0), ("v", 0), ("v", 2), ("qs", 2), ("ks", 2), ("ks", 0)):
        assert torch.equal(_call(pkg, dict(t, **{name: pad(t[name], dim)})), want), (name, dim)


def test_short_state_is_refused(pkg):
    t = _tensors(130, 256, "full")
    _, state = _call(pkg, t, return_state=True, write_o=False)
    _call(pkg, t, state=state)
    for i in range(3):
        with pytest.raises(ValueError):
            _call(pkg, t, state=[_cut(x, 2) if i == j else x for j, x in enumerate(state)])
    with pytest.raises(ValueError):
        _call(pkg, t, state=[x.cpu() for x in state])


@pytest.mark.parametrize("variant", ["full", "half"])
def test_the_prologue_refuses_short_tensors(variant, pkg):
    q, k, v = (torch.ones(B, h, n, D, dtype=torch.float16, device="cuda:0") for h, n in ((H, 130), (HKV, 200), (HKV, 200)))
    pkg.int_flash_attention(q, k, v, True, 0.125, variant=variant)
    for bad in ((q, _cut(k, 0), _cut(v, 0)), (q, k, _cut(v, 2)), (q, k, _cut(v, 0)), (q, _cut(k, 0), v)):
        with pytest.raises(ValueError):
            pkg.int_flash_attention(*bad, True, 0.125, variant=variant)
    for bad in ((q, _cut(k, 0)), (q, k[..., :32].contiguous())):
        with pytest.raises(ValueError):
            pkg.quant_qkv(*bad)
    pkg.check_status()


def test_options_take_any_number(pkg):
    g = torch.Generator().manual_seed(3)
    t = _tensors(130, 200, "full")
    for n in ("q", "k", "v"):
        t[n] = torch.randint(-127, 128, t[n].shape, generator=g).to(torch.int8).cuda()
    t["qs"] *= 0.01
    t["ks"] *= 0.01
    args = [t[n] for n in ("q", "k", "v", "qs", "ks", "vs")]
    want = pkg.attention_full_int8(*args, True, 0.125, G=64, q_offset=70, kv_offset=0, debug_tap=(1, 0))
    got = pkg.attention_full_int8(*args, True, "0.125", G=64.0, q_offset=torch.tensor(70.0), kv_offset=0.0, debug_tap=[1.0, torch.tensor(0)])
    assert torch.equal(got[0], want[0]) and torch.equal(got[1][0], want[1][0])
    for kw in ({"G": "wide"}, {"q_offset": float("nan")}, {"debug_tap": (1, "x")}, {"debug_tap": (1, 2, 3)}):
        with pytest.raises(ValueError):
            pkg.attention_full_int8(*args, True, 0.125, **kw)
    for kw in ({"q_offset": None}, {"debug_tap": 1}, {"debug_tap": ([], 0)}):
        with pytest.raises(TypeError):
            pkg.attention_full_int8(*args, True, 0.125, **kw)
