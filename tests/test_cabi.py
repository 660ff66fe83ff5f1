"""CPU: the C-ABI library loads, exports every symbol include/intfa.h declares, its ctypes mirror
matches the C struct layout, and argument validation answers before anything touches a device."""
import ctypes
import importlib
import os
import re
import subprocess
import sys

import pytest

from conftest import ROOT

HEADER = os.path.join(ROOT, "include", "intfa.h")


@pytest.fixture(scope="module")
def lib():
    L = importlib.import_module("int-flashattention_b200._lib")
    if not os.path.exists(L.LIB_PATH):
        importlib.import_module("int-flashattention_b200.build").build()
    return L


def declared_functions():
    src = open(HEADER).read()
    src = re.sub(r"/\*.*?\*/", "", src, flags=re.S)
    return sorted(set(re.findall(r"\b(intfa_\w+)\s*\(", src)))


def test_every_declared_symbol_is_exported(lib):
    names = declared_functions()
    assert len(names) >= 9
    handle = lib.load()
    for n in names:
        assert hasattr(handle, n), n
    assert sorted(lib.EXPORTS) == [n for n in names if n in lib.EXPORTS]
    missing_in_binding = [n for n in names if n not in lib.EXPORTS]
    assert missing_in_binding == [], missing_in_binding


def test_struct_layout_matches_header(lib, tmp_path):
    fields = [f[0] for f in lib.IntfaFwdParams._fields_]
    c = ['#include <stdio.h>', '#include <stddef.h>', '#include "intfa.h"', 'int main(void){',
         'printf("%zu\\n", sizeof(IntfaFwdParams));']
    c += ['printf("%%zu\\n", offsetof(IntfaFwdParams, %s));' % f for f in fields]
    c += ['return 0;}']
    src = tmp_path / "layout.c"
    src.write_text("\n".join(c))
    exe = tmp_path / "layout"
    subprocess.check_call(["gcc", "-I", os.path.join(ROOT, "include"), str(src), "-o", str(exe)])
    nums = [int(x) for x in subprocess.check_output([str(exe)]).split()]
    assert nums[0] == ctypes.sizeof(lib.IntfaFwdParams)
    for f, off in zip(fields, nums[1:]):
        assert getattr(lib.IntfaFwdParams, f).offset == off, f


def test_version_and_error_text(lib):
    h = lib.load()
    assert h.intfa_version() >= 100
    assert h.intfa_version() == lib.VERSION == int(re.search(r"#define INTFA_VERSION (\d+)", open(HEADER).read()).group(1))
    assert h.intfa_fwd(None, None) == lib.ERR_INVALID_ARG
    assert "NULL" in lib.last_error()


# what the struct ends with in each version: no version has two layouts
LAST_FIELD = {200: ("workspace_bytes", 400)}


def test_every_struct_layout_has_its_own_version(lib):
    last = lib.IntfaFwdParams._fields_[-1][0]
    assert (last, ctypes.sizeof(lib.IntfaFwdParams)) == LAST_FIELD[lib.VERSION]


def test_a_library_of_another_version_is_refused(lib, monkeypatch):
    class Other:
        def __getattr__(self, name):
            f = lambda *a: lib.VERSION - 100
            setattr(self, name, f)
            return f
    monkeypatch.setattr(lib, "_lib", None)
    monkeypatch.setattr(lib.ctypes, "CDLL", lambda path: Other())
    with pytest.raises(RuntimeError, match="version"):
        lib.load()


def test_validation_rejects_before_launch(lib):
    h = lib.load()
    P = lib.IntfaFwdParams()
    P.B, P.H, P.Nq, P.Nk, P.D, P.G = 1, 1, 128, 128, 48, 64
    assert h.intfa_fwd(ctypes.byref(P), None) == lib.ERR_UNSUPPORTED       # head_dim 48: not one of 16, 32, 64, 128, 256
    assert "head_dim" in lib.last_error()
    P.D, P.G, P.variant = 256, 128, lib.VARIANT_HALF
    assert h.intfa_fwd(ctypes.byref(P), None) == lib.ERR_UNSUPPORTED       # half-int8 at head_dim 256: G = 64 only
    P.variant = lib.VARIANT_FULL
    P.D = 128
    P.Nq = 100
    assert h.intfa_fwd(ctypes.byref(P), None) == lib.ERR_INVALID_ARG       # a ragged Nq is fine; q is NULL
    P.Nq = 128
    P.G = 96
    assert h.intfa_fwd(ctypes.byref(P), None) == lib.ERR_UNSUPPORTED       # G must be 64 or 128
    P.D, P.G = 128, 128
    assert h.intfa_fwd(ctypes.byref(P), None) == lib.ERR_INVALID_ARG       # q is NULL
    P.H, P.H_kv = 8, 3
    assert h.intfa_fwd(ctypes.byref(P), None) == lib.ERR_INVALID_ARG       # query heads not a multiple of K/V heads
    assert "H_kv" in lib.last_error()
    P.H_kv = 2
    P.o_dtype = 5
    assert h.intfa_fwd(ctypes.byref(P), None) == lib.ERR_INVALID_ARG       # unknown output type
    assert "o_dtype" in lib.last_error()
    P.o_dtype = 0
    P.variant = 7
    assert h.intfa_fwd(ctypes.byref(P), None) == lib.ERR_INVALID_ARG
    assert h.intfa_quant_pertoken(None, None, None, None, 1, 1, 1, 128, None) == lib.ERR_INVALID_ARG
    assert h.intfa_quant_v_workspace_bytes(2, 3, 128) == 2 * 3 * 128 * 4


@pytest.mark.parametrize("Nk", [128, 200])
def test_k_scale_rows_shorter_than_nk_are_refused(lib, Nk):
    """(No pointer is followed before the strides have been looked at.)"""
    h = lib.load()
    P = lib.IntfaFwdParams()
    P.q = P.k = P.v = P.o = P.q_scale = P.k_scale = P.v_scale = 1 << 20
    for n in ("q_stride", "k_stride", "v_stride", "o_stride"):
        setattr(P, n, lib._i64x3(2 * 256 * 128, 256 * 128, 128))
    P.B, P.H, P.Nq, P.Nk, P.D, P.G, P.sm_scale, P.write_o, P.o_dtype = 2, 2, 256, Nk, 128, 128, 0.1, 1, 0
    for strides in ((2 * Nk, Nk - 1), (Nk - 1, Nk), (0, Nk), (2 * Nk, 0)):
        P.ks_stride = lib._i64x2(*strides)
        assert h.intfa_fwd(ctypes.byref(P), None) == lib.ERR_INVALID_ARG
        assert "k_scale rows" in lib.last_error()
    P.ks_stride, P.o = lib._i64x2(2 * Nk, Nk), None                       # the next thing to be refused
    assert h.intfa_fwd(ctypes.byref(P), None) == lib.ERR_INVALID_ARG
    assert "o is NULL" in lib.last_error()


@pytest.mark.parametrize("D,G,B,H,Hkv,Nq,Nk,few", [
    (128, 64, 64, 8, 1, 24, 200, True),           # 26 us on the few-rows path, 51 on 128-row tiles
    (64, 64, 2, 16, 16, 129, 500, True),          # 12 us, 16
    (64, 128, 16, 32, 8, 1, 4097, True),          # decode
    (128, 128, 4, 32, 8, 256, 1024, False),       # 147 us against 35
    (128, 128, 2, 16, 16, 160, 6000, False),      # 153 against 73
])
def test_full_int8_takes_the_faster_path(lib, D, G, B, H, Hkv, Nq, Nk, few):
    """(Scratch tells which: the few-rows path of full-int8 always needs some, 128-row tiles never.)"""
    P = lib.IntfaFwdParams()
    P.causal, P.sm_scale, P.write_o, P.variant = 1, 0.1, 1, lib.VARIANT_FULL
    P.D, P.G, P.B, P.H, P.H_kv, P.Nq, P.Nk, P.q_offset = D, G, B, H, Hkv, Nq, Nk, Nk - Nq
    assert (lib.load().intfa_fwd_workspace_bytes(ctypes.byref(P)) > 0) == few


def test_scratch_has_a_bound(lib):
    """Batches, heads and lengths of a cache that fills the GPU: 256 MiB are enough, or what one K/V head needs."""
    h = lib.load()
    P = lib.IntfaFwdParams()
    P.causal, P.sm_scale, P.write_o = 1, 0.1, 1
    seen = 0
    for variant in (lib.VARIANT_FULL, lib.VARIANT_HALF):
        for D, G in ((64, 64), (64, 128), (128, 64), (128, 128)):
            for B in (1, 7, 64, 1000):
                for Hkv, ratio in ((1, 1), (8, 4), (32, 1), (8, 8), (1, 64)):
                    for Nq in (1, 4, 16, 256):
                        for Nk in (300, 4097, 65536, 1000003, 5000000):
                            P.variant, P.D, P.G, P.B, P.H, P.H_kv, P.Nq, P.Nk, P.q_offset = variant, D, G, B, Hkv * ratio, Hkv, Nq, Nk, Nk - Nq
                            n = h.intfa_fwd_workspace_bytes(ctypes.byref(P))
                            assert n <= max(256 << 20, 72 * (Nk + 128)), (n, variant, D, G, B, Hkv, ratio, Nq, Nk)
                            seen += n > 64 << 20
    assert seen > 100
    P.variant, P.D, P.G, P.B, P.H, P.H_kv, P.Nq, P.Nk, P.q_offset = lib.VARIANT_FULL, 128, 128, 4, 64, 8, 8, 65536, 65528
    assert 0 < h.intfa_fwd_workspace_bytes(ctypes.byref(P)) <= 256 << 20          # 0.55 GB of scores for 0.54 GB of K and V


def test_python_surface_refuses_cpu_tensors(pkg):
    import torch
    q = torch.zeros(1, 1, 128, 64, dtype=torch.int8)
    s = torch.ones(1, 1, 128)
    with pytest.raises(RuntimeError, match="CUDA"):
        pkg.attention_full_int8(q, q, q, s, s, torch.ones(1, 1), False, 1.0)
    with pytest.raises(RuntimeError, match="CUDA"):
        pkg.quant_pertoken(torch.zeros(1, 1, 128, 64, dtype=torch.float16))
    with pytest.raises(AssertionError):     # the reference's own head-dim assertion
        pkg.attention_int8(torch.zeros(1, 1, 128, 48, dtype=torch.int8), q, q.half(), s, s, False, 1.0)


def test_product_package_never_imports_the_oracle():
    pkg_dir = os.path.join(ROOT, "int-flashattention_b200")
    pat = re.compile(r"^\s*(from|import)\s+\S*oracle", re.M)
    for dirpath, _, files in os.walk(pkg_dir):
        for f in files:
            if f.endswith(".py"):
                assert not pat.search(open(os.path.join(dirpath, f)).read()), f
