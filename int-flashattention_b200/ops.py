"""Python operator surface over libintfa.so, mirroring the reference's operators.

    attention_full_int8(q, k, v, q_scale, k_scale, v_scale, causal, sm_scale) -> o
        (flash_atten_full_int8.py:187,223)
    attention_int8(q, k, v, q_scale, k_scale, causal, sm_scale) -> o
        (flash_atten_int8.py:181,217)
    quant_pertoken / quant_pertensor (benchmark.py:96-107) and quant_perchannel
    int_flash_attention(q16, k16, v16, causal, sm_scale, variant): prologue + forward

Positional arguments and their meaning are the reference's.  Tensors must live on a
CUDA device; launches are asynchronous on torch's current stream of that device.
PyTorch is used for memory and streams only -- every computation runs in libintfa.so, and there is no other path: a
missing library or a CPU tensor raises.  Argument checks, allocation and launches are native code (csrc/intfa_torch.cpp,
module _native); the functions here give them their signatures.
"""
import torch

from . import _lib

_native_mod = None


def _native():
    """The binding, loaded on first use (this package must be importable before it is built)."""
    global _native_mod
    if _native_mod is None:
        _lib.load()
        try:
            from . import _native as mod
        except ImportError as e:
            raise RuntimeError("_native.so is not built (or not for this Python): build it with `python "
                               "int-flashattention_b200/build.py`; there is no non-CUDA fallback. (%s)" % e) from e
        mod.set_error_class(_lib.IntfaError)
        _native_mod = mod
    return _native_mod


def default_G(head_dim, variant="full"):
    """Running-max granularity used when the caller does not choose one.  full-int8: the widest KV
    tile the reference's kernels allow for this head size (BLOCK_N <= HEAD_DIM,
    flash_atten_full_int8.py:88).  half-int8: 128 -- its result does not depend on G beyond fp16
    rounding, and 128-wide KV tiles are the faster ones at both head sizes."""
    if variant == "half":
        return 64 if head_dim == 256 else 128      # (fp16 V tiles of 128 keys x 256 channels do not fit next to K)
    return 128 if head_dim >= 128 else (64 if head_dim >= 64 else 32)


def _status_word(dev):
    """The int32[1] tensor of a device that the kernels report bounded-wait expiry into."""
    return _native().status(dev.index if dev.index is not None else torch.cuda.current_device())


def check_status(device=None):
    """Synchronise and raise if any kernel launched through this module on `device` gave up a
    bounded device-side wait.  Returns the raw status word (0 = fine)."""
    dev = torch.device("cuda", torch.cuda.current_device()) if device is None else torch.device(device)
    word = _status_word(dev)
    val = int(word.item())
    if val != 0:
        word.zero_()
        raise _lib.IntfaError(_lib.ERR_DEVICE_WAIT,
                              "device-side wait expired (wait code %d, CTA %d)" % (val & 0xff, val >> 8))
    return val


def _fwd(variant, q, k, v, q_scale, k_scale, v_scale, causal, sm_scale, **kw):
    """The forward.  Keyword arguments: G, p_round, kv_order, state, q_offset, kv_offset, return_state, return_lse, write_o,
    debug_tap, out_dtype, debug_wait (test hooks of the bounded waits: (limit in kilo-cycles, K step to leave out))."""
    return (_native_mod or _native()).fwd(variant == "full", q, k, v, q_scale, k_scale, v_scale, causal, sm_scale, **kw)


def attention_full_int8(q, k, v, q_scale, k_scale, v_scale, causal, sm_scale, **kw):
    """Full-int8 attention forward (int8 Q/K/V, int8 P).  Mirrors attention_full_int8 of
    flash_atten_full_int8.py:187,223.  With causal=True the running maximum is carried from the
    off-band to the on-band stage (as flash_atten_int8.py:66,157,166 does); the reference's
    full-int8 Triton kernel drops it (flash_atten_full_int8.py:71,166-179).
    Extra keyword arguments (not in the reference): G (running-max granularity, the reference's
    BLOCK_N), p_round ("triton" | "rne"), kv_order ("ascending" | "descending": the CUDA path walks the KV tiles
    last to first, csrc/flash_fwd_kernel_full_qi8.h:331-469), v_scale of shape (B,H,ceil(Nk/G),D) (one row per KV
    tile, the CUDA path's layout), state/q_offset/kv_offset/return_state (ring attention),
    return_lse, debug_tap, out_dtype (torch.float16 | torch.bfloat16).  k, v and their scales may have
    fewer heads than q (grouped-query attention: query head h reads K/V head h // (H // H_kv))."""
    return (_native_mod or _native()).fwd(True, q, k, v, q_scale, k_scale, v_scale, causal, sm_scale, **kw)


def attention_int8(q, k, v, q_scale, k_scale, causal, sm_scale, **kw):
    """Half-int8 attention forward (int8 Q/K, fp16 V and P).  Mirrors attention_int8 of
    flash_atten_int8.py:181,217.  V may also be torch.float8_e5m2: P is then cast to e5m2 as well and P V runs as an
    fp8 matrix product with fp32 accumulation (flash_atten_int8.py:55-56,160)."""
    return (_native_mod or _native()).fwd(False, q, k, v, q_scale, k_scale, None, causal, sm_scale, **kw)


# ---------------------------------------------------------------------------------------------
# quantisation prologue
# ---------------------------------------------------------------------------------------------
def quant_pertoken(X):
    """benchmark.py:96-100.  Returns (int8 [B,H,N,D], scale [B,H,N]); the scale is fp32 holding
    the reference's fp16 value."""
    return (_native_mod or _native()).quant_pertoken(X)


def quant_qkv(q, k, v=None, v_mode="per_channel"):
    """The quantisation prologue of one attention call in one or two launches (one when v is None): per-token q and k
    (benchmark.py:96-100), and v (benchmark.py:102-107 or its per-channel form) with them, or after them where the call is
    larger; where v takes two passes the first, its column absmax, is in the grid of q and k.  Bit-identical to quant_pertoken / quant_perchannel / quant_pertensor called one by one.
    Returns (q8, q_scale, k8, k_scale) and, with v, (v8, v_scale) appended."""
    return (_native_mod or _native()).quant_qkv(q, k, v, _lib.VSCALE_PER_CHANNEL if v_mode == "per_channel" else _lib.VSCALE_PER_TENSOR)


def quant_v_with_allreduce(X, mode, group=None):
    """V quantisation for a token-sharded V: local column absmax, all-reduce(MAX) over `group`
    of the B*H*D fp32 bit patterns (order-preserving as int32 because they are non-negative),
    then the quantising pass.  Equals quantising the unsharded tensor bit for bit."""
    import ctypes
    import torch.distributed as dist
    lib = _lib.load()
    if not X.is_cuda:
        raise RuntimeError("int-flashattention_b200 runs on CUDA tensors only (there is no CPU path)")
    if X.dtype != torch.float16 or X.dim() != 4:
        raise TypeError("quantisers take a float16 [B,H,N,D] tensor")
    if X.stride(-1) != 1 or X.data_ptr() % 16 or any(s % 8 for s in X.stride()[:3]):
        X = X.contiguous()
    stream = ctypes.c_void_p(torch.cuda.current_stream(X.device).cuda_stream)
    B, H, N, D = X.shape
    mode_i = {"per_channel": _lib.VSCALE_PER_CHANNEL, "per_tensor": _lib.VSCALE_PER_TENSOR}.get(mode, mode)
    colmax = torch.zeros(B * H * D, dtype=torch.int32, device=X.device)
    st = _lib._i64x3(*X.stride()[:3])
    with torch.cuda.device(X.device):
        _lib.check(lib.intfa_v_colmax(X.data_ptr(), st, colmax.data_ptr(), B, H, N, D, stream))
    if dist.is_initialized() and dist.get_world_size(group) > 1:
        dist.all_reduce(colmax, op=dist.ReduceOp.MAX, group=group)
    x8 = torch.empty((B, H, N, D), dtype=torch.int8, device=X.device)
    shape = (B, H, D) if mode_i == _lib.VSCALE_PER_CHANNEL else (B, H)
    scale = torch.empty(shape, dtype=torch.float32, device=X.device)
    with torch.cuda.device(X.device):
        _lib.check(lib.intfa_v_quant_from_colmax(X.data_ptr(), st, colmax.data_ptr(), x8.data_ptr(),
                                                 scale.data_ptr(), mode_i, B, H, N, D, stream))
    return x8, scale


def quant_pertensor(X):
    """benchmark.py:102-107: one scale per (batch, head).  Returns (int8, scale [B,H] fp32)."""
    return (_native_mod or _native()).quant_v(X, _lib.VSCALE_PER_TENSOR)


def quant_perchannel(X):
    """Per-channel V quantisation: one scale per (batch, head, channel). Returns (int8, scale [B,H,D] fp32)."""
    return (_native_mod or _native()).quant_v(X, _lib.VSCALE_PER_CHANNEL)


def int_flash_attention(q, k, v, causal, sm_scale, variant="full", v_mode="per_channel", **kw):
    """fp16 Q/K/V in, fp16 O out: fused quantisation prologue (per-token Q/K; per-channel or
    per-(batch,head) V for the full-int8 variant) followed by the INT8 attention forward.
    Argument order follows the reference's attention(q, k, v, causal, sm_scale) (flash_atten_fp.py:155)."""
    return (_native_mod or _native()).flash(q, k, v, causal, sm_scale, variant, v_mode, **kw)
