"""Call site of the TernaSpMM operator: the PyTorch side of the boundary.

Mirrors ``TernaInfer_linear`` / ``SpBitLinear`` / ``get_global_workspace`` of
the reference's ``model.py`` (:37-133 in Gu-J/TernaInfer): same names, same
argument meaning, same checkpoint keys.  Differences, all on this side of the
C ABI: the activation quantiser is a kernel of the library for bf16 activations
on the GPU and torch operators otherwise (no ``torch.compile``, hence no
Triton); rows are not padded to a power of two because the B200 library accepts
any token count >= 1; K splits are reduced on chip, and the workspace serves
``TernaInfer_linear`` at large token counts (the weight, decoded once per
call); ``SpBitLinear`` goes through a native call site (host_call.cpp) that reads a
two-bit copy of its weights, and needs neither in the calls that it takes.

PyTorch is only plumbing here (device memory, the current stream); all
arithmetic of the linear layer happens in ``libternaspmm.so``.  There is no
CPU path: calling with CPU tensors raises.
"""
from __future__ import annotations

import contextlib
import ctypes

import torch
from torch import nn

from .lib import load_host_call, load_library

_GLOBAL_WORKSPACE = {}
_WORKSPACE_BYTES = 13824 * 2560      # the largest BitNet-2B layer as dense int8, as model.py:34 of the reference sizes it


def reserve_workspace(nbytes: int):
    """Raise the size the shared workspace is created with (call before the first forward; a layer
    whose dense int8 copy does not fit simply keeps the on-chip decode at every token count)."""
    global _WORKSPACE_BYTES
    _WORKSPACE_BYTES = max(_WORKSPACE_BYTES, int(nbytes))


def get_global_workspace(device="cuda"):
    """One workspace shared by all layers of a device (model.py:37-42 of the reference).  The
    reference needs it for its split-K partial sums and, at more than 64 tokens, for the dense int8
    copy of the weight its prefill GEMM reads.  Here only large-batch calls use it, the same way:
    the weight is decoded once per call into it and both operands reach the tensor cores by TMA."""
    dev = torch.device(device)
    if dev.index is None and dev.type == "cuda":
        dev = torch.device("cuda", torch.cuda.current_device())
    ws = _GLOBAL_WORKSPACE.get(dev)
    if ws is None or ws.numel() < _WORKSPACE_BYTES:
        ws = _GLOBAL_WORKSPACE[dev] = torch.empty(_WORKSPACE_BYTES, dtype=torch.int8, device=dev)
    return ws


_SAME_DEVICE = contextlib.nullcontext()


def _on(x: torch.Tensor):
    """Context in which launches go to the device of ``x``, as torch operators do by themselves."""
    return _SAME_DEVICE if x.device.index == torch.cuda.current_device() else torch.cuda.device(x.device)


def _stream():
    return torch.cuda.current_stream().cuda_stream


def quant_input(input: torch.Tensor):
    """Per-token absmax int8 quantisation (model.py:120-123):
    s = 127 / clamp(max|x|, 1e-5); x_q = clamp(round(x*s), -128, 127).  bf16 activations on the GPU take one
    kernel (the same values bit for bit; eight torch operators cost 60 us of launches for one token)."""
    K = input.shape[-1]
    if (input.is_cuda and input.dtype == torch.bfloat16 and K % 16 == 0 and K <= 57344 and input.numel() > 0
            and not (input.requires_grad and torch.is_grad_enabled())):
        x = input.contiguous()
        if x.data_ptr() % 16 == 0:
            q = torch.empty(x.shape, dtype=torch.int8, device=x.device)
            s = torch.empty((*x.shape[:-1], 1), dtype=torch.bfloat16, device=x.device)
            with _on(x):
                load_library().ternaspmm_quant(x.data_ptr(), x.numel() // K, K, q.data_ptr(), s.data_ptr(), _stream())
            return q, s
    s = 127 / input.abs().max(dim=-1, keepdim=True).values.clamp_(min=1e-5)
    return (input * s).round().clamp(-128, 127).to(torch.int8), s


def _builtin_segments(segments, out_features, ws_num):
    """Whether explicit scale-segment lengths say the same as the reference's built-in rule (equal
    widths, or 2560/640/640 for 3840 outputs with three scales), which is what the entry points
    without segment arguments apply."""
    if segments is None or len(segments) <= 1:
        return True
    if ws_num == 3 and out_features == 3840:
        return list(segments) == [2560, 640, 640]
    return out_features % ws_num == 0 and all(v == out_features // ws_num for v in segments)


_ENTRY = {"auto": "bitlinear_TernaSpMM", "decode": "bitlinear_TernaSpMM_decode",
          "prefill": "bitlinear_TernaSpMM_prefill"}


def rmsnorm_quant(x: torch.Tensor, norm_weight: torch.Tensor, eps: float, gated: bool = False):
    """One fused kernel for RMSNorm(x) * weight followed by ``quant_input``
    (``gated``: x holds [x1 | x3] and the normalised value is relu(x1)^2 * x3).
    bf16 [..., K or 2K] -> (int8 [..., K], bf16 scale [..., 1])."""
    if not x.is_cuda or norm_weight.device != x.device:
        raise RuntimeError("rmsnorm_quant needs CUDA tensors of one device: the B200 library has no CPU path")
    lib = load_library()
    K = norm_weight.shape[0]
    x2 = x.reshape(-1, x.shape[-1]).contiguous()
    M = x2.shape[0]
    q = torch.empty((M, K), dtype=torch.int8, device=x.device)
    s = torch.empty((M, 1), dtype=torch.bfloat16, device=x.device)
    fn = lib.ternaspmm_relu2_gate_rmsnorm_quant if gated else lib.ternaspmm_rmsnorm_quant
    with _on(x):
        fn(x2.data_ptr(), norm_weight.data_ptr(), float(eps), M, K, q.data_ptr(), s.data_ptr(), _stream())
    return q.reshape(*x.shape[:-1], K), s.reshape(*x.shape[:-1], 1)


def rmsnorm(x: torch.Tensor, norm_weight: torch.Tensor, eps: float) -> torch.Tensor:
    """RMSNorm(x) * weight in one kernel, in the summation order of ``rmsnorm_quant``; bf16 in, bf16 out."""
    if not x.is_cuda or norm_weight.device != x.device:
        raise RuntimeError("rmsnorm needs CUDA tensors of one device: the B200 library has no CPU path")
    lib = load_library()
    K = norm_weight.shape[0]
    x2 = x.reshape(-1, K).contiguous()
    y = torch.empty_like(x2)
    with _on(x):
        lib.ternaspmm_rmsnorm(x2.data_ptr(), norm_weight.data_ptr(), float(eps), x2.shape[0], K, y.data_ptr(), _stream())
    return y.reshape(x.shape)


def rope(x: torch.Tensor, cos: torch.Tensor, sin: torch.Tensor):
    """RoPE on adjacent pairs as one kernel: x bf16 [B, T, H, 128] (heads contiguous), cos / sin fp32 [B, T, 64] equal in
    every sequence (expanded).  None where the kernel does not take the tensors."""
    B, T, H, D = x.shape
    ld = x.stride(1) if T > 1 else x.stride(0)           # (the stride of a dimension of one is anything)
    if not (x.is_cuda and x.device == cos.device == sin.device and x.dtype == torch.bfloat16 and cos.dtype == sin.dtype == torch.float32 and D == 128 and x.numel() > 0
            and x.stride(3) == 1 and x.stride(2) == D and (B == 1 or x.stride(0) == T * ld) and ld % 8 == 0
            and x.data_ptr() % 16 == 0 and cos.shape[1:] == sin.shape[1:] == (T, 64) and (B == 1 or cos.stride(0) == sin.stride(0) == 0)
            and (T == 1 or cos.stride(1) == sin.stride(1) == 64) and cos.stride(2) == sin.stride(2) == 1 and cos.data_ptr() % 16 == 0 and sin.data_ptr() % 16 == 0):
        return None
    out = torch.empty((B, T, H, D), dtype=torch.bfloat16, device=x.device)
    with _on(x):
        load_library().ternaspmm_rope(x.data_ptr(), ld, cos.data_ptr(), sin.data_ptr(), out.data_ptr(), B, T, H, _stream())
    return out


def relu2_gate(x13: torch.Tensor):
    """relu(x1)^2 * x3 of bf16 [..., x1 | x3] as one kernel, rounded as the torch operators; None where it does not apply."""
    K = x13.shape[-1] // 2
    if not (x13.is_cuda and x13.dtype == torch.bfloat16 and x13.is_contiguous() and K % 8 == 0 and x13.numel() > 0 and x13.data_ptr() % 16 == 0):
        return None
    out = torch.empty((*x13.shape[:-1], K), dtype=torch.bfloat16, device=x13.device)
    with _on(x13):
        load_library().ternaspmm_relu2_gate(x13.data_ptr(), out.data_ptr(), x13.numel() // (2 * K), K, _stream())
    return out


def to_float(x: torch.Tensor) -> torch.Tensor:
    """x.float(); bf16 on the GPU by the library (at the copy rate; torch's casting kernel reaches a third of it)."""
    if not (x.is_cuda and x.dtype == torch.bfloat16 and x.is_contiguous() and x.numel() > 0 and x.data_ptr() % 16 == 0
            and not (x.requires_grad and torch.is_grad_enabled())):
        return x.float()
    out = torch.empty(x.shape, dtype=torch.float32, device=x.device)
    with _on(x):
        load_library().ternaspmm_bf16_to_f32(x.data_ptr(), out.data_ptr(), x.numel(), _stream())
    return out


def _attn_takes(qkv, k_cache, v_cache, cos, sin, pos, heads, kv_heads):
    """What both attention kernels ask of their tensors; they get addresses and can check none of it."""
    return (qkv.is_cuda and qkv.device == k_cache.device == v_cache.device == cos.device == sin.device == pos.device
            and qkv.dtype == k_cache.dtype == v_cache.dtype == cos.dtype == sin.dtype == torch.bfloat16 and pos.dtype == torch.int64
            and qkv.dim() == 3 and k_cache.dim() == 4 and k_cache.shape == v_cache.shape and kv_heads > 0
            and k_cache.shape[0] == qkv.shape[0] and k_cache.shape[2:] == (kv_heads, 128) and qkv.shape[2] == (heads + 2 * kv_heads) * 128
            and pos.numel() == qkv.shape[1] <= k_cache.shape[1] and qkv.numel() > 0
            and all(t.is_contiguous() for t in (qkv, k_cache, v_cache, cos, sin, pos)))


def attn_decode(qkv, k_cache, v_cache, cos_row, sin_row, pos, heads: int, kv_heads: int):
    """RoPE, cache append and attention of one new token per sequence in one kernel: qkv bf16 [B, 1, (heads + 2 *
    kv_heads) * 128], caches bf16 [B, L, kv_heads, 128], ``pos`` int64 [1] on the device, ``cos_row`` / ``sin_row`` bf16
    [1, 64] the rotation of that position.  bf16 [B, 1, heads * 128], or
    None where the kernel does not take the tensors."""
    if not (_attn_takes(qkv, k_cache, v_cache, cos_row, sin_row, pos, heads, kv_heads) and qkv.shape[1] == 1
            and heads in (4 * kv_heads, 8 * kv_heads) and cos_row.numel() == sin_row.numel() == 64):
        return None
    B, D = qkv.shape[0], k_cache.shape[-1]
    out = torch.empty((B, 1, heads * D), dtype=torch.bfloat16, device=qkv.device)
    with _on(qkv):
        status = load_library().ternaspmm_attn_decode(qkv.data_ptr(), k_cache.data_ptr(), v_cache.data_ptr(), cos_row.data_ptr(),
                                                      sin_row.data_ptr(), pos.data_ptr(), out.data_ptr(), B, heads, kv_heads, D,
                                                      k_cache.shape[1], _stream())
    return out if status == 0 else None


def attn_decode_by_head(qkv, k_cache, v_cache, cos_row, sin_row, pos, heads: int, kv_heads: int):
    """``attn_decode`` on caches [B, kv_heads, L, 128], rotation fp32 [64] of that position in the arithmetic of ``rope``: the
    default glue's RoPE, ``index_copy_`` and masked attention of one new token per sequence.  Not under autograd.  A position outside of the
    cache gives NaN and leaves the caches as they are (status 1 of the library)."""
    if not (qkv.is_cuda and qkv.device == k_cache.device == v_cache.device == cos_row.device == sin_row.device == pos.device
            and qkv.dtype == k_cache.dtype == v_cache.dtype == torch.bfloat16 and cos_row.dtype == sin_row.dtype == torch.float32
            and pos.dtype == torch.int64 and pos.numel() == 1 and qkv.dim() == 3 and qkv.shape[1] == 1 and k_cache.dim() == 4
            and k_cache.shape == v_cache.shape and k_cache.shape[:2] == (qkv.shape[0], kv_heads) and k_cache.shape[3] == 128
            and k_cache.numel() > 0 and heads in (4 * kv_heads, 8 * kv_heads) and qkv.shape[2] == (heads + 2 * kv_heads) * 128
            and cos_row.numel() == sin_row.numel() == 64 and all(t.is_contiguous() for t in (qkv, k_cache, v_cache, cos_row, sin_row))
            and not torch.is_grad_enabled()):
        return None
    B = qkv.shape[0]
    out = torch.empty((B, 1, heads * 128), dtype=torch.bfloat16, device=qkv.device)
    with _on(qkv):
        status = load_library().ternaspmm_attn_decode_by_head(qkv.data_ptr(), k_cache.data_ptr(), v_cache.data_ptr(), cos_row.data_ptr(),
                                                              sin_row.data_ptr(), pos.data_ptr(), out.data_ptr(), B, heads, kv_heads, 128,
                                                              k_cache.shape[2], _stream())
    return out if status == 0 else None


def attn_prefill(qkv, k_cache, v_cache, cos_tab, sin_tab, pos, heads: int, kv_heads: int):
    """``attn_decode`` for T new tokens per sequence at consecutive positions (``pos`` int64 [T]), causal: qkv bf16
    [B, T, (heads + 2 * kv_heads) * 128], tables bf16 [>= L, 64].  bf16 [B, T, heads * 128], or None."""
    if not (_attn_takes(qkv, k_cache, v_cache, cos_tab, sin_tab, pos, heads, kv_heads) and heads % (4 * kv_heads) == 0
            and cos_tab.shape == sin_tab.shape and cos_tab.dim() == 2 and cos_tab.shape[1] == 64 and k_cache.shape[1] <= cos_tab.shape[0]):
        return None
    B, T, D = qkv.shape[0], qkv.shape[1], k_cache.shape[-1]
    out = torch.empty((B, T, heads * D), dtype=torch.bfloat16, device=qkv.device)
    with _on(qkv):
        status = load_library().ternaspmm_attn_prefill(qkv.data_ptr(), k_cache.data_ptr(), v_cache.data_ptr(), cos_tab.data_ptr(),
                                                       sin_tab.data_ptr(), pos.data_ptr(), out.data_ptr(), B, T, heads, kv_heads, D,
                                                       k_cache.shape[1], _stream())
    return out if status == 0 else None


_HEAD_SCRATCH = {}


def lm_head_argmax(h: torch.Tensor, embedding: torch.Tensor, want_logits: bool = True, want_argmax: bool = True):
    """Output head for up to 8 rows: (fp32 logits [M, V] or None, int64 greedy tokens [M] or None).
    One kernel that reads the embedding once; the logits carry the bf16 rounding of the reference's
    bf16 linear and the arg-max is taken over them (smallest index on ties)."""
    if not h.is_cuda:
        raise RuntimeError("lm_head_argmax needs CUDA tensors: the B200 library has no CPU path")
    lib = load_library()
    V, K = embedding.shape
    h2 = h.reshape(-1, K).contiguous()
    M = h2.shape[0]
    assert 1 <= M <= 8 and h2.dtype == torch.bfloat16 and embedding.dtype == torch.bfloat16 and embedding.is_contiguous()
    assert embedding.device == h2.device
    dev = h.device
    scratch = _HEAD_SCRATCH.get(dev)
    if scratch is None:   # one zero-initialised scratch area per device (calls on one device run in stream order)
        scratch = _HEAD_SCRATCH[dev] = torch.zeros(int(lib.ternaspmm_lm_head_scratch_bytes()), dtype=torch.uint8, device=dev)
    logits = torch.empty((M, V), dtype=torch.float32, device=dev) if want_logits else None
    tokens = torch.empty((M,), dtype=torch.int64, device=dev) if want_argmax else None
    with _on(h2):
        lib.ternaspmm_lm_head_argmax(h2.data_ptr(), embedding.data_ptr(), M, V, K, logits.data_ptr() if want_logits else None,
                                     tokens.data_ptr() if want_argmax else None, 1, scratch.data_ptr(), _stream())
    return logits, tokens


def TernaInfer_linear(input, compressed_val, TileOffsets_global, TileOffsets_median, bitmap,
                      workspace, s, ws, ws_num, out_features, mode: str = "auto", residual=None, segments=None):
    """out = TernaSpMM(input_int8, packed weight) as bf16 (model.py:45-92).
    ``input`` is int8 [..., K] on the GPU, ``s`` its per-token bf16 scale,
    ``ws`` the 4-slot bf16 weight scale with ``ws_num`` non-zero slots.
    ``segments`` (optional, not in the reference): lengths of the scale segments;
    without it the reference's built-in rule decides (equal widths, or
    2560/640/640 for 3840 outputs)."""
    if not input.is_cuda:
        raise RuntimeError("TernaInfer_linear needs CUDA tensors: the B200 library has no CPU path")
    if input.device.index != torch.cuda.current_device():
        with torch.cuda.device(input.device):
            return TernaInfer_linear(input, compressed_val, TileOffsets_global, TileOffsets_median, bitmap, workspace, s, ws, ws_num,
                                     out_features, mode, residual, segments)
    lib = load_library()
    out_shape = list(input.shape)
    out_shape[-1] = out_features
    K = input.shape[-1]
    M = input.numel() // K
    x2 = input.reshape(M, K)
    if not x2.is_contiguous():
        x2 = x2.contiguous()
    if s.dtype != torch.bfloat16:
        s = s.to(torch.bfloat16)
    s = s.contiguous()
    ret = torch.empty((M, out_features), dtype=torch.bfloat16, device=input.device)
    stream = torch.cuda.current_stream()
    if (workspace is not None and mode == "auto" and M > 64 and _builtin_segments(segments, out_features, ws_num)
            and workspace.numel() * workspace.element_size() >= out_features * K):
        # large batch with the reference-sized workspace: decode once into it, both operands by TMA
        res = None
        if residual is not None:
            res = residual.reshape(M, out_features)
            assert res.is_contiguous() and res.dtype == torch.bfloat16
        lib.bitlinear_TernaSpMM_ws(x2.data_ptr(), bitmap.data_ptr(), TileOffsets_global.data_ptr(),
                                   TileOffsets_median.data_ptr(), compressed_val.data_ptr(), ret.data_ptr(), s.data_ptr(),
                                   ws.data_ptr(), ws_num, M, out_features, K, res.data_ptr() if res is not None else None,
                                   workspace.data_ptr(), workspace.numel() * workspace.element_size(), 0, stream.cuda_stream)
        return ret.reshape(*out_shape)
    if segments is not None and len(segments) > 1 and residual is None:
        bounds = [sum(segments[:i + 1]) for i in range(len(segments) - 1)] + [2 ** 31 - 1] * 3
        form = {"auto": -1, "decode": 0, "prefill": 1}[mode]
        lib.ternaspmm_linear_segments(x2.data_ptr(), bitmap.data_ptr(), TileOffsets_global.data_ptr(),
                                      TileOffsets_median.data_ptr(), compressed_val.data_ptr(), ret.data_ptr(),
                                      s.data_ptr(), ws.data_ptr(), ws_num, M, out_features, K, bounds[0], bounds[1],
                                      bounds[2], form, stream.cuda_stream)
        return ret.reshape(*out_shape)
    if residual is not None:
        res = residual.reshape(M, out_features)
        assert mode == "auto" and res.is_contiguous() and res.dtype == torch.bfloat16
        lib.bitlinear_TernaSpMM_residual(x2.data_ptr(), bitmap.data_ptr(), TileOffsets_global.data_ptr(),
                                         TileOffsets_median.data_ptr(), compressed_val.data_ptr(), ret.data_ptr(),
                                         s.data_ptr(), ws.data_ptr(), ws_num, M, out_features, K, res.data_ptr(),
                                         stream.cuda_stream)
        return ret.reshape(*out_shape)
    getattr(lib, _ENTRY[mode])(
        ctypes.c_void_p(x2.data_ptr()),
        ctypes.c_void_p(bitmap.data_ptr()),
        ctypes.c_void_p(TileOffsets_global.data_ptr()),
        ctypes.c_void_p(TileOffsets_median.data_ptr()),
        ctypes.c_void_p(compressed_val.data_ptr()),
        ctypes.c_void_p(ret.data_ptr()),
        ctypes.c_void_p(s.data_ptr()),
        ctypes.c_void_p(ws.data_ptr()),
        ctypes.c_int(ws_num),
        ctypes.c_int(M), ctypes.c_int(out_features), ctypes.c_int(K),
        ctypes.c_int(1), ctypes.c_void_p(workspace.data_ptr() if workspace is not None else 0),
        ctypes.c_void_p(stream.cuda_stream),
    )
    return ret.reshape(*out_shape)


class _OwnedParameters(dict):
    """Parameters of an ``SpBitLinear``.  Whatever gets hold of one - an attribute of the module, ``parameters()``,
    ``state_dict()``, ``to()`` ... - reads it here, and that invalidates the layer's two-bit copy of the weights, since
    the values may change from then on without a trace.  The next call takes the copy up again when the module alone holds
    every parameter (host_call.cpp); hence lists instead of views, which would hand parameters out later."""

    __slots__ = ("layer",)

    def __init__(self, layer, items=()):
        super().__init__(items)
        self.layer = layer

    def _handing_out(name):
        read = getattr(dict, name)

        def method(self, *args):
            self.layer.invalidate()
            out = read(self, *args)
            return list(out) if name in ("items", "values") else out
        method.__name__ = name
        return method

    def _replacing(name):
        write = getattr(dict, name)

        def method(self, *args, **kwargs):
            self.layer.replace()
            return write(self, *args, **kwargs)
        method.__name__ = name
        return method

    for _name in ("__getitem__", "get", "items", "values", "copy", "__or__", "__ror__"):
        locals()[_name] = _handing_out(_name)
    for _name in ("__setitem__", "__delitem__", "__ior__", "pop", "popitem", "setdefault", "update", "clear"):
        locals()[_name] = _replacing(_name)
    del _name, _handing_out, _replacing

    def __iter__(self):          # (its own, so that dict(self) reads through __getitem__)
        return super().__iter__()

    def __reduce__(self):
        return dict, (dict(self),)


class SpBitLinear(nn.Module):
    """Ternary linear layer bound to packed checkpoint tensors (model.py:96-133):
    ``<key>.weight_compressed_val`` (uint32), ``_TileOffsets_global`` (int32),
    ``_TileOffsets_median`` (uint16), ``_bitmap`` (uint64), ``.weight_scale``
    (bf16[4]).

    The packed tensors are parameters, copied from ``dic``; besides them the module keeps the weights in the two-bit
    layout of its kernels (N*K/4 bytes more).  Calls use that copy while nothing outside of the module holds a parameter
    or a tensor that shares its memory, and lay it out again after something did; otherwise they read the packed tensors.
    A captured graph goes on reading what it was captured with.  ``load_state_dict`` and ``relayout()`` write the copy in
    place, so that replays follow; after any other change of the weights, and after writes through a raw pointer, call ``relayout()``."""

    def __init__(self, in_features: int, out_features: int, dic: dict, key: str, bias: bool = False):
        super().__init__()
        self.in_features = in_features
        self.out_features = out_features
        dev = "cuda"

        def own(name):           # on the GPU, in memory that nothing else shares
            t = dic[key + "." + name]
            return nn.Parameter(t.clone() if t.is_cuda else t.to(dev), requires_grad=False)
        self.weight_compressed_val = own("weight_compressed_val")
        self.weight_TileOffsets_global = own("weight_TileOffsets_global")
        self.weight_TileOffsets_median = own("weight_TileOffsets_median")
        self.weight_bitmap = own("weight_bitmap")
        ws = dic[key + ".weight_scale"]
        self.weight_scale = nn.Parameter(ws.to(dev), requires_grad=False)
        self.ws_num = int((ws != 0).sum().item())
        # explicit scale-segment lengths when the checkpoint carries them (written by this
        # library's converter); absent in checkpoints converted by the reference
        seg = dic.get(key + ".weight_segments")
        self.segments = [int(v) for v in seg] if seg is not None else None
        if self.segments is not None:
            assert sum(self.segments) == out_features and len(self.segments) == self.ws_num
        self._attach()

    def _attach(self):
        """The native call site; it keeps the weights in the layout of the small-batch kernel, laid out here once."""
        bounds = [0, 0, 0]
        if not _builtin_segments(self.segments, self.out_features, self.ws_num):
            bounds = [sum(self.segments[:i + 1]) for i in range(len(self.segments) - 1)] + [2 ** 31 - 1] * 3
        self._native = load_host_call().Layer(self.in_features, self.out_features, self.ws_num, *bounds[:3])
        self.__dict__["_parameters"] = _OwnedParameters(self._native, self._parameters)
        self._native.prepare(self._parameters)

    def __getstate__(self):      # copies and pickles carry what checkpoints carry; the call site is made again from it
        state = self.__dict__.copy()
        state.pop("_native", None)
        state["_parameters"] = dict(self._parameters)
        return state

    def __setstate__(self, state):
        super().__setstate__(state)
        self._attach()

    quant_input = staticmethod(quant_input)

    def _apply(self, fn, recurse=True):
        super()._apply(fn, recurse)
        self._native.prepare(self._parameters)
        return self

    def _load_from_state_dict(self, state_dict, prefix, *args):
        errors, before = args[-1], len(args[-1])
        super()._load_from_state_dict(state_dict, prefix, *args)
        # laid out at once, for the sake of captured graphs; a part of the tensors (one shard of several) is not a weight yet
        if len(errors) == before and all(prefix + n in state_dict for n in self._PACKED):
            self._native.relayout(self._parameters)

    def relayout(self):
        """Lay the two-bit copy out again from the packed parameters, which have changed, and wait for it.  In the
        copy's memory, so that captured graphs follow.  Not while a stream is being captured."""
        if torch.cuda.is_current_stream_capturing():
            raise RuntimeError("SpBitLinear.relayout while the stream is being captured")
        self._native.relayout(self._parameters)

    _PACKED = ("weight_compressed_val", "weight_TileOffsets_global", "weight_TileOffsets_median", "weight_bitmap")

    def _weights(self):
        """The packed tensors and the scale, for a call to read."""
        names = (*self._PACKED, "weight_scale")
        p = self._parameters
        return [dict.__getitem__(p, n) for n in names] if isinstance(p, _OwnedParameters) else [getattr(self, n) for n in names]

    def forward_quantized(self, input_q, s, residual=None):
        """Already quantised input (int8 + per-token scale), optional fused residual add."""
        out = self._native.forward_quantized(self._parameters, input_q, s, residual)
        if out is not None:
            return out
        *packed, ws = self._weights()
        return TernaInfer_linear(input_q, *packed, get_global_workspace(input_q.device), s, ws, self.ws_num, self.out_features,
                                 residual=residual, segments=self.segments)

    def forward_normed(self, x, norm_weight, eps, gated=False, residual=None):
        """forward_quantized(*rmsnorm_quant(x, norm_weight, eps, gated), residual): the front-end runs inside the
        linear's kernel for the smallest calls."""
        out = self._native.forward_normed(self._parameters, x, norm_weight, eps, gated, residual)
        if out is not None:
            return out
        xq, s = rmsnorm_quant(x, norm_weight, eps, gated)
        return self.forward_quantized(xq, s, residual=residual)

    def forward(self, input):
        out = self._native.forward(self._parameters, input)
        if out is not None:
            return out
        input, s = quant_input(input)
        *packed, ws = self._weights()
        return TernaInfer_linear(input, *packed, get_global_workspace(input.device), s, ws, self.ws_num, self.out_features,
                                 segments=self.segments)
