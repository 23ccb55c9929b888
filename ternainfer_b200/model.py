"""BitNet-b1.58 style decoder around the TernaSpMM call site.

Thin PyTorch glue so that a decoder block and the full model can be run and
timed end to end; only the four ternary linears per layer (``wqkv``, ``wo``,
``w13``, ``w2``) are the hand-written path.  Shapes and order of operations
follow ``model.py`` of Gu-J/TernaInfer (:155-386): GQA attention with RoPE on
adjacent pairs, RMSNorm before each sub-block, a sub-layer norm before ``wo``
and ``w2``, ReLU^2 gated FFN, tied bf16 embedding / output head.  The
reference's xformers ops are replaced by plain torch (RMSNorm, RoPE, SDPA over
a dense per-sequence KV cache), and nothing goes through ``torch.compile``.
With ``tp`` > 1 the linears are the column-/row-parallel versions of
``ternainfer_b200.tp``.
"""
from __future__ import annotations

from dataclasses import dataclass
from typing import List, Optional, Tuple

import torch
from torch import nn
from torch.nn import functional as F

from .linear import SpBitLinear, attn_decode, attn_decode_by_head, attn_prefill, lm_head_argmax, quant_input, relu2_gate, rmsnorm, rope, to_float


@dataclass
class ModelArgs:
    dim: int = 2560
    n_layers: int = 30
    n_heads: int = 20
    n_kv_heads: int = 5
    vocab_size: int = 128256
    ffn_dim: int = 6912
    norm_eps: float = 1e-5
    rope_theta: float = 500000.0
    use_kernel: bool = True
    fused_glue: bool = False     # fused norm+quantiser kernels and residual add in the linear epilogue
    flash_attention: Optional[bool] = None   # attention glue through flash_attn's kv-cache kernel; None = with fused_glue

    @property
    def head_dim(self) -> int:
        return self.dim // self.n_heads


LayerCache = Tuple[torch.Tensor, torch.Tensor]


class RMSNorm(nn.Module):
    def __init__(self, dim: int, eps: float = 1e-5):
        super().__init__()
        self.eps = eps
        self.weight = nn.Parameter(torch.ones(dim))

    def forward(self, x):
        if (x.is_cuda and x.device == self.weight.device and x.dtype == self.weight.dtype == torch.bfloat16 and x.shape[-1] % 16 == 0
                and x.shape[-1] <= 57344 and x.numel() > 0 and not torch.is_grad_enabled()):
            return rmsnorm(x, self.weight, self.eps)       # one launch instead of seven, the fused front-ends' summation order
        xf = x.float()
        y = xf * torch.rsqrt(xf.pow(2).mean(-1, keepdim=True) + self.eps)
        return (y * self.weight.float()).to(x.dtype)


class BF16BitLinear(nn.Module):
    """Dense comparator (model.py:135-153 of the reference): same quantiser,
    bf16 GEMM on the de-quantised ternary weight, division by the scale."""

    def __init__(self, in_features, out_features, dic, key, bias=False):
        super().__init__()
        self.weight = nn.Parameter(dic[key + ".weight"].cuda(), requires_grad=False)

    def forward(self, input):
        xq, s = quant_input(input)
        return F.linear(xq.to(torch.bfloat16), self.weight) / s


def rope_tables(head_dim: int, max_len: int, theta: float, device):
    inv = 1.0 / (theta ** (torch.arange(0, head_dim, 2, device=device).float() / head_dim))
    ang = torch.outer(torch.arange(max_len, device=device).float(), inv)
    return ang.cos(), ang.sin()


def apply_rope(x, cos, sin):
    """Rotate adjacent pairs (2i, 2i+1); x [B, T, H, D], cos/sin [B, T, D/2]."""
    out = rope(x, cos, sin) if not torch.is_grad_enabled() else None
    if out is not None:
        return out
    xf = x.float().unflatten(-1, (-1, 2))
    a, b = xf[..., 0], xf[..., 1]
    c, s = cos.unsqueeze(2), sin.unsqueeze(2)
    return torch.stack((a * c - b * s, a * s + b * c), dim=-1).flatten(-2).to(x.dtype)


CAUSAL = object()                # in place of a mask: every position up to that of the (one) new token


def causal_mask(pos, length):
    """[1, 1, T, L]: the cache positions that queries at ``pos`` attend to."""
    keys = torch.arange(length, device=pos.device)
    return (keys[None, :] <= pos[:, None])[None, None]


class Attention(nn.Module):
    def __init__(self, args: ModelArgs, dic: dict, prefix: str, linear_cls, tp_group=None, tp: int = 1):
        super().__init__()
        self.head_dim = args.head_dim
        self.n_heads = args.n_heads // tp
        self.n_kv_heads = args.n_kv_heads // tp
        qkv_out = (args.n_heads + 2 * args.n_kv_heads) * self.head_dim
        if tp > 1:
            from .tp import ColumnParallelSpBitLinear, RowParallelSpBitLinear
            self.wqkv = ColumnParallelSpBitLinear(args.dim, qkv_out // tp, dic, prefix + ".wqkv")
            self.wo = RowParallelSpBitLinear(args.dim // tp, args.dim, dic, prefix + ".wo", tp_group,
                                             norm_weight=dic[prefix + ".attn_sub_norm.weight"], eps=args.norm_eps)
            self.attn_sub_norm = None
        else:
            self.wqkv = linear_cls(args.dim, qkv_out, dic, prefix + ".wqkv")
            self.wo = linear_cls(args.dim, args.dim, dic, prefix + ".wo")
            self.attn_sub_norm = RMSNorm(args.dim, args.norm_eps)
            with torch.no_grad():
                self.attn_sub_norm.weight.copy_(dic[prefix + ".attn_sub_norm.weight"])

    def forward(self, x, cache: LayerCache, pos, cos, sin, mask, fused=None):
        """``fused`` = (norm weight, eps): the norm in front of wqkv runs in its front-end, x is wo's residual.  ``mask``: [1, 1,
        T, L], or CAUSAL for one token per sequence, all at the same position (rotation, append and attention in one kernel)."""
        B, T = x.shape[0], x.shape[1]
        H, Hkv, D = self.n_heads, self.n_kv_heads, self.head_dim
        qkv = self.wqkv(x) if fused is None else self.wqkv.forward_normed(x, fused[0], fused[1])
        if mask is CAUSAL:
            o = attn_decode_by_head(qkv, cache[0], cache[1], cos[0, 0], sin[0, 0], pos, H, Hkv)
            if o is not None:
                return self._project(o, x, fused)
            mask = causal_mask(pos, cache[0].shape[2])
        q = qkv[..., : H * D].view(B, T, H, D)
        k = qkv[..., H * D: (H + Hkv) * D].view(B, T, Hkv, D)
        v = qkv[..., (H + Hkv) * D:].view(B, T, Hkv, D)
        q, k = apply_rope(q, cos, sin), apply_rope(k, cos, sin)
        ck, cv = cache                                  # [B, Hkv, L, D]
        ck.index_copy_(2, pos, k.transpose(1, 2))
        cv.index_copy_(2, pos, v.transpose(1, 2))
        o = F.scaled_dot_product_attention(q.transpose(1, 2), ck, cv, attn_mask=mask, enable_gqa=True)
        o = o.transpose(1, 2).reshape(B, T, H * D)
        return self._project(o, x, fused)

    def forward_flash(self, x, cache: LayerCache, pos, rope, rope_row, fused):
        """Attention glue in the cache layout [B, L, Hkv, D]: RoPE on adjacent pairs, cache append and causal
        attention - the library's kernels for one token or a prompt per sequence, flash_attn's kv-cache kernel for head
        shapes that they do not take."""
        B, T = x.shape[0], x.shape[1]
        H, Hkv, D = self.n_heads, self.n_kv_heads, self.head_dim
        qkv = self.wqkv(x) if fused is None else self.wqkv.forward_normed(x, fused[0], fused[1])
        if rope_row is not None:
            o = attn_decode(qkv, cache[0], cache[1], *rope_row, pos, H, Hkv)
        else:
            o = attn_prefill(qkv, cache[0], cache[1], *rope, pos, H, Hkv)
        if o is not None:
            return self._project(o, x, fused)
        from flash_attn import flash_attn_with_kvcache
        q = qkv[..., : H * D].view(B, T, H, D)
        k = qkv[..., H * D: (H + Hkv) * D].view(B, T, Hkv, D)
        v = qkv[..., (H + Hkv) * D:].view(B, T, Hkv, D)
        seqlens = pos[:1].to(torch.int32).expand(B).contiguous()
        o = flash_attn_with_kvcache(q, cache[0], cache[1], k=k, v=v, rotary_cos=rope[0], rotary_sin=rope[1],
                                    cache_seqlens=seqlens, causal=True, rotary_interleaved=True)
        return self._project(o.reshape(B, T, H * D), x, fused)

    def _project(self, o, x, fused):
        if fused is not None:
            return self.wo.forward_normed(o, self.attn_sub_norm.weight, fused[1], residual=x)
        if self.attn_sub_norm is not None:
            o = self.attn_sub_norm(o)
        return self.wo(o)


class FeedForward(nn.Module):
    def __init__(self, args: ModelArgs, dic: dict, prefix: str, linear_cls, tp_group=None, tp: int = 1):
        super().__init__()
        if tp > 1:
            from .tp import ColumnParallelSpBitLinear, RowParallelSpBitLinear
            self.w13 = ColumnParallelSpBitLinear(args.dim, 2 * args.ffn_dim // tp, dic, prefix + ".w13")
            self.w2 = RowParallelSpBitLinear(args.ffn_dim // tp, args.dim, dic, prefix + ".w2", tp_group,
                                             norm_weight=dic[prefix + ".ffn_sub_norm.weight"], eps=args.norm_eps)
            self.ffn_sub_norm = None
        else:
            self.w13 = linear_cls(args.dim, 2 * args.ffn_dim, dic, prefix + ".w13")
            self.w2 = linear_cls(args.ffn_dim, args.dim, dic, prefix + ".w2")
            self.ffn_sub_norm = RMSNorm(args.ffn_dim, args.norm_eps)
            with torch.no_grad():
                self.ffn_sub_norm.weight.copy_(dic[prefix + ".ffn_sub_norm.weight"])

    def forward_fused(self, h, norm_weight, eps):
        x13 = self.w13.forward_normed(h, norm_weight, eps)
        return self.w2.forward_normed(x13, self.ffn_sub_norm.weight, eps, gated=True, residual=h)

    def forward(self, x):
        x13 = self.w13(x)
        inner = relu2_gate(x13) if not torch.is_grad_enabled() else None
        if inner is None:
            x1, x3 = x13.chunk(2, -1)
            inner = F.relu(x1) ** 2 * x3
        if self.ffn_sub_norm is not None:
            inner = self.ffn_sub_norm(inner)
        return self.w2(inner)


class TransformerBlock(nn.Module):
    def __init__(self, args: ModelArgs, dic: dict, prefix: str, linear_cls, tp_group=None, tp: int = 1):
        super().__init__()
        self.attention = Attention(args, dic, prefix + ".attention", linear_cls, tp_group, tp)
        self.feed_forward = FeedForward(args, dic, prefix + ".feed_forward", linear_cls, tp_group, tp)
        self.attention_norm = RMSNorm(args.dim, args.norm_eps)
        self.ffn_norm = RMSNorm(args.dim, args.norm_eps)
        with torch.no_grad():
            self.attention_norm.weight.copy_(dic[prefix + ".attention_norm.weight"])
            self.ffn_norm.weight.copy_(dic[prefix + ".ffn_norm.weight"])

    def forward(self, x, cache, pos, cos, sin, mask, fused: bool = False, flash=None):
        if fused:
            eps = self.attention_norm.eps
            fused = (self.attention_norm.weight, eps)
            if flash is not None:
                h = self.attention.forward_flash(x, cache, *flash, fused)
            else:
                h = self.attention(x, cache, pos, cos, sin, mask, fused=fused)
            return self.feed_forward.forward_fused(h, self.ffn_norm.weight, eps)
        if flash is not None:
            h = x + self.attention.forward_flash(self.attention_norm(x), cache, *flash, None)
        else:
            h = x + self.attention(self.attention_norm(x), cache, pos, cos, sin, mask)
        return h + self.feed_forward(self.ffn_norm(h))


class Transformer(nn.Module):
    """``dic`` holds the checkpoint tensors under the reference's key names
    (``layers.<i>.attention.wqkv.weight_bitmap`` ... ``tok_embeddings.weight``,
    ``norm.weight``); the output head is tied to the embedding."""

    def __init__(self, args: ModelArgs, dic: dict, linear_cls=None, max_seq_len: int = 2048, tp_group=None,
                 tp: int = 1):
        super().__init__()
        self.args = args
        linear_cls = linear_cls or (SpBitLinear if args.use_kernel else BF16BitLinear)
        self.tok_embeddings = nn.Embedding(args.vocab_size, args.dim)
        with torch.no_grad():
            self.tok_embeddings.weight.copy_(dic["tok_embeddings.weight"])
        self.layers = nn.ModuleList([TransformerBlock(args, dic, f"layers.{i}", linear_cls, tp_group, tp)
                                     for i in range(args.n_layers)])
        self.norm = RMSNorm(args.dim, args.norm_eps)
        with torch.no_grad():
            self.norm.weight.copy_(dic["norm.weight"])
        self.max_seq_len = max_seq_len
        self.tp = tp
        self._rope = None
        self.flash = False
        want_flash = args.fused_glue if args.flash_attention is None else args.flash_attention
        if want_flash and tp == 1:
            try:
                import flash_attn  # noqa: F401
                self.flash = True
            except Exception:
                if args.flash_attention:
                    raise
                self.flash = False

    def make_cache(self, batch: int, device, dtype=torch.bfloat16) -> List[LayerCache]:
        a = self.args
        shape = (batch, a.n_kv_heads // self.tp, self.max_seq_len, a.head_dim)
        if self.flash:
            shape = (batch, self.max_seq_len, a.n_kv_heads, a.head_dim)
        return [(torch.zeros(shape, device=device, dtype=dtype), torch.zeros(shape, device=device, dtype=dtype))
                for _ in range(a.n_layers)]

    def head(self, h: torch.Tensor, greedy: bool = False):
        """Final norm + tied output head.  fp32 logits [B, T, vocab] (model.py:380-386 of the
        reference); with ``greedy`` -> (None, int64 tokens [B, T]) without materialising the logits.
        Up to 8 rows run on the library's head kernel (one pass over the embedding, arg-max fused);
        more rows use the dense bf16 GEMM."""
        B, T = h.shape[0], h.shape[1]
        if self.args.fused_glue and h.is_cuda and h.dtype == torch.bfloat16 and h.shape[-1] % 16 == 0:
            h = rmsnorm(h, self.norm.weight, self.norm.eps)   # one launch, the fused front-ends' summation order
        else:
            h = self.norm(h)
        emb = self.tok_embeddings.weight
        if h.is_cuda and B * T <= 8 and emb.dtype == torch.bfloat16 and h.dtype == torch.bfloat16 and h.shape[-1] % 32 == 0:
            logits, toks = lm_head_argmax(h, emb, want_logits=not greedy, want_argmax=greedy)
            return (None, toks.view(B, T)) if greedy else logits.view(B, T, -1)
        logits = F.linear(h, emb)
        logits = logits.float() if greedy else to_float(logits)
        return (None, logits.argmax(-1)) if greedy else logits

    def forward(self, tokens: torch.Tensor, cache: List[LayerCache], pos: torch.Tensor, greedy_last: bool = False):
        """tokens [B, T]; pos [T] (device int64) = positions written in the cache.
        Returns fp32 logits [B, T, vocab] (model.py:380-386 of the reference); with ``greedy_last``
        only the greedy token of every sequence's last position, int64 [B] (what the generation
        loop needs: generate.py:274, :283, :305 of the reference)."""
        if self._rope is None or self._rope[0].device != tokens.device:
            self._rope = rope_tables(self.args.head_dim, self.max_seq_len, self.args.rope_theta, tokens.device)
            self._rope_lp = (self._rope[0].to(torch.bfloat16), self._rope[1].to(torch.bfloat16))
        B, T = tokens.shape
        h = self.tok_embeddings(tokens)
        fused = self.args.fused_glue and self.tp == 1
        flash, cos, sin, mask = None, None, None, None
        if self.flash:   # the attention kernels apply RoPE from the tables and mask by position themselves
            flash = (pos, self._rope_lp, tuple(t.index_select(0, pos) for t in self._rope_lp) if T == 1 else None)
        else:
            cos, sin = self._rope[0][pos].expand(B, T, -1), self._rope[1][pos].expand(B, T, -1)
            mask = CAUSAL if T == 1 else causal_mask(pos, self.max_seq_len)
        for layer, c in zip(self.layers, cache):
            h = layer(h, c, pos, cos, sin, mask, fused, flash)
        if greedy_last:
            return self.head(h[:, -1:], greedy=True)[1][:, 0]
        return self.head(h)
