"""GPU: the attention glue of a decode step against a float64 restatement, at the edges of its split over a cluster and
of its key tiles."""
import pytest
import torch

from ternainfer_b200.linear import attn_decode, attn_prefill
from ternainfer_b200.model import apply_rope, rope_tables

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H,Hkv", [(20, 5), (64, 8)])
@pytest.mark.parametrize("B,pos,L", [(1, 0, 8), (1, 1, 8), (2, 7, 8), (1, 9, 64), (1, 127, 640), (3, 600, 640), (8, 255, 300),
                                     (8, 1100, 1101), (1, 2047, 2500), (1, 2300, 2500), (16, 513, 600), (70, 300, 320)])
def test_decode_attention(lib, B, pos, L, H, Hkv):
    D = 128
    g = torch.Generator(device="cuda").manual_seed(pos + B)
    qkv = torch.randn((B, 1, (H + 2 * Hkv) * D), generator=g, device="cuda").to(torch.bfloat16)
    kc, vc = (torch.randn((B, L, Hkv, D), generator=g, device="cuda").to(torch.bfloat16) for _ in range(2))
    kc[:, pos + 1:], vc[:, pos + 1:] = float('nan'), float('nan')       # rows that hold no token yet
    k0, v0 = kc.clone(), vc.clone()
    cos, sin = (t.to(torch.bfloat16) for t in rope_tables(D, L, 500000.0, "cuda"))
    p = torch.tensor([pos], device="cuda")
    out = attn_decode(qkv, kc, vc, cos[p], sin[p], p, H, Hkv)
    q, k, v = (t.view(B, 1, -1, D) for t in qkv.split([H * D, Hkv * D, Hkv * D], -1))
    c, s = cos[p].float().expand(B, 1, -1), sin[p].float().expand(B, 1, -1)
    q, k = apply_rope(q, c, s), apply_rope(k, c, s)
    k0[:, pos], v0[:, pos] = k[:, 0], v[:, 0]
    assert torch.equal(kc.view(torch.int16), k0.view(torch.int16)) and torch.equal(vc.view(torch.int16), v0.view(torch.int16)), "the caches differ from an append of the rotated key and the value"
    kk, vv = (t[:, :pos + 1].double().repeat_interleave(H // Hkv, 2) for t in (k0, v0))
    a = torch.softmax(torch.einsum("bhd,blhd->bhl", q[:, 0].double(), kk) / D ** 0.5, -1)
    want = torch.einsum("bhl,blhd->bhd", a, vv).reshape(B, 1, H * D)
    assert ((out.double() - want).norm() / want.norm()).item() < 3e-3
    assert (out.double() - want).abs().max().item() < 1.2e-2 * want.abs().max().item()
    assert torch.equal(attn_decode(qkv, kc, vc, cos[p], sin[p], p, H, Hkv), out)


@pytest.mark.parametrize("H,Hkv", [(20, 5), (64, 8)])
@pytest.mark.parametrize("B,pos,L", [(1, 0, 8), (3, 7, 8), (2, 127, 640), (3, 333, 461), (8, 1100, 1101), (1, 2300, 2500), (70, 300, 320)])
@torch.no_grad()
def test_decode_attention_by_head(lib, B, pos, L, H, Hkv):
    """On the default glue's caches: bytes appended as torch's rotation and index_copy_ leave them, result as close to float64 as torch's
    masked attention (both round the probabilities to bf16 and the result once), rows without a token unread."""
    from ternainfer_b200.linear import attn_decode_by_head
    from ternainfer_b200.model import causal_mask
    D = 128
    g = torch.Generator(device="cuda").manual_seed(pos + B)
    qkv = torch.randn((B, 1, (H + 2 * Hkv) * D), generator=g, device="cuda").to(torch.bfloat16)
    kc, vc = (torch.randn((B, Hkv, L, D), generator=g, device="cuda").to(torch.bfloat16) for _ in range(2))
    k0, v0 = kc.clone(), vc.clone()
    kc[:, :, pos + 1:], vc[:, :, pos + 1:] = float("nan"), float("nan")
    cos, sin = rope_tables(D, L, 500000.0, "cuda")
    p = torch.tensor([pos], device="cuda")
    out = attn_decode_by_head(qkv, kc, vc, cos[p], sin[p], p, H, Hkv)
    q, k, v = (t.view(B, 1, -1, D) for t in qkv.split([H * D, Hkv * D, Hkv * D], -1))
    with torch.enable_grad():                               # (torch's operators)
        q, k = (apply_rope(t, cos[p].expand(B, 1, -1), sin[p].expand(B, 1, -1)).detach() for t in (q, k))
    k0[:, :, pos], v0[:, :, pos] = k[:, 0], v[:, 0]
    assert torch.equal(kc[:, :, :pos + 1], k0[:, :, :pos + 1]) and torch.equal(vc[:, :, :pos + 1], v0[:, :, :pos + 1])
    assert kc[:, :, pos + 1:].isnan().all() and vc[:, :, pos + 1:].isnan().all()
    kk, vv = (t[:, :, :pos + 1].double().repeat_interleave(H // Hkv, 1) for t in (k0, v0))
    a = torch.softmax(torch.einsum("bhd,bhld->bhl", q[:, 0].double(), kk) / D ** 0.5, -1)
    want = torch.einsum("bhl,bhld->bhd", a, vv).reshape(B, 1, H * D)
    plain = torch.nn.functional.scaled_dot_product_attention(q.transpose(1, 2), k0, v0, attn_mask=causal_mask(p, L), enable_gqa=True)
    err, theirs = (((t.double() - want).norm() / want.norm()).item() for t in (out, plain.transpose(1, 2).reshape(B, 1, H * D)))
    print(f"error against float64 {err:.2e}, torch {theirs:.2e}")
    assert err < max(1.05 * theirs, 2.1e-3)                 # (one rounding to bf16 is 1.7e-3 of normally distributed values)


@pytest.mark.parametrize("B,pos,L", [(1, 8, 8), (3, -1, 40), (2, 2 ** 40, 600), (1, -2 ** 33, 16)])
@torch.no_grad()
def test_decode_attention_by_head_refuses_a_position_outside_of_the_cache(lib, B, pos, L):
    """As index_copy_ did: nothing is written, the result is no number, and the library says so once."""
    from ternainfer_b200.linear import attn_decode_by_head
    H, Hkv, D = 20, 5, 128
    qkv = torch.randn((B, 1, (H + 2 * Hkv) * D), device="cuda").to(torch.bfloat16)
    kc, vc = (torch.randn((B, Hkv, L, D), device="cuda").to(torch.bfloat16) for _ in range(2))
    k0, v0 = kc.clone(), vc.clone()
    cos, sin = (t[0] for t in rope_tables(D, L, 500000.0, "cuda"))
    out = attn_decode_by_head(qkv, kc, vc, cos, sin, torch.tensor([pos], device="cuda"), H, Hkv)
    assert lib.ternaspmm_last_status() == 1 and lib.ternaspmm_last_status() == 0
    assert out.isnan().all() and torch.equal(kc, k0) and torch.equal(vc, v0)
    out = attn_decode_by_head(qkv, kc, vc, cos, sin, torch.tensor([L - 1], device="cuda"), H, Hkv)
    assert lib.ternaspmm_last_status() == 0 and not out.isnan().any()


@pytest.mark.parametrize("H,Hkv", [(20, 5), (64, 8)])
@pytest.mark.parametrize("B,T,past,L", [(1, 2, 0, 8), (2, 16, 0, 16), (1, 17, 0, 64), (3, 64, 0, 64), (1, 65, 1, 80), (2, 200, 63, 300), (1, 613, 0, 613),
                                        (1, 40, 1000, 1040), (1, 129, 0, 200), (2, 500, 37, 640)])
def test_prompt_attention(lib, B, T, past, L, H, Hkv):
    D = 128
    g = torch.Generator(device="cuda").manual_seed(T + past)
    qkv = torch.randn((B, T, (H + 2 * Hkv) * D), generator=g, device="cuda").to(torch.bfloat16)
    kc, vc = (torch.randn((B, L, Hkv, D), generator=g, device="cuda").to(torch.bfloat16) for _ in range(2))
    kc[:, past:], vc[:, past:] = float("nan"), float("nan")
    k0, v0 = kc.clone(), vc.clone()
    cos, sin = (t.to(torch.bfloat16) for t in rope_tables(D, L, 500000.0, "cuda"))
    p = torch.arange(past, past + T, device="cuda")
    out = attn_prefill(qkv, kc, vc, cos, sin, p, H, Hkv)
    q, k, v = (t.view(B, T, -1, D) for t in qkv.split([H * D, Hkv * D, Hkv * D], -1))
    c, s = cos[p].float().expand(B, T, -1), sin[p].float().expand(B, T, -1)
    q, k = apply_rope(q, c, s), apply_rope(k, c, s)
    k0[:, past:past + T], v0[:, past:past + T] = k, v
    assert torch.equal(kc.view(torch.int16), k0.view(torch.int16)) and torch.equal(vc.view(torch.int16), v0.view(torch.int16))
    kk, vv = (t[:, :past + T].double().repeat_interleave(H // Hkv, 2) for t in (k0, v0))
    a = torch.einsum("bthd,blhd->bhtl", q.double(), kk) / D ** 0.5
    a = a.masked_fill(torch.arange(past + T, device="cuda")[None, :] > p[:, None], float("-inf")).softmax(-1)
    want = torch.einsum("bhtl,blhd->bthd", a, vv).reshape(B, T, H * D)
    assert ((out.double() - want).norm() / want.norm()).item() < 4e-3
    assert (out.double() - want).abs().max().item() < 1.2e-2 * want.abs().max().item()


def test_attention_refuses_what_its_kernels_cannot_check(lib, monkeypatch):
    """Tensors on other devices, of other shapes or strides: None (and the caller's general path), without a launch."""
    from ternainfer_b200 import linear
    H, Hkv, D, B, L = 20, 5, 128, 2, 16

    def args(T, **other):
        a = dict(qkv=torch.zeros((B, T, (H + 2 * Hkv) * D), dtype=torch.bfloat16, device="cuda"), pos=torch.arange(T, device="cuda"),
                 k=torch.zeros((B, L, Hkv, D), dtype=torch.bfloat16, device="cuda"), v=torch.zeros((B, L, Hkv, D), dtype=torch.bfloat16, device="cuda"),
                 cos=torch.zeros((1 if T == 1 else L, 64), dtype=torch.bfloat16, device="cuda"), heads=H, kv_heads=Hkv)
        a["sin"] = a["cos"].clone()
        a.update((k, f(a[k])) for k, f in other.items())
        return a["qkv"], a["k"], a["v"], a["cos"], a["sin"], a["pos"], a["heads"], a["kv_heads"]

    assert attn_decode(*args(1)) is not None and attn_prefill(*args(3)) is not None
    monkeypatch.setattr(linear, "load_library", lambda: pytest.fail("launched"))
    bad = [dict(pos=torch.Tensor.cpu), dict(k=torch.Tensor.cpu), dict(v=torch.Tensor.cpu), dict(cos=torch.Tensor.cpu), dict(sin=torch.Tensor.cpu),
           dict(sin=torch.Tensor.float), dict(pos=torch.Tensor.int), dict(qkv=lambda t: t[..., :-128].contiguous()), dict(qkv=lambda t: t[:1].contiguous()),
           dict(k=lambda t: t[:1].contiguous()), dict(v=lambda t: t[:, :8].contiguous()), dict(k=lambda t: t[:, :, :4].contiguous(), v=lambda t: t[:, :, :4].contiguous()),
           dict(v=lambda t: t.transpose(1, 2).contiguous().transpose(1, 2)), dict(pos=lambda t: torch.arange(len(t) + 1, device="cuda")),
           dict(heads=lambda h: h + 4), dict(kv_heads=lambda h: 0), dict(cos=lambda t: t[:, :32].contiguous(), sin=lambda t: t[:, :32].contiguous()),
           dict(pos=lambda t: torch.arange(2 * len(t), device="cuda")[::2])]
    for T, f in ((1, attn_decode), (3, attn_prefill)):
        for other in bad:
            if T == 1 and list(other) == ["pos"] and other is bad[-1]:
                continue                                                    # (one element is contiguous)
            assert f(*args(T, **other)) is None, (T, list(other))
    assert attn_prefill(*args(17, cos=lambda t: t[:1].expand(17, 64).contiguous(), sin=lambda t: t[:1].expand(17, 64).contiguous())) is None, "more tokens than rows of the cache"
    assert attn_decode(*args(2)) is None


@pytest.mark.parametrize("B,T,past,L", [(1, 1, 600, 640), (8, 1, 1100, 1101), (2, 613, 0, 613), (1, 200, 1000, 1200), (1, 1024, 0, 1024)])
def test_attention_is_as_exact_as_flash_attn(lib, B, T, past, L):
    """Error against float64 beside that of the kernel which the model called before, on the same inputs."""
    flash_attn = pytest.importorskip("flash_attn")
    H, Hkv, D = 20, 5, 128
    g = torch.Generator(device="cuda").manual_seed(T + past)
    qkv = torch.randn((B, T, (H + 2 * Hkv) * D), generator=g, device="cuda").to(torch.bfloat16)
    kc, vc = (torch.randn((B, L, Hkv, D), generator=g, device="cuda").to(torch.bfloat16) for _ in range(2))
    k0, v0 = kc.clone(), vc.clone()
    cos, sin = (t.to(torch.bfloat16) for t in rope_tables(D, L, 500000.0, "cuda"))
    p = torch.arange(past, past + T, device="cuda")
    ours = attn_decode(qkv, kc, vc, cos[p], sin[p], p, H, Hkv) if T == 1 else attn_prefill(qkv, kc, vc, cos, sin, p, H, Hkv)
    q, k, v = (t.view(B, T, -1, D) for t in qkv.split([H * D, Hkv * D, Hkv * D], -1))
    theirs = flash_attn.flash_attn_with_kvcache(q, k0, v0, k=k, v=v, rotary_cos=cos, rotary_sin=sin, causal=True, rotary_interleaved=True,
                                                cache_seqlens=torch.full((B,), past, dtype=torch.int32, device="cuda")).reshape(B, T, H * D)
    qr = apply_rope(q, cos[p].float().expand(B, T, -1), sin[p].float().expand(B, T, -1)).double()
    kk, vv = (t[:, :past + T].double().repeat_interleave(H // Hkv, 2) for t in (kc, vc))
    a = torch.einsum("bthd,blhd->bhtl", qr, kk) / D ** 0.5
    a = a.masked_fill(torch.arange(past + T, device="cuda")[None, :] > p[:, None], float("-inf")).softmax(-1)
    want = torch.einsum("bhtl,blhd->bthd", a, vv).reshape(B, T, H * D)
    e_ours, e_theirs = (((t.double() - want).norm() / want.norm()).item() for t in (ours, theirs))
    # the same formats (bf16 operands and probabilities, fp32 sums) and 2e5 to 6e6 outputs: the two norms agree to a per cent
    assert e_ours <= 1.02 * e_theirs


@pytest.mark.parametrize("B,pos,L", [(2, 17, 40), (3, 333, 461), (8, 1100, 1101), (1, 2300, 2500)])
@torch.no_grad()
def test_default_glue_attention_is_no_less_exact_than_torch(lib, B, pos, L):
    """Error against float64 beside that of the operators which the model called before, on the same inputs: both round the rotated query, the
    probabilities and the result to bf16, torch its intermediate sums as well, so the kernel's is the smaller one (2.0e-3 and 2.2e-3)."""
    from ternainfer_b200.linear import attn_decode_by_head
    from ternainfer_b200.model import causal_mask
    H, Hkv, D = 20, 5, 128
    g = torch.Generator(device="cuda").manual_seed(7 * pos + B)
    qkv = torch.randn((B, 1, (H + 2 * Hkv) * D), generator=g, device="cuda").to(torch.bfloat16)
    kc, vc = (torch.randn((B, Hkv, L, D), generator=g, device="cuda").to(torch.bfloat16) for _ in range(2))
    cos, sin = rope_tables(D, L, 500000.0, "cuda")
    p = torch.tensor([pos], device="cuda")
    ours = attn_decode_by_head(qkv, kc, vc, cos[p], sin[p], p, H, Hkv)
    q = apply_rope(qkv[..., :H * D].view(B, 1, H, D), cos[p].expand(B, 1, -1), sin[p].expand(B, 1, -1))
    theirs = torch.nn.functional.scaled_dot_product_attention(q.transpose(1, 2), kc, vc, attn_mask=causal_mask(p, L), enable_gqa=True).transpose(1, 2).reshape(B, 1, H * D)
    kk, vv = (t[:, :, :pos + 1].double().repeat_interleave(H // Hkv, 1) for t in (kc, vc))
    a = torch.softmax(torch.einsum("bhd,bhld->bhl", q[:, 0].double(), kk) / D ** 0.5, -1)
    want = torch.einsum("bhl,bhld->bhd", a, vv).reshape(B, 1, H * D)
    e_ours, e_theirs = (((t.double() - want).norm() / want.norm()).item() for t in (ours, theirs))
    assert e_ours <= e_theirs


def test_default_glue_attention_refuses_what_its_kernel_cannot_check(lib, monkeypatch):
    """Tensors on other devices, of other types, shapes or strides, and under autograd: None (and the caller's general path), without a launch."""
    from ternainfer_b200 import linear
    H, Hkv, D, B, L = 20, 5, 128, 2, 16

    def args(**other):
        a = dict(qkv=torch.zeros((B, 1, (H + 2 * Hkv) * D), dtype=torch.bfloat16, device="cuda"), k=torch.zeros((B, Hkv, L, D), dtype=torch.bfloat16, device="cuda"),
                 v=torch.zeros((B, Hkv, L, D), dtype=torch.bfloat16, device="cuda"), cos=torch.zeros(64, device="cuda"), sin=torch.zeros(64, device="cuda"),
                 pos=torch.arange(1, device="cuda"), heads=H, kv_heads=Hkv)
        a.update((k, f(a[k])) for k, f in other.items())
        return a.values()

    with torch.no_grad():
        assert linear.attn_decode_by_head(*args()) is not None
    monkeypatch.setattr(linear, "load_library", lambda: pytest.fail("launched"))
    assert linear.attn_decode_by_head(*args()) is None, "under autograd"
    bad = [dict(pos=torch.Tensor.cpu), dict(k=torch.Tensor.cpu), dict(v=torch.Tensor.cpu), dict(cos=torch.Tensor.cpu), dict(sin=torch.Tensor.cpu),
           dict(cos=torch.Tensor.bfloat16), dict(sin=torch.Tensor.double), dict(k=torch.Tensor.float), dict(v=torch.Tensor.half), dict(qkv=torch.Tensor.float),
           dict(pos=torch.Tensor.int), dict(pos=lambda t: torch.arange(2, device="cuda")), dict(qkv=lambda t: t[..., :-128].contiguous()),
           dict(qkv=lambda t: t[:1].contiguous()), dict(qkv=lambda t: torch.cat([t, t], 1)), dict(qkv=lambda t: t[:, 0]), dict(k=lambda t: t[:1].contiguous()),
           dict(v=lambda t: t[:, :, :8].contiguous()), dict(k=lambda t: t[:, :4].contiguous(), v=lambda t: t[:, :4].contiguous()),
           dict(k=lambda t: t[..., :64].contiguous(), v=lambda t: t[..., :64].contiguous()), dict(k=lambda t: t[:, :, :0], v=lambda t: t[:, :, :0]),
           dict(v=lambda t: t.transpose(1, 2).contiguous().transpose(1, 2)), dict(cos=lambda t: t[:32], sin=lambda t: t[:32]),
           dict(cos=lambda t: torch.zeros(128, device="cuda")[::2]), dict(heads=lambda h: h + 4), dict(kv_heads=lambda h: 4), dict(kv_heads=lambda h: 0)]
    with torch.no_grad():
        for other in bad:
            assert linear.attn_decode_by_head(*args(**other)) is None, list(other)
