"""GPU: linears on two-bit weights (the layout SpBitLinear keeps) against the CPU oracle, bit for bit, at the edges of
the kernel's tiles: odd numbers of 64-column blocks, fewer blocks than warps, one strip group too many, token blocks with
one row, weights larger than the shared-memory ring."""
import copy
import ctypes

import numpy as np
import pytest
import torch

import ternaspmm_oracle as o
import c_oracle
from gpu_util import Packed, dev
from ternainfer_b200.convert import compress_weight
from ternainfer_b200.linear import SpBitLinear, quant_input, rmsnorm_quant

pytestmark = pytest.mark.gpu


def w2_of(lib, pk):
    w2 = torch.empty(lib.ternaspmm_w2_bytes(pk.N, pk.K), dtype=torch.uint8, device="cuda")
    lib.ternaspmm_w2_relayout(pk.bm.data_ptr(), pk.tg.data_ptr(), pk.tm.data_ptr(), pk.cv.data_ptr(), pk.N, pk.K, w2.data_ptr(),
                              torch.cuda.current_stream().cuda_stream)
    return w2


@pytest.mark.parametrize("N,K,ws_num", [(64, 64, 1), (128, 192, 2), (192, 1088, 1), (3840, 2560, 3), (2560, 6912, 1), (64, 28672, 1),
                                        (13824, 320, 2), (38464, 128, 2), (9536, 8192, 1)])
@pytest.mark.parametrize("M", [1, 7, 9, 17, 33, 64, 65, 130])
def test_linear_on_two_bit_weights(lib, M, N, K, ws_num):
    check_linear(lib, M, N, K, ws_num)


def check_linear(lib, M, N, K, ws_num):
    w = o.make_ternary(N, K, 0.45, N + K)
    pk = Packed(w, [t.cpu().numpy() for t in compress_weight(torch.from_numpy(w).cuda())])
    xq, s = o.make_activations(M, K, M + 1)
    xq[0, :64] = -128
    ws = o.make_ws(ws_num, M + 2)
    sb, wb = o.f32_to_bf16_bits(s.reshape(-1)), o.f32_to_bf16_bits(ws)
    _, want = c_oracle.ternaspmm(xq, w, sb, wb, ws_num, -1)
    w2, x_d, s_d, ws_d = w2_of(lib, pk), dev(xq), dev(sb), dev(wb)
    for residual, skew in ((False, 0), (True, 0), (True, 3)):
        res_d, exp = None, want
        if residual:
            res = o.bf16_round(np.random.default_rng(M).standard_normal((M, N)).astype(np.float32))
            res_d, exp = dev(o.f32_to_bf16_bits(res)), o.f32_to_bf16_bits(res + o.bf16_bits_to_f32(want))
        out = torch.full((M * N + 128,), 0x7B7B, dtype=torch.int16, device="cuda")
        lib.ternaspmm_w2_linear(x_d.data_ptr(), 0, None, 0.0, w2.data_ptr(), out.data_ptr() + 2 * skew, s_d.data_ptr(), ws_d.data_ptr(),
                                ws_num, M, N, K, 0, 0, 0, -1, res_d.data_ptr() if residual else None,
                                torch.cuda.current_stream().cuda_stream)
        torch.cuda.synchronize()
        assert lib.ternaspmm_last_status() == 0
        got = out.cpu().numpy().view(np.uint16)
        assert (got[:skew] == 0x7B7B).all() and (got[skew + M * N:] == 0x7B7B).all(), "wrote outside the output"
        assert (got[skew:skew + M * N].reshape(M, N) == exp).all()


@pytest.mark.parametrize("M,N,K", [(40, 64, 64), (257, 320, 192), (700, 320, 128), (2049, 2560, 192), (1000, 13824, 320), (300, 2560, 6912),
                                   (1226, 3840, 2560), (4096, 192, 64), (150, 57344, 128)])
def test_pairs_with_several_tiles_and_ragged_edges(lib, M, N, K):
    """Several tiles per pair, a last row block of 64 rows, half a last stage; small and deep layers, which single tiles take (heights: below)."""
    check_linear(lib, M, N, K, 2)


@pytest.mark.parametrize("M,N,K", [(9, 64, 64), (16, 128, 640), (33, 192, 1088), (64, 2560, 2560), (48, 2560, 6912), (80, 1024, 16384), (129, 1344, 1344),
                                   (250, 2560, 2560), (190, 320, 8256), (256, 13824, 320), (1025, 128, 192)])
def test_tiles_in_tensor_memory(lib, M, N, K):
    """One to eight slices of K (uneven ones, half a last block pair), one to several blocks of tokens, half a last row tile (heights: below)."""
    check_linear(lib, M, N, K, 3)


@pytest.mark.parametrize("M,N,K", [(24, 320, 640), (70, 3840, 2560), (600, 320, 640)])
def test_scales_out_of_the_usual_range_and_segments(lib, M, N, K):
    """Scales that the epilogue's short division does not take (tiny, huge, zero) beside usual ones; one scale segment, and several inside a row tile."""
    w = o.make_ternary(N, K, 0.45, N + K)
    pk = Packed(w, [t.cpu().numpy() for t in compress_weight(torch.from_numpy(w).cuda())])
    w2, stream = w2_of(lib, pk), torch.cuda.current_stream().cuda_stream
    xq, s = o.make_activations(M, K, M + 1)
    s = s.reshape(-1)
    odd = s.copy()
    odd[::5], odd[1::7], odd[2::11] = 1e-20, 3e15, 0.0
    wb = o.f32_to_bf16_bits(o.make_ws(4, M + 2))
    for scales in (s, odd):
        for prefill in (0, 1):
            for seg in ((N, N, N), (40, 104, 200)):
                sb = o.f32_to_bf16_bits(scales)
                out = torch.empty((M, N), dtype=torch.int16, device="cuda")
                x_d, s_d, ws_d = dev(xq), dev(sb), dev(wb)
                lib.ternaspmm_w2_linear(x_d.data_ptr(), 0, None, 0.0, w2.data_ptr(), out.data_ptr(), s_d.data_ptr(), ws_d.data_ptr(), 4, M, N, K,
                                        *seg, prefill, None, stream)
                want = torch.empty_like(out)
                lib.ternaspmm_linear_segments(x_d.data_ptr(), pk.bm.data_ptr(), pk.tg.data_ptr(), pk.tm.data_ptr(), pk.cv.data_ptr(), want.data_ptr(),
                                              s_d.data_ptr(), ws_d.data_ptr(), 4, M, N, K, *seg, prefill, stream)
                torch.cuda.synchronize()
                assert lib.ternaspmm_last_status() == 0
                a, b = out.cpu().numpy().view(np.uint16), want.cpu().numpy().view(np.uint16)
                nan = np.isnan(o.bf16_bits_to_f32(b))
                assert (np.isnan(o.bf16_bits_to_f32(a)) == nan).all() and (a == b)[~nan].all()


@pytest.mark.parametrize("M,N,K", [(3, 320, 640), (6, 192, 1088), (24, 320, 640), (70, 3840, 2560), (1000, 13824, 320)])
@pytest.mark.parametrize("skew", [0, 1])
def test_scales_at_the_ends_of_the_number_range(lib, M, N, K, skew):
    """Every scale that bf16 has is a valid one: the largest, infinity and subnormals beside usual ones, by each kernel, with outputs at odd
    addresses too: the quotient of the packed kernels, bit for bit."""
    w = o.make_ternary(N, K, 0.45, N + K)
    pk = Packed(w, [t.cpu().numpy() for t in compress_weight(torch.from_numpy(w).cuda())])
    w2, stream = w2_of(lib, pk), torch.cuda.current_stream().cuda_stream
    xq, s = o.make_activations(M, K, M + 1)
    s = s.reshape(-1).copy()
    s[::3], s[1::7], s[2::11], s[-1] = 1e37, np.finfo(np.float32).max / 2, 1e-39, np.inf
    ws = o.make_ws(2, M + 2)
    ws[:2] *= 1e30                                     # (so that outputs under the largest scales are not zero)
    x_d, s_d, ws_d = dev(xq), dev(o.f32_to_bf16_bits(s)), dev(o.f32_to_bf16_bits(ws))
    for prefill in (0, 1):
        for seg in ((N, N, N), (40, 104, 200)):
            got, want = (torch.empty(M * N + 8, dtype=torch.int16, device="cuda")[skew:skew + M * N] for _ in range(2))
            lib.ternaspmm_w2_linear(x_d.data_ptr(), 0, None, 0.0, w2.data_ptr(), got.data_ptr(), s_d.data_ptr(), ws_d.data_ptr(), 2, M, N, K,
                                    *seg, prefill, None, stream)
            lib.ternaspmm_linear_segments(x_d.data_ptr(), pk.bm.data_ptr(), pk.tg.data_ptr(), pk.tm.data_ptr(), pk.cv.data_ptr(), want.data_ptr(),
                                          s_d.data_ptr(), ws_d.data_ptr(), 2, M, N, K, *seg, prefill, stream)
            torch.cuda.synchronize()
            assert lib.ternaspmm_last_status() == 0
            a, b = got.cpu().numpy().view(np.uint16), want.cpu().numpy().view(np.uint16)
            nan = np.isnan(o.bf16_bits_to_f32(b))
            assert (np.isnan(o.bf16_bits_to_f32(a)) == nan).all() and (a == b)[~nan].all()
            assert ((b.reshape(M, N)[::3] & 0x7FFF) != 0).any()


@pytest.mark.parametrize("M,N,K,kernel", [(5, 64, 640, 8), (5, 64, 576, 9), (8, 4736, 1024, 8), (8, 4800, 1024, 9), (6, 7104, 1088, 8), (6, 7168, 1088, 9), (9, 64, 640, 9),
                                          (7, 128, 17408, 8), (7, 128, 17536, 9), (5, 192, 2496, 8), (4, 7168, 256, 8), (8, 2432, 7104, 8), (8, 2432, 7168, 9), (8, 2368, 7168, 8)])
def test_five_to_eight_tokens_by_either_kernel(lib, M, N, K, kernel):
    """Either side of each line of the rule (on 148 SMs): the kernel that was measured to be the faster one there, and the oracle's bits."""
    check_linear(lib, M, N, K, 2)
    shape = (ctypes.c_int * 6)()
    lib.ternaspmm_last_launch_shape(shape)
    assert shape[0] == kernel or torch.cuda.get_device_properties(0).multi_processor_count != 148


def check_against_packed(lib, M, N, K):
    g = torch.Generator(device="cuda").manual_seed(N + K + M)
    w = torch.randint(-1, 2, (N, K), generator=g, device="cuda", dtype=torch.int8)
    pk = Packed(np.empty((N, K), np.int8), [t.cpu().numpy() for t in compress_weight(w)])
    w2, stream = w2_of(lib, pk), torch.cuda.current_stream().cuda_stream
    x = torch.randint(-128, 128, (M, K), generator=g, device="cuda", dtype=torch.int8)
    s = (20 + 10 * torch.rand(M, generator=g, device="cuda")).to(torch.bfloat16)
    ws = torch.tensor([0.5, 2.0, 0, 0], device="cuda").to(torch.bfloat16)
    got, want = (torch.full((M, N), float("nan"), dtype=torch.bfloat16, device="cuda") for _ in range(2))
    lib.ternaspmm_w2_linear(x.data_ptr(), 0, None, 0.0, w2.data_ptr(), got.data_ptr(), s.data_ptr(), ws.data_ptr(), 2, M, N, K, 0, 0, 0, -1, None, stream)
    shape = (ctypes.c_int * 6)()
    lib.ternaspmm_last_launch_shape(shape)
    res, summed = torch.randn((M, N), generator=g, device="cuda").to(torch.bfloat16), torch.full((M, N), float("nan"), dtype=torch.bfloat16, device="cuda")
    lib.ternaspmm_w2_linear(x.data_ptr(), 0, None, 0.0, w2.data_ptr(), summed.data_ptr(), s.data_ptr(), ws.data_ptr(), 2, M, N, K, 0, 0, 0, -1, res.data_ptr(), stream)
    lib.bitlinear_TernaSpMM(x.data_ptr(), pk.bm.data_ptr(), pk.tg.data_ptr(), pk.tm.data_ptr(), pk.cv.data_ptr(), want.data_ptr(), s.data_ptr(),
                            ws.data_ptr(), 2, M, N, K, 1, None, stream)
    assert lib.ternaspmm_last_status() == 0 and torch.equal(got, want) and torch.equal(summed, (res.float() + want.float()).to(torch.bfloat16))
    return list(shape)


@pytest.mark.parametrize("M,N,K", [(1, 4800, 3072), (4, 7104, 3072), (4, 7168, 384), (2, 9536, 2624), (3, 11840, 640), (4, 11904, 4096), (1, 14208, 2560), (2, 14272, 7680), (3, 4800, 8256)])
def test_strips_at_a_time(lib, M, N, K):
    """CTAs of three to seven strips, some with one less, one and three strips at a time: the bits of the packed kernels."""
    check_against_packed(lib, M, N, K)


@pytest.mark.parametrize("M,N,K,warps", [(1, 11840, 8192, 16), (2, 11840, 8128, 10), (2, 11904, 8192, 10), (4, 11904, 8192, 10), (3, 19008, 8192, 10), (4, 19008, 8192, 16), (4, 18944, 8192, 10),
                                         (1, 11904, 12288, 20), (1, 11904, 12224, 10), (3, 128, 28672, 19)])
def test_ten_and_twenty_warps(lib, M, N, K, warps):
    """Either side of each line of the rule (on 148 SMs): the warps that were measured to be faster there, the bits of the packed kernels."""
    shape = check_against_packed(lib, M, N, K)
    assert shape[0] == 8 and (shape[3] == warps or torch.cuda.get_device_properties(0).multi_processor_count != 148)


@pytest.mark.parametrize("M,N,K,tokens", [(65, 38208, 1216, 96), (4170, 1088, 64, 96), (2691, 2368, 1216, 128), (1807, 2496, 1216, 160), (2249, 2368, 1216, 192), (1603, 1600, 2368, 192),
                                          (1926, 1600, 4544, 224), (193, 28800, 3264, 224), (1541, 2560, 6912, 224), (2249, 1600, 9152, 256), (225, 28800, 4544, 256), (2402, 3392, 9152, 256)])
def test_pairs_by_tokens_per_tile(lib, M, N, K, tokens):
    """Every height of the pair kernel's tiles (on 148 SMs), one tile per pair and several, one accumulator buffer and two, ragged in every dimension: the
    bits of the packed kernels."""
    shape = check_against_packed(lib, M, N, K)
    assert shape[:2] == [7, tokens] or torch.cuda.get_device_properties(0).multi_processor_count != 148


@pytest.mark.parametrize("M,N,K,tokens,slices", [(9, 64, 64, 16, 1), (17, 320, 1216, 32, 2), (577, 448, 2368, 64, 3), (33, 192, 1984, 48, 4), (257, 576, 9152, 64, 5), (1569, 64, 5184, 64, 5),
                                                 (100, 448, 5184, 64, 6), (9, 64, 7104, 16, 7), (23, 192, 16448, 32, 8), (129, 13120, 1216, 80, 1), (257, 7616, 1216, 96, 1),
                                                 (770, 2880, 1216, 112, 1), (1671, 1344, 1216, 128, 1), (5000, 448, 64, 128, 1)])
def test_tiles_by_tokens_and_slices(lib, M, N, K, tokens, slices):
    """Every height of the tile kernel's tiles and every number of K slices (on 148 SMs), the bits of the packed kernels."""
    shape = check_against_packed(lib, M, N, K)
    assert shape[:3] == [9, tokens, slices] or torch.cuda.get_device_properties(0).multi_processor_count != 148


def test_layout_and_linear_on_one_stream(lib):
    """Two weights and two norm weights in turn through the same memory, layout and linear in stream order: never the other's values."""
    N, K = 13824, 2560
    ws = [o.make_ternary(N, K, 0.45, i) for i in (1, 2)]
    pks = [Packed(w, [t.cpu().numpy() for t in compress_weight(torch.from_numpy(w).cuda())]) for w in ws]
    g = torch.Generator(device="cuda").manual_seed(1)
    x = torch.randn((1, K), generator=g, device="cuda").to(torch.bfloat16)
    norms = [(1 + 0.3 * torch.randn(K, generator=g, device="cuda")).to(torch.bfloat16) for _ in range(2)]
    scale = torch.tensor([0.5, 2.0, 0, 0], device="cuda").to(torch.bfloat16)
    w2, norm = torch.empty(lib.ternaspmm_w2_bytes(N, K), dtype=torch.uint8, device="cuda"), torch.empty_like(norms[0])
    outs = torch.empty((80, 1, N), dtype=torch.bfloat16, device="cuda")
    stream = torch.cuda.current_stream().cuda_stream
    for i in range(80):
        pk = pks[i & 1]
        norm.copy_(norms[i & 1])
        lib.ternaspmm_w2_relayout(pk.bm.data_ptr(), pk.tg.data_ptr(), pk.tm.data_ptr(), pk.cv.data_ptr(), N, K, w2.data_ptr(), stream)
        for _ in range(1 + i % 3):
            lib.ternaspmm_w2_linear(x.data_ptr(), 2, norm.data_ptr(), 1e-5, w2.data_ptr(), outs[i].data_ptr(), None, scale.data_ptr(), 2, 1, N, K,
                                    0, 0, 0, -1, None, stream)
    for i in (0, 1):
        xq, s = rmsnorm_quant(x, norms[i], 1e-5)
        _, want = c_oracle.ternaspmm(xq.cpu().numpy(), ws[i], s.view(torch.int16).cpu().numpy().view(np.uint16).reshape(-1),
                                     scale.view(torch.int16).cpu().numpy().view(np.uint16), 2, -1)
        got = outs[i::2].view(torch.int16).cpu().numpy().view(np.uint16)
        assert (got == want[None]).all()


def make_layer(N, K, ws_num, seed, segments=None):
    w = o.make_ternary(N, K, 0.45, seed)
    cv, tg, tm, bm = compress_weight(torch.from_numpy(w))
    dic = {"l.weight_compressed_val": cv, "l.weight_TileOffsets_global": tg, "l.weight_TileOffsets_median": tm, "l.weight_bitmap": bm,
           "l.weight_scale": torch.from_numpy(o.make_ws(ws_num, seed)).to(torch.bfloat16)}
    if segments:
        dic["l.weight_segments"] = torch.tensor(segments)
    return SpBitLinear(K, N, dic, "l"), dic


@pytest.mark.parametrize("N,K", [(2560, 2560), (64, 64), (192, 6912), (128, 28672), (64, 8256), (64, 8128), (128, 8192)])
@pytest.mark.parametrize("M", [1, 2, 3, 4, 5, 8, 20, 64, 70])
@pytest.mark.parametrize("kind", ["plain", "norm", "gated"])
def test_front_end_inside_the_linear(lib, M, N, K, kind):
    """bf16 activations: one kernel or two, always the values of the separate front-end followed by the linear."""
    layer, _ = make_layer(N, K, 1, N + K)
    g = torch.Generator(device="cuda").manual_seed(M)
    x = torch.randn((M, 2 * K if kind == "gated" else K), generator=g, device="cuda").to(torch.bfloat16)
    w = (1 + 0.1 * torch.randn(K, generator=g, device="cuda")).to(torch.bfloat16)
    res = torch.randn((M, N), generator=g, device="cuda").to(torch.bfloat16)
    if kind == "plain":
        xf = (127 / x.abs().max(dim=-1, keepdim=True).values.clamp_(min=1e-5))
        xq, s = (x * xf).round().clamp(-128, 127).to(torch.int8), xf
        assert all(torch.equal(a, b) for a, b in zip(quant_input(x), (xq, s)))
        got, want = layer(x), layer.forward_quantized(xq, s)
    else:
        xq, s = rmsnorm_quant(x, w, 1e-5, gated=kind == "gated")
        got = layer.forward_normed(x, w, 1e-5, gated=kind == "gated", residual=res)
        want = layer.forward_quantized(xq, s, residual=res)
    assert torch.equal(got, want)


@pytest.mark.parametrize("M,N,K", [(2, 64, 5120), (2, 64, 5184), (2, 4800, 4096), (3, 64, 3392), (3, 128, 3456), (4, 64, 2560), (4, 64, 2624)])
def test_quantiser_inside_the_linear_or_before_it(lib, M, N, K):
    """Either side of the line up to which a few rows are quantised inside: the values of the separate launch."""
    layer, _ = make_layer(N, K, 1, N + K)
    x = torch.randn((M, K), generator=torch.Generator(device="cuda").manual_seed(M), device="cuda").to(torch.bfloat16)
    x[-1] *= 100
    assert torch.equal(layer(x), layer.forward_quantized(*quant_input(x)))


def test_layer_follows_its_weights(lib):
    """New values in place, a loaded state dict, a replaced parameter and copies: the layout is never stale."""
    layer, dic = make_layer(128, 192, 2, 1, segments=[64, 64])
    other, dic2 = make_layer(128, 192, 2, 1, segments=[64, 64])
    x = torch.randn((5, 192), generator=torch.Generator().manual_seed(1)).to(torch.bfloat16).cuda()
    y = layer(x)
    twin = copy.deepcopy(layer)
    assert torch.equal(twin(x), y)
    signs = layer.weight_compressed_val
    layer.weight_compressed_val.data.view(torch.int32).copy_(~signs.data.view(torch.int32))      # every sign flipped
    assert torch.equal(layer(x), -y)
    assert torch.equal(twin(x), y)
    layer.load_state_dict(other.state_dict())
    assert torch.equal(layer(x), y)
    layer.weight_compressed_val = torch.nn.Parameter((~dic["l.weight_compressed_val"].view(torch.int32)).view(torch.uint32).cuda(),
                                                     requires_grad=False)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):                  # not laid out again inside a capture: reads the packed tensors
        z = layer(x)
    graph.replay()
    assert torch.equal(z, -y) and torch.equal(layer(x), -y)


@pytest.mark.parametrize("N,K", [(64, 64), (2560, 2560), (192, 6912), (320, 8128), (13824, 8192)])
@pytest.mark.parametrize("M", [1, 2, 3, 4, 5, 7, 8])
def test_front_end_of_several_rows_through_the_c_abi(lib, M, N, K):
    """Front-ends 1-3 up to ternaspmm_w2_fused_rows(K) tokens, rows of very different size: the values of the separate launch."""
    assert lib.ternaspmm_w2_fused_rows(K) == 8 and lib.ternaspmm_w2_fused_rows(8256) == 0
    w = torch.from_numpy(o.make_ternary(N, K, 0.45, N + K)).cuda()
    pk = Packed(np.empty((N, K), np.int8), [t.cpu().numpy() for t in compress_weight(w)])
    w2, stream = w2_of(lib, pk), torch.cuda.current_stream().cuda_stream
    g = torch.Generator(device="cuda").manual_seed(M)
    norm = (1 + 0.1 * torch.randn(K, generator=g, device="cuda")).to(torch.bfloat16)
    ws = torch.tensor([0.5, 2.0, 0, 0], device="cuda").to(torch.bfloat16)
    res = torch.randn((M, N), generator=g, device="cuda").to(torch.bfloat16)
    size = torch.logspace(-2, 2, M, device="cuda")[:, None]
    for front_end in (1, 2, 3):
        x = (torch.randn((M, K if front_end < 3 else 2 * K), generator=g, device="cuda") * size).to(torch.bfloat16)
        xq, s = quant_input(x) if front_end == 1 else rmsnorm_quant(x, norm, 1e-5, gated=front_end == 3)
        outs = [torch.full((M, N), float("nan"), dtype=torch.bfloat16, device="cuda") for _ in range(2)]
        for out, (t, fe, sc) in zip(outs, ((x, front_end, None), (xq, 0, s.data_ptr()))):
            lib.ternaspmm_w2_linear(t.data_ptr(), fe, norm.data_ptr(), 1e-5, w2.data_ptr(), out.data_ptr(), sc, ws.data_ptr(), 2, M, N, K, 0, 0, 0, -1,
                                    res.data_ptr() if front_end > 1 else None, stream)
        assert lib.ternaspmm_last_status() == 0 and torch.equal(*outs)


def flip(t):
    t = t.view(torch.int32)
    t.copy_(~t)


def by_data(layer):
    flip(layer.weight_compressed_val.data)


def in_inference_mode(layer):
    with torch.inference_mode():
        flip(layer.weight_compressed_val)


def by_state_dict(layer):
    flip(layer.state_dict()["weight_compressed_val"].data)


def by_iteration(layer):
    for name, p in layer.named_parameters():
        if name == "weight_compressed_val":
            flip(p.data)


def on_the_way(layer):          # the memory on the GPU is given back and taken again, at the same address as it may be
    layer.cpu()
    flip(layer.weight_compressed_val.data)
    layer.cuda()


def by_swap(layer):
    layer.weight_compressed_val.data = ~layer.weight_compressed_val.data.view(torch.int32)
    layer.weight_compressed_val.data = layer.weight_compressed_val.data.view(torch.uint32)


@pytest.mark.parametrize("write", [by_data, in_inference_mode, by_state_dict, by_iteration, on_the_way, by_swap])
@pytest.mark.parametrize("inference", [False, True])
def test_layer_sees_weights_written_in_any_way(lib, write, inference):
    with torch.inference_mode(inference):
        layer, _ = make_layer(128, 192, 2, 1)
        x = torch.randn((5, 192), generator=torch.Generator().manual_seed(1)).to(torch.bfloat16).cuda()
        y = layer(x)
        write(layer)
        assert torch.equal(layer(x), -y)
        write(layer)
        assert torch.equal(layer(x), y)


def test_layer_sees_writes_through_tensors_that_somebody_keeps(lib):
    """As long as one is kept there is nothing to tell a write by: the packed tensors are read, in captures too."""
    layer, dic = make_layer(128, 192, 2, 1)
    x = torch.randn((5, 192), generator=torch.Generator().manual_seed(1)).to(torch.bfloat16).cuda()
    y = layer(x)
    assert layer._native.prepare(layer._parameters)
    for kept in (layer.weight_compressed_val, layer.weight_compressed_val.detach(), layer.state_dict()["weight_compressed_val"],
                 torch.from_dlpack(layer.weight_compressed_val.view(torch.int32)), layer.weight_compressed_val.untyped_storage()):
        assert not layer._native.prepare(layer._parameters)
        alias = torch.empty(0, dtype=torch.int32, device="cuda").set_(kept) if isinstance(kept, torch.UntypedStorage) else kept.data
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            z = layer(x)
        flip(alias)
        graph.replay()
        assert torch.equal(layer(x), -y) and torch.equal(z, -y)
        flip(alias)
        graph.replay()
        assert torch.equal(layer(x), y) and torch.equal(z, y)
        del graph, z
    del kept, alias
    assert torch.equal(layer(x), y) and layer._native.prepare(layer._parameters)
    twin = copy.copy(layer)                        # two modules, one set of parameters
    assert torch.equal(twin(x), y) and not twin._native.prepare(twin._parameters) and not layer._native.prepare(layer._parameters)
    flip(twin.weight_compressed_val.data)
    assert torch.equal(layer(x), -y)


def test_no_copy_of_tensors_that_cannot_be_laid_out(lib):
    """A bitmap that does not start on 16 bytes, offsets of another size: no copy, instead of one that nothing has written."""
    layer, _ = make_layer(128, 192, 2, 1)
    whole = {k: v.clone() for k, v in layer.state_dict().items()}
    bitmap, offsets, quarters = (whole["weight_" + n] for n in ("bitmap", "TileOffsets_global", "TileOffsets_median"))
    for name, bad in (("weight_bitmap", lambda: torch.empty(bitmap.numel() + 1, dtype=torch.int64, device="cuda").view(torch.uint64)[1:]),
                      ("weight_bitmap", lambda: bitmap[:-64].clone()), ("weight_TileOffsets_global", lambda: offsets[:-1].clone()),
                      ("weight_TileOffsets_median", lambda: quarters[:-1].clone())):
        setattr(layer, name, torch.nn.Parameter(bad(), requires_grad=False))
        assert not layer._native.prepare(layer._parameters)
        setattr(layer, name, torch.nn.Parameter(whole[name].clone(), requires_grad=False))
        assert layer._native.prepare(layer._parameters)


def test_graphs_follow_loaded_weights(lib):
    """A replay after load_state_dict and after relayout() computes with the new weights; a part of the tensors, as from
    one file of several, is not laid out."""
    layer, _ = make_layer(128, 192, 2, 1)
    x = torch.randn((5, 192), generator=torch.Generator().manual_seed(1)).to(torch.bfloat16).cuda()
    y = layer(x)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        z = layer(x)
    old = {k: v.clone() for k, v in layer.state_dict().items()}
    new = {k: v.clone() for k, v in old.items()}
    flip(new["weight_compressed_val"])
    layer.load_state_dict(new)
    graph.replay()
    assert torch.equal(z, -y)
    kept = layer.weight_compressed_val             # as an optimiser would
    layer.load_state_dict(old)
    graph.replay()
    assert torch.equal(z, y)
    flip(kept.data)
    layer.relayout()
    graph.replay()
    assert torch.equal(z, -y) and torch.equal(layer(x), -y)
    del kept
    layer.load_state_dict({"weight_compressed_val": old["weight_compressed_val"]}, strict=False)
    graph.replay()
    assert torch.equal(z, -y) and torch.equal(layer(x), y)
    layer.weight_bitmap = torch.nn.Parameter(old["weight_bitmap"].clone(), requires_grad=False)   # (the graph's copy stays where it is)
    assert torch.equal(layer(x), y)
    graph.replay()
    assert torch.equal(z, y)
    with pytest.raises(RuntimeError, match="captured"):
        with torch.cuda.graph(torch.cuda.CUDAGraph()):
            layer.relayout()


@torch.inference_mode()
def test_generation_follows_its_weights(lib):
    """FastGen replays graphs: weights changed in place, and a parameter that somebody keeps, between two prompts."""
    from ternainfer_b200.generate import FastGen, GenArgs
    from ternainfer_b200.model import ModelArgs, Transformer
    from ternainfer_b200.convert.convert_TernaInfer import random_checkpoint
    args = ModelArgs(n_layers=1, vocab_size=1024, fused_glue=True)
    dic = random_checkpoint(args.dim, 1, args.n_heads, args.n_kv_heads, args.ffn_dim, 1024, seed=7)

    def model(d):
        with torch.device("cuda"):
            return Transformer(args, d, max_seq_len=96).to(torch.bfloat16)
    a = model(dic)
    prompt = torch.randint(0, 1024, (2, 64), generator=torch.Generator(device="cuda").manual_seed(3), device="cuda")
    gen = FastGen(a, GenArgs(16, 2, 64, True))
    first, _ = gen.generate(prompt)
    wo = a.layers[0].attention.wo
    flip(wo.weight_compressed_val.data)
    b = model(dic)
    flip(b.layers[0].attention.wo.weight_compressed_val.data)
    want, _ = FastGen(b, GenArgs(16, 2, 64, False)).generate(prompt)
    assert torch.equal(gen.generate(prompt)[0], want) and not torch.equal(first, want)
    kept = wo.weight_compressed_val
    flip(kept.data)
    assert torch.equal(gen.generate(prompt)[0], first)
    flip(kept.data)
    assert torch.equal(gen.generate(prompt)[0], want)


@pytest.mark.parametrize("K", [64, 1040, 2560, 8192])
def test_norms_of_many_rows_are_the_norms_of_each(lib, K):
    """From two rows per SM on, a kernel that keeps a row in registers takes over: the same bits as a few rows at a time."""
    from ternainfer_b200.linear import rmsnorm
    M = 2 * torch.cuda.get_device_properties(0).multi_processor_count + 3
    g = torch.Generator(device="cuda").manual_seed(K)
    x = (torch.randn((M, K), generator=g, device="cuda") * torch.logspace(-3, 3, M, device="cuda")[:, None]).to(torch.bfloat16)
    x[7, K // 2], x[9] = float("nan"), 0.0
    w = (1 + 0.1 * torch.randn(K, generator=g, device="cuda")).to(torch.bfloat16)

    def bits(ts):
        return [t.view(torch.int16) if t.dtype == torch.bfloat16 else t for t in ts]

    for f in (lambda v: rmsnorm_quant(v, w, 1e-5), quant_input, lambda v: (rmsnorm(v, w, 1e-5),)):
        parts = [bits(f(x[i:i + 50])) for i in range(0, M, 50)]
        for k, got in enumerate(bits(f(x))):
            want = torch.cat([p[k] for p in parts])
            keep = torch.ones(M, dtype=torch.bool, device="cuda")
            keep[7] = False                                   # (a NaN's payload and its int8 values are not part of the contract)
            assert torch.equal(got[keep], want[keep])
    assert torch.isnan(rmsnorm_quant(x, w, 1e-5)[1].reshape(-1)[7]) and torch.isnan(quant_input(x)[1].reshape(-1)[7])
