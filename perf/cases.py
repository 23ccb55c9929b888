"""The work that a user of this framework has it do, as cases that can be timed.

Sizes are the two architectures that the tests and bench.py run: the 2560-wide decoder (fused QKV 3840 x 2560,
O 2560 x 2560, gate-up 13824 x 2560, down 2560 x 6912, vocabulary 128256, 30 layers) and the 8192-wide one with its
tensor-parallel shards, plus generic multiples of 64.  Weights are ternary with about 45 % zeros, as such
checkpoints have them; activations are normally distributed bf16.

Kinds of case:
  linear   one SpBitLinear layer called eagerly: "module" hands it bf16 activations (quantise + linear), "quantized"
           hands it int8 activations with their scales and the residual stream (what a decoder block does)
  sweep    many linears through the C entry points with raw pointers, replayed from a CUDA graph, one call each, or
           all of them as one work list
  decode   one token per sequence through Transformer.forward, replayed from a CUDA graph as the generation loop does
  prefill  a prompt through Transformer.forward, logits of every position (scoring a text), from a CUDA graph
  head     output head and greedy token for a few rows
  pack     conversion: int8 ternary weights to the packed format, on the GPU
"""
import ctypes

import torch

from ternainfer_b200 import load_library
from ternainfer_b200.convert import compress_weight
from ternainfer_b200.convert.convert_TernaInfer import random_checkpoint
from ternainfer_b200.lib import ListItem
from ternainfer_b200.linear import SpBitLinear, lm_head_argmax, quant_input
from ternainfer_b200.model import ModelArgs, Transformer

DEV = "cuda"
VOCAB = 128256
# rows, columns, weight scales of the four linears of a layer
SMALL_MODEL = [(3840, 2560, 3), (2560, 2560, 1), (13824, 2560, 2), (2560, 6912, 1)]
# the 8192-wide model's linears and their shards for 2, 4 and 8 GPUs
WIDE_MODEL = [(n // (t if col else 1), k // (1 if col else t), ws)
              for t in (1, 2, 4, 8) for n, k, ws, col in ((10240, 8192, 3, True), (8192, 8192, 1, False),
                                                          (57344, 8192, 2, True), (8192, 28672, 1, False))]
DIM, HEADS, KV_HEADS, HEAD_DIM, FFN = 2560, 20, 5, 128, 6912
# Scales of the two projections into the residual stream, relative to random_checkpoint's.  A trained network's sub-layers
# change the residual stream by a little; with random_checkpoint's own scales every sub-layer overwrites it, and such a
# network amplifies one differently rounded bf16 value to a tenth of its logits, so that no two implementations agree.
# The factor brings one sub-layer to about one per cent of the stream.  It does not change the work.
RESIDUAL_SCALE = 2.5e-4


def listed():
    return [
        # the smallest call: one token through one layer, called from an eager program
        dict(name="linear_o_1", kind="linear", entry="module", tokens=1, out=2560, inp=2560, scales=1, zeros=0.45),
        # a few sequences' worth of tokens (speculative or batched decoding) through the widest layer
        dict(name="linear_gateup_48", kind="linear", entry="quantized", tokens=48, out=13824, inp=2560, scales=2, zeros=0.45),
        # a short prompt, ragged
        dict(name="linear_qkv_333", kind="linear", entry="module", tokens=333, out=3840, inp=2560, scales=3, zeros=0.45),
        # a long prompt or a batch of prompts
        dict(name="linear_down_2048", kind="linear", entry="quantized", tokens=2048, out=2560, inp=6912, scales=1, zeros=0.45),
        # decoding with a big model: the layer that streams the most weights
        dict(name="linear_wide_4", kind="linear", entry="module", tokens=4, out=57344, inp=8192, scales=2, zeros=0.45),
        # every linear of the 30-layer model at 8 tokens through the C entry point: more weight bytes than L2 holds
        dict(name="sweep_calls_8", kind="sweep", tokens=8, layers=30, as_list=False),
        # interactive decoding, one sequence
        dict(name="decode_1", kind="decode", batch=1, past=600, layers=30, fused=True),
        # batched decoding
        dict(name="decode_8", kind="decode", batch=8, past=1100, layers=30, fused=True),
        # the same loop with the default glue between the linears (plain torch operators)
        dict(name="decode_plain_3", kind="decode", batch=3, past=333, layers=10, fused=False),
        # two prompts of odd length
        dict(name="prefill_2x613", kind="prefill", batch=2, tokens=613, layers=30),
        # output head of a decode step: three sequences
        dict(name="head_3", kind="head", rows=3, vocab=VOCAB, inp=2560),
        # converting a checkpoint: one layer
        dict(name="pack_qkv", kind="pack", out=3840, inp=2560, zeros=0.45),
    ]


def _log(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["linear"] * 5 + ["sweep", "decode", "decode", "prefill", "head", "pack"])
    if kind == "linear":
        if rng.random() < 0.75:
            out, inp, scales = rng.choice(SMALL_MODEL * 2 + WIDE_MODEL)
        else:
            out, inp, scales = 64 * _log(rng, 4, 256), 64 * _log(rng, 4, 256), rng.choice([1, 2])
        most = max(1, min(4096, int(7e11 / (2 * out * inp))))     # below the prompt case's work
        return dict(kind=kind, entry=rng.choice(["module", "quantized"]), tokens=_log(rng, 1, most), out=out, inp=inp,
                    scales=scales, zeros=round(rng.uniform(0.35, 0.55), 2))
    if kind == "sweep":
        return dict(kind=kind, tokens=_log(rng, 1, 16), layers=_log(rng, 2, 30), as_list=rng.random() < 0.5)
    if kind == "decode":
        fused = rng.random() < 0.75
        return dict(kind=kind, batch=_log(rng, 1, 16), past=_log(rng, 20, 2000), layers=_log(rng, 2, 30 if fused else 10), fused=fused)
    if kind == "prefill":
        batch = rng.choice([1, 1, 2, 4])
        return dict(kind=kind, batch=batch, tokens=_log(rng, 16, 1226 // batch), layers=_log(rng, 2, 30))
    if kind == "head":
        return dict(kind=kind, rows=rng.randint(1, 8), vocab=_log(rng, 8000, VOCAB), inp=rng.choice([2560, 2560, 4096]))
    return dict(kind=kind, out=64 * _log(rng, 8, 216), inp=64 * _log(rng, 8, 108), zeros=round(rng.uniform(0.35, 0.55), 2))


def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(seed)


def _ternary(out, inp, zeros, g):
    sign = torch.randint(0, 2, (out, inp), generator=g, device=DEV, dtype=torch.int8) * 2 - 1
    return sign.masked_fill_(torch.rand((out, inp), generator=g, device=DEV, dtype=torch.bfloat16 if out * inp > 1 << 28 else None) < zeros, 0)


def _packed_linear(out, inp, scales, zeros, g):
    """Checkpoint tensors of one layer under the key "l"."""
    cv, tg, tm, bm = compress_weight(_ternary(out, inp, zeros, g))
    ws = torch.zeros(4, device=DEV)
    ws[:scales] = torch.rand(scales, generator=g, device=DEV) * 0.04 + 0.01
    return {"l.weight_compressed_val": cv, "l.weight_TileOffsets_global": tg, "l.weight_TileOffsets_median": tm,
            "l.weight_bitmap": bm, "l.weight_scale": ws.to(torch.bfloat16)}


def _prepare_linear(c, g):
    layer = SpBitLinear(c["inp"], c["out"], _packed_linear(c["out"], c["inp"], c["scales"], c["zeros"], g), "l")
    x = torch.randn((c["tokens"], c["inp"]), generator=g, device=DEV).to(torch.bfloat16)
    if c["entry"] == "module":
        return lambda: layer(x)
    xq, s = quant_input(x)
    residual = torch.randn((c["tokens"], c["out"]), generator=g, device=DEV).to(torch.bfloat16)
    return lambda: layer.forward_quantized(xq, s, residual=residual)


def _capture(fn):
    """fn's result and a CUDA graph that computes it again, as the generation loop captures its steps."""
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        fn()
    torch.cuda.current_stream().wait_stream(side)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = fn()
    return graph, out


def _prepare_sweep(c, g):
    lib, M = load_library(), c["tokens"]
    xs = {K: quant_input(torch.randn((M, K), generator=g, device=DEV).to(torch.bfloat16)) for K in (2560, 6912)}
    shapes = [s for _ in range(c["layers"]) for s in SMALL_MODEL]
    weights = [_packed_linear(N, K, ws, 0.45, g) for N, K, ws in shapes]
    out = torch.empty(M * sum(N for N, _, _ in shapes), dtype=torch.bfloat16, device=DEV)
    items, at = (ListItem * len(shapes))(), 0
    for it, (N, K, ws), w in zip(items, shapes, weights):
        it.x, it.s = xs[K][0].data_ptr(), xs[K][1].data_ptr()
        it.bitmap, it.tile_offsets = w["l.weight_bitmap"].data_ptr(), w["l.weight_TileOffsets_global"].data_ptr()
        it.quarter_offsets, it.sign_words = w["l.weight_TileOffsets_median"].data_ptr(), w["l.weight_compressed_val"].data_ptr()
        it.out, it.ws, it.residual = out.data_ptr() + 2 * at, w["l.weight_scale"].data_ptr(), None
        it.ws_num, it.M, it.N, it.K, it.prefill_form = ws, M, N, K, -1
        at += M * N
    if c["as_list"]:
        tb, sb = ctypes.c_longlong(), ctypes.c_longlong()
        lib.ternaspmm_list_plan(items, len(items), ctypes.byref(tb), ctypes.byref(sb))
        table = torch.empty(tb.value, dtype=torch.uint8, device=DEV)
        scratch = torch.empty(sb.value, dtype=torch.uint8, device=DEV)
        handle = lib.ternaspmm_list_create(items, len(items), table.data_ptr(), scratch.data_ptr(),
                                           torch.cuda.current_stream().cuda_stream)
        keep = (xs, weights, table, scratch)

        def launch():
            lib.ternaspmm_list_run(handle, torch.cuda.current_stream().cuda_stream)
    else:
        keep = (xs, weights)

        def launch():
            stream = torch.cuda.current_stream().cuda_stream
            for it in items:
                lib.bitlinear_TernaSpMM(it.x, it.bitmap, it.tile_offsets, it.quarter_offsets, it.sign_words, it.out, it.s, it.ws,
                                        it.ws_num, it.M, it.N, it.K, 1, None, stream)
    graph, _ = _capture(launch)

    def step(keep=keep):
        graph.replay()
        return out
    return step


def _model(c, g, max_len):
    args = ModelArgs(n_layers=c["layers"], fused_glue=c.get("fused", True))
    dic = random_checkpoint(args.dim, args.n_layers, args.n_heads, args.n_kv_heads, args.ffn_dim, args.vocab_size,
                            seed=g.initial_seed())
    for key in dic:
        if key.endswith(("wo.weight_scale", "w2.weight_scale")):
            dic[key] = dic[key] * RESIDUAL_SCALE
    with torch.device(DEV):
        model = Transformer(args, dic, max_seq_len=max_len)
    model = model.to(device=DEV, dtype=torch.bfloat16)
    return model


def _cache(model, batch, past, g):
    """Key / value caches in one allocation, with `past` earlier tokens in them."""
    layout = model.make_cache(batch, DEV)
    kv = torch.zeros((len(layout), 2) + tuple(layout[0][0].shape), dtype=torch.bfloat16, device=DEV)
    length_dim = 3 if model.flash else 4
    if past:
        kv.narrow(length_dim, 0, past).normal_(generator=g)
    return kv, [(kv[i, 0], kv[i, 1]) for i in range(len(layout))]


@torch.inference_mode()
def _prepare_forward(c, g):
    past = c.get("past", 0)
    T = 1 if c["kind"] == "decode" else c["tokens"]
    model = _model(c, g, past + 128 if c["kind"] == "decode" else T)
    kv, cache = _cache(model, c["batch"], past, g)
    tokens = torch.randint(0, VOCAB, (c["batch"], T), generator=g, device=DEV)
    pos = torch.arange(past, past + T, device=DEV)
    graph, logits = _capture(lambda: model(tokens, cache, pos))

    def step(keep=(model, cache, tokens, pos)):
        graph.replay()
        return {"logits": logits, "cache": kv}
    return step


def _prepare_head(c, g):
    emb = (0.02 * torch.randn((c["vocab"], c["inp"]), generator=g, device=DEV)).to(torch.bfloat16)
    h = torch.randn((c["rows"], c["inp"]), generator=g, device=DEV).to(torch.bfloat16)
    return lambda: lm_head_argmax(h, emb)


def _prepare_pack(c, g):
    w = _ternary(c["out"], c["inp"], c["zeros"], g)
    signs = torch.zeros(c["out"] * c["inp"] // 32 + 4, dtype=torch.int32, device=DEV)   # their number depends on the zeros

    def pack():
        cv, tg, tm, bm = compress_weight(w)
        signs[:cv.numel()].copy_(cv.view(torch.int32))
        return [signs, tg, tm.view(torch.int16), bm.view(torch.int64)]
    return pack


def prepare(case, seed):
    g = _gen(seed)
    return {"linear": _prepare_linear, "sweep": _prepare_sweep, "decode": _prepare_forward, "prefill": _prepare_forward,
            "head": _prepare_head, "pack": _prepare_pack}[case["kind"]](case, g)


def run(state):
    return state()


def _weight_bytes(out, inp, zeros):
    """Packed size: bitmap, sign bits of the non-zeros (padded to 32 per 64 x 64 tile), offsets."""
    tiles = out * inp // 4096
    return out * inp / 8 + out * inp * (1 - zeros) / 8 + tiles * (2 + 10)


def _linear_work(tokens, out, inp, zeros, x_bytes, residual=False):
    b = _weight_bytes(out, inp, zeros) + tokens * inp * x_bytes + 2 * tokens * out * (2 if residual else 1)
    return b, 2.0 * tokens * out * inp


def work(case):
    c = case
    if c["kind"] == "linear":
        q = c["entry"] == "quantized"
        b, f = _linear_work(c["tokens"], c["out"], c["inp"], c["zeros"], 1 if q else 2, q)
    elif c["kind"] == "sweep":
        each = [_linear_work(c["tokens"], N, K, 0.45, 1) for N, K, _ in SMALL_MODEL]
        b, f = (c["layers"] * sum(e[i] for e in each) for i in (0, 1))
    elif c["kind"] in ("decode", "prefill"):
        T = 1 if c["kind"] == "decode" else c["tokens"]
        M, past = c["batch"] * T, c.get("past", 0)
        keys = sum(past + t + 1 for t in range(T)) * c["batch"]           # attended positions over all queries
        b = c["layers"] * (sum(_weight_bytes(N, K, 0.45) for N, K, _ in SMALL_MODEL)
                           + c["batch"] * (past + T) * 2 * KV_HEADS * HEAD_DIM * 2)
        f = c["layers"] * (sum(2.0 * M * N * K for N, K, _ in SMALL_MODEL) + 4.0 * keys * HEADS * HEAD_DIM)
        b += 2.0 * VOCAB * DIM + 4.0 * M * VOCAB
        f += 2.0 * M * VOCAB * DIM
    elif c["kind"] == "head":
        b = 2.0 * c["vocab"] * c["inp"] + c["rows"] * (2.0 * c["inp"] + 4.0 * c["vocab"] + 8)
        f = 2.0 * c["rows"] * c["vocab"] * c["inp"]
    else:
        b, f = c["out"] * c["inp"] + _weight_bytes(c["out"], c["inp"], c["zeros"]), 0.0
    return {"bytes": b, "flops": f}


def tolerance(case):
    if case["kind"] == "pack":
        return "exact"
    if case["kind"] in ("decode", "prefill"):
        # bf16 activations through up to 30 layers, each with four int8 quantisers: a rounding that falls the other
        # way moves an activation by a whole quantisation step (two attention kernels, exact linears: 1e-2, 0.1)
        return {"rel": 2e-2, "max": 0.2}
    # integer contraction, then one or two bf16 roundings (a unit in the last place is 2^-8 of the value)
    return {"rel": 4e-3, "max": 1e-2}
