"""GPU: the elementwise kernels of the glue at the edges of their vectors and chunks, and on the device of their tensors."""
import pytest
import torch

import ternaspmm_oracle as o
from ternainfer_b200 import linear
from ternainfer_b200.convert import compress_weight
from ternainfer_b200.linear import to_float
from ternainfer_b200.model import RMSNorm

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 3, 4, 7, 1023, 4096, 4099, 148 * 8 * 4096 + 5])
def test_bf16_to_fp32(lib, n):
    x = torch.randn(n, device="cuda").to(torch.bfloat16)
    y = to_float(x)
    assert y.dtype == torch.float32 and torch.equal(y, x.float())


def test_bf16_to_fp32_keeps_the_gradient(lib):
    """Logits of a prompt under autograd."""
    x = torch.randn(4096, device="cuda").to(torch.bfloat16).requires_grad_()
    to_float(x).sum().backward()
    assert torch.equal(x.grad, torch.ones_like(x))


def calls():
    def t(*shape):
        return torch.zeros(shape, dtype=torch.bfloat16, device="cuda")
    qkv, kv, pos = t(1, 1, 30 * 128), t(1, 8, 5, 128), torch.zeros(1, dtype=torch.int64, device="cuda")
    cv, tg, tm, bm = compress_weight(torch.from_numpy(o.make_ternary(64, 64, 0.45, 1)).cuda())
    return {"quant_input": lambda: linear.quant_input(t(1, 64)), "rmsnorm_quant": lambda: linear.rmsnorm_quant(t(1, 64), t(64), 1e-5),
            "rmsnorm": lambda: linear.rmsnorm(t(1, 64), t(64), 1e-5), "RMSNorm": lambda: RMSNorm(64).to("cuda", torch.bfloat16)(t(1, 64)),
            "rope": lambda: linear.rope(t(1, 1, 1, 128), t(1, 1, 64).float(), t(1, 1, 64).float()), "relu2_gate": lambda: linear.relu2_gate(t(1, 128)),
            "to_float": lambda: to_float(t(1, 64)), "attn_decode": lambda: linear.attn_decode(qkv, kv, kv, t(1, 64), t(1, 64), pos, 20, 5),
            "attn_decode_by_head": lambda: linear.attn_decode_by_head(qkv, kv.transpose(1, 2).contiguous(), kv.transpose(1, 2).contiguous(), t(64).float(), t(64).float(), pos, 20, 5),
            "attn_prefill": lambda: linear.attn_prefill(qkv, kv, kv, t(8, 64), t(8, 64), pos, 20, 5),
            "lm_head_argmax": lambda: linear.lm_head_argmax(t(1, 64), t(128, 64)),
            "TernaInfer_linear": lambda: linear.TernaInfer_linear(torch.zeros((1, 64), dtype=torch.int8, device="cuda"), cv, tg, tm, bm, None, t(1), t(4), 1, 64)}


@pytest.mark.parametrize("name", ["quant_input", "rmsnorm_quant", "rmsnorm", "RMSNorm", "rope", "relu2_gate", "to_float", "attn_decode", "attn_prefill",
                                  "lm_head_argmax", "TernaInfer_linear", "attn_decode_by_head"])
def test_launches_go_to_the_device_of_the_tensors(lib, monkeypatch, name):
    """With another device current (here by its number only), a call switches to its tensors' device, as torch operators do."""
    call, entered, real = calls()[name], [], torch.cuda.current_device()

    class Device:
        def __init__(self, device):
            self.device = device

        def __enter__(self):
            entered.append(torch.device(self.device))
            monkeypatch.setattr(torch.cuda, "current_device", lambda: real)

        def __exit__(self, *exc):
            monkeypatch.setattr(torch.cuda, "current_device", lambda: real + 1)
    with torch.no_grad():
        call()
        assert not entered
        monkeypatch.setattr(torch.cuda, "device", Device)
        monkeypatch.setattr(torch.cuda, "current_device", lambda: real + 1)
        call()
    assert torch.device("cuda", real) in entered
