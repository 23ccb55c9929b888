"""CPU: the Python side of the call site - what a module's copies and pickles carry, what its parameters may share."""
import copy
import gc
import io
import subprocess
import sys

import pytest
import torch
from torch import nn

from conftest import ROOT
import ternaspmm_oracle as o
from ternainfer_b200.convert import compress_weight
from ternainfer_b200.linear import SpBitLinear


@pytest.fixture
def layer(lib):
    """A 128 x 192 layer whose parameters are CPU tensors (its constructor puts them on the GPU)."""
    cv, tg, tm, bm = compress_weight(torch.from_numpy(o.make_ternary(128, 192, 0.45, 1)))
    m = SpBitLinear.__new__(SpBitLinear)
    nn.Module.__init__(m)
    m.__dict__.update(in_features=192, out_features=128, ws_num=2, segments=[64, 64])
    for name, t in (("weight_compressed_val", cv), ("weight_TileOffsets_global", tg), ("weight_TileOffsets_median", tm), ("weight_bitmap", bm),
                    ("weight_scale", torch.tensor([0.5, 2.0, 0, 0]).to(torch.bfloat16))):
        m.register_parameter(name, nn.Parameter(t, requires_grad=False))
    m._attach()
    return m


def test_saved_module_loads_in_a_fresh_process(layer, tmp_path):
    path = tmp_path / "layer.pt"       # (torch.save: torch's plain pickles do not take unsigned dtypes)
    torch.save(nn.Sequential(layer), path)
    code = f"import sys, torch; sys.path.insert(0, {ROOT!r}); m = torch.load({str(path)!r}, weights_only=False)[0]; " \
           "print(m.out_features, m.segments, m.weight_bitmap.numel(), m._native.prepare(m._parameters))"
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    assert r.stdout.split() == ["128", "[64,", "64]", str(layer.weight_bitmap.numel()), "0"]


HOLDS = {"attribute": lambda m: m.weight_bitmap, "detached": lambda m: m.weight_compressed_val.detach(), "state_dict": lambda m: m.state_dict(),
         "parameters": lambda m: list(m.parameters()), "iterator": lambda m: iter(m._parameters.items()), "dict": lambda m: dict(m._parameters),
         "view": lambda m: m.weight_bitmap.view(torch.uint8)[3:], "numpy": lambda m: m.weight_TileOffsets_global.numpy(),
         "storage": lambda m: m.weight_TileOffsets_median.untyped_storage(), "get": lambda m: m._parameters.get("weight_bitmap"),
         "unpacked": lambda m: {**m._parameters}, "shallow copy": lambda m: copy.copy(m)}


@pytest.mark.parametrize("how", HOLDS)
def test_a_parameter_in_other_hands_is_noticed(layer, how):
    """Handing one out invalidates the two-bit copy, and it stays so while the module is not alone with its parameters."""
    calls = []

    class Spy:
        def invalidate(self):
            calls.append(1)
    own = layer._native
    assert own.exclusive(layer._parameters)
    layer._parameters.layer = Spy()
    held = HOLDS[how](layer)
    layer._parameters.layer = own
    assert calls and not own.exclusive(layer._parameters)
    del held
    gc.collect()
    torch.save(layer.state_dict(), io.BytesIO())
    assert own.exclusive(layer._parameters)


def test_replaced_parameters_and_replaced_dicts_are_noticed(layer):
    calls = []

    class Spy:
        def invalidate(self):
            pass

        def replace(self):
            calls.append(1)
    own = layer._native
    layer._parameters.layer = Spy()
    layer.weight_bitmap = nn.Parameter(torch.zeros(4), requires_grad=False)
    assert len(calls) == 1
    layer._parameters.layer = own
    assert own.exclusive(layer._parameters)
    assert not own.exclusive(dict(layer._parameters)) and not own.exclusive(copy.deepcopy(layer)._parameters)
    assert copy.deepcopy(layer)._native.exclusive(layer._parameters) is False
