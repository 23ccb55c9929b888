"""CPU: the Python side of the call site - what a module's copies and pickles carry, what its parameters may share."""
import subprocess
import sys

import pytest
import torch
from torch import nn

from conftest import ROOT
import ternaspmm_oracle as o
from ternainfer_b200.convert import compress_weight
from ternainfer_b200.lib import load_host_call
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
    m._native = load_host_call().Layer(192, 128, 2, 0, 0, 0)
    return m


def test_saved_module_loads_in_a_fresh_process(layer, tmp_path):
    path = tmp_path / "layer.pt"       # (torch.save: torch's plain pickles do not take unsigned dtypes)
    torch.save(nn.Sequential(layer), path)
    code = f"import sys, torch; sys.path.insert(0, {ROOT!r}); m = torch.load({str(path)!r}, weights_only=False)[0]; " \
           "print(m.out_features, m.segments, m.weight_bitmap.numel(), m._native.prepare(m._parameters))"
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    assert r.stdout.split() == ["128", "[64,", "64]", str(layer.weight_bitmap.numel()), "False"]
