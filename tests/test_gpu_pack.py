"""GPU: the packer's kernels give the host packer's arrays, bytes for bytes."""
import numpy as np
import pytest
import torch

import ternaspmm_oracle as o
from ternainfer_b200.convert import compress_weight

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,K,p_zero", [(64, 64, 0.45), (64, 64, 1.0), (128, 192, 0.0), (192, 4096, 0.9), (3840, 2560, 0.45), (64, 64 * 4097, 0.45),
                                        (8192, 2112, 0.3)])
def test_gpu_packer_equals_host_packer(lib, N, K, p_zero):
    w = torch.from_numpy(o.make_ternary(N, K, p_zero, N + K))
    w[0, :8] = torch.tensor([-128, 127, -1, 1, 0, -2, 2, 0], dtype=torch.int8)      # any sign counts, as on the host
    for got, want in zip(compress_weight(w.cuda()), compress_weight(w)):
        assert got.dtype == want.dtype and got.shape == want.shape
        assert np.array_equal(got.cpu().numpy(), want.numpy())


def test_gpu_packer_in_two_steps_without_scratch(lib):
    """The entry points that extract the signs at their places: the same arrays."""
    N, K = 192, 4160
    w = torch.from_numpy(o.make_ternary(N, K, 0.45, 5)).cuda()
    cv, tg, tm, bm = compress_weight(w)
    a, b, c = torch.empty_like(bm), torch.empty_like(tg), torch.empty_like(tm)
    stream = torch.cuda.current_stream().cuda_stream
    words = lib.ternaspmm_pack_gpu_layout(w.data_ptr(), N, K, a.data_ptr(), b.data_ptr(), c.data_ptr(), stream)
    assert words + 4 == cv.numel()
    d = torch.empty_like(cv)
    lib.ternaspmm_pack_gpu_signs(w.data_ptr(), N, K, b.data_ptr(), d.data_ptr(), stream)
    for x, y in ((a, bm), (b, tg), (c, tm), (d, cv)):
        assert torch.equal(x.view(torch.int8), y.view(torch.int8))


def test_gpu_packer_takes_views(lib):
    w = torch.from_numpy(o.make_ternary(129, 128, 0.45, 3)).cuda()
    a, b = compress_weight(w[1:]), compress_weight(w.t().contiguous().t()[1:])
    c = compress_weight(w.view(-1)[8:8 + 64 * 128].view(64, 128))               # not 16-byte aligned
    for x, y, z in zip(a, b, compress_weight(w[1:].cpu())):
        assert torch.equal(x.view(torch.int8), y.view(torch.int8)) and torch.equal(x.view(torch.int8).cpu(), z.view(torch.int8))
    for x, z in zip(c, compress_weight(w.view(-1)[8:8 + 64 * 128].view(64, 128).cpu())):
        assert torch.equal(x.view(torch.int8).cpu(), z.view(torch.int8))
