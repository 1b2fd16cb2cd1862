"""The fp32 convolution past 65535 blocks in a grid dimension.  Rows and weights
of small whole numbers: every sum is exact."""
import numpy as np
import pytest
import torch

from cumm import tensorview as tv
from cumm.conv.main import ConvMainUnitTest
from cumm.tensorview.gemm import ConvOpType, ConvParams

from helpers import find_desp

pytestmark = pytest.mark.gpu


def _run(op, desp, x, w, y, indices, mask, order, mask_width=-1):
    p = ConvParams(3, op)
    p.conv_algo_desp = desp
    p.input, p.weight, p.output = tv.Tensor(x), tv.Tensor(w), tv.Tensor(y)
    p.indices, p.mask_argsort = tv.Tensor(indices), tv.Tensor(order)
    p.mask = tv.Tensor(mask, tv.uint32)
    p.mask_width = mask_width
    ConvMainUnitTest(sync_check=True).implicit_gemm2(p)


def test_wgrad_many_rows():
    """67,107,905 rows: 65,536 blocks of 1024 rows, the last with 65."""
    n = 65535 * 1024 + 65
    rng = np.random.default_rng(0)
    at = torch.from_numpy(np.concatenate([rng.choice(n, 1000, replace=False), np.arange(n - 65, n)])).cuda().unique()
    x = torch.zeros((n, 1), device="cuda")
    x[at, 0] = (at % 7).float() + 1
    dy = torch.ones((n, 1), device="cuda")
    dy[::2] = 2
    order = torch.arange(n, dtype=torch.int32, device="cuda")
    words = torch.ones((n + 127) // 128, dtype=torch.int32, device="cuda")
    dw = torch.zeros((1, 1, 1), device="cuda")
    desp = find_desp(ConvOpType.kBackwardWeight, "Simt", tv.float32, tv.float32, tv.float32, 32)
    _run(ConvOpType.kBackwardWeight, desp, x, dw, dy, order[None], words, order, mask_width=128)
    assert dw.item() == (x.double() * dy.double()).sum().item()


def test_many_columns():
    """2,097,121 columns: 65,536 column blocks of 32, the last with one."""
    n = 65535 * 32 + 1
    one = torch.zeros((1,), dtype=torch.int32, device="cuda")
    mask = torch.ones((1,), dtype=torch.int32, device="cuda")
    w = (torch.arange(n, device="cuda") % 1000).float()
    x = torch.full((1, 1), 3.0, device="cuda")
    y = torch.zeros((1, n), device="cuda")
    f = find_desp(ConvOpType.kForward, "Simt", tv.float32, tv.float32, tv.float32, 32)
    _run(ConvOpType.kForward, f, x, w.view(n, 1, 1), y, one[None], mask, one)
    assert torch.equal(y[0], 3 * w)
    y.zero_()
    d = find_desp(ConvOpType.kBackwardInput, "Simt", tv.float32, tv.float32, tv.float32, 32)
    _run(ConvOpType.kBackwardInput, d, y, w.view(1, 1, n), x, one[None], mask, one)
    assert torch.equal(y[0], 3 * w)
