"""The scale-and-bias epilogue rounds once: act(scale * acc + alpha * bias) with
the sum of the exact product and the rounded alpha * bias.  Whole-number
operands make acc exact, and scale * acc + bias fits 53 bits, so the FP64 value
rounded to fp32 is the only right answer."""
import numpy as np
import pytest
import torch

from cumm import tensorview as tv
from cumm import voxelgen as vg
from cumm.tensorview.gemm import ConvOpType
from oracle import conv_oracle as co
from oracle import pairs_oracle as po

from helpers import conv, dev, find_desp, to64

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,C,K,srt", [(129, 16, 48, False), (600, 64, 64, True), (600, 64, 64, False), (1001, 32, 128, False)])
@pytest.mark.parametrize("with_bias", [True, False])
def test_scale_and_bias_round_once(n, C, K, srt, with_bias):
    grid = max(4, int(round((n * 4) ** (1 / 3))))
    coords = vg.uniform_voxels(n, grid, n)
    pf, _, m = po.subm_pairs(coords, (grid,) * 3)
    ms, order = po.sort_by_key_split(m, 0xffffffff)
    rng = np.random.default_rng(n + K)
    x = rng.integers(-8, 9, (n, C)).astype(np.float32)
    w = rng.integers(-8, 9, (K, 27, C)).astype(np.float32)
    scale = (rng.integers(1 << 15, 1 << 16, K) / 65536).astype(np.float32)
    bias = (100 * rng.standard_normal(K)).astype(np.float32) if with_bias else np.zeros(K, np.float32)
    bf = torch.bfloat16
    f = find_desp(ConvOpType.kForward, "Tcgen05", tv.bfloat16, tv.bfloat16, tv.float32)
    out = torch.zeros((n, K), device="cuda")
    conv(ConvOpType.kForward, f, dev(x, bf), dev(w, bf), out, pf, ms, order, scale=dev(scale),
         bias=dev(bias) if with_bias else None, sorted_indices=srt)
    acc = co.conv_fwd_masked(x.astype(np.float64), w.astype(np.float64), pf, ms, order, 128)[0]
    assert np.array_equal(acc, np.rint(acc))
    ref = (scale.astype(np.float64) * acc + bias.astype(np.float64)).astype(np.float32)
    assert np.array_equal(to64(out), ref.astype(np.float64))
