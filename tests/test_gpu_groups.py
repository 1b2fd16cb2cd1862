"""The convolution kernels' producer groups, split rounding and the row
scatter's rows per thread, at the sizes where their rules turn: layouts of 1, 2
and 4 warps a group (several column blocks, packed rows, a dOut ring of two
buffers), one tile, a ragged last tile and more tiles than CTAs.

Tolerance: bf16 operands with fp32 sums and one bf16 rounding of the result (up
to 2^-8 a value, about 2^-8 / 2.3 in norm over many): 2e-3 as the other tests; fp32 dW: 1e-5 of the terms' norm."""
import numpy as np
import pytest
import torch

from cumm import tensorview as tv
from cumm import voxelgen as vg
from cumm.gemm.gather import ScatterAll
from cumm.tensorview.gemm import ConvOpType
from oracle import conv_oracle as co
from oracle import pairs_oracle as po

from helpers import conv, dev, find_desp, to64

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,C,K", [(1, 64, 64), (129, 16, 32), (4004, 32, 32), (4004, 128, 64), (2051, 64, 128),
                                   (3000, 128, 256), (2500, 256, 64), (19012, 64, 32)])
def test_producer_groups(n, C, K):
    grid = max(4, int(round((n * 4) ** (1 / 3))))
    coords = vg.uniform_voxels(n, grid, n)
    pf, pb, m = po.subm_pairs(coords, (grid,) * 3)
    ms, order = po.sort_by_key_split(m, 0xffffffff)
    rng = np.random.default_rng(n + C)
    bf = torch.bfloat16
    x = dev(rng.standard_normal((n, C)).astype(np.float32), bf)
    dy = dev(rng.standard_normal((n, K)).astype(np.float32), bf)
    w = dev(vg.kaiming_uniform(K, 27, C, n), bf)
    f = find_desp(ConvOpType.kForward, "Tcgen05", tv.bfloat16, tv.bfloat16, tv.bfloat16)
    d = find_desp(ConvOpType.kBackwardInput, "Tcgen05", tv.bfloat16, tv.bfloat16, tv.bfloat16)
    ref = co.conv_fwd_masked(to64(x), to64(w), pf, ms, order, 128)[0]
    refd = co.conv_dgrad_masked(to64(dy), to64(w), pb, ms, order, 128, reverse_mask=True)
    for srt in (False, True):
        out = torch.zeros((n, K), dtype=bf, device="cuda")
        conv(ConvOpType.kForward, f, x, w, out, pf, ms, order, sorted_indices=srt)
        assert co.rel_err(to64(out), ref)[0] < 2e-3
        din = torch.zeros((n, C), dtype=bf, device="cuda")
        conv(ConvOpType.kBackwardInput, d, din, w, dy, pb, ms, order, reverse_mask=True, sorted_indices=srt)
        assert co.rel_err(to64(din), refd)[0] < 2e-3
    g = find_desp(ConvOpType.kBackwardWeight, "Tcgen05", tv.bfloat16, tv.float32, tv.bfloat16)
    words = co.tile_masks(ms, 128).astype(np.uint32)
    dw = torch.zeros((K, 27, C), device="cuda")
    conv(ConvOpType.kBackwardWeight, g, x, dw, dy, pf, words, order, mask_width=128)
    refw = co.conv_wgrad_masked(to64(dy), to64(x), pf, words, 128, order, 27)
    assert np.linalg.norm(to64(dw) - refw) <= 1e-5 * np.linalg.norm(refw)


@pytest.mark.parametrize("c", [2, 8, 62, 64, 66, 128])
@pytest.mark.parametrize("n", [1, 7, 4097])
def test_scatter_rows_per_thread(n, c):
    """Distinct target rows and small whole numbers: exact."""
    rng = np.random.default_rng(n + c)
    x = dev(rng.integers(-8, 9, (n, c)).astype(np.float32), torch.bfloat16)
    inds = dev(rng.permutation(2 * n)[:n].astype(np.int32))
    out = torch.ones((2 * n, c), dtype=torch.bfloat16, device="cuda")
    ScatterAll().scatter(tv.Tensor(out), tv.Tensor(x), tv.Tensor(inds))
    ref = np.ones((2 * n, c))
    ref[inds.cpu().numpy()] += to64(x)
    assert np.array_equal(to64(out), ref)


@pytest.mark.parametrize("n", [28284, 28420])
@pytest.mark.parametrize("C,K", [(64, 256), (32, 256)])
def test_strands_per_cta(n, C, K):
    """884 and 892 (row, column) tiles of 64 columns: one strand per CTA below
    three tiles a CTA, two from there, with a last tile of four rows."""
    coords = vg.uniform_voxels(n, 48, n)
    pf, pb, m = po.subm_pairs(coords, (48,) * 3)
    ms, order = po.sort_by_key_split(m, 0xffffffff)
    rng = np.random.default_rng(n)
    bf = torch.bfloat16
    x = dev(rng.standard_normal((n, C)).astype(np.float32), bf)
    w = dev(vg.kaiming_uniform(K, 27, C, n), bf)
    f = find_desp(ConvOpType.kForward, "Tcgen05", tv.bfloat16, tv.bfloat16, tv.bfloat16)
    out = torch.zeros((n, K), dtype=bf, device="cuda")
    conv(ConvOpType.kForward, f, x, w, out, pf, ms, order, sorted_indices=True, tile_n=64)
    assert co.rel_err(to64(out), co.conv_fwd_masked(to64(x), to64(w), pf, ms, order, 128)[0])[0] < 2e-3
    # the transposed layer's input gradient: rows of C values of dOut, K columns
    wt = w.permute(2, 1, 0).contiguous()
    d = find_desp(ConvOpType.kBackwardInput, "Tcgen05", tv.bfloat16, tv.bfloat16, tv.bfloat16)
    din = torch.zeros((n, K), dtype=bf, device="cuda")
    conv(ConvOpType.kBackwardInput, d, din, wt, x, pb, ms, order, reverse_mask=True, sorted_indices=True, tile_n=64)
    ref = co.conv_dgrad_masked(to64(x), to64(wt), pb, ms, order, 128, reverse_mask=True)
    assert co.rel_err(to64(din), ref)[0] < 2e-3
