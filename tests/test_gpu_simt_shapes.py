"""The fp32 SIMT convolution at the edges of its tiles and copies: every mask
tile, ragged rows and channels (4-byte copies), unaligned base pointers,
several column tiles and row ranges; against the FP64 oracle.

Tolerance: a sum of up to 27 * 70 fp32 products and additions is off by about
sqrt(27 * 70) * 2^-24 = 2.6e-6 of the terms' norm; 1e-5 as the other fp32 tests."""
import numpy as np
import pytest
import torch

from cumm import tensorview as tv
from cumm import voxelgen as vg
from cumm.tensorview.gemm import ConvOpType
from oracle import conv_oracle as co
from oracle import pairs_oracle as po

from helpers import conv, dev, find_desp, to64, u32

pytestmark = pytest.mark.gpu
TOL = 1e-5


def _unaligned(a):
    buf = torch.empty(a.size + 1, device="cuda")
    t = buf[1:].view(a.shape)
    t.copy_(torch.from_numpy(a))
    return t


def _close(got, ref):
    assert np.isfinite(got).all()
    assert np.linalg.norm(got - ref) <= TOL * np.linalg.norm(ref)


@pytest.mark.parametrize("n,C,K,tile_m,aligned", [
    (1, 4, 4, 32, True), (63, 32, 32, 64, True), (65, 33, 31, 128, True), (2000, 32, 64, 128, False),
    (2049, 64, 36, 64, True), (3000, 5, 70, 32, True), (19001, 36, 64, 128, True), (19001, 64, 100, 32, True),
])
def test_simt_shapes(n, C, K, tile_m, aligned):
    grid = max(4, int(round((n * 4) ** (1 / 3))))
    coords = vg.uniform_voxels(n, grid, n)
    pf, pb, m = po.subm_pairs(coords, (grid,) * 3)
    ms, order = po.sort_by_key_split(m, 0xffffffff)
    rng = np.random.default_rng(n)
    x = rng.standard_normal((n, C)).astype(np.float32)
    dy = rng.standard_normal((n, K)).astype(np.float32)
    w = vg.kaiming_uniform(K, 27, C, n)
    put = dev if aligned else _unaligned

    f = find_desp(ConvOpType.kForward, "Simt", tv.float32, tv.float32, tv.float32, tile_m)
    out = torch.zeros((n, K), device="cuda")
    mo = u32(np.zeros((n + tile_m - 1) // tile_m))
    conv(ConvOpType.kForward, f, put(x), put(w), out, pf, ms, order, mask_output=mo)
    ref, ref_mo = co.conv_fwd_masked(x, w, pf, ms, order, tile_m)
    _close(to64(out), ref)
    assert np.array_equal(mo.torch().cpu().numpy().view(np.uint32), np.asarray(ref_mo, np.uint32))

    d = find_desp(ConvOpType.kBackwardInput, "Simt", tv.float32, tv.float32, tv.float32, tile_m)
    din = torch.zeros((n, C), device="cuda")
    conv(ConvOpType.kBackwardInput, d, din, put(w), put(dy), pb, ms, order, reverse_mask=True)
    _close(to64(din), co.conv_dgrad_masked(dy, w, pb, ms, order, tile_m, reverse_mask=True))

    g = find_desp(ConvOpType.kBackwardWeight, "Simt", tv.float32, tv.float32, tv.float32, 32)
    words = co.tile_masks(ms, tile_m).astype(np.uint32)
    dw = torch.zeros((K, 27, C), device="cuda")
    conv(ConvOpType.kBackwardWeight, g, put(x), dw, put(dy), pf, words, order, mask_width=tile_m)
    _close(to64(dw), co.conv_wgrad_masked(dy, x, pf, words, tile_m, order, 27))
