"""Routes of the GPU pair builder and the mask sort, bit-exact against the CPU
oracle: group-hash lookups at group and grid edges, rows in any order, equal
coordinates, unaligned coordinates; strided builds through the output bitmap
and through the hash table (grids too large for the bitmap, batch indices
outside the given batch size); the sort at the edges of its tiles."""
import numpy as np
import pytest
import torch

from cumm import voxelgen as vg
from cumm.spconv_ops import SpconvOps, build_pair_table
from oracle import pairs_oracle as po

pytestmark = pytest.mark.gpu


def _coords(n, spatial, seed, batch=1, order="hash"):
    rng = np.random.default_rng(seed)
    cells = batch * int(np.prod(spatial))
    lin = np.sort(rng.choice(cells, n, replace=False))
    if order == "hash":
        rng.shuffle(lin)
    x, r = lin % spatial[2], lin // spatial[2]
    y, r = r % spatial[1], r // spatial[1]
    return np.stack([r // spatial[0], r % spatial[0], y, x], 1).astype(np.int32)


def _cuda(c, aligned=True):
    if aligned:
        return torch.from_numpy(c).cuda()
    buf = torch.empty(c.size + 1, dtype=torch.int32, device="cuda")
    t = buf[1:].view(c.shape)
    t.copy_(torch.from_numpy(c))
    return t


def _u(t):
    return t.cpu().numpy().view(np.uint32)


@pytest.mark.parametrize("n,spatial,ksize,dil,batch,aligned", [
    (1, (3, 3, 3), (3, 3, 3), 1, 1, True),
    (90, (3, 6, 5), (3, 3, 3), 1, 1, False),
    (200, (4, 8, 8), (3, 3, 3), 1, 1, True),      # all but full, W a whole number of groups
    (3000, (9, 31, 27), (3, 3, 3), 1, 2, True),
    (3000, (9, 31, 27), (3, 3, 3), 2, 2, True),
    (1000, (9, 11, 13), (5, 1, 3), 1, 2, False),
    (1000, (9, 11, 14), (1, 1, 9), 1, 1, True),
])
def test_subm_lookup_edges(n, spatial, ksize, dil, batch, aligned):
    c = _coords(n, spatial, 3, batch)
    pt = build_pair_table(_cuda(c, aligned), spatial, ksize=ksize, dilation=(dil,) * 3)
    pf, pb, m = po.subm_pairs(c, spatial, ksize, (dil,) * 3)
    assert np.array_equal(pt.pairs_fwd.cpu().numpy(), pf)
    assert np.array_equal(pt.pairs_bwd.cpu().numpy(), pb)
    ms, order = po.sort_by_key_split(m, 0xffffffff)
    assert np.array_equal(_u(pt.masks_fwd[0]), ms)
    assert np.array_equal(pt.argsorts_fwd[0].cpu().numpy(), order)
    assert np.array_equal(pt.sorted_indices("fwd").cpu().numpy(), pf[:, order])


def test_subm_equal_coordinates():
    """The smallest index of equal coordinates is everyone's neighbour; the
    others are nobody's."""
    c = _coords(500, (6, 9, 10), 5)
    c = np.concatenate([c, c[:40]], 0)
    pt = build_pair_table(_cuda(c), (6, 9, 10))
    pf, _, _ = po.subm_pairs(c, (6, 9, 10))
    got, bwd = pt.pairs_fwd.cpu().numpy(), pt.pairs_bwd.cpu().numpy()
    assert np.array_equal(got, pf)
    assert (bwd[:, 500:] == -1).all()
    for k in range(27):
        i = np.nonzero(bwd[k] >= 0)[0]
        assert np.array_equal(got[k, bwd[k, i]], i)
        assert np.array_equal(np.unique(i), np.unique(got[k][got[k] >= 0]))


def _check_strided(c, spatial, batch_arg, aligned=True, **kw):
    args = dict(ksize=(3, 3, 3), stride=(2, 2, 2), padding=(1, 1, 1), dilation=(1, 1, 1))
    args.update(kw)
    pt = build_pair_table(_cuda(c, aligned), spatial, subm=False, batch_size=batch_arg, **args)
    out, pf, pb, mf, mb, osp = po.conv_pairs(c, batch_arg, spatial, args["ksize"], args["stride"], args["padding"],
                                             args["dilation"])
    assert pt.out_spatial == osp
    assert np.array_equal(pt.out_inds.cpu().numpy(), out)
    assert np.array_equal(pt.pairs_fwd.cpu().numpy(), pf)
    assert np.array_equal(pt.pairs_bwd.cpu().numpy(), pb)
    for got, srt, m in ((pt.masks_fwd[0], pt.argsorts_fwd[0], mf), (pt.masks_bwd[0], pt.argsorts_bwd[0], mb)):
        ms, order = po.sort_by_key_split(m, 0xffffffff)
        assert np.array_equal(_u(got), ms)
        assert np.array_equal(srt.cpu().numpy(), order)


@pytest.mark.parametrize("n,spatial,batch,aligned,kw", [
    (1, (3, 3, 3), 1, True, {}),
    (400, (7, 8, 9), 1, False, {}),
    (4000, (9, 31, 40), 3, True, {}),
    (4000, (9, 31, 40), 3, True, dict(ksize=(2, 2, 2), padding=(0, 0, 0))),
    (2000, (9, 31, 40), 2, True, dict(ksize=(3, 1, 3), stride=(1, 2, 3), padding=(2, 0, 1))),
    (2000, (12, 31, 40), 1, True, dict(dilation=(2, 1, 3), padding=(0, 1, 2))),
])
def test_strided_bitmap(n, spatial, batch, aligned, kw):
    _check_strided(_coords(n, spatial, 7, batch), spatial, batch, aligned, **kw)


def test_strided_grid_beyond_the_bitmap():
    """1.6e9 output cells against 3000 voxels: the hash route."""
    spatial = (400, 8000, 4000)
    rng = np.random.default_rng(9)
    c = np.unique(np.concatenate([np.zeros((3000, 1)), rng.integers(0, spatial, (3000, 3)) // 40 * 3], 1).astype(np.int32),
                  axis=0)
    _check_strided(c, spatial, 1)


def test_strided_batch_index_outside_the_batch_size():
    """Accepted as before, through the hash route.  65 output cells a batch; the
    second batch's voxels stay below key 128, inside the sorted bits."""
    spatial = (1, 9, 25)
    c = _coords(120, spatial, 11, 2, order="scan")
    c = c[(c[:, 0] == 0) | (c[:, 2] < 6)]
    _check_strided(c, spatial, 1)


@pytest.mark.parametrize("n", [1, 31, 1023, 1024, 1025, 131072, 131073, 524288, 524289, 1048576, 1048577, 1300000])
def test_mask_sort_tile_edges(n):
    rng = np.random.default_rng(n)
    # few distinct words, as masks of real clouds: long runs of equal digits
    data = (rng.integers(0, 1 << 27, 5000)[rng.integers(0, 5000, n)] | (1 << 13)).astype(np.uint32)
    for sm in (0xffffffff, (1 << 27) - 1, 0b1111111111111 << 14, 1 << 31, 0):
        t = torch.from_numpy(data.view(np.int32)).cuda()
        order = SpconvOps.sort_1d_by_key_split(t, sm)
        s, o = po.sort_by_key_split(data, sm)
        assert np.array_equal(order.cpu().numpy(), o), hex(sm)
        assert np.array_equal(_u(t), s), hex(sm)


@pytest.mark.parametrize("n,order", [(777, "hash"), (20000, "scan")])
def test_sorted_tables_by_mask(n, order):
    """Tables sorted with the masks at hand equal the plain gather, all four of them."""
    c = _coords(n, (9, 60, 70), 13, order=order)
    for pt in (build_pair_table(_cuda(c), (9, 60, 70)),
               build_pair_table(_cuda(c), (9, 60, 70), num_split=2),
               build_pair_table(_cuda(c), (9, 60, 70), stride=(2, 2, 2), subm=False)):
        for j in range(len(pt.argsorts_fwd)):
            back = pt.argsorts_fwd[j] if pt.subm else pt.argsorts_bwd[j]
            assert torch.equal(pt.sorted_indices("fwd", j), pt.pairs_fwd[:, pt.argsorts_fwd[j].long()])
            assert torch.equal(pt.sorted_indices("bwd", j), pt.pairs_bwd[:, back.long()])
            assert torch.equal(SpconvOps.sort_indices(pt.pairs_bwd, back), pt.sorted_indices("bwd", j))
