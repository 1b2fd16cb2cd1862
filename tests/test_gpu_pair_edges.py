"""Submanifold pairs where the lookups' short cuts end: rows beside a voxel
outside the grid, whose linear key is that of another row's group, and buckets
of the group table that overflow."""
import numpy as np
import pytest
import torch

from cumm import _lib
from cumm.spconv_ops import build_pair_table
from oracle import pairs_oracle as po

pytestmark = pytest.mark.gpu


def _neighbours(c, spatial):
    """pairs_fwd by the definition: the voxel of the grid at coord + offset - 1."""
    at = {tuple(v): i for i, v in reversed(list(enumerate(c.tolist()))) if all(0 <= v[d + 1] < spatial[d] for d in range(3))}
    out = np.full((27, len(c)), -1, np.int32)
    for i, (b, z, y, x) in enumerate(c.tolist()):
        for k in range(27):
            out[k, i] = at.get((b, z + k // 9 - 1, y + k // 3 % 3 - 1, x + k % 3 - 1), -1)
    return out


@pytest.mark.parametrize("outside", [(0, 1, 1, 8), (0, 1, 1, 9), (0, 0, 6, 0), (0, 0, 5, 8), (0, 2, -2, 0), (0, 1, 3, -3),
                                     (-1, 7, 2, 3)])
@pytest.mark.parametrize("first", [True, False])
def test_rows_beside_a_voxel_outside_the_grid(outside, first):
    """Every voxel of a 4 x 4 x 8 grid once, in scan order, with a voxel outside
    the grid before or after each row: the voxels of the grid keep their
    neighbours, and the call leaves its error bit."""
    spatial = (4, 4, 8)
    c = np.stack(np.meshgrid([0], range(4), range(4), range(8), indexing="ij"), -1).reshape(-1, 4).astype(np.int32)
    for at in range(0, len(c) + 1):
        rows = np.insert(c, at, outside, axis=0)
        if not first:
            rows = rows[::-1].copy()
        pt = build_pair_table(torch.from_numpy(rows).cuda(), spatial)
        assert _lib.device_error_bits() == 1
        inside = np.delete(np.arange(len(rows)), at if first else len(c) - at)
        assert np.array_equal(pt.pairs_fwd.cpu().numpy()[:, inside], _neighbours(rows, spatial)[:, inside]), at


def _bucket(key, log2cap):
    """The hash of pairs.cu's group table: the bucket of eight slots of a key."""
    m = np.uint64(0xffffffff)
    h = (key & m) + (((key >> np.uint64(32)) * np.uint64(0x85ebca6b)) & m) & m
    h = h * np.uint64(0x9e3779b1) & m
    h ^= h >> np.uint64(15)
    h = h * np.uint64(0x2c1b3c6d) & m
    return (h >> np.uint64(32 - log2cap)) >> np.uint64(3)


@pytest.mark.parametrize("ksize", [(3, 3, 3), (5, 1, 3)])
def test_full_buckets(ksize):
    """As many groups as the table takes of one size (5456 of 8192 slots): about
    one bucket in ten has more than eight and overflows into the next."""
    n, spatial = 5456, (20, 30, 40)
    rng = np.random.default_rng(1)
    group = rng.choice(20 * 30 * 10, n, replace=False)
    c = np.stack([np.zeros(n, np.int64), group // 300, group // 10 % 30, group % 10 * 4 + rng.integers(0, 4, n)], 1).astype(np.int32)
    assert np.bincount(_bucket(group.astype(np.uint64), 13).astype(np.int64), minlength=1024).max() > 8
    pt = build_pair_table(torch.from_numpy(c).cuda(), spatial, ksize=ksize)
    pf, pb, _ = po.subm_pairs(c, spatial, ksize)
    assert np.array_equal(pt.pairs_fwd.cpu().numpy(), pf)
    assert np.array_equal(pt.pairs_bwd.cpu().numpy(), pb)


@pytest.mark.parametrize("ksize", [(3, 3, 3), (1, 1, 5)])
@pytest.mark.parametrize("width", [2 ** 31 - 1, 2 ** 31 - 3])
def test_widest_rows(width, ksize):
    """Rows as wide as int32 coordinates allow, voxels at both ends."""
    x = np.concatenate([np.arange(6), width - 1 - np.arange(6)])
    c = np.stack([np.zeros(24, np.int64), np.zeros(24, np.int64), np.repeat([0, 1], 12), np.tile(x, 2)], 1).astype(np.int32)
    pt = build_pair_table(torch.from_numpy(c).cuda(), (1, 2, width), ksize=ksize)
    pf, pb, _ = po.subm_pairs(c, (1, 2, width), ksize)
    assert np.array_equal(pt.pairs_fwd.cpu().numpy(), pf)
    assert np.array_equal(pt.pairs_bwd.cpu().numpy(), pb)
