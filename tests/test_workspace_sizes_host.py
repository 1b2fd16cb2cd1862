"""Workspace queries: a workspace that was sized for the largest call serves
every smaller one, and an empty call needs none of the caller."""
import ctypes

import pytest

from cumm import _lib


def _sort_bytes(n):
    b = ctypes.c_int64(-1)
    assert _lib.load().sc_sort_workspace_size(n, ctypes.byref(b)) == 0
    return b.value


def _pair_bytes(n, kv, subm):
    b = ctypes.c_int64(-1)
    assert _lib.load().sc_pairs_workspace_size(n, kv, subm, ctypes.byref(b)) == 0
    return b.value


# around every size at which the sort's tiles or the tables' capacities change
SIZES = sorted({max(0, b + d) for b in [0, 1 << 10, 1 << 17, 1 << 18, 1 << 19, 1 << 20, 150000, 175000, 1398090, 2600000]
                for d in (-1, 0, 1, 1024)})


def test_sort_workspace_grows_with_n():
    got = [_sort_bytes(n) for n in SIZES]
    assert got == sorted(got)


@pytest.mark.parametrize("kv", [1, 27, 32])
@pytest.mark.parametrize("subm", [0, 1])
def test_pair_workspace_grows_with_n(kv, subm):
    got = [_pair_bytes(n, kv, subm) for n in SIZES]
    assert got == sorted(got)


def test_empty_sort_takes_no_workspace():
    assert _sort_bytes(0) == 0
    assert _lib.load().sc_sort_masks_split(None, 0, 0xffffffff, None, None, 0, None) == 0
