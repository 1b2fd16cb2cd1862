"""Host side of the pair builder's calls, with the native library replaced by a
recorder: which addresses a call hands over, and what it refuses before that."""
import dataclasses
import pickle

import numpy as np
import pytest
import torch

from cumm import _lib
from cumm import tensorview as tv
from cumm.spconv_ops import PairTable, SpconvOps, build_pair_table


class Recorder:
    """Every entry point returns SC_OK and leaves its arguments in `calls`."""

    def __init__(self):
        self.calls = {}

    def __getattr__(self, name):
        def call(*args):
            self.calls[name] = args
            return 0
        return call


@pytest.fixture
def lib(monkeypatch):
    rec = Recorder()
    monkeypatch.setattr(_lib, "require_cuda", lambda: None)
    monkeypatch.setattr(_lib, "load", lambda: rec)
    monkeypatch.setattr(_lib, "current_stream", lambda: 0)
    return rec


def _subm(mask, n=8):
    coords = torch.zeros((n, 4), dtype=torch.int32)
    pairs = torch.empty((2, 27, n), dtype=torch.int32)
    SpconvOps.generate_subm_conv_inds(coords, pairs, mask, (4, 4, 4), (3, 3, 3))


def _mask_address(lib):
    return lib.calls["sc_build_subm_pairs"][7].value


def test_subm_mask_row_written_in_place(lib):
    mask = torch.zeros((1, 8), dtype=torch.int32)
    _subm(mask)
    assert _mask_address(lib) == mask.data_ptr()


@pytest.mark.parametrize("words", [5, 9])
def test_subm_mask_of_another_length(lib, words):
    """The kernel writes one word per voxel: a row of another length is never
    handed to it, and is an error."""
    mask = torch.zeros((1, words), dtype=torch.int32)
    with pytest.raises(RuntimeError):
        _subm(mask)
    assert _mask_address(lib) != mask.data_ptr()


@pytest.mark.parametrize("mask", [torch.zeros((1, 8), dtype=torch.int64),
                                  torch.zeros((1, 8, 2), dtype=torch.int32)[..., 0],
                                  torch.empty((1, 8), dtype=torch.int32, device="meta")])
def test_subm_mask_elsewhere_or_of_another_form(lib, mask):
    """Another dtype, stride or device: the kernel's words go through a buffer
    beside the coordinates and are copied."""
    _subm(mask)
    address = _mask_address(lib)
    assert address is not None
    assert mask.device.type == "meta" or address != mask.data_ptr()


@pytest.mark.parametrize("mask", [torch.zeros(7, dtype=torch.int32), torch.zeros(9, dtype=torch.int32),
                                  torch.zeros(8, dtype=torch.int64), torch.zeros(8, dtype=torch.float32),
                                  torch.zeros(16, dtype=torch.int32)[::2],
                                  torch.empty(8, dtype=torch.int32, device="meta")])
def test_sort_indices_refuses_other_masks(lib, mask):
    """The kernel reads N 32-bit words of the mask."""
    with pytest.raises(ValueError, match="mask"):
        SpconvOps.sort_indices(torch.zeros((27, 8), dtype=torch.int32), torch.arange(8, dtype=torch.int32), mask=mask)
    assert not lib.calls


@pytest.mark.parametrize("wrap", [lambda t: t, lambda t: tv.Tensor(t, tv.uint32)])
def test_sort_indices_takes_a_mask(lib, wrap):
    mask = torch.zeros(8, dtype=torch.int32)
    SpconvOps.sort_indices(torch.zeros((27, 8), dtype=torch.int32), torch.arange(8, dtype=torch.int32), mask=wrap(mask))
    assert lib.calls["sc_sort_indices_masked"][4].value == mask.data_ptr()


def _table(n=8, **kw):
    row = lambda: torch.arange(n, dtype=torch.int32)
    pairs = lambda: torch.zeros((27, n), dtype=torch.int32)
    return PairTable(n, n, 27, False, pairs(), pairs(), [row()], [row()], **kw)


def _sorted_with(lib, pt, which):
    lib.calls.clear()
    pt.sorted_indices(which)
    mask = lib.calls["sc_sort_indices_masked"][4]
    return None if mask is None else mask.value


def test_tables_made_by_the_caller_are_sorted_whole(lib):
    """Masks that did not come with the tables may name fewer pairs than these
    hold (rows of one split, merged words) or be absent: every entry is read."""
    assert _sorted_with(lib, _table(), "fwd") is None
    pt = _table(argsorts_bwd=[torch.arange(8, dtype=torch.int32)])
    assert _sorted_with(lib, pt, "bwd") is None


@pytest.mark.parametrize("change", [lambda m: m[0].bitwise_and_(1), lambda m: m.__setitem__(0, m[0] & 1)])
def test_built_tables_are_sorted_by_their_own_masks(lib, change):
    coords = torch.zeros((8, 4), dtype=torch.int32)
    pt = build_pair_table(coords, (4, 4, 4))
    assert _sorted_with(lib, pt, "bwd") == pt.masks_fwd[0].data_ptr()
    change(pt.masks_fwd)
    assert _sorted_with(lib, pt, "fwd") is None
    # the forward's table without the backward's
    pt = build_pair_table(coords, (4, 4, 4))
    pt.pairs_bwd = None
    assert _sorted_with(lib, pt, "fwd") is None
    # a copy with other masks is a table made by the caller, and a copy of the
    # tensors is not what the builder left
    assert _sorted_with(lib, pickle.loads(pickle.dumps(build_pair_table(coords, (4, 4, 4)))), "fwd") is None
    pt = build_pair_table(coords, (4, 4, 4))
    assert _sorted_with(lib, dataclasses.replace(pt, masks_fwd=[pt.masks_fwd[0] & 1]), "fwd") is None


@pytest.mark.parametrize("v", [(2 ** 31, 4, 4), (4, 2 ** 32 + 4, 4), (4, 4, -2 ** 31 - 1), (4, 4)])
def test_sizes_outside_int32_are_refused(lib, v):
    """A size that 32 bits do not hold is an error and not another size."""
    coords = torch.zeros((8, 4), dtype=torch.int32)
    with pytest.raises((RuntimeError, ValueError)):
        build_pair_table(coords, v)
    with pytest.raises((RuntimeError, ValueError)):
        build_pair_table(coords, v, subm=False)
    assert not {"sc_build_subm_pairs", "sc_build_conv_outputs"} & set(lib.calls)


def test_sizes_of_any_integer_kind(lib):
    coords = torch.zeros((8, 4), dtype=torch.int32)
    for v in (torch.tensor([4, 5, 6]), np.array([4, 5, 6]), (4.0, 5, 6), (4, 5, 6, 7)):
        build_pair_table(coords, v)
        assert list(lib.calls["sc_build_subm_pairs"][2])[:3] == [4, 5, 6]
