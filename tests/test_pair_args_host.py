"""Host side of the pair builder's calls, with the native library replaced by a
recorder: which addresses a call hands over, and what it refuses before that."""
import pytest
import torch

from cumm import _lib
from cumm import tensorview as tv
from cumm.spconv_ops import SpconvOps


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
