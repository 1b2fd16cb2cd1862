"""Indice-pair / mask builder and mask argsort for the mask-implicit-GEMM
convolution, on the GPU kernels of libcumm_b200.so.

The reference consumes these from spconv (``SpconvOps.generate_subm_conv_inds``
and ``SpconvOps.sort_1d_by_key_split``, called at
cumm/conv/main_real_spconv.py:79-145); spconv is not part of the reference
tree, so the semantics are defined here (and restated on the CPU in
oracle/pairs_oracle.py):

* offsets k = (kz * KY + ky) * KX + kx over the kernel box, cross-correlation
  (the same indexing as ``torch.nn.functional.conv3d`` with a [K, C, kz, ky, kx]
  weight);
* ``pairs[0][k][o]`` = input index feeding output o through offset k (-1 if
  none), ``pairs[1][k][i]`` = output index fed by input i through offset k;
* ``mask_fwd[o]`` bit k <=> pairs[0][k][o] >= 0, ``mask_bwd[i]`` bit k <=>
  pairs[1][k][i] >= 0; for submanifold convs mask_bwd is the bit-reversed
  mask_fwd, which the backward-input kernel derives with ``reverse_mask``;
* strided-conv outputs are numbered in ascending (batch, z, y, x) order.
"""
import ctypes
import weakref
from dataclasses import dataclass, field
from typing import List, Optional, Sequence

import torch

from . import _lib
from . import tensorview as tv

# split masks of spconv's two-way MaskSplitImplicitGemm (main_real_spconv.py:120-121)
SPLIT_MASKS_27 = (0b11111111111111, 0b1111111111111 << 14)


def _vp(t: torch.Tensor):
    return ctypes.c_void_p(t.data_ptr()) if t is not None and t.numel() > 0 else None


_I32x3 = ctypes.c_int32 * 3
_LO, _HI = -(1 << 31), (1 << 31) - 1


def _i32x3(v: Sequence[int]):
    """The first three ints as a host array (an argument of the C entry
    points).  ctypes wraps a value that 32 bits do not hold."""
    a, b, c = map(int, v if len(v) == 3 else list(v)[:3])
    if not (_LO <= a <= _HI and _LO <= b <= _HI and _LO <= c <= _HI):
        raise ValueError(f"{a}, {b}, {c}: a value does not fit 32 bits")
    return _I32x3(a, b, c)


def _stream(stream: int):
    return ctypes.c_void_p(stream if stream else _lib.current_stream())


def _ws(nbytes: int, device) -> torch.Tensor:
    return torch.empty(max(int(nbytes), 256), dtype=torch.uint8, device=device)


def _t(x):
    return x.torch() if isinstance(x, tv.Tensor) else x


class SpconvOps:
    """GPU pair builder with spconv's operation names."""

    @staticmethod
    def generate_subm_conv_inds(indices, indice_pairs, indice_pair_mask, spatial_shape: Sequence[int],
                                ksize: Sequence[int], dilation: Sequence[int] = (1, 1, 1),
                                indice_num_per_loc=None, split_masks: Optional[Sequence[int]] = None,
                                stream: int = 0) -> int:
        """Fills ``indice_pairs`` [2, kv, N] int32 and ``indice_pair_mask``
        [S, N] uint32 (S = 1, or 2 with ``split_masks``: row j holds
        mask & split_masks[j]) for a submanifold conv; returns N."""
        _lib.require_cuda()
        lib = _lib.load()
        coords = _t(indices)
        pairs = _t(indice_pairs)
        masks = _t(indice_pair_mask)
        n = coords.shape[0]
        kv = int(ksize[0] * ksize[1] * ksize[2])
        if tuple(pairs.shape) != (2, kv, n) or pairs.dtype != torch.int32:
            raise ValueError(f"indice_pairs must be int32 [2, {kv}, {n}]")
        dev = coords.device
        need = ctypes.c_int64(0)
        _lib.check(lib.sc_pairs_workspace_size(n, kv, 1, ctypes.byref(need)))
        ws = _ws(need.value, dev)
        sp, ks, dl = _i32x3(spatial_shape), _i32x3(ksize), _i32x3(dilation)
        # without a split the kernel writes the caller's mask row itself, where
        # that is n plain words beside the coordinates (else copy_ converts,
        # moves or refuses)
        row = masks[0]
        direct = (split_masks is None and row.dtype == torch.int32 and row.shape == (n,) and row.device == dev and
                  row.is_contiguous())
        mask_full = row if direct else torch.empty(n, dtype=torch.int32, device=dev)
        s = _stream(stream)
        fwd = pairs.data_ptr() if n else None
        bwd = fwd + 4 * pairs.stride(0) if n else None
        _lib.check(lib.sc_build_subm_pairs(
            _vp(coords), n, sp, ks, dl, fwd, bwd, _vp(mask_full), _vp(ws), ws.numel(), s))
        if split_masks is None:
            if not direct:
                row.copy_(mask_full)
        else:
            for j, sm in enumerate(split_masks):
                masks[j].copy_(mask_full & _as_i32(sm))
        if indice_num_per_loc is not None:
            _t(indice_num_per_loc).copy_((pairs[0] >= 0).sum(1).to(torch.int32))
        return n

    @staticmethod
    def generate_conv_inds(indices, batch_size: int, spatial_shape: Sequence[int],
                           ksize: Sequence[int], stride: Sequence[int], padding: Sequence[int],
                           dilation: Sequence[int] = (1, 1, 1), stream: int = 0):
        """Regular (strided) sparse conv: returns (out_inds [n_out, 4],
        pairs_fwd [kv, n_out], pairs_bwd [kv, n_in], mask_fwd [n_out],
        mask_bwd [n_in], out_spatial_shape).  Synchronises once (n_out sizes
        the outputs)."""
        _lib.require_cuda()
        lib = _lib.load()
        coords = _t(indices)
        n = coords.shape[0]
        dev = coords.device
        kv = int(ksize[0] * ksize[1] * ksize[2])
        need = ctypes.c_int64(0)
        _lib.check(lib.sc_pairs_workspace_size(n, kv, 0, ctypes.byref(need)))
        ws = _ws(need.value, dev)
        sp, ks, st, pd, dl = (_i32x3(spatial_shape), _i32x3(ksize), _i32x3(stride), _i32x3(padding),
                              _i32x3(dilation))
        out_sp = _I32x3()
        n_out = ctypes.c_int64(0)
        s = _stream(stream)
        args = (sp, ks, st, pd, dl)
        _lib.check(lib.sc_build_conv_outputs(_vp(coords), n, batch_size, *args, out_sp,
                                             ctypes.byref(n_out), _vp(ws), ws.numel(), s))
        no = int(n_out.value)
        out_inds = torch.empty((no, 4), dtype=torch.int32, device=dev)
        pf = torch.empty((kv, no), dtype=torch.int32, device=dev)
        pb = torch.empty((kv, n), dtype=torch.int32, device=dev)
        mf = torch.empty(no, dtype=torch.int32, device=dev)
        mb = torch.empty(n, dtype=torch.int32, device=dev)
        _lib.check(lib.sc_build_conv_pairs(_vp(coords), n, batch_size, *args, no, _vp(out_inds),
                                           _vp(pf), _vp(pb), _vp(mf), _vp(mb), _vp(ws), ws.numel(),
                                           s))
        return out_inds, pf, pb, mf, mb, list(out_sp)

    @staticmethod
    def sort_1d_by_key_split(data, mask, stream: int = 0):
        """Stable sort of ``data`` (uint32 [N], in place) by ``data & mask``;
        returns the argsort (int32 [N]).  ``mask`` is an int or a one-element
        tensor (reference call: main_real_spconv.py:141-145)."""
        _lib.require_cuda()
        lib = _lib.load()
        d = _t(data)
        if isinstance(mask, (tv.Tensor, torch.Tensor)):
            m = int(_t(mask).reshape(-1)[0].item()) & 0xffffffff
        else:
            m = int(mask) & 0xffffffff
        n = d.numel()
        out = torch.empty(n, dtype=torch.int32, device=d.device)
        need = ctypes.c_int64(0)
        _lib.check(lib.sc_sort_workspace_size(n, ctypes.byref(need)))
        ws = _ws(need.value, d.device)
        _lib.check(lib.sc_sort_masks_split(_vp(d), n, ctypes.c_uint32(m), _vp(out), _vp(ws),
                                           ws.numel(), _stream(stream)))
        if isinstance(data, tv.Tensor):
            return tv.Tensor(out, tv.int32)
        return out

    @staticmethod
    def sort_1d_by_key(data, stream: int = 0):
        return SpconvOps.sort_1d_by_key_split(data, 0xffffffff, stream)

    @staticmethod
    def sort_indices(indices, argsort, stream: int = 0, mask=None, reverse: bool = False):
        """indices [kv, N] permuted into argsort order: out[k][r] =
        indices[k][argsort[r]] (the optional ConvParams.indices_sorted).
        ``mask``: the sorted masks [N], bit k (of the kv-bit reversed word with
        ``reverse``) set exactly where out[k][r] != -1; absent entries are then
        not read."""
        ind, srt, msk = _t(indices), _t(argsort), _t(mask)
        n = ind.shape[1]
        if msk is not None and not (msk.numel() == n and msk.dtype in (torch.int32, torch.uint32) and
                                    msk.device == ind.device and msk.is_contiguous()):
            raise ValueError(f"mask must be {n} contiguous 32-bit words on the device of indices")
        out = _sort_indices(ind, srt, msk, reverse, stream)
        if isinstance(indices, tv.Tensor):
            return tv.Tensor(out, tv.int32)
        return out


    @staticmethod
    def tile_order(mask, kv: int, mask_filter: int = 0xffffffff, reverse: bool = False,
                   stream: int = 0):
        """Largest-first order of the 128-row tiles of the sorted masks (the
        optional ConvParams.tile_order): tiles by the number of offsets their
        OR-ed masks visit, heaviest first."""
        _lib.require_cuda()
        lib = _lib.load()
        m = _t(mask)
        n = int(m.numel())
        out = torch.empty(((n + 127) // 128,), dtype=torch.int32, device=m.device)
        need = ctypes.c_int64(0)
        _lib.check(lib.sc_tile_order_workspace_size(n, ctypes.byref(need)))
        ws = torch.empty((max(int(need.value), 1),), dtype=torch.uint8, device=m.device)
        _lib.check(lib.sc_tile_order(_vp(m), n, ctypes.c_uint32(mask_filter & 0xffffffff), kv,
                                     1 if reverse else 0, _vp(out), _vp(ws), ws.numel(),
                                     _stream(stream)))
        if isinstance(mask, tv.Tensor):
            return tv.Tensor(out, tv.int32)
        return out


def _sort_indices(ind: torch.Tensor, order: torch.Tensor, mask, reverse: bool, stream: int) -> torch.Tensor:
    """sort_indices of a mask that fits."""
    _lib.require_cuda()
    kv, n = ind.shape
    out = torch.empty_like(ind)
    _lib.check(_lib.load().sc_sort_indices_masked(_vp(ind), kv, n, _vp(order), _vp(mask), 1 if reverse else 0,
                                                  _vp(out), _stream(stream)))
    return out


def _as_i32(v: int) -> int:
    v &= 0xffffffff
    return v - (1 << 32) if v >= (1 << 31) else v


def _versions(tensors):
    """torch's counts of the writes to the tensors (None: inference tensors, or
    a table that the caller dropped)."""
    try:
        return [t._version for t in tensors]
    except (RuntimeError, AttributeError):
        return None


@dataclass
class PairTable:
    """Device-resident pair tables of one sparse conv layer (the inputs of
    ConvParams for fwd / dgrad / wgrad)."""
    n_in: int
    n_out: int
    kv: int
    subm: bool
    pairs_fwd: torch.Tensor            # [kv, n_out] int32
    pairs_bwd: torch.Tensor            # [kv, n_in] int32
    masks_fwd: List[torch.Tensor]      # per split: sorted masks [n_out] (int32 storage of uint32)
    argsorts_fwd: List[torch.Tensor]   # per split: [n_out] int32
    masks_bwd: List[torch.Tensor] = field(default_factory=list)   # strided only
    argsorts_bwd: List[torch.Tensor] = field(default_factory=list)
    split_masks: List[int] = field(default_factory=list)
    out_inds: Optional[torch.Tensor] = None
    out_spatial: Optional[List[int]] = None

    def pair_count(self) -> int:
        """P = number of valid (input, output) pairs."""
        return int((self.pairs_fwd >= 0).sum().item())

    def _tables(self):
        return (self.pairs_fwd, self.pairs_bwd, *self.masks_fwd, *self.argsorts_fwd, *self.masks_bwd,
                *self.argsorts_bwd)

    def _mark_built(self):
        """Notes that the masks name exactly the pairs of the tables, in their
        argsort's order, as the builder leaves them.  Another tensor in their
        place, and a write to one through torch (inference tensors do not
        count those), end that."""
        tables = self._tables()
        self._built = [*map(weakref.ref, tables)], _versions(tables)

    def _as_built(self) -> bool:
        built = self.__dict__.get("_built")
        if built is None:
            return False
        tables = self._tables()
        return [id(r()) for r in built[0]] == [*map(id, tables)] and _versions(tables) == built[1]

    def __getstate__(self):
        return {k: v for k, v in self.__dict__.items() if k != "_built"}

    def sorted_indices(self, which: str = "fwd", split: int = 0) -> torch.Tensor:
        """Index table of `which` ('fwd' or 'bwd') permuted into the argsort
        order the matching convolution uses: forward and backward-weight walk
        pairs_fwd in argsorts_fwd order; backward-input walks pairs_bwd in
        argsorts_fwd order (submanifold, reverse_mask) or argsorts_bwd order
        (strided).  Cached per (which, split)."""
        cache = self.__dict__.setdefault("_sorted_cache", {})
        key = (which, split)
        if key not in cache:
            fwd, subm = which == "fwd", self.subm
            pairs = self.pairs_fwd if fwd else self.pairs_bwd
            order = (self.argsorts_fwd if fwd or subm else self.argsorts_bwd)[split]
            # the masks that the builder left say which entries exist; others
            # may disagree with the tables
            mask = (self.masks_fwd if fwd or subm else self.masks_bwd)[split] if self._as_built() else None
            cache[key] = _sort_indices(pairs, order, mask, not fwd and subm, 0)
        return cache[key]

    def tile_order(self, which: str = "fwd", split: int = 0) -> torch.Tensor:
        """Largest-first tile order (ConvParams.tile_order) for the masks
        `which` uses: forward and (submanifold) backward-input share
        masks_fwd[split], whose offset counts are the same in both directions;
        a strided backward-input uses masks_bwd[split].  Cached per (which,
        split)."""
        cache = self.__dict__.setdefault("_order_cache", {})
        key = ("fwd" if which == "fwd" or self.subm else "bwd", split)
        if key not in cache:
            masks = self.masks_fwd if key[0] == "fwd" else self.masks_bwd
            cache[key] = SpconvOps.tile_order(masks[split], self.kv, self.split_masks[split]
                                              if self.split_masks else 0xffffffff)
        return cache[key]


def _sorted_masks(mask: torch.Tensor, splits: Sequence[int], kv: int, stream: int):
    """Per split: the masks sorted by their split bits, and the argsort.  `mask`
    itself is sorted for the last split.  Bits past kv are never set, so the
    sort skips their digits."""
    masks, sorts = [], []
    for j, sm in enumerate(splits):
        mm = mask if j == len(splits) - 1 else mask.clone()
        sorts.append(SpconvOps.sort_1d_by_key_split(mm, sm & ((1 << kv) - 1), stream))
        masks.append(mm)
    return masks, sorts


def build_pair_table(coords: torch.Tensor, spatial_shape: Sequence[int], ksize=(3, 3, 3),
                     stride=(1, 1, 1), padding=(1, 1, 1), dilation=(1, 1, 1), subm: bool = True,
                     batch_size: int = 1, num_split: int = 1, stream: int = 0) -> PairTable:
    """Builds pairs, masks and (split) argsorts for one layer on the GPU, the
    way spconv's get_indice_pairs_implicit_gemm prepares them for
    MaskImplicitGemm (num_split 1) or MaskSplitImplicitGemm (num_split 2)."""
    kv = int(ksize[0] * ksize[1] * ksize[2])
    if num_split == 1:
        splits = [0xffffffff]
    elif num_split == 2:
        half = kv // 2 + 1
        splits = [(1 << half) - 1, ((1 << kv) - 1) & ~((1 << half) - 1)]
    else:
        raise ValueError("num_split must be 1 or 2")
    dev = coords.device
    n = coords.shape[0]
    if subm:
        pairs = torch.empty((2, kv, n), dtype=torch.int32, device=dev)
        m = torch.empty((1, n), dtype=torch.int32, device=dev)
        SpconvOps.generate_subm_conv_inds(coords, pairs, m, spatial_shape, ksize, dilation,
                                          stream=stream)
        masks, sorts = _sorted_masks(m[0], splits, kv, stream)
        pt = PairTable(n, n, kv, True, pairs[0], pairs[1], masks, sorts, split_masks=splits,
                       out_inds=coords, out_spatial=list(spatial_shape))
        pt._mark_built()
        return pt
    out_inds, pf, pb, mf, mb, out_sp = SpconvOps.generate_conv_inds(
        coords, batch_size, spatial_shape, ksize, stride, padding, dilation, stream)
    masks, sorts = _sorted_masks(mf, splits, kv, stream)
    masks_b, sorts_b = _sorted_masks(mb, splits, kv, stream)
    pt = PairTable(n, out_inds.shape[0], kv, False, pf, pb, masks, sorts, masks_b, sorts_b,
                   splits, out_inds, out_sp)
    pt._mark_built()
    return pt
