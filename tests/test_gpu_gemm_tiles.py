"""The dense tcgen05 GEMM where its tiles can go wrong: CTA pairs (256 x 256
tiles, K of at least 1024 per split) and single CTAs (128 x 256, 128 or 64 by
the columns), at the edges of rows, columns and K, more tiles than CTAs, and every output type through the
epilogue's shared-memory lines (whole, cut by n, rows that start off 16 bytes).

Tolerance: an fp32 sum is rounded once per 16 products, at most K / 16 * 2^-23
of the sums' norm: 1e-5 for K <= 1344 (one split).  A 16-bit output is rounded
once more: 2^-8 of the value (bf16, half a step of its 8 bits) or 2^-11 (fp16),
element by element."""
import numpy as np
import pytest
import torch

from cumm import tensorview as tv
from cumm.tensorview.gemm import ShuffleStrideType
from oracle import conv_oracle as co

from test_gpu_gemm import TVD, _desp, _f64, _run, _t

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dt,dc", [(torch.bfloat16, torch.bfloat16), (torch.float16, torch.float16),
                                   (torch.bfloat16, torch.float32)])
@pytest.mark.parametrize("ta,tb", [(False, False), (False, True), (True, False), (True, True)])
@pytest.mark.parametrize("m,n,k,split", [
    (8, 8, 1024, 1), (128, 136, 1024, 1), (264, 512, 1032, 1), (248, 256, 1344, 1), (520, 328, 1096, 1),
    (384, 264, 2176, 2), (256, 256, 1016, 1), (136, 520, 960, 1),
    (40, 8, 64, 1), (1000, 64, 72, 1), (264, 72, 136, 1), (1000, 128, 960, 1), (300 * 128, 64, 136, 1),
    (298 * 128 + 8, 96, 200, 1), (200, 120, 520, 2),
])
def test_dense_tile_edges(dt, dc, ta, tb, m, n, k, split):
    rng = np.random.default_rng(m + n + k)
    a = rng.standard_normal((k, m) if ta else (m, k)).astype(np.float32)
    b = rng.standard_normal((n, k) if tb else (k, n)).astype(np.float32)
    d = rng.standard_normal((m, n)).astype(np.float32)
    at, bt, dd = _t(a, dt), _t(b, dt), _t(d, dc)
    c = torch.full((m, n), 7.0, dtype=dc, device="cuda")
    desp = _desp("Tcgen05", TVD[dt], TVD[dc], ta, tb, ShuffleStrideType.kNoShuffle)
    _run(desp, at, bt, c, d=dd, alpha=0.5, beta=2.0, act=1, split_k=split)
    ref = co.gemm(_f64(at), _f64(bt), ta, tb, d=_f64(dd), alpha=0.5, beta=2.0, act_type=1)
    err = np.abs(_f64(c) - ref)
    step = {torch.float32: 0.0, torch.bfloat16: 2.0 ** -8, torch.float16: 2.0 ** -11}[dc]
    assert np.linalg.norm(np.maximum(err - step * np.abs(ref), 0)) <= 1e-5 * split * np.linalg.norm(ref)


@pytest.mark.parametrize("m,n", [(1280, 8192), (1152, 8192), (4104, 2568)])
def test_dense_many_tiles(m, n):
    """More tiles than pairs (3 a pair: both accumulators twice) and the row
    count whose 256-row tiles would need another wave; rows of zeros and ones
    make every sum a small whole number, so the outputs are exact."""
    k = 1024
    rng = np.random.default_rng(n)
    a = torch.from_numpy(rng.integers(-1, 2, (m, k)).astype(np.float32)).cuda()
    b = torch.from_numpy((rng.random((k, n)) < 0.02).astype(np.float32)).cuda()
    c = torch.zeros((m, n), device="cuda")
    desp = _desp("Tcgen05", tv.bfloat16, tv.float32, False, False, ShuffleStrideType.kNoShuffle)
    _run(desp, a.bfloat16(), b.bfloat16(), c)
    ref = _f64(a.cpu()) @ _f64(b.cpu())
    assert np.array_equal(_f64(c), ref)


def test_dense_unaligned_rows():
    """An fp32 output of 1,001 columns: rows start off 16 bytes (store by row)."""
    rng = np.random.default_rng(2)
    m, n, k = 300, 1001, 1024
    a = rng.standard_normal((m, k)).astype(np.float32)
    b = rng.standard_normal((n, k)).astype(np.float32)
    at, bt = _t(a, torch.bfloat16), _t(b, torch.bfloat16)
    c = torch.zeros((m, n), device="cuda")
    desp = _desp("Tcgen05", tv.bfloat16, tv.float32, False, True, ShuffleStrideType.kNoShuffle)
    if not desp.supported(m, n, k):
        with pytest.raises(ValueError, match="misaligned"):
            _run(desp, at, bt, c)
        return
    _run(desp, at, bt, c)
    assert co.rel_err(_f64(c), co.gemm(_f64(at), _f64(bt), False, True))[0] < 1e-5
