"""The dense tcgen05 GEMM with C and D that start off 16 bytes: rows are stored
by their own threads and D is read element by element.  Single CTAs of 64, 128
and 256 columns, one and two per SM, and CTA pairs; D beside C and D = C.

Tolerance as in test_gpu_gemm_tiles.py: 1e-5 of the norm beside one rounding of
the output's type."""
import numpy as np
import pytest
import torch

from cumm.tensorview.gemm import ShuffleStrideType
from oracle import conv_oracle as co

from test_gpu_gemm import TVD, _desp, _f64, _run, _t

pytestmark = pytest.mark.gpu


def _offset(x, dt):
    """x one element into a larger buffer of sevens, and the buffer."""
    buf = torch.full((x.size + 2,), 7.0, dtype=dt, device="cuda")
    t = buf[1:-1].view(x.shape)
    t.copy_(torch.from_numpy(x))
    assert t.data_ptr() % 16
    return t, buf


@pytest.mark.parametrize("dt,dc", [(torch.bfloat16, torch.bfloat16), (torch.float16, torch.float16),
                                   (torch.bfloat16, torch.float32)])
@pytest.mark.parametrize("m,n,k", [(264, 72, 136), (40, 64, 72), (136, 520, 960), (298 * 128 + 8, 96, 200), (264, 512, 1032)])
@pytest.mark.parametrize("alias", [False, True])
def test_unaligned_outputs(dt, dc, m, n, k, alias):
    rng = np.random.default_rng(m + n + k)
    at = _t(rng.standard_normal((m, k)).astype(np.float32), dt)
    bt = _t(rng.standard_normal((n, k)).astype(np.float32), dt)
    d, d_buf = _offset(rng.standard_normal((m, n)).astype(np.float32), dc)
    d0 = _f64(d)
    c, c_buf = (d, d_buf) if alias else _offset(np.zeros((m, n), np.float32), dc)
    desp = _desp("Tcgen05", TVD[dt], TVD[dc], False, True, ShuffleStrideType.kNoShuffle)
    assert desp.supported(m, n, k)
    _run(desp, at, bt, c, d=d, alpha=0.5, beta=2.0, act=1)
    ref = co.gemm(_f64(at), _f64(bt), False, True, d=d0, alpha=0.5, beta=2.0, act_type=1)
    step = {torch.float32: 0.0, torch.bfloat16: 2.0 ** -8, torch.float16: 2.0 ** -11}[dc]
    err = np.maximum(np.abs(_f64(c) - ref) - step * np.abs(ref), 0)
    assert np.linalg.norm(err) <= 1e-5 * np.linalg.norm(ref)
    assert c_buf[0] == 7 and c_buf[-1] == 7
    assert alias or np.array_equal(_f64(d), d0)
