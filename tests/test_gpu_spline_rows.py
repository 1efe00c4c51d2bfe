"""few_spline_build's CTA-per-series form against its thread-per-series form, bit
for bit: the first series of a batch too large for the former, built again on
their own.  Shortest systems, one row a thread and a row more, several rows a
thread, the longest that shared memory takes and one more; nearly even and very
uneven knots; both layouts; knots shared and per series; split strided input."""
import numpy as np
import pytest
import torch

from fastemriwaveforms_b200 import _lib
from fastemriwaveforms_b200.summation import _ptr, _stream

pytestmark = pytest.mark.gpu

FEW = 3


def build(t, t_rs, y, sk, sp, split, off2, ni, N, layout):
    out = torch.empty((4, N, ni) if layout == _lib.FEW_LAYOUT_KNOT_MAJOR else (4, ni, N), dtype=torch.float64, device=y.device)
    _lib.call("few_spline_build", _ptr(t), t_rs, _ptr(y), sk, sp, split, off2, ni, N, _ptr(out), layout,
              _stream(y.device))
    return out


@pytest.mark.parametrize("N", [4, 5, 6, 65, 66, 67, 130, 131, 258, 1000, 6400, 6401])
@pytest.mark.parametrize("uneven", [False, True])
@pytest.mark.parametrize("own", [False, True])
def test_rows_equal_threads(cuda, N, uneven, own):
    rng = np.random.default_rng(N)
    big = 1024 + 3 * N + 1
    shape = (big if own else 1, N)
    gaps = 10.0 ** rng.uniform(-5, 0, shape) if uneven else rng.uniform(0.2, 1.0, shape)
    t = torch.tensor(np.cumsum(gaps, axis=1), device=cuda)
    y = torch.tensor(rng.standard_normal((big, N)), device=cuda)
    rs = N if own else 0
    for layout in (_lib.FEW_LAYOUT_KNOT_MAJOR, _lib.FEW_LAYOUT_INTERP_MAJOR):
        many = build(t, rs, y, 1, N, big, 0, big, N, layout)
        few = build(t, rs, y, 1, N, FEW, 0, FEW, N, layout)
        want = many[:, :, :FEW] if layout == _lib.FEW_LAYOUT_KNOT_MAJOR else many[:, :FEW]
        assert torch.isfinite(few).all()
        assert torch.equal(few, want), layout
    # complex series read in place: real parts, then imaginary parts
    z = torch.complex(y[:FEW], y[FEW:2 * FEW]).T.contiguous()  # (N, FEW)
    got = build(t[:1], 0, torch.view_as_real(z), 2 * FEW, 2, FEW, 1, 2 * FEW, N, _lib.FEW_LAYOUT_KNOT_MAJOR)
    want = build(t[:1], 0, y, 1, N, big, 0, big, N, _lib.FEW_LAYOUT_KNOT_MAJOR)[:, :, :2 * FEW]
    assert torch.equal(got, want)
