"""Series whose runs do not join bitwise in few_spline_build's CTA-per-series form (pulses,
steps, values many orders apart, NaN): swept there by one thread where few series go to
an SM, left to the thread form where many do; either way the thread form's result, to the
last bit, and every other series' of the same batch too."""
import numpy as np
import pytest
import torch

from fastemriwaveforms_b200 import _lib
from test_gpu_spline_rows import build

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ni", [24, 2700])
@pytest.mark.parametrize("own", [False, True])
def test_unjoined_series_equal_the_thread_form(cuda, ni, own):
    N = 1000
    big = 1024 + 3 * N + 1  # thread form
    rng = np.random.default_rng(ni)
    t = torch.tensor(np.cumsum(rng.uniform(0.2, 1.0, (big if own else 1, N)), axis=1), device=cuda)
    y = np.sin(rng.uniform(1.0, 7.0, (big, 1)) * np.arange(N) / N)
    y[0] = 0.0
    y[1] = np.arange(N) == 500
    y[2] = np.arange(N) > 77
    y[3] = np.exp(-2.0 * np.minimum(np.arange(N), 330))
    y[4] = np.exp(2.0 * np.minimum(np.arange(N)[::-1], 330))
    y[5, 40] = np.nan
    y[6, 0] = np.nan
    y[7, N - 1] = np.inf
    y[20] = np.arange(N) == N - 2
    yd = torch.tensor(y, device=cuda)
    rs = N if own else 0
    for layout in (_lib.FEW_LAYOUT_KNOT_MAJOR, _lib.FEW_LAYOUT_INTERP_MAJOR):
        want = build(t, rs, yd, 1, N, big, 0, big, N, layout)
        want = want[:, :, :ni] if layout == _lib.FEW_LAYOUT_KNOT_MAJOR else want[:, :ni]
        got = build(t, rs, yd, 1, N, ni, 0, ni, N, layout)
        a, b = (torch.nan_to_num(v, nan=1.25e99) for v in (got, want))
        assert torch.equal(a, b), layout
