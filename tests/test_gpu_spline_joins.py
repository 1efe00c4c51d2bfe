"""The spline build over independent runs of knots (few_spline_build_joined) where a run's
far ends matter: values that are not finite, and values so far apart that what a run
leaves out would show.  There the coefficients are few_spline_build_factored's to the
last bit, for the whole series, at knot counts on both sides of the one from which
CubicSplineInterpolant takes this build; elsewhere the two agree to rounding, also where a
series passes an extremum at a join (slopes close to 0 beside the largest)."""
import numpy as np
import pytest
import torch

from fastemriwaveforms_b200 import CubicSplineInterpolant, _lib
from fastemriwaveforms_b200.summation import (ONE_PASS_KNOTS, _ptr, _stream, build_splines, spline_factor,
                                              spline_factor_host, spline_factor_table)

pytestmark = pytest.mark.gpu


def overlap_of(t):
    fac = spline_factor_host(t)
    return int(_lib.load().few_spline_overlap(fac.ctypes.data, len(t)))


def both(cuda, t, y, layout=_lib.FEW_LAYOUT_KNOT_MAJOR):
    """(scan, joined) coefficients (4, N * ni) of the series y (ni, N)."""
    ni, N = y.shape
    fac, yd, st = spline_factor_table(t, cuda), torch.tensor(y, device=cuda), _stream(cuda)
    a, b = (torch.full((4, N * ni), 7.0, dtype=torch.float64, device=cuda) for _ in range(2))
    scratch = torch.full((int(_lib.load().few_spline_joined_scratch(ni, N)),), float("nan"), dtype=torch.float64,
                         device=cuda)
    _lib.call("few_spline_build_factored", _ptr(fac), _ptr(yd), 1, N, ni, 0, ni, N, _ptr(a), layout, st)
    _lib.call("few_spline_build_joined", _ptr(fac), overlap_of(t), _ptr(yd), 1, N, ni, 0, ni, N, _ptr(b), layout,
              _ptr(scratch), st)
    return a, b


def same_bits(a, b):
    return torch.equal(a.view(torch.int64), b.view(torch.int64))


def wild(kind, N, rng):
    y = rng.standard_normal(N)
    i = np.arange(N)
    if kind == "pulse":
        y = (i == N // 2).astype(float)
    elif kind == "spike":
        y[N // 3] = 1e30
    elif kind == "decay":
        y = np.exp(-2.0 * np.minimum(i, 330))
    elif kind == "growth":
        y = np.exp(2.0 * np.minimum(i, 330))
    elif kind == "odd":  # what the two sides of a join leave out of a slope is equal
        y = np.sinh(2.0 * np.clip(i - (1 + 32 * (N // 64)), -330, 330))
    elif kind == "step":
        y = (i > N // 2).astype(float)
    else:
        y[{"first": 0, "second": 1, "middle": N // 2, "last": N - 1}[kind.split()[1]]] = (
            np.nan if kind.startswith("nan") else np.inf)
    return y


WILD = ["pulse", "spike", "decay", "growth", "odd", "step", "nan first", "nan second", "nan middle", "nan last",
        "inf middle", "inf last"]


@pytest.mark.parametrize("uneven", [False, True])
@pytest.mark.parametrize("N", [150, 162, 226, 387, 1000])
@pytest.mark.parametrize("kind", WILD)
def test_wild_series_get_the_scan_forms_bits(cuda, kind, N, uneven):
    rng = np.random.default_rng(N)
    t = np.cumsum(10.0 ** rng.uniform(-0.7, 0.0, N) if uneven else np.ones(N))
    y = np.stack([wild(kind, N, rng)] + [np.sin(0.01 * (q + 1) * t) for q in range(3)])
    for layout in (_lib.FEW_LAYOUT_KNOT_MAJOR, _lib.FEW_LAYOUT_INTERP_MAJOR):
        a, b = both(cuda, t, y, layout)
        assert same_bits(a, b), (kind, N)
    c = a.reshape(4, 4, N)
    if not np.isfinite(y).all():
        assert not torch.isfinite(c[1:, 0]).any()  # the whole series
    assert torch.isfinite(c[:, 1:]).all()  # and no other


@pytest.mark.parametrize("N", [ONE_PASS_KNOTS - 1, ONE_PASS_KNOTS, ONE_PASS_KNOTS + 1, 1000])
@pytest.mark.parametrize("at", [0, 1, 5, -2, -1])
def test_interpolant_of_a_nan_is_nan_at_every_knot_count(cuda, N, at):
    t = np.cumsum(np.random.default_rng(3).uniform(0.2, 1.0, N))
    y = np.stack([np.sin(t), np.cos(t)])
    y[0, at] = np.nan
    s = CubicSplineInterpolant(t, y)
    for c in (s.c1, s.c2, s.c3):
        assert torch.isnan(c[0]).all() and torch.isfinite(c[1]).all()


@pytest.mark.parametrize("N", [150, 163, 1000, 2000])
@pytest.mark.parametrize("ni", [1, 31, 33, 70])
def test_ordinary_series_agree_to_rounding(cuda, N, ni):
    rng = np.random.default_rng(N + ni)
    t = np.cumsum(10.0 ** rng.uniform(-0.7, 0.0, N))
    # slow sines: at 1, 33, 65, ... some series' slopes pass 0
    w = rng.uniform(1.0, 9.0, (ni, 1))
    at = t[1 + 32 * rng.integers(0, (N - 2) // 32 + 1, (ni, 1))]
    y = np.cos(w * (t - at) / t[-1]) * (1.0 + 0.1 * np.arange(ni)[:, None])
    a, b = both(cuda, t, y)
    for q in range(2):  # values and slopes, from which both forms make c2 and c3 alike
        assert (a[q] - b[q]).abs().max() <= 1e-13 * a[q].abs().max(), q


def test_the_scan_form_through_the_shared_builder(cuda):
    """build_splines without an overlap (what spline_factor gives below ONE_PASS_KNOTS, and
    would for knots of a larger overlap than the joined build takes) is the scan form."""
    N, ni = 2 * ONE_PASS_KNOTS, 40
    t = np.cumsum(10.0 ** np.random.default_rng(1).uniform(-6, 0, N))
    fac, ov = spline_factor(t, cuda)
    assert 1 <= ov <= _lib.load().few_spline_max_overlap()
    y = np.sin(40.0 * t / t[-1] + np.arange(ni)[:, None])
    want, _ = both(cuda, t, y)
    yd = torch.tensor(y, device=cuda)
    c = torch.full((4, N, ni), float("nan"), dtype=torch.float64, device=cuda)
    build_splines(fac, 0, _ptr(yd), (1, N, ni, 0), ni, N, c, _stream(cuda))
    assert same_bits(c.reshape(4, N * ni), want)


def test_many_knots(cuda):
    """More runs of knots than a grid's second dimension takes (65,535 tiles of 128)."""
    N, ni = 128 * 65536 + 5, 1
    t = np.arange(N, dtype=np.float64)
    y = np.sin(1e-3 * t)[None]
    a, b = both(cuda, t, y)
    for q in range(2):
        assert (a[q] - b[q]).abs().max() <= 1e-13 * a[q].abs().max(), q
