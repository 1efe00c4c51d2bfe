"""few_spline_overlap on the host, at the knot counts that use it: every product of that
many successive sweep factors is below 2^-70 and some product of two fewer is not; and
knots of every kind of unevenness stay below the largest overlap that the joined build
takes."""
import numpy as np
import pytest

from fastemriwaveforms_b200 import _lib
from fastemriwaveforms_b200.summation import ONE_PASS_KNOTS, spline_factor_host


def knots(kind, N, rng):
    s = rng.uniform(0.0, 8.0)
    if kind == "even":
        gaps = np.ones(N)
    elif kind == "random":
        gaps = 10.0 ** rng.uniform(-s, 0.0, N)
    elif kind == "geometric":
        gaps = rng.uniform(1.001, 3.0) ** np.minimum(np.arange(N), 200)
        gaps = gaps[:: rng.choice([1, -1])]
    elif kind == "two sizes":
        gaps = np.where(rng.random(N) < rng.random(), 1.0, 10.0**-s)
    else:
        gaps = 10.0 ** (np.cumsum(rng.normal(0.0, s / 3, N)) % 8.0 - 8.0)
    t = np.cumsum(gaps)
    return t if (np.diff(t) > 0).all() else None


@pytest.mark.parametrize("kind", ["even", "random", "geometric", "two sizes", "wandering"])
def test_overlap(kind):
    lib = _lib.load()
    rng = np.random.default_rng(len(kind))
    for _ in range(40):
        N = int(rng.integers(ONE_PASS_KNOTS, 800))
        t = knots(kind, N, rng)
        if t is None:
            continue
        fac = spline_factor_host(t)
        w = int(lib.few_spline_overlap(fac.ctypes.data, N))
        assert 1 <= w <= lib.few_spline_max_overlap(), (kind, N)
        rows = np.abs(fac[: _lib.FEW_FAC_WIDTH * N].reshape(N, -1)[1 : N - 1])
        factors = rows[:, 0] * rows[:, 1], rows[:, 2]
        products = [np.lib.stride_tricks.sliding_window_view(f, n).prod(axis=1).max() for n in (w, w - 2)
                    for f in factors]
        assert max(products[:2]) < 2.0**-70 <= max(products[2:]), (kind, N)


def test_bad_arguments_are_refused_on_the_host():
    import ctypes

    lib = _lib.load()
    d = ctypes.c_void_p(16)  # never read
    for fn, tail in ((lib.few_spline_build_chunked, ()), (lib.few_spline_build_joined, (d,))):
        call = lambda fac=d, ov=40, y=d, split=1, ni=1, n=400, out=d, layout=0: fn(  # noqa: E731
            fac, ov, y, 1, 1, split, 0, ni, n, out, layout, *tail, None)
        assert call(fac=None) == call(y=None) == call(out=None) == _lib.FEW_ERR_ARG
        assert call(layout=2) == call(split=2) == _lib.FEW_ERR_ARG
        assert call(ov=0) == call(ov=97) == call(ni=0) == call(n=3) == _lib.FEW_ERR_SIZE
    assert lib.few_spline_build_joined(d, 40, d, 1, 1, 1, 0, 1, 400, d, 0, None, None) == _lib.FEW_ERR_ARG
