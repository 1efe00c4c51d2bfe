"""The one-pass spline builds, the fold from slopes and the two evaluations, at the
sizes where their forms change.

* few_spline_build_chunked against the scan build, for knot counts around a chunk (32 rows), a CTA's four chunks and one row more, with even and
  uneven knots and both layouts.  Tolerance: the two differ by the rounding of their
  sweeps (a few units in the last place of the slopes, which the divided differences of
  c2 and c3 pass on as the same share of each plane's largest value): 1e-13.
* few_spline_slopes against the scan build's c1 plane (but for its end knot), and few_fold_slopes against
  few_fold_coeffs on its coefficients: equal to the last bit.
* Knots too uneven for the one-pass form keep the scan, through the same entry points.
* few_spline_eval's shared form against its per-series form (the same knots given once
  and repeated for every series): equal to the last bit."""
import numpy as np
import pytest
import torch

from fastemriwaveforms_b200 import CubicSplineInterpolant, _lib
from fastemriwaveforms_b200.summation import ONE_PASS_KNOTS, _ptr, _stream, spline_factor, spline_factor_table

pytestmark = pytest.mark.gpu


def overlap_of(t):
    fac = np.zeros(_lib.FEW_FAC_WIDTH * (len(t) + 1))
    _lib.call("few_spline_factor", t.ctypes.data, len(t), fac.ctypes.data)
    return int(_lib.load().few_spline_overlap(fac.ctypes.data, len(t)))


def knots(N, uneven):
    rng = np.random.default_rng(N)
    return np.cumsum(10.0 ** rng.uniform(-0.7, 0.0, N) if uneven else np.ones(N))


@pytest.mark.parametrize("N", [4, 5, 33, 34, 35, 66, 130, 131, 162, 258, 259, 1000, 1025])
@pytest.mark.parametrize("uneven", [False, True])
@pytest.mark.parametrize("ni", [1, 31, 33, 70])
def test_one_pass_builds_match_scan(cuda, N, uneven, ni):
    t = knots(N, uneven)
    ov = overlap_of(t)
    assert 1 <= ov <= _lib.load().few_spline_max_overlap()
    fac = spline_factor_table(t, cuda)
    y = torch.tensor(np.random.default_rng(ni).standard_normal((ni, N)), device=cuda)
    st = _stream(cuda)
    for layout in (_lib.FEW_LAYOUT_KNOT_MAJOR, _lib.FEW_LAYOUT_INTERP_MAJOR):
        a, b = (torch.zeros(4, N * ni, dtype=torch.float64, device=cuda) for _ in range(2))
        _lib.call("few_spline_build_factored", _ptr(fac), _ptr(y), 1, N, ni, 0, ni, N, _ptr(a), layout, st)
        _lib.call("few_spline_build_chunked", _ptr(fac), ov, _ptr(y), 1, N, ni, 0, ni, N, _ptr(b), layout, st)
        for q in range(4):
            assert (a[q] - b[q]).abs().max() <= 1e-13 * a[q].abs().max(), (layout, q)
        if layout == _lib.FEW_LAYOUT_KNOT_MAJOR:
            s = torch.zeros(N, ni, dtype=torch.float64, device=cuda)
            yt = y.T.contiguous()
            _lib.call("few_spline_slopes", _ptr(fac), _ptr(yt), ni, N, _ptr(s), st)
            c1 = a[1].reshape(N, ni)
            assert torch.equal(s[:-1], c1[:-1])
            # the c1 plane ends with the last segment's derivative, formed from its coefficients
            assert (s[-1] - c1[-1]).abs().max() <= 1e-13 * c1.abs().max()


@pytest.mark.parametrize("N,nseg", [(4, 3), (6, 5), (66, 64), (163, 162), (163, 151)])
@pytest.mark.parametrize("R,NN", [(1, 1), (3, 43), (5, 61)])
def test_fold_from_slopes_matches_fold_of_coefficients(cuda, N, nseg, R, NN):
    rng = np.random.default_rng(N * 100 + R)
    K = 2 * R * NN + 3
    fac = spline_factor_table(knots(N, True), cuda)
    teuk = torch.tensor(rng.standard_normal((N, K)) + 1j * rng.standard_normal((N, K)), device=cuda)
    ylm = torch.tensor(rng.standard_normal(2 * K) + 1j * rng.standard_normal(2 * K), device=cuda)
    keys = R * NN
    owner = rng.integers(0, keys, 2 * K)  # some keys stay empty
    order = np.argsort(owner, kind="stable")
    ptr = np.concatenate([[0], np.cumsum(np.bincount(owner, minlength=keys))]).astype(np.int32)
    lst = (2 * (order % K) + (order // K)).astype(np.int32)
    ptr_d, lst_d = torch.tensor(ptr, device=cuda), torch.tensor(lst, device=cuda)
    st = _stream(cuda)
    co = torch.zeros(4, N, 2 * K, dtype=torch.float64, device=cuda)
    _lib.call("few_spline_build_factored", _ptr(fac), _ptr(teuk), 2 * K, 2, K, 1, 2 * K, N, _ptr(co),
              _lib.FEW_LAYOUT_KNOT_MAJOR, st)
    s = torch.zeros(N, 2 * K, dtype=torch.float64, device=cuda)
    _lib.call("few_spline_slopes", _ptr(fac), _ptr(teuk), 2 * K, N, _ptr(s), st)
    a, b = (torch.full((nseg, keys, 4), float("nan"), dtype=torch.complex128, device=cuda) for _ in range(2))
    _lib.call("few_fold_coeffs", _ptr(co), _ptr(ylm), _ptr(ptr_d), _ptr(lst_d), K, N, nseg, R, NN, _ptr(a), st)
    _lib.call("few_fold_slopes", _ptr(teuk), _ptr(s), _ptr(fac), _ptr(ylm), _ptr(ptr_d), _ptr(lst_d), K, N, nseg, R,
              NN, _ptr(b), st)
    assert torch.equal(a, b)


def test_very_uneven_knots_keep_the_scan(cuda):
    N = 2 * ONE_PASS_KNOTS
    gaps = np.where(np.arange(N) < N // 2, 1.6 ** np.arange(N), 1.0)  # growing gaps: slow forgetting one way
    gaps = gaps / gaps.max() + 1e-12
    t = np.cumsum(gaps)
    assert spline_factor(np.cumsum(np.ones(N)), cuda)[1] > 0
    assert spline_factor(np.cumsum(np.ones(ONE_PASS_KNOTS - 1)), cuda)[1] == 0
    y = np.sin(3 * t)
    s = CubicSplineInterpolant(t, y)
    if overlap_of(t) > _lib.load().few_spline_max_overlap():
        assert spline_factor(t, cuda)[1] == 0
    from scipy.interpolate import CubicSpline

    want = CubicSpline(t, y, bc_type="not-a-knot")(0.5 * (t[1:] + t[:-1]))
    got = s(0.5 * (t[1:] + t[:-1])).cpu().numpy()
    np.testing.assert_allclose(got, want, rtol=0, atol=1e-10 * np.abs(want).max())


@pytest.mark.parametrize("ni", [16, 31, 33, 70])
@pytest.mark.parametrize("N,M", [(4, 1), (5, 63), (9, 64), (40, 65), (300, 1000), (4097, 129)])
def test_shared_evaluation_equals_per_series(cuda, ni, N, M):
    rng = np.random.default_rng(N + M)
    t = knots(N, True)
    td = torch.tensor(t, device=cuda)
    co = torch.tensor(rng.standard_normal((4, N, ni)), device=cuda)
    tn = rng.uniform(t[0], t[-1], M)
    tn[0] = t[-1]
    if M > 3:
        tn[1:4] = t[0], t[1], t[0] - 1.0
    if M > 60:
        tn[-1] = t[-1] + 2.0
    tn = torch.tensor(tn, device=cuda)
    many, tnm = td[None].expand(ni, N).contiguous(), tn[None].expand(ni, M).contiguous()
    st = _stream(cuda)
    for deriv in range(4):
        outs, flags = [], []
        for tt, trs, nn, nrs in ((td, 0, tn, 0), (many, N, tn, 0), (many, N, tnm, M)):
            out = torch.full((ni, M), float("nan"), dtype=torch.float64, device=cuda)
            fl = torch.zeros(2, dtype=torch.int32, device=cuda)
            _lib.call("few_spline_eval", _ptr(tt), trs, _ptr(co), ni, N, _ptr(nn), nrs, M, deriv, _ptr(out), _ptr(fl),
                      st)
            outs.append(out)
            flags.append(fl.tolist())
        assert torch.isfinite(outs[0]).all()
        assert torch.equal(outs[0], outs[1]) and torch.equal(outs[0], outs[2])
        assert flags[0] == flags[1] == flags[2] == [int(M > 3), int(M > 60)]
