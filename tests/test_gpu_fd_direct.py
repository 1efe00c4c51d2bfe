"""The stationary-phase sum's two ways to a bin's root against the CPU oracle,
which takes Cardano's formula for every bin: segments of hundreds of bins (two
bins a lane), about one warp's width, just above and below the mean number of
bins per segment at which the sum stops forming a segment's shared terms, less
than one bin a segment; few and many knots (strongly curved and nearly straight
frequency tracks), turning tracks, k != 0 modes, negative slopes, +m only.

Tolerance: the phases reach 2 pi f span ~ 1e5 rad, whose last place is 1.5e-11;
a term's phase is rounded three times on each side, so 5e-11 bounds the relative
L2 difference.  The tracks end at p = 8.3: at p = 8 these frequencies hold
f_phi = 2 f_r exactly, which puts the root of the zero bin on the last knot, where
rounding alone decides whether it counts."""
import numpy as np
import pytest
import torch

from fastemriwaveforms_b200 import FDInterpolatedModeSum
from fastemriwaveforms_b200 import synthetic as S

pytestmark = pytest.mark.gpu

REL = 5e-11


def frequencies(M, a, p, e, x):
    f = p ** -1.5 / (2 * np.pi * M * 4.9254909491978065e-06)
    return np.stack([f, f * (1 - 0.5 / p), f * np.sqrt(1 - 6 / p)])


# K, N, span (s), kmax, nmax, options
CASES = {
    "long_segments": (40, 12, 2e6, 0, 5, {}),
    "warp_width": (60, 60, 2e6, 0, 5, {}),
    "above_the_rule": (60, 100, 1.5e6, 0, 5, {}),
    "below_the_rule": (60, 200, 4e5, 0, 5, {}),
    "less_than_one_bin": (50, 300, 6e4, 0, 5, {"mask_positive": True}),
    "inclined": (99, 40, 1e6, 1, 5, {"include_minus_m": False}),
    "wide_n": (244, 25, 5e5, 0, 30, {}),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_fd_sum_matches_oracle(cuda, oracle, name):
    K, N, span, kmax, nmax, opts = CASES[name]
    inp, tr = S.fd_case(K=K, N=N, span=span, seed=71, lmax=3 if nmax < 30 else 2, kmax=kmax, nmax=nmax,
                        x=1.0 if kmax == 0 else 0.8, p_range=(12.0, 8.3), frequencies=frequencies)
    fk = frequencies(tr.M, tr.a, tr.p, tr.e, tr.xI)
    fd = FDInterpolatedModeSum(pad_output=True)
    num, pad = S.output_length(inp.t, inp.T, inp.dt, True, True)
    fd.num_pts, fd.num_pts_pad = num, pad
    want, freq, start, end = oracle.fd_sum(inp, fk, L=num + pad, **opts)
    got = {}
    for shape in (1, 2, 3):
        fd.sum_ctas_per_sm = shape
        fd.sum_with_frequencies(*inp.call_args(), fk, dt=inp.dt, **opts)
        torch.cuda.synchronize()
        got[shape] = fd.waveform.cpu().numpy()
    assert np.array_equal(fd.seg_start_inds.cpu().numpy(), start) and np.array_equal(fd.seg_end_inds.cpu().numpy(), end)
    bins = int(fd.total_bins.item())
    for shape, h in got.items():
        err = np.linalg.norm(h - want) / np.linalg.norm(want)
        print(f"\n{name}: {bins / (inp.num_modes * (N - 1)):.1f} bins a segment, shape {shape}: rel L2 {err:.2e}")
        assert err <= REL
