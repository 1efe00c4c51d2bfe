"""The Bessel combinations that k_aak interpolates over a CTA's range of e, against the
recurrence it runs per sample where e moves too far: the same trajectory sampled at dt
(6, 8 or 12 nodes) and at 2^k dt (the recurrence), compared at the common samples, whose
times, phases and orientations are formed from the same bits.

Tolerance: a recurrence value at fl(n e) errs by about n 2^-53 of itself for each of the
two roundings of the argument, so two values by at most 2 nmodes 2^-52, of the largest
sample."""
import numpy as np
import pytest

from fastemriwaveforms_b200 import AAKSummation
from fastemriwaveforms_b200 import synthetic as S

pytestmark = pytest.mark.gpu

# samples (one a thread, 128 to a CTA), e range, nmodes, nodes, k
CASES = {
    "six": (32769, (0.6, 0.45), 18, 6, 10),
    "six_low": (32769, (0.4, 0.2), 9, 6, 10),
    "eight": (4097, (0.6, 0.50), 18, 8, 7),
    "eight_24": (8193, (0.5, 0.30), 24, 8, 8),
    "twelve": (2049, (0.6, 0.35), 24, 12, 6),
    "twelve_low": (2049, (0.45, 0.2), 18, 12, 6),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_interpolated_values_match_the_recurrence(cuda, name):
    samples, e, nmodes, nodes, k = CASES[name]
    dt = 4.0
    half = nmodes * (e[0] - e[1]) / (samples - 1) * 127 / 2  # n times the half width of e over a CTA's samples
    assert nodes == (6 if half <= 7.8e-3 else 8 if half <= 0.052 else 12) and half <= 0.38
    assert (samples - 1) >> k < 128 and nmodes * (e[0] - e[1]) / 2 > 0.38
    inp = S.aak_case(N=30, span=(samples - 1) * dt, seed=7, e_range=e, nmodes=nmodes, dt=dt)
    fine = AAKSummation()(*inp.call_args(), mich=False, T=inp.T, dt=dt).cpu().numpy()
    step = 1 << k
    T = ((samples - 1) * dt + step * dt) / S.YRSID_SI
    coarse = AAKSummation()(*inp.call_args(), mich=False, T=T, dt=dt * step).cpu().numpy()
    fine = fine[::step]
    n = min(len(fine), len(coarse)) - 1
    assert n >= 31
    err = np.abs(fine[:n] - coarse[:n]).max() / np.abs(coarse).max()
    print(f"\n{name}: {err:.2e} (tolerance {2 * nmodes * 2.0**-52:.1e})")
    assert err <= 2 * nmodes * 2.0**-52
