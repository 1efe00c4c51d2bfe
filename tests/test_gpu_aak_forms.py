"""k_aak's forms against the numpy restatement (scipy's Bessel functions): one and
several samples a thread, with and without the response; 6, 8 and 12 interpolation
nodes and the recurrence per sample (e still, slow, fast and very fast over a CTA);
one harmonic, odd counts, one group of 24 and one more; circular orbits; phases
past the first-order rounding factor.

Tolerance: the two sides evaluate Phi_r in other operations and so differ by its
last place, which harmonic n multiplies by n; the harmonics' rounded phases are
formed alike.  2 nmodes ulp(Phi_max) + 1e-13 bounds the relative L2 difference."""
import numpy as np
import pytest
import torch

from fastemriwaveforms_b200 import AAKSummation
from fastemriwaveforms_b200 import synthetic as S

pytestmark = pytest.mark.gpu

# N, samples, dt, e range, nmodes, mich, f0
CASES = {
    "still_e": (12, 3000, 10.0, (0.3, 0.3), 9, False, 1.5e-3),
    "six_nodes": (20, 20011, 10.0, (0.5, 0.45), 18, False, 1.5e-3),
    "eight_nodes": (20, 5003, 10.0, (0.5, 0.45), 18, True, 1.5e-3),
    "twelve_nodes": (20, 2001, 10.0, (0.6, 0.35), 24, False, 1.5e-3),
    "recurrence": (20, 300, 10.0, (0.7, 0.05), 24, True, 1.5e-3),
    "one_harmonic": (10, 1000, 10.0, (0.2, 0.1), 1, False, 1.5e-3),
    "one_group": (10, 2000, 10.0, (0.6, 0.5), 24, False, 1.5e-3),
    "group_and_one": (10, 2000, 10.0, (0.6, 0.5), 25, True, 1.5e-3),
    "three_groups": (10, 1200, 10.0, (0.6, 0.5), 51, False, 1.5e-3),
    "circular": (10, 1500, 10.0, (0.0, 0.0), 5, False, 1.5e-3),
    "four_a_thread": (50, 151_553, 1.0, (0.4, 0.3), 3, False, 1.5e-3),
    "two_a_thread": (50, 151_553, 1.0, (0.4, 0.3), 3, True, 1.5e-3),
    "long_phases": (12, 1000, 10.0, (0.4, 0.3), 20, False, 4e1),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_aak_forms_match_oracle(cuda, oracle, name):
    N, samples, dt, e, nmodes, mich, f0 = CASES[name]
    inp = S.aak_case(N=N, span=(samples - 1) * dt, seed=81, e_range=e, nmodes=nmodes, dt=dt, f0=f0)
    got = AAKSummation()(*inp.call_args(), mich=mich, T=inp.T, dt=dt)
    torch.cuda.synchronize()
    got = got.cpu().numpy()
    want = oracle.aak_waveform(inp.t, inp.interp_coeffs, inp.m1, inp.a, inp.m2, inp.qS, inp.phiS, inp.qK, inp.phiK,
                               inp.dist, inp.nmodes, mich, len(got), dt)
    tol = 2 * nmodes * np.spacing(np.abs(inp.interp_coeffs[:, 5, 0]).max()) + 1e-13
    err = np.linalg.norm(got - want) / np.linalg.norm(want)
    print(f"\n{name}: rel L2 {err:.2e} (tolerance {tol:.1e})")
    assert err <= tol
