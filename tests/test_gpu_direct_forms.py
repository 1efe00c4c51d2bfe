"""Both lane splits of the direct mode sum (8 lanes per sample; 32 for few samples of
many modes) against the sum in numpy, at the edges of a block's samples, of a lane's modes
and of the rule between the splits, with phases above 2^30 and non-finite ones.

The bound, per sample: each term's products and phasor lie within 8 roundings of 2^-53 on
either side and a sum of 2 K terms within 2 K more, so 2 (2 K + 8) 2^-53 sum |Y| |A|."""
import numpy as np
import pytest
import torch

from fastemriwaveforms_b200 import DirectModeSum

pytestmark = pytest.mark.gpu


def _case(T, K, scale):
    rng = np.random.default_rng(T + 1000 * K)
    A = rng.standard_normal((T, K)) + 1j * rng.standard_normal((T, K))
    y = rng.standard_normal(2 * K) + 1j * rng.standard_normal(2 * K)
    phases = rng.uniform(-scale, scale, (3, T))
    l, m = rng.integers(2, 7, K), rng.integers(0, 4, K)
    k, n = rng.integers(-2, 3, K), rng.integers(-9, 10, K)
    return A, y, phases, l, m, k, n


def _numpy(A, y, phases, l, m, k, n):
    K = len(l)
    P = phases[:, :, None]
    ph = (m * P[0] + k * P[1]) + n * P[2]
    e = np.cos(ph) - 1j * np.sin(ph)
    ym = y[K:] * np.where(l % 2 == 0, 1.0, -1.0) * (m > 0)
    b = A * e
    size = ((np.abs(y[:K]) + np.abs(ym)) * np.abs(A)).sum(axis=1)
    return (y[:K] * b).sum(axis=1) + (ym * b.conj()).sum(axis=1), 2 * (2 * K + 8) * 2.0**-53 * size


@pytest.mark.parametrize("T,K", [(2, 1), (2, 33), (31, 8), (32, 9), (33, 7), (7, 64), (4095, 65), (11999, 33),
                                 (12000, 33), (12001, 32)])
@pytest.mark.parametrize("scale", [1e3, 3e8])
def test_against_numpy(cuda, T, K, scale):
    x = _case(T, K, scale)
    t = np.arange(T) * 10.0
    A, y, phases, *modes = x
    got = DirectModeSum()(t, A, y, t, phases, *modes).cpu().numpy()
    want, bound = _numpy(*x)
    assert np.all(np.abs(got - want) <= bound)


@pytest.mark.parametrize("T,K", [(50, 5), (50, 40)])
def test_non_finite_phase_stays_in_its_sample(cuda, T, K):
    A, y, phases, *modes = _case(T, K, 1e3)
    phases[0, 17], phases[2, 30] = np.inf, np.nan
    modes[1][0] = 1
    t = np.arange(T) * 10.0
    got = DirectModeSum()(t, A, y, t, torch.as_tensor(phases), *modes).cpu().numpy()
    phases[0, 17] = phases[2, 30] = 0.0
    want, bound = _numpy(A, y, phases, *modes)
    bad = np.isin(np.arange(T), (17, 30))
    assert np.isnan(got[bad]).all()
    assert np.all(np.abs(got - want)[~bad] <= bound[~bad])
