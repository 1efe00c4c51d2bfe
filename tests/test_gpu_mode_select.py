"""The mode selection's kernels against numpy in the same order of operations, so
equal to the last bit: the power estimates at the edges of a tile of knots and of a
warp of modes, with and without weights; the order with ties, zeros of both signs,
NaN and infinities; the kept modes, their harmonics' indices and ranks, up to the
longest list the kernel takes."""
import numpy as np
import pytest
import torch

from fastemriwaveforms_b200 import _lib
from fastemriwaveforms_b200.summation import _ptr, _stream

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [1, 2, 72, 73, 74, 145, 217])
@pytest.mark.parametrize("K", [1, 31, 32, 33, 70])
def test_power_estimates(cuda, N, K):
    rng = np.random.default_rng(100 * N + K)
    teuk = rng.standard_normal((N, K)) + 1j * rng.standard_normal((N, K))
    ylms = rng.standard_normal(2 * K) + 1j * rng.standard_normal(2 * K)
    minus = np.where(rng.random(K) < 0.3, -1, K + np.arange(K)).astype(np.int32)
    t = np.cumsum(rng.uniform(0.5, 2.0, N))
    psd = rng.uniform(0.5, 2.0, (N, K))
    dev = {k: torch.tensor(v, device=cuda) for k, v in (("A", teuk), ("y", ylms), ("i", minus), ("t", t), ("p", psd))}
    for weighted in (False, True):
        got = torch.empty(K, dtype=torch.float64, device=cuda)
        _lib.call("few_mode_snr2", _ptr(dev["A"]), N, K, _ptr(dev["y"]), _ptr(dev["i"]),
                  _ptr(dev["p"]) if weighted else None, _ptr(dev["t"]), _ptr(got), _stream(cuda))

        def power(a, b):  # |a b|^2 with the product's parts rounded one by one
            z = torch.hypot(a.real * b.real - a.imag * b.imag, a.real * b.imag + a.imag * b.real)
            return z * z

        A = dev["A"]
        p = power(A, dev["y"][:K])
        ym = dev["y"][dev["i"].clamp(min=0).long()]
        p = torch.where(dev["i"] >= 0, p + power(torch.conj_physical(A), ym), p)
        if weighted:
            p = p / dev["p"]
        want = torch.zeros(K, dtype=torch.float64, device=cuda)
        for n in range(N - 1):
            want = want + p[n] * (dev["t"][n + 1] - dev["t"][n])
        assert torch.equal(got, want), (weighted, (got - want).abs().max())


def reference(snr, threshold, m0, m1):
    """numpy's stable descending order with NaN first, the keep rule, the kept modes."""
    v = np.where(np.isnan(snr), np.inf, snr)
    order = np.lexsort((np.arange(len(snr)), -v, ~np.isnan(snr)))
    run = np.cumsum(snr[order])
    with np.errstate(invalid="ignore"):
        keep = np.concatenate([[True], run[:-1] < run[-1] * ((1.0 - threshold) * (1.0 - threshold))])
    kept = np.sort(order[keep])
    rank = np.searchsorted(kept, order[keep])
    return kept, np.concatenate([kept, np.where(kept < m0, kept, kept + m1)]), rank


@pytest.mark.parametrize("K", [1, 2, 3, 31, 33, 1023, 1025, 3843, 8192])
@pytest.mark.parametrize("kind", ["spread", "ties", "zeros", "special", "negative"])
def test_selection(cuda, K, kind):
    rng = np.random.default_rng(K)
    snr = np.exp(rng.uniform(-12, 0, K))
    if kind == "ties":
        snr = np.round(snr * 8) / 8 + 0.125
    if kind == "zeros":
        snr[rng.random(K) < 0.5] = 0.0
        snr[rng.random(K) < 0.2] = -0.0
    if kind == "special" and K > 2:
        snr[K // 2] = np.nan
        snr[K // 3] = np.inf
    if kind == "negative":  # sums that fall again: the rule then keeps no prefix
        snr[rng.random(K) < 0.4] *= -1.0
    m0, m1 = K // 4, K - K // 4
    d = torch.tensor(snr, device=cuda)
    for threshold in (1e-5, 1e-2, 0.5):
        buf = torch.full((6, K), -7, dtype=torch.int64, device=cuda)
        count = torch.zeros(1, dtype=torch.int32, device=cuda)
        _lib.call("few_mode_select", _ptr(d), K, threshold, m0, m1, _ptr(buf[4]), _ptr(buf[0]), _ptr(buf[1]),
                  _ptr(buf[3]), _ptr(count), _stream(cuda))
        kept, ylm, rank = reference(snr, threshold, m0, m1)
        c = int(count.item())
        assert c == len(kept)
        assert np.array_equal(buf[0, :c].cpu().numpy(), kept)
        assert np.array_equal(buf[1:3].reshape(-1)[:2 * c].cpu().numpy(), ylm)
        assert np.array_equal(buf[3, :c].cpu().numpy(), rank)


def test_limits(cuda):
    K = _lib.load().few_mode_select_max()
    buf = torch.zeros((6, K + 1), dtype=torch.int64, device=cuda)
    for bad in (0, K + 1):
        with pytest.raises(ValueError):
            _lib.call("few_mode_select", _ptr(buf), bad, 0.1, 0, 0, _ptr(buf), _ptr(buf), _ptr(buf), _ptr(buf),
                      _ptr(buf), _stream(cuda))
