"""The FP64 sum's row blocks against the CPU oracle: every number of rows up to two
full blocks and one more of either form (blocks of one row to seven, of equal and
unequal size), one column and many, k' != 0 rows, and so many columns that the row
blocks go through shared memory in several passes; the batched form of each equal to
the single one to the last bit.  Tolerances as in test_gpu_sum.py."""
import numpy as np
import pytest
import torch

from fastemriwaveforms_b200 import InterpolatedModeSum
from fastemriwaveforms_b200 import synthetic as S
from fastemriwaveforms_b200.batched import BatchedInterpolatedModeSum

pytestmark = pytest.mark.gpu

TOL = 1e-12


def case(rows, nmax, theta, out_len=700, seed=3):
    """Modes whose fold has `rows` (m', k') rows: m = 0 gives one, each (m > 0, k) two."""
    base = S.small_case(K=4, N=6, out_len=out_len, seed=seed, theta=theta)
    rng = np.random.default_rng(seed + rows)
    mk = [(0, 0)] if rows % 2 else []
    mk += [(1 + q // (2 if theta else 1), q % 2 if theta else 0) for q in range(rows // 2)]
    ns = sorted({-nmax, nmax} | set(rng.integers(-nmax, nmax + 1, 3).tolist()))
    modes = np.array([(max(2, m), m, k, n) for m, k in mk for n in ns], np.int32)
    l, m, k, n = (np.ascontiguousarray(modes[:, i]) for i in range(4))
    K = len(modes)
    frac = (base.t / base.t[-1])[:, None]
    lo, hi = rng.uniform(-1, 1, (2, 2, K))
    teuk = (lo[0] + (hi[0] - lo[0]) * frac) + 1j * (lo[1] + (hi[1] - lo[1]) * frac)
    ylms = rng.standard_normal(2 * K) + 1j * rng.standard_normal(2 * K)
    return S.ModeSumInputs(t=base.t, teuk_modes=np.ascontiguousarray(teuk), ylms=ylms, phase_t=base.t.copy(),
                           phase_coeffs=base.phase_coeffs, l=l, m=m, k=k, n=n, dt=base.dt, T=base.T)


def check(oracle, inp, rows):
    for precision in ("faithful", "exact"):
        ims = InterpolatedModeSum(precision=precision)
        got = ims(*inp.call_args(), T=inp.T, dt=inp.dt)
        assert ims._last_plan[0].R == rows
        want = oracle.mode_sum(inp, extended=precision == "exact")
        err = np.linalg.norm(got.cpu().numpy() - want) / np.linalg.norm(want)
        assert err < TOL, (precision, rows, err)
        batch = BatchedInterpolatedModeSum(precision=precision, autotune=False).setup([inp, inp])
        for out in batch.forward():
            assert torch.equal(out, got), precision


@pytest.mark.parametrize("rows", list(range(1, 17)) + [21, 22])
@pytest.mark.parametrize("nmax", [0, 5])
def test_row_counts(cuda, oracle, rows, nmax):
    check(oracle, case(rows, nmax, theta=False), rows)


@pytest.mark.parametrize("rows", [2, 7, 12, 13, 15])
def test_row_counts_with_theta(cuda, oracle, rows):
    check(oracle, case(rows, 4, theta=True), rows)


@pytest.mark.parametrize("rows,nmax", [(8, 199), (15, 120), (9, 215)])
def test_several_passes(cuda, oracle, rows, nmax):
    check(oracle, case(rows, nmax, theta=False, out_len=520), rows)
