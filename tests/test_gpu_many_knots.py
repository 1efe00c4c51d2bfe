"""Trajectories of very many knots with few modes: more pairs of segments than one
dimension of a grid takes beside its first (65,535), which the fold from slopes has to
cover as the fold of coefficients does, to the last bit."""
import numpy as np
import pytest
import torch

from fastemriwaveforms_b200 import _lib
from fastemriwaveforms_b200.summation import _ptr, _stream, spline_factor_table

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nseg", [2 * 65535, 2 * 65535 + 1, 200_001])
@pytest.mark.parametrize("R,NN", [(1, 1), (3, 45)])
def test_fold_of_many_segments(cuda, nseg, R, NN):
    N, K = nseg + 1, 2
    rng = np.random.default_rng(nseg)
    t = np.cumsum(rng.uniform(0.5, 1.5, N))
    fac = spline_factor_table(t, cuda)
    teuk = torch.tensor(rng.standard_normal((N, K)) + 1j * rng.standard_normal((N, K)), device=cuda)
    ylm = torch.tensor(rng.standard_normal(2 * K) + 1j * rng.standard_normal(2 * K), device=cuda)
    keys = R * NN
    ptr = np.zeros(keys + 1, np.int32)
    ptr[1:] = 2  # both modes' + terms on the first key, their - terms on the last
    ptr[keys] = 4
    ptr_d, lst_d = torch.tensor(ptr, device=cuda), torch.tensor(np.array([0, 2, 1, 3], np.int32), device=cuda)
    st = _stream(cuda)
    co = torch.empty(4, N, 2 * K, dtype=torch.float64, device=cuda)
    _lib.call("few_spline_build_factored", _ptr(fac), _ptr(teuk), 2 * K, 2, K, 1, 2 * K, N, _ptr(co),
              _lib.FEW_LAYOUT_KNOT_MAJOR, st)
    s = torch.empty(N, 2 * K, dtype=torch.float64, device=cuda)
    _lib.call("few_spline_slopes", _ptr(fac), _ptr(teuk), 2 * K, N, _ptr(s), st)
    a, b = (torch.full((nseg, keys, 4), float("nan"), dtype=torch.complex128, device=cuda) for _ in range(2))
    _lib.call("few_fold_coeffs", _ptr(co), _ptr(ylm), _ptr(ptr_d), _ptr(lst_d), K, N, nseg, R, NN, _ptr(a), st)
    _lib.call("few_fold_slopes", _ptr(teuk), _ptr(s), _ptr(fac), _ptr(ylm), _ptr(ptr_d), _ptr(lst_d), K, N, nseg, R,
              NN, _ptr(b), st)
    assert torch.equal(a, b)
