"""The tensor-core sum with a tile written ahead of the previous one's epilogue (a stage
for every chunk of a tile: up to 2 chunks with one stage per producer half, up to 4 with
two) gives bitwise what it gives without, for 1 to 5 chunks of 16 n', units of one short
tile, of whole tiles and of a remainder, and waveforms of different chunk counts in turn."""
import numpy as np
import pytest
import torch

from fastemriwaveforms_b200 import InterpolatedModeSum
from fastemriwaveforms_b200 import synthetic as S
from fastemriwaveforms_b200.batched import BatchedInterpolatedModeSum

pytestmark = pytest.mark.gpu


def _wave(nmax, N, samples):
    span = (samples - 1) * 10.0
    return S.make_inputs(K=150, N=N, span=span, t_c=span * 1.05, lmax=4, nmax=nmax, seed=nmax, name=f"n{nmax}")


@pytest.mark.parametrize("chunk", [100, 128, 1024])
@pytest.mark.parametrize("nmaxs", [(7,), (15,), (23,), (31,), (35,), (31, 7, 35, 15)])
def test_ahead_gives_the_same_bits(cuda, chunk, nmaxs):
    waves = [_wave(n, 6, 9000 + 77 * n) for n in nmaxs]
    ref = None
    for astages in (1, 2):
        b = BatchedInterpolatedModeSum(precision="mixed", chunk=chunk, ctas_per_sm=2, astages=astages,
                                       bstages=2).setup(waves)
        outs = [o.cpu().numpy() for o in b.forward()]
        torch.cuda.synchronize()
        assert not b.mixed_error()
        ref = ref or outs
        assert all(np.array_equal(x, y) for x, y in zip(ref, outs))
    for inp, got in zip(waves, ref):
        ims = InterpolatedModeSum(precision="mixed", chunk=chunk)
        assert np.array_equal(ims(*inp.call_args(), T=inp.T, dt=inp.dt).cpu().numpy(), got)
        assert not ims.mixed_error()
