"""The FP64 sum's split of (m, k) rows into blocks (a host rule, and the persistent
kernel's loop counts): every pass takes at least one block, as many as the shared memory
surely holds, whatever the number of columns; only when not one row fits are there no
blocks, and then the calls are refused.  On a GPU: column counts at which one block of
the usual size does not fit, against the CPU oracle."""
import numpy as np
import pytest

from fastemriwaveforms_b200 import _lib

BUDGET = 200 * 1024
ROWS = {_lib.FEW_SUM_FAITHFUL: 7, _lib.FEW_SUM_EXACT: 6}  # rows of a block at most


def blocks_of(R, NN, smem, mode):
    out = np.full(2, -1, np.int32)
    _lib.call("few_sum_row_blocks", R, NN, smem, mode, out.ctypes.data)
    return out.tolist()


@pytest.mark.parametrize("mode", sorted(ROWS))
def test_every_pass_takes_a_block_that_fits(mode):
    for NN in [1, 2, 61, 399, 400, 401, 457, 458, 533, 534, 600, 640, 641, 800, 801, 1000, 1067, 1600, 1601, 3199, 3200]:
        for R in [1, 2, 4, 5, 6, 7, 8, 9, 12, 13, 14, 15, 21, 43, 64, 255, 256]:
            for smem in {BUDGET, min(BUDGET, (R + 7) // 8 * 8 * NN * 64)}:
                nblk, per_pass = blocks_of(R, NN, smem, mode)
                edges = [b * R // nblk for b in range(nblk + 1)]
                sizes = np.diff(edges)
                assert sizes.min() >= 1 and sizes.max() <= ROWS[mode] and sizes.max() - sizes.min() <= 1
                assert 1 <= per_pass <= nblk
                for b in range(0, nblk, per_pass):
                    rows = edges[min(b + per_pass, nblk)] - edges[b]
                    assert rows * NN * 64 <= smem, (R, NN, smem)
                if R * NN * 64 <= smem:  # one pass, in the fewest blocks
                    assert per_pass == nblk == -(-R // ROWS[mode])


@pytest.mark.parametrize("mode", sorted(ROWS))
def test_no_blocks_when_no_row_fits(mode):
    assert blocks_of(5, 3201, BUDGET, mode) == [0, 0]
    assert blocks_of(5, 61, 61 * 64 - 1, mode) == [0, 0]
    dummy = np.zeros(1)
    with pytest.raises(ValueError, match="NN=3201 too large"):
        _lib.call("few_sum_folded", *[dummy.ctypes.data] * 3, 10, *[dummy.ctypes.data] * 2, 1, *[dummy.ctypes.data] * 2, 5,
                  0, 3201, 10.0, mode, 0, None)


@pytest.mark.gpu
@pytest.mark.parametrize("rows,nmax", [(5, 300), (6, 290), (9, 300), (7, 229), (9, 460)])
def test_wide_column_ranges(cuda, oracle, rows, nmax):
    import torch

    from fastemriwaveforms_b200 import InterpolatedModeSum
    from fastemriwaveforms_b200.batched import BatchedInterpolatedModeSum
    from test_gpu_sum_rows import TOL, case

    inp = case(rows, nmax, theta=False, out_len=300)
    for precision in ("faithful", "exact"):
        ims = InterpolatedModeSum(precision=precision)
        got = ims(*inp.call_args(), T=inp.T, dt=inp.dt)
        assert ims._last_plan[0].R == rows and ims._last_plan[0].NN == 2 * nmax + 1
        want = oracle.mode_sum(inp, extended=precision == "exact")
        assert np.linalg.norm(got.cpu().numpy() - want) / np.linalg.norm(want) < TOL
        for out in BatchedInterpolatedModeSum(precision=precision, autotune=False).setup([inp, inp]).forward():
            assert torch.equal(out, got), precision


@pytest.mark.gpu
def test_batch_refuses_what_does_not_fit(cuda):
    from fastemriwaveforms_b200.batched import BatchedInterpolatedModeSum
    from test_gpu_sum_rows import case

    inp = case(2, 1600, theta=False, out_len=300)
    for precision in ("faithful", "exact"):
        with pytest.raises(ValueError, match="3200"):
            BatchedInterpolatedModeSum(precision=precision, autotune=False).setup([inp])
