"""The autotuner and shapes that the library refuses (no GPU): they are left out, the best of
the others is kept, and only when every shape is refused does the refusal reach the caller.
On a GPU: a tensor-core batch of more (m, k) rows than the widest ring holds, set up with
the default tuning."""
import pytest

from fastemriwaveforms_b200 import autotune


def test_refused_shapes_are_left_out(tmp_path, monkeypatch):
    monkeypatch.setenv("FEW_B200_TUNE_CACHE", str(tmp_path / "tune.json"))
    monkeypatch.setattr(autotune, "time_ms", lambda fn, reps=3: fn())

    def runner(bstages):
        def run():
            if bstages > 2:
                raise ValueError(f"{bstages} B stages exceed shared memory")
            return float(bstages)
        return run

    shapes = [{"bstages": b} for b in (4, 2, 3)]
    choice = autotune.tune("k", runner, shapes)
    assert choice["bstages"] == 2 and len(choice["tried"]) == 1
    with pytest.raises(ValueError, match="exceed shared memory"):
        autotune.tune("k", runner, [{"bstages": 3}, {"bstages": 4}])


@pytest.mark.gpu
def test_many_rows_are_tuned(cuda, tmp_path, monkeypatch):
    import torch

    from fastemriwaveforms_b200 import InterpolatedModeSum
    from fastemriwaveforms_b200.batched import BatchedInterpolatedModeSum
    from test_gpu_sum_rows import case

    monkeypatch.setenv("FEW_B200_TUNE_CACHE", str(tmp_path / "tune.json"))
    inp = case(63, 5, theta=True)
    batch = BatchedInterpolatedModeSum(precision="mixed").setup([inp])
    assert batch.max_R == 63 and 0 < len(batch.tuning["tried"]) < 24
    want = InterpolatedModeSum(precision="mixed")(*inp.call_args(), T=inp.T, dt=inp.dt)
    assert torch.equal(batch.forward()[0], want) and not batch.mixed_error()
