"""The operand ring of the tensor-core sum, a host rule (no GPU): two CTAs share an SM
wherever the accumulators and some ring of at least one A stage and two B slots let
them; a second A stage is taken only beside the second CTA; an asked shape is kept, and
one part of it never makes the other too large; and the autotuner's keys name the form
of the kernels they were timed on."""
import numpy as np
import pytest

from fastemriwaveforms_b200 import _lib, autotune

SM_SHARED = 228 * 1024   # shared memory of an SM (sm_100)
RESERVED = 1024          # per resident CTA, by the driver
MAX_DYNAMIC = 220 * 1024
TMEM_COLS = 512
A_STAGE = 16 * 1024      # 128 samples x 32 values, two BF16 planes


def ring(R, nchunks, astages=0, bstages=0):
    shape = np.zeros(5, np.int32)
    _lib.call("few_mixed_ring", R, nchunks, astages, bstages, shape.ctypes.data)
    nas, nbs, dyn, static, cols = shape.tolist()
    return nas, nbs, dyn, static, cols


def two_fit(dyn, static):
    return 2 * (dyn + static + RESERVED) <= SM_SHARED


def b_slot(R):
    return 2 * ((8 * R + 15) // 16 * 16) * 32 * 2


@pytest.mark.parametrize("nchunks", [0, 1, 2, 3, 4, 5])
def test_two_ctas_share_an_sm(nchunks):
    for R in range(1, 65):
        nas, nbs, dyn, static, cols = ring(R, nchunks)
        assert dyn == 2 * nas * A_STAGE + nbs * b_slot(R) <= MAX_DYNAMIC
        assert nas in (1, 2) and 2 <= nbs <= 4
        if 2 * cols > TMEM_COLS:
            continue  # one CTA per SM whatever the ring
        assert two_fit(dyn, static), (R, nchunks, nas, nbs, dyn)
        ahead = nchunks in (0, 3, 4) and two_fit(4 * A_STAGE + 2 * b_slot(R), static)
        assert nas == (2 if ahead else 1), (R, nchunks)
        if nbs < 4:  # no slot was left out that would have fitted
            assert not two_fit(dyn + b_slot(R), static), (R, nchunks)


def test_an_asked_shape_is_kept_and_one_part_leaves_room_for_the_other():
    for R in range(1, 65):
        for nchunks in range(6):
            for bstages in (2, 3, 4):
                for astages in (1, 2):
                    assert ring(R, nchunks, astages, bstages)[:2] == (astages, bstages)
                nas, nbs, dyn, _, _ = ring(R, nchunks, 0, bstages)
                assert nbs == bstages
                if ring(R, nchunks, 1, bstages)[2] <= MAX_DYNAMIC:
                    assert dyn <= MAX_DYNAMIC, (R, nchunks, bstages)
            for astages in (1, 2):
                assert ring(R, nchunks, astages, 0)[0] == astages


def test_tuned_choices_belong_to_the_form_of_the_kernels(monkeypatch):
    monkeypatch.setattr(autotune.torch.cuda, "get_device_name", lambda device: "B200")
    key = autotune.key_of(None, "mixed", 21, 61, 3000.0, 12)
    assert key.endswith(f"|v{autotune.KERNEL_FORM}")
    monkeypatch.setattr(autotune, "KERNEL_FORM", autotune.KERNEL_FORM + 1)
    assert autotune.key_of(None, "mixed", 21, 61, 3000.0, 12) != key
