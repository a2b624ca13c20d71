"""The autotuner's choice without a GPU: a fake plan says which schedule bits
matter, a fake clock how long each schedule takes."""

import json

import numpy as np
import pytest

from deconlib_b200 import batch

FUSED, NO_PIPE, NO_TMA, LEAN_OFF, ODD, HALF = 1, 2, 4, 8, 16, 32


class FakeConv:
    bits = FUSED | NO_TMA

    def __init__(self, psf, sig, fft_shape=None):
        self.fft_shape, self.sched = fft_shape, 0

    def set_schedule(self, s):
        self.sched = s

    @property
    def fused_yz(self):
        return bool(self.sched & self.bits & FUSED)

    @property
    def schedule_bits(self):
        return self.bits


@pytest.fixture
def tuner(monkeypatch, tmp_path):
    class X:
        def fill_(self, v):
            pass

    timed = []
    cost = {}

    def clock(conv, x, reps):
        timed.append((conv.fft_shape, conv.sched))
        return cost.get(conv.sched, 1.0)

    monkeypatch.setenv("DECON_AUTOTUNE_CACHE", str(tmp_path / "tune.json"))
    monkeypatch.setattr(batch, "_TUNED", {})
    monkeypatch.setattr(batch, "_CACHE_LOADED", False)
    monkeypatch.setattr(batch, "_device_tag", lambda: "fake")
    monkeypatch.setattr(batch, "empty", lambda s: X())
    monkeypatch.setattr(batch, "LinearFFTConvolver", FakeConv)
    monkeypatch.setattr(batch, "_time_pair", clock)
    return timed, cost, tmp_path / "tune.json"


PSF, SIG, CANVAS = np.zeros((3, 5, 5), np.float32), (30, 60, 50), (32, 64, 54)


@pytest.mark.parametrize("bits,want", [(0, [0]), (NO_TMA, [0, NO_TMA]), (FUSED | NO_TMA, [0, FUSED, NO_TMA]),
                                       (ODD | HALF, [0, ODD, HALF])])
def test_each_family_is_timed_once(tuner, monkeypatch, bits, want):
    timed, cost, _ = tuner
    monkeypatch.setattr(FakeConv, "bits", bits)
    assert batch.autotune_schedule(SIG, PSF, [CANVAS]) == (CANVAS, 0)
    assert [s for _, s in timed] == want


def test_default_unless_clearly_slower(tuner):
    timed, cost, _ = tuner
    cost[NO_TMA] = 0.99  # within the scatter of a timing
    assert batch.autotune_schedule(SIG, PSF, [CANVAS]) == (CANVAS, 0)
    batch._TUNED.clear()
    cost[FUSED] = 0.9
    assert batch.autotune_schedule(SIG, PSF, [CANVAS]) == (CANVAS, FUSED)


def test_choices_of_other_kernels_are_not_used(tuner, monkeypatch):
    timed, cost, path = tuner
    old = {"fft_shape": [64, 64, 64], "schedule": NO_PIPE, "ms": 0.1}
    path.write_text(json.dumps({f"fake|{SIG}|{PSF.shape}": old}))
    assert batch.autotune_schedule(SIG, PSF, [CANVAS]) == (CANVAS, 0)
    n = len(timed)
    assert n > 0
    # the new choice is read back, and not under the next kernels
    monkeypatch.setattr(batch, "_TUNED", {})
    monkeypatch.setattr(batch, "_CACHE_LOADED", False)
    assert batch.autotune_schedule(SIG, PSF, [CANVAS]) == (CANVAS, 0) and len(timed) == n
    monkeypatch.setattr(batch, "TUNE_KERNELS", batch.TUNE_KERNELS + 1)
    batch.autotune_schedule(SIG, PSF, [CANVAS])
    assert len(timed) == 2 * n
