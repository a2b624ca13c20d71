"""X lines of 513 to 1024 complex points (even Fx from 1080 to 2048): each 5-smooth
length has register kernels like the shorter ones, with every prologue and
epilogue.  Tolerance as in test_gpu_fft_lengths.py."""

import numpy as np
import pytest
import torch

from test_gpu_fft_lengths import TOL, D, check, half, rel, smooth  # noqa: F401

pytestmark = pytest.mark.gpu

LENGTHS = smooth(513, 1024)


def test_every_length_vs_fp64(D):  # noqa: F811
    bad = []
    for i, L in enumerate(LENGTHS):
        fft = (16, 18, 2 * L)
        c, x, err = check(D, tuple(half(f) for f in fft), fft, i)
        if not err < TOL:
            bad.append((fft, err))
        # a register kernel has one radix order: the schedule's odd radices first
        # would round differently on the runtime-radix passes
        y = c.forward(x)
        if not torch.equal(c.set_schedule(16).forward(x), y):
            bad.append((fft, "runtime radices"))
    assert not bad, bad


@pytest.mark.parametrize("L", LENGTHS)
def test_area_sums_and_crops_equal_the_operators(D, L):  # noqa: F811
    fft, shape = (16, 18, 2 * L), (6, 10, (L // 2) * 2)
    c, x, _ = check(D, shape, fft, L)
    down = D.FractionalAreaDownsample(2.0)
    A = D.compose(down, c)
    assert torch.equal(A.forward(x), down.forward(c.forward(x)))
    y = down.forward(x)
    assert torch.equal(A.adjoint(y), c.adjoint(down.adjoint(y)))
    crop = D.Crop(shape, (5, 7, L // 2 + 1), start=(1, 2, 3))
    B = D.compose(crop, c)
    z = crop.forward(x)
    assert torch.equal(B.forward(x), crop.forward(c.forward(x)))
    assert torch.equal(B.adjoint(z), c.adjoint(crop.adjoint(z)))


@pytest.mark.parametrize("L", [540, 625, 640, 768, 800, 900, 960, 1000, 1024])
def test_rl_epilogues_equal_the_operator_form(D, L):  # noqa: F811
    fft = (16, 18, 2 * L)
    shape = tuple(half(f) for f in fft)
    c, x, _ = check(D, shape, fft, 3)
    obs = torch.poisson(200 * x)
    a = D.richardson_lucy_with_operator(obs, c, num_iter=4, background=3.0, eval_interval=2)
    b = D.richardson_lucy_with_operator(obs, D.compose(D.Crop(shape, shape), c), num_iter=4, background=3.0,
                                        eval_interval=2)
    assert rel(a.restored, b.restored.double()) < 1e-6
    assert rel(a.pred, b.pred.double()) < 1e-6
    np.testing.assert_allclose(a.loss_history, b.loss_history, rtol=1e-6)
