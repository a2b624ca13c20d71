"""Schedules of a convolution plan other than the default one.

A schedule changes which kernels run and how many rows or columns a CTA takes,
so per-row values keep their bits wherever the kernels are the same, and sums
over a volume change by the order of their FP64 additions only.
"""

import os
import subprocess
import sys

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

FUSED, NO_TMA, HALF_LINES = 1, 4, 32


@pytest.fixture(scope="module")
def D():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import deconlib_b200.deconvolution as d

    return d


# X lines of the runtime-radix pass with four, two and one row per CTA.  Half the
# lines mean twice the CTAs (1200, 1600 and 1400), each with a loss partial of its
# own: more than the 1184 that every plan holds.
@pytest.mark.parametrize("sig,fft", [((8, 300, 1030), (8, 320, 2100)), ((4, 400, 2100), (4, 400, 4200)),
                                     ((4, 350, 4200), (4, 350, 8400))])
def test_loss_under_half_lines(D, sig, fft):
    rng = np.random.default_rng(5)
    psf = rng.random((1, 1, 5)).astype(np.float32)
    obs = rng.poisson(20.0, sig).astype(np.float32)
    runs = []
    for sched in (0, HALF_LINES):
        conv = D.LinearFFTConvolver(psf, sig, fft_shape=fft, schedule=sched)
        runs.append(D.richardson_lucy_with_operator(obs, conv, num_iter=2, background=1.0, eval_interval=1))
    a, b = runs
    assert torch.equal(a.restored, b.restored)
    # 6e6 terms of one sign in another order: below 6e6 eps64 of the sum
    assert len(a.loss_history) == 2
    np.testing.assert_allclose(a.loss_history, b.loss_history, rtol=1e-9)


FIRST_PLANS = """
import threading
import numpy as np, torch
import deconlib_b200.deconvolution as D

psf = np.random.default_rng(0).random((5, 9, 9)).astype(np.float32)
x = torch.rand((40, 100, 90), device="cuda")
torch.cuda.synchronize()
gate, plans = threading.Barrier(12), [None] * 12

def make(i):
    gate.wait()
    plans[i] = D.LinearFFTConvolver(psf, (40, 100, 90))

threads = [threading.Thread(target=make, args=(i,)) for i in range(12)]
for t in threads:
    t.start()
for t in threads:
    t.join()
y = D.LinearFFTConvolver(psf, (40, 100, 90)).forward(x)
assert all(torch.equal(p.forward(x), y) for p in plans)
"""


def test_first_plans_of_a_process_by_several_threads(D):
    # every thread's plan gets the kernels of a plan made alone: the same bits
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    for _ in range(3):
        subprocess.run([sys.executable, "-c", FIRST_PLANS], check=True, timeout=120, cwd=root)


# tiles of 16 and 8 columns, whole and with planes side by side, one plane, short
# and 1024-point axes, and a 7-smooth one (runtime radices on every schedule)
@pytest.mark.parametrize("sig,fft", [((20, 40, 60), (40, 80, 120)), ((8, 9, 9), (16, 18, 18)), ((70, 180, 33), (135, 360, 64)),
                                     ((1, 300, 100), (1, 600, 200)), ((5, 30, 500), (10, 60, 1000)),
                                     ((3, 500, 30), (16, 1024, 48)), ((500, 9, 30), (1000, 18, 50)), ((10, 20, 30), (20, 42, 60))])
def test_plain_loads_give_the_same_bits(D, monkeypatch, sig, fft):
    rng = np.random.default_rng(1)
    psf = rng.random(tuple(f - n + 1 for n, f in zip(sig, fft))).astype(np.float32)
    x = torch.from_numpy(rng.random(sig).astype(np.float32)).cuda()
    c = D.LinearFFTConvolver(psf, sig, fft_shape=fft)
    y, z = c.forward(x), c.adjoint(x)
    c.set_schedule(NO_TMA)
    assert torch.equal(c.forward(x), y) and torch.equal(c.adjoint(x), z)
    monkeypatch.setenv("DECON_NO_TMA", "1")
    p = D.LinearFFTConvolver(psf, sig, fft_shape=fft)
    assert torch.equal(p.otf, c.otf)
    assert torch.equal(p.forward(x), y) and torch.equal(p.adjoint(x), z)


# X lines with a kx-major kernel of their own, and others (runtime radices)
@pytest.mark.parametrize("L", [64, 80, 96, 128, 160, 192, 240, 256, 320, 384, 480, 512, 640, 768, 960, 1024, 50, 63, 600])
def test_fused_pass_at_every_x_length(D, L):
    # FP32 transforms of the same canvas, factored differently: twice the 1e-6
    # that the repository allows each of them against FP64
    sig, fft = (5, 18, L // 2 * 2), (128, 256, 2 * L)
    rng = np.random.default_rng(L)
    psf = rng.random((9, 31, L // 2)).astype(np.float32) ** 4
    x = torch.from_numpy(rng.random(sig).astype(np.float32)).cuda()
    c0 = D.LinearFFTConvolver(psf, sig, fft_shape=fft)
    c = D.LinearFFTConvolver(psf, sig, fft_shape=fft, schedule=FUSED)
    assert c.fused_yz
    rel = lambda a, b: float((a.double() - b.double()).norm() / b.double().norm())  # noqa: E731
    assert rel(c.forward(x), c0.forward(x)) < 2e-6 and rel(c.adjoint(x), c0.adjoint(x)) < 2e-6
    # the same plan's epilogues and windows are the operators in turn, bit for bit
    crop = D.Crop(sig, (3, 7, L // 2 + 1), start=(1, 2, 3))
    A = D.compose(crop, c)
    z = crop.forward(x)
    assert torch.equal(A.forward(x), crop.forward(c.forward(x)))
    assert torch.equal(A.adjoint(z), c.adjoint(crop.adjoint(z)))
    obs = torch.poisson(100 * x)
    a = D.richardson_lucy_with_operator(obs, c, num_iter=3, background=2.0, eval_interval=1)
    b = D.richardson_lucy_with_operator(obs, c0, num_iter=3, background=2.0, eval_interval=1)
    assert rel(a.restored, b.restored) < 1e-5  # as test_gpu_yz.py allows RL
    np.testing.assert_allclose(a.loss_history, b.loss_history, rtol=1e-6)


@pytest.mark.parametrize("L", [64, 80, 240, 256, 640, 1024, 50])
def test_fused_area_sum_at_x_lengths(D, L):
    sig, fft = (6, 32, L // 2 * 2), (128, 256, 2 * L)
    rng = np.random.default_rng(L)
    c = D.LinearFFTConvolver(rng.random((9, 31, L // 2)).astype(np.float32), sig, fft_shape=fft, schedule=FUSED)
    down = D.FractionalAreaDownsample(2.0)
    A = D.compose(down, c)
    x = torch.from_numpy(rng.random(sig).astype(np.float32)).cuda()
    y = down.forward(x)
    assert torch.equal(A.forward(x), down.forward(c.forward(x)))
    assert torch.equal(A.adjoint(y), c.adjoint(down.adjoint(y)))


def test_schedule_bits_are_those_that_change_the_result_or_the_kernels(D, monkeypatch):
    psf = np.ones((3, 5, 5), np.float32)
    bits = lambda sig, fft, **kw: D.LinearFFTConvolver(psf, sig, fft_shape=fft, **kw).schedule_bits  # noqa: E731
    assert bits((20, 40, 60), (40, 80, 120)) == NO_TMA
    assert bits((40, 120, 100), (128, 256, 200)) == NO_TMA | FUSED
    # the fused pass leaves the column kernels out; rows of 100 points run on runtime radices there
    assert bits((40, 120, 100), (128, 256, 256), schedule=FUSED) == FUSED
    assert bits((40, 120, 90), (128, 256, 200), schedule=FUSED) == FUSED | 16 | HALF_LINES
    assert bits((20, 16, 30), (40, 21, 120)) == NO_TMA | 16 | HALF_LINES  # a 7-smooth axis
    assert bits((3, 16, 30), (7, 21, 42)) == 16 | HALF_LINES
    assert bits((30, 40, 60), (64, 80, 120), precision="mixed") == NO_TMA | 2
    monkeypatch.setenv("DECON_NO_TMA", "1")
    assert bits((20, 40, 60), (40, 80, 120)) == 0
