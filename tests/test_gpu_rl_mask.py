"""The active-support mask of composed RL above the number of voxels at which
its maximum takes every partial of the reduction workspace."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

FULL = 1183 * 2048  # voxels of 1183 CTAs of the reduction


@pytest.mark.parametrize("n", [FULL, FULL + 1, 1184 * 2048 + 1, 3 * FULL + 7])
def test_mask_is_exact(n):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from deconlib_b200 import _lib
    from deconlib_b200.deconvolution._device import stream, workspace

    g = torch.Generator(device="cuda").manual_seed(n)
    x = torch.rand(n, generator=g, device="cuda") * 2e-6
    sens = torch.rand(n, generator=g, device="cuda") * 2e-6
    sens[-1] = 1.0  # the largest value is the last one
    floor = np.float32(max(np.float32(1.0) * np.float32(1e-6), np.float32(1e-10)))
    on = sens > float(floor)
    want_s = torch.where(on, sens, torch.zeros_like(sens))
    want_x = torch.where(on, x.clamp_min(1e-6), torch.zeros_like(x))
    _lib.call("decon_rl_mask", _lib.ptr(x), _lib.ptr(sens), n, _lib.ptr(workspace()), stream())
    assert torch.equal(sens, want_s) and torch.equal(x, want_x)


def test_composed_rl_above_the_limit():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import deconlib_b200.deconvolution as D

    big, small = (40, 256, 256), (36, 250, 252)  # 2.6 M and 2.3 M voxels
    assert np.prod(big) > FULL
    rng = np.random.default_rng(2)
    psf = rng.random((3, 5, 5)).astype(np.float32)
    obs = rng.poisson(30.0, small).astype(np.float32)
    op = D.compose(D.Crop(big, small), D.LinearFFTConvolver(psf, big))
    r = D.richardson_lucy_with_operator(obs, op, num_iter=4, background=1.0, eval_interval=1)
    assert tuple(r.restored.shape) == big and bool(torch.isfinite(r.restored).all())
    assert all(b < a for a, b in zip(r.loss_history, r.loss_history[1:]))
