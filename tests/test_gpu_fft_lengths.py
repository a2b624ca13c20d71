"""Every axis length with a register FFT kernel, on every axis, against FP64.

The passes are compiled per length (two register DFTs of lengths r1 x r2), so
each length is a kernel of its own: all 5-smooth lengths from 16 to 1024 along
y and z, all even Fx up to 1024 and all odd 5-smooth Fx.  Signal extents are
odd numbers around half the canvas, so rows end inside a butterfly, the last
column tile is a partial one and rows are not a multiple of the CTA's lines.

Tolerance: an FP32 FFT of N points has a relative L2 error of about 0.6 eps
sqrt(log2 N) (eps = 2^-24); two transforms over up to 2^19 canvas points and the
product give about 4e-7; the repository's convolution tests allow 1e-6.
"""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

TOL = 1e-6


def smooth(lo, hi):
    out = []
    for n in range(lo, hi + 1):
        m = n
        for p in (2, 3, 5):
            while m % p == 0:
                m //= p
        if m == 1:
            out.append(n)
    return out


@pytest.fixture(scope="module")
def D():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import deconlib_b200.deconvolution as d

    return d


def rel(a, b):
    return float((a.double() - b).norm() / b.norm())


def reference(k, x, fft, adjoint):
    """Zero-boundary convolution with a corner-origin kernel, torch float64."""
    big = torch.zeros(fft, dtype=torch.float64, device="cuda")
    k = k.double() / float(np.float32(k.double().sum().item()))
    idx = []
    for m, f in zip(k.shape, fft):
        i = torch.arange(m, device="cuda")
        idx.append(torch.where(i < (m + 1) // 2, i, f - (m - i)))
    big[idx[0][:, None, None], idx[1][None, :, None], idx[2][None, None, :]] = k
    otf = torch.fft.rfftn(big)
    y = torch.fft.irfftn(torch.fft.rfftn(x.double(), s=fft) * (otf.conj() if adjoint else otf), s=fft)
    return y[tuple(slice(0, n) for n in x.shape)]


def check(D, shape, fft, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    k = torch.rand(tuple(f - n + 1 for n, f in zip(shape, fft)), generator=g, device="cuda") ** 4
    x = torch.rand(shape, generator=g, device="cuda")
    c = D.LinearFFTConvolver(k, shape, fft_shape=fft)
    return c, x, max(rel(c.forward(x), reference(k, x, fft, False)), rel(c.adjoint(x), reference(k, x, fft, True)))


def half(n):
    return max(2, (n // 2) | 1)


AXES = {
    "z": [(L, 20, 30) for L in smooth(16, 1024)],
    "y": [(18, L, 50) for L in smooth(16, 1024)],
    "x_even": [(16, 18, 2 * L) for L in smooth(16, 512)],
    "x_odd": [(16, 18, L) for L in smooth(25, 729) if L % 2],
    # shorter, longer and 7-smooth axes take the runtime-radix passes
    "other": [(8, 12, 14), (15, 1080, 28), (21, 36, 49), (1, 512, 640), (5, 35, 2160)],
}


@pytest.mark.parametrize("axis", list(AXES))
def test_every_length_vs_fp64(D, axis):
    bad = []
    for i, fft in enumerate(AXES[axis]):
        shape = tuple(half(f) if f > 1 else 1 for f in fft)
        err = check(D, shape, fft, i)[2]
        if not err < TOL:
            bad.append((fft, err))
    assert not bad, bad
    from deconlib_b200 import _lib

    _lib.call("decon_device_status", _lib.stream_ptr())


@pytest.mark.parametrize("fft", [(32, 64, 64), (48, 375, 90), (64, 60, 225), (20, 27, 405), (128, 40, 192)])
def test_rl_epilogues_equal_the_operator_form(D, fft):
    # the ratio and update carried by the last X pass against the element-wise
    # kernels on the same convolutions (odd Nx, odd Fx, odd row counts)
    shape = tuple(half(f) for f in fft)
    c, x, _ = check(D, shape, fft, 3)
    obs = torch.poisson(200 * x)
    a = D.richardson_lucy_with_operator(obs, c, num_iter=4, background=3.0, eval_interval=2)
    b = D.richardson_lucy_with_operator(obs, D.compose(D.Crop(shape, shape), c), num_iter=4, background=3.0,
                                        eval_interval=2)
    assert rel(a.restored, b.restored.double()) < 1e-6
    assert rel(a.pred, b.pred.double()) < 1e-6
    np.testing.assert_allclose(a.loss_history, b.loss_history, rtol=1e-6)


@pytest.mark.parametrize("L", [16, 25, 27, 64, 135, 250, 256, 375, 400, 486, 512])
def test_fused_area_sum_equals_operators_at_every_kind_of_length(D, L):
    fft, shape = (16, 18, 2 * L), (6, 10, (L // 2) * 2)
    c, x, _ = check(D, shape, fft, L)
    down = D.FractionalAreaDownsample(2.0)
    A = D.compose(down, c)
    assert torch.equal(A.forward(x), down.forward(c.forward(x)))
    y = down.forward(x)
    assert torch.equal(A.adjoint(y), c.adjoint(down.adjoint(y)))
    assert A._down2 is not None


@pytest.mark.parametrize("shape", [(3, 16, 18), (2, 27, 25), (5, 96, 75), (2, 225, 320), (2, 729, 48), (3, 21, 28)])
def test_psf_lengths_and_support(shape):
    # pupils that fill the plane, fill a disc, and are zero but for one column
    from deconlib_b200.psf import pupil_to_psf

    nz, ny, nx = shape
    g = torch.Generator(device="cuda").manual_seed(ny)
    full = torch.randn(ny, nx, 2, generator=g, device="cuda", dtype=torch.float64)
    full = torch.view_as_complex(full)
    kz = torch.rand(ny, nx, generator=g, device="cuda", dtype=torch.float64) * 3
    z = np.linspace(-1, 1, nz)
    ky = torch.fft.fftfreq(ny, device="cuda")[:, None]
    kx = torch.fft.fftfreq(nx, device="cuda")[None, :]
    one = torch.zeros_like(full)
    one[:, nx // 2] = full[:, nx // 2]
    for pupil in (full, full * (ky * ky + kx * kx < 0.04), one):
        p = pupil_to_psf(pupil, kz, z)
        a = torch.stack([torch.fft.ifft2(pupil * torch.exp(2j * np.pi * kz * v)) for v in z])
        ref = a.real ** 2 + a.imag ** 2
        assert rel(p, ref / ref.sum()) < TOL


@pytest.mark.parametrize("fft,ext", [((32, 64, 64), None), ((32, 64, 64), (3, 7, 10)), ((48, 375, 90), (11, 100, 31)),
                                     ((20, 27, 405), (5, 3, 101)), ((64, 60, 225), (1, 1, 1)), ((15, 27, 28), (4, 9, 8)),
                                     ((90, 128), (20, 33)), ((96,), (17,)), ((21, 36, 49), (6, 11, 13))])
def test_crop_of_a_convolution_equals_the_operators_in_turn(D, fft, ext):
    shape = tuple(half(f) for f in fft)
    ext = ext or shape
    g = torch.Generator(device="cuda").manual_seed(len(fft))
    c = D.LinearFFTConvolver(torch.rand(tuple(f - n + 1 for n, f in zip(shape, fft)), generator=g, device="cuda"),
                             shape, fft_shape=fft)
    x = torch.rand(shape, generator=g, device="cuda")
    y = torch.rand(ext, generator=g, device="cuda")
    for starts in (None, tuple(0 for _ in ext), tuple(n - e for n, e in zip(shape, ext)),
                   tuple(min(1, n - e) for n, e in zip(shape, ext))):
        crop = D.Crop(shape, ext, start=starts)
        A = D.compose(crop, c)
        assert torch.equal(A.forward(x), crop.forward(c.forward(x)))
        assert torch.equal(A.adjoint(y), c.adjoint(crop.adjoint(y)))
    with pytest.raises(ValueError):
        A.forward(y if ext != shape else x[..., :-1])
