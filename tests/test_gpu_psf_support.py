"""PSF of pupils whose non-zeros lie in a few rows, so that each part of the support
search holds some columns and misses others."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("ny,nx", [(16, 16), (64, 35), (70, 32), (135, 75), (729, 48), (1050, 28), (1400, 98)])
@pytest.mark.parametrize("normalize", [True, False])
def test_psf_of_scattered_pupils(ny, nx, normalize):
    """Relative error of an FP32 FFT of N points <= about log2(N) 2^-23 in the L2
    norm of the field (N <= 2^18: 2.2e-6), twice that in the intensity: 1e-5."""
    from deconlib_b200.psf import pupil_to_psf

    rng = np.random.default_rng(ny)
    z = np.array([-0.4, 0.0, 0.7])
    kz = rng.uniform(0, 3, (ny, nx))
    rows = sorted({0, ny // 3, ny // 2, ny - 1})
    for use in (rows, rows[-1:], rows[:1]):
        p = np.zeros((ny, nx), np.complex64)
        for i, y in enumerate(use):
            cols = rng.choice(nx, size=max(1, nx // 7), replace=False)
            p[y, cols] = rng.standard_normal(len(cols)) + 1j * rng.standard_normal(len(cols))
        got = pupil_to_psf(p, kz, z, normalize=normalize).double().cpu().numpy()
        a = np.fft.ifft2(p[None].astype(np.complex128) * np.exp(2j * np.pi * kz[None] * z[:, None, None]))
        want = np.abs(a) ** 2
        if normalize:
            want /= want.sum()
        assert np.linalg.norm(got - want) <= 1e-5 * np.linalg.norm(want)
