"""Band sums along rows, one row per block and rows side by side in a block."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("rows,n_in,n_out", [(1, 100001, 50000), (1, 600, 257), (3, 4096, 2048), (2400, 450, 225),
                                             (2400, 453, 224), (5000, 400, 129), (20000, 60, 31)])
def test_band_sums_equal_float64(rows, n_in, n_out):
    """At most ceil(scale) + 2 <= 6 products of weights <= 1, summed in order:
    relative error <= 8 * 2^-24 of the sum of magnitudes."""
    import deconlib_b200.deconvolution as D

    s = n_in / n_out
    x = np.random.default_rng(6).uniform(0.5, 1.5, (rows, n_in)).astype(np.float32)
    op = D.FractionalAreaDownsample(scale=(1.0, s), in_shape=(rows, n_in))
    assert tuple(op.out_shape) == (rows, n_out)
    got = op.forward(torch.from_numpy(x).cuda()).cpu().numpy().astype(np.float64)
    # the integral of the piecewise constant row at the coarse edges
    c = np.concatenate([np.zeros((rows, 1)), np.cumsum(x.astype(np.float64), axis=1)], axis=1)
    e = np.arange(n_out + 1) * s
    i = np.minimum(e.astype(np.int64), n_in - 1)
    at = c[:, i] + (e - i) * x.astype(np.float64)[:, i]
    want = np.diff(at, axis=1)
    assert np.all(np.abs(got - want) <= 8 * 2.0**-24 * want)
