"""Window copies and band sums along rows at the edges of their thread layouts."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.fixture(scope="module")
def D():
    import deconlib_b200.deconvolution as D

    return D


@pytest.mark.parametrize("shape,ext,start", [
    ((1,), (1,), (0,)), ((7,), (3,), (4,)), ((100003,), (99990,), (5,)), ((513, 1), (511, 1), (1, 0)),
    ((33, 31), (32, 8), (0, 23)), ((5, 9, 32), (1, 9, 32), (4, 0, 0)), ((6, 70, 129), (5, 67, 128), (1, 2, 1)),
    ((3, 5, 520), (3, 1, 513), (0, 4, 7)), ((2, 3, 4, 5), (1, 2, 3, 4), (1, 0, 1, 1)),
])
def test_windows_copy_whole_values(D, shape, ext, start):
    rng = np.random.default_rng(3)
    x = rng.standard_normal(shape).astype(np.float32)
    y = rng.standard_normal(ext).astype(np.float32)
    box = tuple(slice(s, s + e) for s, e in zip(start, ext))
    crop = D.Crop(shape, ext, start=start)
    assert np.array_equal(crop.forward(torch.from_numpy(x).cuda()).cpu().numpy(), x[box])
    want = np.zeros(shape, np.float32)
    want[box] = y
    assert np.array_equal(crop.adjoint(torch.from_numpy(y).cuda()).cpu().numpy(), want)


@pytest.mark.parametrize("rows,n_in,n_out", [(1, 2, 1), (7, 66, 33), (1000, 63, 32), (257, 520, 257), (33, 900, 256),
                                             (65, 45, 30)])
def test_band_sums_along_rows_equal_float64(D, rows, n_in, n_out):
    """Area sums: at most ceil(scale) + 2 <= 6 products of weights <= 1, summed
    in order: relative error <= 8 * 2^-24 of the sum of magnitudes."""
    rng = np.random.default_rng(4)
    x = rng.uniform(0.5, 1.5, (rows, n_in)).astype(np.float32)
    op = D.FractionalAreaDownsample(scale=(1.0, n_in / n_out), in_shape=(rows, n_in))
    assert tuple(op.out_shape) == (rows, n_out)
    got = op.forward(torch.from_numpy(x).cuda()).cpu().numpy().astype(np.float64)
    s = n_in / n_out
    edges = np.arange(n_out + 1) * s
    w = np.clip(np.minimum(edges[1:, None], np.arange(n_in)[None] + 1) - np.maximum(edges[:-1, None],
                                                                                 np.arange(n_in)[None]), 0, None)
    want = x.astype(np.float64) @ w.T
    assert np.all(np.abs(got - want) <= 8 * 2.0**-24 * want)
