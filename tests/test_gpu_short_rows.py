"""Window copies of very short rows, more of them than one sweep of the grid takes."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("n,last,ext", [(1300007, 1, 1), (1300007, 3, 2), (1300007, 4, 3), (700001, 5, 5),
                                        (700001, 8, 7), (400009, 9, 4), (300007, 16, 15), (170003, 17, 17)])
def test_short_rows_are_copied_whole(n, last, ext):
    import deconlib_b200.deconvolution as D

    src, dst, start = (n, last), (n - 6, ext), (5, last - ext)
    crop = D.Crop(src, dst, start=start)
    x = torch.arange(n * last, device="cuda", dtype=torch.float32).reshape(src)
    box = x[5:n - 1, last - ext:]
    assert torch.equal(crop.forward(x), box)
    want = torch.zeros_like(x)
    want[5:n - 1, last - ext:] = box
    assert torch.equal(crop.adjoint(box.contiguous()), want)
