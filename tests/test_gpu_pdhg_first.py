"""PDHG with the identity or gradient regulariser evaluated on the fly, against
the same iteration through the operators (``fused=False``).

Both form the same float32 values; the FP64 sums are folded in another order,
so the step sizes agree to rounding and the iterates to the tolerance that the
Hessian forms are held to (1e-6).  Shapes: one plane, one row, one column, rows
and planes that end inside a tile of 64 x 4 x 8, and an image and a line for the
identity.
"""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def D():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import deconlib_b200.deconvolution as d

    return d


CASES = [("gradient", s) for s in ((1, 9, 70), (9, 1, 64), (17, 5, 1), (8, 4, 128), (23, 31, 65), (2, 2, 2))]
CASES += [("identity", s) for s in ((9, 7, 66), (40, 130), (500,), (1, 1, 3))]


@pytest.mark.parametrize("norm", ["L1", "L1_2"])
@pytest.mark.parametrize("kind,shape", CASES)
def test_on_the_fly_equals_operators(D, kind, shape, norm):
    from deconlib_b200.deconvolution.pdhg import GradientRegularizer, IdentityRegularizer, PDHGRunner

    g = torch.Generator(device="cuda").manual_seed(sum(shape))
    psf = torch.rand(tuple(min(3, s) for s in shape), device="cuda", generator=g)
    obs = torch.poisson(100 * torch.rand(shape, device="cuda", generator=g) + 5)
    A = D.LinearFFTConvolver(psf, shape)
    reg = IdentityRegularizer(norm) if kind == "identity" else GradientRegularizer(3, 0.7, norm)
    out = []
    for fused in (True, False):
        run = PDHGRunner(obs, A, reg, obs.clone(), 2e-2, "gaussian", 20, 5.0, 0.99, 0.5, 5, 0.0, 100, 5, fused=fused)
        assert (run.first is not None) == fused
        out.append(run.run().result())
    a, b = out[0][0].double(), out[1][0].double()
    assert float((a - b).norm()) <= 1e-6 * float(b.norm())
    for i in (3, 4, 5):  # tau, sigma, loss histories
        for u, v in zip(out[0][i], out[1][i]):
            assert abs(u - v) <= 1e-6 * abs(v)
