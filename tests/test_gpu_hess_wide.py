"""The four-voxels-per-thread Hessian stencils (16-byte aligned rows).

The dual update must give the bits of the one-voxel walk inside
decon_pdhg_hess_dual_primal; the trajectory, which also depends on
||H (x_new - x)||^2, must follow the operator-by-operator path to FP32
rounding (the tolerance of the same comparison for the one-voxel walk).
Shapes: rows that end inside a piece of 128 voxels, rows of several pieces,
one-plane, one-row and eight-row volumes, z extents around the tile depths,
and an unaligned base and an unaligned row length, which keep the old walk.
"""

import ctypes as C

import pytest
import torch

pytestmark = pytest.mark.gpu

SHAPES = [(1, 8, 96), (5, 1, 80), (2, 30, 384), (17, 9, 128), (33, 17, 204), (128, 16, 256), (7, 23, 110)]


@pytest.fixture(scope="module")
def lib():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from deconlib_b200 import _lib

    return _lib


@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("norm", [0, 1])
@pytest.mark.parametrize("shape", SHAPES)
def test_dual_update_bits(lib, shape, norm, offset):
    g = torch.Generator(device="cuda").manual_seed(sum(shape))

    def field(n, scale):
        # a view whose base is `offset` floats past an aligned address
        return (scale * torch.randn(n + offset, device="cuda", generator=g))[offset:]

    n = shape[0] * shape[1] * shape[2]
    xc, xp, aty, y2 = field(n, 1.0), field(n, 1.0), field(n, 1.0), field(6 * n, 0.01)
    shp, st = lib.i64arr(shape), lib.stream_ptr()
    dll = lib.load()
    h = C.c_void_p()
    lib.check(dll.decon_pdhg_create(4, 0.3, 0.99, 0.5, 0.0, 0, 1, C.byref(h)))
    ref, xn = torch.empty_like(y2), torch.empty_like(xc)
    lib.check(dll.decon_pdhg_hess_dual_primal(h, lib.ptr(y2), lib.ptr(ref), lib.ptr(xc), lib.ptr(xp), lib.ptr(aty),
                                              lib.ptr(xn), shp, C.c_float(0.7), C.c_float(0.02), norm, st))
    lib.check(dll.decon_pdhg_hess_dual(h, lib.ptr(y2), lib.ptr(xc), lib.ptr(xp), shp, C.c_float(0.7),
                                       C.c_float(0.02), norm, st))
    torch.cuda.synchronize()
    dll.decon_pdhg_destroy(h)
    assert torch.equal(y2, ref)


@pytest.mark.parametrize("shape", [(6, 9, 80), (19, 20, 132), (9, 33, 256)])
def test_trajectory_follows_the_operator_path(lib, shape):
    import deconlib_b200.deconvolution as D
    from deconlib_b200.deconvolution.pdhg import HessianRegularizer, PDHGRunner

    g = torch.Generator(device="cuda").manual_seed(shape[2])
    psf = torch.rand((3, 5, 5), device="cuda", generator=g)
    obs = torch.poisson(200 * torch.rand(shape, device="cuda", generator=g) + 5)
    A = D.LinearFFTConvolver(psf, shape)
    reg = HessianRegularizer(3, 0.8, "L1")
    out = []
    for fused in (True, False):
        run = PDHGRunner(obs, A, reg, obs.clone(), 1e-2, "poisson", 25, 5.0, 0.99, 0.5, 10, 0.0, 100, 5, fused=fused)
        out.append(run.run().result())
    a, b = out[0][0].double(), out[1][0].double()
    assert float((a - b).norm() / b.norm()) < 1e-6
    for u, v in zip(out[0][3], out[1][3]):
        assert abs(u - v) <= 1e-6 * abs(v)
