"""A CTA whose wait gave up leaves only when its copies have landed: the kernels'
bounded wait with no polls at all, then their drain, on a copy that does arrive."""

import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [4, 100, 8192])
def test_copies_have_landed_when_a_cta_gives_up(n):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from deconlib_b200 import _lib

    lib, st = _lib.load(), _lib.stream_ptr()
    src = torch.arange(1, n + 1, device="cuda", dtype=torch.float32)
    dst = torch.zeros_like(src)
    assert lib.decon_device_status_clear(st) == _lib.OK
    assert lib.decon_test_wait_drain(_lib.ptr(src), _lib.ptr(dst), n, st) == _lib.OK
    assert lib.decon_device_status(st) == _lib.ERR_TIMEOUT
    assert lib.decon_device_status_clear(st) == _lib.OK
    assert torch.equal(src, dst)
    for bad in (0, 3, 8196):
        assert lib.decon_test_wait_drain(_lib.ptr(src), _lib.ptr(dst), bad, st) == _lib.ERR_VALUE
