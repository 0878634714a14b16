"""The U-Net's convolution with one halo copy for all nine taps (images whose
rows are whole 128-pixel tiles) against the copy-loop kernel: the same products
summed in the same order, so the same bits.  Odd heights take one row per tile,
even ones two; one to three channel blocks; every tile width; FP32 and BF16
outputs with and without ReLU."""
import ctypes

import numpy as np
import pytest

from elastic_isotropic_operators_b200 import _lib

pytestmark = pytest.mark.gpu


def _p(t):
    return ctypes.c_void_p(int(t.data_ptr()))


@pytest.mark.parametrize("n,h,w,cin,cout", [
    (1, 1, 128, 16, 16), (2, 5, 128, 16, 32), (1, 6, 256, 32, 32), (3, 4, 384, 32, 16), (1, 7, 256, 48, 32),
    (1, 4, 128, 96, 32), (2, 2, 256, 32, 96), (1, 8, 128, 64, 64), (1, 40, 1024, 32, 48), (20, 16, 256, 16, 32)])
def test_halo_convolution_equals_the_copy_loop(n, h, w, cin, cout):
    torch = pytest.importorskip("torch")
    L = _lib.lib()
    rng = np.random.default_rng(h * w + cin)
    bf = lambda *s: torch.as_tensor(rng.standard_normal(s).astype(np.float32), device="cuda").to(torch.bfloat16)  # noqa: E731
    x, wt = bf(n, h, w, cin), bf(cout, 9, cin)
    mode = ctypes.c_int()
    _lib.check(L.eio_unet_get_tma(ctypes.byref(mode)))
    out = []
    try:
        for m in (3, 0):
            _lib.check(L.eio_unet_set_tma(m))
            for relu in (0, 1):
                y32 = torch.full((n, h, w, cout), float("nan"), device="cuda")
                y16 = torch.full((n, h, w, cout), float("nan"), dtype=torch.bfloat16, device="cuda")
                _lib.check(L.eio_unet_conv3x3(n, h, w, cin, cout, _p(x), _p(wt), _p(y32), _p(y16), relu, None))
                torch.cuda.synchronize()
                out += [y32, y16]
    finally:
        _lib.check(L.eio_unet_set_tma(mode.value))
    for a, b in zip(out[:4], out[4:]):
        assert torch.isfinite(b.float()).all()
        assert torch.equal(a, b)


def test_halo_convolution_wait_timeout_reports_and_recovers():
    torch = pytest.importorskip("torch")
    L = _lib.lib()
    n, h, w, c = 2, 16, 256, 32
    x = torch.randn(n, h, w, c, device="cuda").to(torch.bfloat16)
    wt = torch.randn(c, 9, c, device="cuda").to(torch.bfloat16)
    y = torch.empty(n, h, w, c, device="cuda")
    err = ctypes.c_int()

    def conv():
        _lib.check(L.eio_unet_conv3x3(n, h, w, c, c, _p(x), _p(wt), _p(y), None, 0, None))
        torch.cuda.synchronize()
        _lib.check(L.eio_gemm_status(1, ctypes.byref(err)))
        return err.value, y.clone()

    _lib.check(L.eio_gemm_status(1, ctypes.byref(err)))
    e, ref = conv()
    assert e == 0
    try:
        _lib.check(L.eio_gemm_set_wait_limit(0))
        e, _ = conv()
        assert e == 1                      # timed out, drained (not 2)
    finally:
        _lib.check(L.eio_gemm_set_wait_limit(-1))
    e, got = conv()
    assert e == 0 and torch.equal(got, ref)
