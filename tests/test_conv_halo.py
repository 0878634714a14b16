"""The U-Net's convolution with one halo copy for all nine taps (images whose
rows are whole 128-pixel tiles) against the copy-loop kernel: the same products
summed in the same order, so the same bits.  Odd heights take one row per tile,
even ones two; one to three channel blocks; every tile width; FP32 and BF16
outputs with and without ReLU."""
import ctypes
import threading

import numpy as np
import pytest

from elastic_isotropic_operators_b200 import _lib

pytestmark = pytest.mark.gpu


def _p(t):
    return ctypes.c_void_p(int(t.data_ptr()))


@pytest.mark.parametrize("n,h,w,cin,cout", [
    (1, 1, 128, 16, 16), (2, 5, 128, 16, 32), (1, 6, 256, 32, 32), (3, 4, 384, 32, 16), (1, 7, 256, 48, 32),
    (1, 4, 128, 96, 32), (2, 2, 256, 32, 96), (1, 8, 128, 64, 64), (1, 40, 1024, 32, 48), (20, 16, 256, 16, 32),
    # one CTA an SM: a tile each, and two or more
    (1, 37, 512, 96, 32), (1, 75, 256, 96, 32), (2, 148, 128, 64, 32), (2, 149, 128, 64, 64), (4, 76, 256, 64, 64),
    (1, 149, 128, 64, 96), (3, 100, 128, 48, 48)])
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


@pytest.mark.parametrize("n,h,w,ca,cb", [(1, 1, 1, 8, 8), (2, 3, 5, 64, 32), (3, 8, 16, 256, 128), (1, 40, 24, 16, 48)])
def test_up_concat_equals_its_two_passes(n, h, w, ca, cb):
    torch = pytest.importorskip("torch")
    L = _lib.lib()
    bf = lambda *s: torch.randn(*s, device="cuda").to(torch.bfloat16)  # noqa: E731
    a, b, z = bf(n, h, w, ca), bf(n, 2 * h, 2 * w, cb), bf(n, 2 * h, 2 * w, ca + cb)
    up, z1, z2 = bf(n, 2 * h, 2 * w, ca), torch.empty_like(z), torch.empty_like(z)
    _lib.check(L.eio_unet_resample(2, n, h, w, ca, _p(a), _p(up), 0, None))
    _lib.check(L.eio_unet_concat(0, 4 * n * h * w, ca, cb, _p(up), 0, _p(b), 0, _p(z1), None))
    _lib.check(L.eio_unet_up_concat(0, n, h, w, ca, cb, _p(a), _p(b), _p(z2), None))
    assert torch.equal(z1, z2)
    a1, b1, a2, b2 = (torch.empty_like(t) for t in (a, b, a, b))
    _lib.check(L.eio_unet_concat(1, 4 * n * h * w, ca, cb, _p(up), 0, _p(b1), 0, _p(z), None))
    _lib.check(L.eio_unet_resample(3, n, h, w, ca, _p(up), _p(a1), 0, None))
    _lib.check(L.eio_unet_up_concat(1, n, h, w, ca, cb, _p(a2), _p(b2), _p(z), None))
    assert torch.equal(a1, a2) and torch.equal(b1, b2)


@pytest.mark.parametrize("npix,c,nc", [(1, 8, 1), (777, 16, 3), (5000, 24, 17), (300000, 16, 16), (1000, 12, 3)])
def test_loss_and_its_derivative(npix, c, nc):
    torch = pytest.importorskip("torch")
    L = _lib.lib()
    y, t = torch.randn(npix, c, device="cuda"), torch.randn(npix, nc, device="cuda")
    dz = torch.full((npix, c), float("nan"), dtype=torch.bfloat16, device="cuda")
    part = torch.zeros(1024, dtype=torch.float64, device="cuda")
    loss = torch.zeros(1, dtype=torch.float64, device="cuda")
    _lib.check(L.eio_cnn_mse(npix, c, nc, _p(y), _p(t), _p(dz), _p(part), _p(loss), None))
    d = y[:, :nc] - t
    want = torch.zeros_like(dz)
    want[:, :nc] = (d * np.float32(1.0 / (npix * nc))).to(torch.bfloat16)
    assert torch.equal(dz, want)
    ref = 0.5 * d.double().square().mean().item()      # the same FP32 differences, summed in FP64
    assert abs(loss.item() - ref) <= 1e-12 * ref


@pytest.mark.parametrize("n,h,w,cin,cout", [      # small images take the split GEMM
    (300, 1, 128, 16, 16), (100, 5, 128, 16, 32), (5, 120, 128, 32, 32), (4, 50, 384, 32, 16), (3, 151, 256, 48, 32),
    (2, 150, 128, 96, 32), (2, 302, 128, 64, 64), (2, 101, 256, 64, 16), (20, 32, 256, 32, 32), (1, 6, 256, 32, 32),
    # both sides of the rule: 4 rows of 128 pixels an SM, 12 where one CTA fits; dz after slabs of odd size
    (592, 1, 128, 16, 64), (591, 1, 128, 16, 64), (120, 5, 128, 32, 64), (37, 16, 128, 32, 16), (37, 16, 128, 16, 32),
    (8, 111, 256, 64, 64), (6, 148, 256, 64, 32), (7, 127, 256, 96, 32), (6, 148, 256, 32, 64), (592, 1, 128, 48, 32)])
def test_halo_weight_gradient(n, h, w, cin, cout):
    """Against FP64 products of the same BF16 values: FP32 sums of n h w terms, relative L2 <= 1e-5 (as the
    other weight-gradient kernels); reproducible."""
    torch = pytest.importorskip("torch")
    L = _lib.lib()
    rng = np.random.default_rng(h * w + cin)
    bf = lambda *s: torch.as_tensor(rng.standard_normal(s).astype(np.float32), device="cuda").to(torch.bfloat16)  # noqa: E731
    x, dz = bf(n, h, w, cin), bf(n, h, w, cout)
    need = ctypes.c_longlong()
    _lib.check(L.eio_unet_wgrad_scratch(n, h, w, cin, cout, ctypes.byref(need)))
    scratch = torch.full((need.value,), float("nan"), device="cuda")
    dw = [torch.full((cout, 9, cin), float("nan"), device="cuda") for _ in range(2)]
    for d in dw:
        _lib.check(L.eio_unet_conv3x3_wgrad(n, h, w, cin, cout, _p(x), _p(dz), _p(d), _p(scratch), need.value, None))
    xp = torch.nn.functional.pad(x.double(), (0, 0, 1, 1, 1, 1))
    ref = torch.stack([torch.einsum("nhwo,nhwi->oi", dz.double(), xp[:, i:i + h, j:j + w])
                       for i in range(3) for j in range(3)], 1)
    assert torch.equal(dw[0], dw[1])
    assert ((dw[0].double() - ref).norm() / ref.norm()).item() < 1e-5


def test_halo_kernels_on_threads():
    """Layers of different channel counts share a kernel and take different shared memory.  Host threads that
    run them at once, each on its own stream: every launch is accepted and gives the bits of a serial run."""
    torch = pytest.importorskip("torch")
    L = _lib.lib()
    n, h, w, cout = 1800, 1, 128, 32
    bf = lambda *s: torch.randn(*s, device="cuda").to(torch.bfloat16)  # noqa: E731
    jobs = []
    for cin in (16, 32, 64):
        x, wt, dz = bf(n, h, w, cin), bf(cout, 9, cin), bf(n, h, w, cout)
        need = ctypes.c_longlong()
        _lib.check(L.eio_unet_wgrad_scratch(n, h, w, cin, cout, ctypes.byref(need)))
        y, dw = torch.empty(n, h, w, cout, device="cuda"), torch.empty(cout, 9, cin, device="cuda")
        scratch = torch.empty(need.value, device="cuda")

        def conv(st, cin=cin, x=x, wt=wt, y=y):    # one image: the launches are what counts
            _lib.check(L.eio_unet_conv3x3(1, h, w, cin, cout, _p(x), _p(wt), _p(y), None, 0, st))

        def wgrad(st, cin=cin, x=x, dz=dz, dw=dw, scratch=scratch):
            _lib.check(L.eio_unet_conv3x3_wgrad(n, h, w, cin, cout, _p(x), _p(dz), _p(dw), _p(scratch),
                                                scratch.numel(), st))
        jobs += [(conv, y[:1], 20000), (wgrad, dw, 3000)]
    want = []
    for f, o, _ in jobs:
        f(None)
        torch.cuda.synchronize()
        want.append(o.clone())
        o.fill_(float("nan"))
    err = []

    def work(f, passes):
        torch.zeros(1, device="cuda")      # the device's context is this thread's too
        st = torch.cuda.Stream()
        try:
            for _ in range(passes):
                f(ctypes.c_void_p(st.cuda_stream))
        except Exception as e:     # noqa: BLE001
            err.append(e)
        st.synchronize()

    torch.cuda.synchronize()
    th = [threading.Thread(target=work, args=(f, k)) for f, _, k in jobs]
    for t in th:
        t.start()
    for t in th:
        t.join()
    assert not err, err
    for (_, o, _), ref in zip(jobs, want):
        assert torch.equal(o, ref)


def test_convolution_as_a_threads_first_call():
    torch = pytest.importorskip("torch")
    L = _lib.lib()
    x = torch.randn(1, 4, 128, 16, device="cuda").to(torch.bfloat16)
    wt = torch.randn(16, 9, 16, device="cuda").to(torch.bfloat16)
    y = [torch.empty(1, 4, 128, 16, device="cuda") for _ in range(2)]
    rc = []

    def conv(o):
        rc.append(L.eio_unet_conv3x3(1, 4, 128, 16, 16, _p(x), _p(wt), _p(o), None, 0, None))

    conv(y[0])
    torch.cuda.synchronize()
    th = threading.Thread(target=conv, args=(y[1],))
    th.start()
    th.join()
    torch.cuda.synchronize()
    assert rc == [0, 0] and torch.equal(y[0], y[1])
