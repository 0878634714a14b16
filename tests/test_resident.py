"""The resident time loop of the nonlinear operators (small grids, whole
propagation in one cooperative launch) against the per-step launches.

A pinned kernel (eio_ctx_set_kernel) keeps the per-step launches, so each case
runs once by default and once pinned to the tile kernel; both do the same
operations in the same order, so their traces are the same bits.  Sizes: the
smallest grid, one-row and ragged rectangles, both unit widths, both sides of
the size rule, windows of different widths, several shots, sub > 1."""
import ctypes
import threading

import numpy as np
import pytest

from elastic_isotropic_operators_b200 import _lib, prop, synthetic
from helpers import Ctx, reg_inputs

pytestmark = pytest.mark.gpu


def _pair(w, windows=None):
    ops = []
    for pinned in (False, True):
        src, rec = w.geometry()
        op = prop.nonlinearPropElasticShotsGpu(w.elastic, w.par, *src, *rec)
        if windows is not None:
            op.setShotWindows(*windows)
        if pinned:
            _lib.check(op._L.eio_ctx_set_kernel(op.ctx, 0, 64, 16, 0))
        ops.append(op)
    return ops


def _run(op, w, seed=3):
    rng = np.random.default_rng(seed)
    m, d = op.modelSpace(), op.dataSpace()
    m.getNdArray()[...] = w.source_signal()[None]
    op.forward(False, m, d)
    a, b = op.modelSpace(), op.dataSpace()
    b.getNdArray()[...] = rng.standard_normal(b.getNdArray().shape).astype(np.float32)
    op.adjoint(False, a, b)
    return d.getNdArray().copy(), a.getNdArray().copy()


@pytest.mark.parametrize("nz,nx,nts,shots,sub", [
    (40, 56, 40, 1, 1),      # smallest: rectangles of one float4 row or four columns
    (72, 104, 61, 2, 1), (72, 104, 30, 3, 3), (104, 72, 40, 5, 2), (136, 264, 30, 8, 1),
    (312, 520, 25, 1, 1),    # one unit per thread
    (312, 424, 21, 3, 2),    # two columns per unit, several rounds (forward)
    (328, 616, 21, 1, 1),    # adjoint just above its size rule
    (56, 1256, 21, 1, 1), (1256, 56, 21, 2, 1)])
def test_resident_equals_step_launches(nz, nx, nts, shots, sub):
    w = synthetic.small(nz=nz, nx=nx, nts=nts, nshots=shots, nrec=min(20, (nx - 40) // 2), sub=sub, seed=nz + nx)
    got, ref = (_run(op, w) for op in _pair(w))
    for a, b in zip(got, ref):
        assert np.abs(b).max() > 0
        np.testing.assert_array_equal(a, b)


def test_resident_windows():
    w = synthetic.small(nz=72, nx=264, nts=60, nshots=2, nrec=20)
    wins = ([0, 10], [8 + 16 * 16, 8 + 15 * 16])
    got, ref = (_run(op, w) for op in _pair(w, wins))
    for a, b in zip(got, ref):
        np.testing.assert_array_equal(a, b)


def test_resident_repeated_points_take_the_step_launches():
    # a position given twice: its sources add up and both receivers record
    w = synthetic.small(nts=40)
    r = reg_inputs(w, "f", seed=4)
    rep = lambda lists: [np.concatenate([p, p[:1]]) for p in lists]     # noqa: E731
    sp, rp = rep(r["sp"]), rep(r["rp"])
    model = [np.concatenate([m, m[:1]]) for m in r["model"]]
    data = [np.concatenate([d, d[:1]]) for d in r["data"]]
    out = []
    for kind in (None, 0):
        c = Ctx(w)
        try:
            if kind is not None:
                c.set_kernel(kind)
            out.append([c.nl(adj, model, data, sp, rp)[0 if adj else 1] for adj in (0, 1)])
        finally:
            c.close()
    for a, b in zip(out[0], out[1]):
        for x, y in zip(a, b):
            np.testing.assert_allclose(x, y, rtol=0, atol=1e-6 * max(np.abs(y).max(), 1e-30))


def test_resident_wait_timeout_reports_and_recovers():
    w = synthetic.small(nts=60)
    c = Ctx(w)
    try:
        r = reg_inputs(w, "f", seed=3)
        for adj in (0, 1):
            ref = c.nl(adj, r["model"], r["data"], r["sp"], r["rp"])[0 if adj else 1]
            _lib.check(c.L.eio_ctx_set_wait_limit(c.h, 0))
            with pytest.raises(prop.EioError) as ex:
                c.nl(adj, r["model"], r["data"], r["sp"], r["rp"])
            assert ex.value.code == -7
            _lib.check(c.L.eio_ctx_set_wait_limit(c.h, -1))
            got = c.nl(adj, r["model"], r["data"], r["sp"], r["rp"])[0 if adj else 1]
            for a, b in zip(got, ref):
                np.testing.assert_array_equal(a, b)
    finally:
        c.close()


def test_resident_counts_fine_steps():
    w = synthetic.small(nts=60, nshots=1)
    op = _pair(w)[0]
    m, d = op.modelSpace(), op.dataSpace()
    m.getNdArray()[...] = w.source_signal()[None]
    L, n, s, c = op._L, ctypes.c_longlong(), ctypes.c_longlong(), ctypes.c_longlong()
    ms = ctypes.c_double()
    _lib.check(L.eio_ctx_stats(op.ctx, 1, 1, None, None, None))
    op.forward(False, m, d)
    _lib.check(L.eio_ctx_stats(op.ctx, 1, 0, ctypes.byref(n), ctypes.byref(s), ctypes.byref(ms)))
    _lib.check(L.eio_ctx_step_cells(op.ctx, ctypes.byref(c)))
    assert s.value == w.fine_steps and n.value < 60 and ms.value > 0
    assert c.value == w.fine_steps * w.cells


def test_resident_contexts_on_threads():
    # contexts of several host threads share the device; their cooperative launches take turns
    w = synthetic.small(nz=104, nx=136, nts=80, nshots=2)
    ref = _run(_pair(w)[0], w)
    out, err = [None] * 4, []

    def work(k):
        try:
            op = _pair(w)[0]
            for _ in range(3):
                out[k] = _run(op, w)
        except Exception as e:     # noqa: BLE001
            err.append(e)

    th = [threading.Thread(target=work, args=(k,)) for k in range(4)]
    for t in th:
        t.start()
    for t in th:
        t.join()
    assert not err, err
    for o in out:
        for a, b in zip(o, ref):
            np.testing.assert_array_equal(a, b)


def test_resident_beside_the_persistent_born_groups():
    # the other cooperative launch of the library, on another context and host thread
    w = synthetic.small(nz=104, nx=136, nts=60, nshots=3)
    src, rec = w.geometry()
    nl = _pair(w)[0]
    born = prop.BornElasticShotsGpu(w.elastic, w.par, [w.source_signal()], *src, *rec)
    born.setBornBatch(3)
    born.setLanes(3)
    _lib.check(born._L.eio_ctx_set_kernel(born.ctx, 3, 64, 16, 0))
    born.setPersistent(7)

    def run_born():
        m, d = born.modelSpace(), born.dataSpace()
        m.getNdArray()[...] = w.extra["dmodel"]
        born.forward(False, m, d)
        a = born.modelSpace()
        born.adjoint(False, a, d)
        return d.getNdArray().copy(), a.getNdArray().copy()

    jobs = [lambda: _run(nl, w), run_born]
    ref = [f() for f in jobs]
    out, err = [[], []], []

    def work(k):
        try:
            for _ in range(5):
                out[k].append(jobs[k]())
        except Exception as e:     # noqa: BLE001
            err.append(e)

    th = [threading.Thread(target=work, args=(k,)) for k in range(2)]
    for t in th:
        t.start()
    for t in th:
        t.join()
    assert not err, err
    for k in range(2):
        for o in out[k]:
            for a, b in zip(o, ref[k]):
                np.testing.assert_array_equal(a, b)


UNTUNED = (1, 64, 8, 8)     # what eio_ctx_get_kernel says before any timing


def _kernel(op):
    v = [ctypes.c_int() for _ in range(4)]
    _lib.check(op._L.eio_ctx_get_kernel(op.ctx, *[ctypes.byref(x) for x in v]))
    return tuple(x.value for x in v)


def test_lanes_choose_their_kernel_before_they_run():
    # the saved wavefield's shot takes the step launches, on the second lane here: the first lane timed
    # the kernels beforehand, alone, and both use its choice
    w = synthetic.small(nts=40, nshots=4)
    w.par.set("saveWavefield", "1")
    w.par.set("wavefieldShotNumber", "1")
    op = _pair(w)[0]
    m, d = op.modelSpace(), op.dataSpace()
    m.getNdArray()[...] = w.source_signal()[None]
    op.forwardWavefield(False, m, d)
    assert _kernel(op) != UNTUNED
    ref = _run(op, w)[0]
    np.testing.assert_array_equal(d.getNdArray(), ref)


@pytest.mark.parametrize("nz,nx,shots,fwd,adj", [
    (312, 520, 1, False, False), (312, 424, 3, False, True), (72, 104, 2, False, False), (600, 1000, 1, True, True),
    # the adjoint where its plan has two columns a unit: not faster than its launches
    (312, 600, 1, False, True), (56, 3400, 1, False, True), (1000, 200, 1, False, True), (72, 344, 8, False, True)])
def test_resident_calls_time_no_kernel(nz, nx, shots, fwd, adj):
    w = synthetic.small(nz=nz, nx=nx, nts=5, nshots=shots)
    for direction, timed in (("forward", fwd), ("adjoint", adj)):
        op = _pair(w)[0]
        m, d = op.modelSpace(), op.dataSpace()
        m.getNdArray()[...] = w.source_signal()[None]
        getattr(op, direction)(False, m, d)
        assert (_kernel(op) != UNTUNED) == timed, direction


def _resident(op, call):
    """Whether the call's fine steps were one launch (counters: launches of any kind, fine steps)."""
    n, s = ctypes.c_longlong(), ctypes.c_longlong()
    _lib.check(op._L.eio_ctx_stats(op.ctx, 0, 1, None, None, None))
    call()
    _lib.check(op._L.eio_ctx_stats(op.ctx, 0, 0, ctypes.byref(n), ctypes.byref(s), None))
    assert s.value > 0
    return n.value < s.value


@pytest.mark.parametrize("lanes,resident", [(2, True), (3, False), (4, False)])
def test_more_than_two_lanes_keep_their_overlapping_launches(lanes, resident):
    w = synthetic.small(nts=60, nshots=4)
    op = _pair(w)[0]
    ref = _run(op, w)
    op.setShotBatch(1)
    op.setLanes(lanes)
    assert _resident(op, lambda: _run(op, w)) == resident
    for a, b in zip(_run(op, w), ref):
        np.testing.assert_allclose(a, b, rtol=0, atol=1e-6 * np.abs(b).max())
    op.setLanes(1)
    assert _resident(op, lambda: _run(op, w))


def test_autotune_takes_the_choice_back():
    w = synthetic.small(nts=60, nshots=1)
    op = _pair(w)[1]
    assert not _resident(op, lambda: _run(op, w))      # the caller's kernel
    _lib.check(op._L.eio_ctx_autotune(op.ctx, None, None, None, None))
    assert _resident(op, lambda: _run(op, w))


@pytest.mark.parametrize("value", [np.nan, np.inf])
def test_non_finite_samples_spread_as_with_step_launches(value):
    # a sample is part of every fine step between its neighbours, also where its time weight is zero
    w = synthetic.small(nts=60, nshots=1)
    out = []
    for op in _pair(w):
        m, d, a, b = op.modelSpace(), op.dataSpace(), op.modelSpace(), op.dataSpace()
        m.getNdArray()[...] = w.source_signal()[None]
        m.getNdArray().reshape(5, -1)[2, 30] = value
        op.forward(False, m, d)
        b.getNdArray()[...] = 1.0
        b.getNdArray().reshape(5, 20, 60)[3, 7, 25] = value
        op.adjoint(False, a, b)
        out.append((d.getNdArray().copy(), a.getNdArray().copy()))
    for got, ref in zip(*out):
        assert 0 < np.isfinite(ref).sum() < ref.size
        np.testing.assert_array_equal(got, ref)


def test_resident_without_memory_for_its_slots_takes_the_step_launches():
    # 6 MB of edge slots, and a context that has no more than its step launches needed
    w = synthetic.small(nz=312, nx=520, nts=20, nshots=1)
    op = _pair(w)[1]
    ref = _run(op, w)
    L = op._L
    _lib.check(L.eio_ctx_autotune(op.ctx, None, None, None, None))     # no longer pinned
    used = ctypes.c_longlong()
    try:
        _lib.check(L.eio_get_device_memory_used(ctypes.byref(used)))
        _lib.check(L.eio_set_device_memory_cap(used.value + (1 << 20)))
        got = []
        assert not _resident(op, lambda: got.extend(_run(op, w)))
        for a, b in zip(got, ref):
            np.testing.assert_allclose(a, b, rtol=0, atol=1e-6 * np.abs(b).max())
    finally:
        _lib.check(L.eio_set_device_memory_cap(0))
    assert _resident(op, lambda: _run(op, w))


@pytest.mark.parametrize("nz,nx,shots,fwd,adj", [
    # one column a unit: both directions (the adjoint's last size along z)
    (40, 56, 1, True, True), (104, 72, 5, True, True), (312, 520, 1, True, True), (1256, 56, 2, True, True),
    (136, 264, 5, True, True), (2504, 72, 1, True, True),
    # two columns a unit, one and two rounds: the forward only
    (312, 600, 1, True, False), (216, 440, 2, True, False), (600, 72, 6, True, False), (72, 344, 8, True, False),
    (408, 1016, 1, True, False), (600, 696, 1, True, False),
    # just above the size rule
    (408, 1032, 1, False, False)])
def test_resident_route_and_bits(nz, nx, shots, fwd, adj):
    """Each direction takes the resident loop where the size rule says so, and gives the step launches' bits."""
    # more fine steps than the shots' other launches, which is what the counters tell apart
    w = synthetic.small(nz=nz, nx=nx, nts=12 + 20 * shots, nshots=shots, nrec=min(20, (nx - 40) // 2), seed=nz + nx)
    op, pinned = _pair(w)
    for name, resident in (("forward", fwd), ("adjoint", adj)):
        out = []
        for o in (op, pinned):
            m, d = o.modelSpace(), o.dataSpace()
            m.getNdArray()[...] = w.source_signal()[None]
            d.getNdArray()[...] = np.random.default_rng(3).standard_normal(d.getNdArray().shape).astype(np.float32)
            call = lambda: getattr(o, name)(False, m, d)     # noqa: B023,E731
            call()                                           # a first call may time kernels
            assert _resident(o, call) == (resident and o is op), name
            out.append((d if name == "forward" else m).getNdArray().copy())
        assert np.abs(out[1]).max() > 0
        np.testing.assert_array_equal(*out)
