"""The C handle's getters: what they hold on the device, and several threads reading one handle."""
import ctypes
import threading

import numpy as np
import pytest

from activemodelbplus.integrator import _native as N

pytestmark = pytest.mark.gpu
STENCIL = N.amb_stencil(1e-3, 1, 1)
MODEL = N.amb_model(-0.25, 0, 0.25, 1, -1, -4, 0.05)


def _handle(field, precision, seed=7):
    h = ctypes.c_void_p()
    field = np.ascontiguousarray(field, dtype=np.float64)
    rc = N.lib().amb_integrator_create(field.ctypes.data, *field.shape, ctypes.byref(STENCIL), ctypes.byref(MODEL), precision,
                                       seed, ctypes.byref(h))
    assert rc == 0, N.last_error()
    return h


def _used():
    import torch
    torch.cuda.synchronize()
    free, total = torch.cuda.mem_get_info()
    return total - free


def _current(h, which, shape):
    out = np.empty((2,) + shape)
    assert N.lib().amb_integrator_get_current(h, which, out[0].ctypes.data, out[1].ctypes.data) == 0, N.last_error()
    return out


def _potential(h, which, shape):
    out = np.empty(shape)
    assert N.lib().amb_integrator_get_chemical_potential(h, which, out.ctypes.data) == 0, N.last_error()
    return out


@pytest.mark.parametrize("precision", [N.AMB_F64, N.AMB_F32, N.AMB_F32C])
@pytest.mark.parametrize("shape", [(1, 1), (33, 70)])
def test_getters_leave_the_run_as_it_was(shape, precision):
    """Every current and potential is the sum of its terms to the bit, and a run goes on as without them."""
    lib, field = N.lib(), np.random.default_rng(1).normal(-0.4, 0.1, shape)
    a, b = _handle(field, precision), _handle(field, precision)
    for h in (a, b):
        assert lib.amb_integrator_run(h, 3) == 0
    t = {k: _current(a, w, shape) for k, w in N.CURRENTS.items()}
    assert np.array_equal(t["active"], t["circulating"] + t["lambda"])
    assert np.array_equal(t["deterministic"], t["active"] + t["passive"])
    assert np.array_equal(t["total"], t["deterministic"] + t["random"])
    assert np.array_equal(_potential(a, 0, shape), _potential(a, 1, shape) + _potential(a, 2, shape))
    fields = []
    for h in (a, b):
        assert lib.amb_integrator_run(h, 4) == 0
        out = np.empty(shape)
        assert lib.amb_integrator_get_field(h, out.ctypes.data) == 0
        fields.append(out)
        lib.amb_integrator_destroy(h)
    assert np.array_equal(*fields)


@pytest.mark.parametrize("precision", [N.AMB_F64, N.AMB_F32C])
def test_getters_allocate_the_term_planes_only(precision):
    import torch
    side, shape = 2048, (2048, 2048)
    plane = side * side * 8
    torch.cuda.empty_cache()
    h = _handle(np.random.default_rng(2).normal(-0.4, 0.1, shape), precision)
    assert N.lib().amb_integrator_run(h, 1) == 0
    _current_before = _used()
    _current(h, N.CURRENTS["total"], shape)
    _potential(h, 0, shape)
    assert _used() - _current_before < 10.5 * plane
    N.lib().amb_integrator_destroy(h)


def test_threads_read_one_handle():
    """Getters of one state from several threads (every call its own arrays) give what one thread gets."""
    shape, lib = (300, 400), N.lib()
    h = _handle(np.random.default_rng(3).normal(-0.4, 0.1, shape), N.AMB_F64)
    assert lib.amb_integrator_run(h, 2) == 0
    want = [_current(h, w, shape) for w in range(7)]
    bad = []

    def work(w):
        for _ in range(30):
            if not np.array_equal(_current(h, w, shape), want[w]):
                bad.append(w)
    threads = [threading.Thread(target=work, args=(w,)) for w in range(7)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    lib.amb_integrator_destroy(h)
    assert not bad


def test_runs_share_and_give_back_their_workspace():
    """Four FP64 handles that have run hold their two planes each and one workspace of eight together; no handle, no
    workspace."""
    import torch
    side = 2048
    plane, field = side * side * 8, np.random.default_rng(4).normal(-0.4, 0.1, (side, side))
    warm = _handle(field[:8, :8], N.AMB_F64)  # what the library holds with any handle
    assert N.lib().amb_integrator_run(warm, 1) == 0
    torch.cuda.empty_cache()
    before = _used()
    handles = [_handle(field, N.AMB_F64, seed=i) for i in range(4)]
    for h in handles:
        assert N.lib().amb_integrator_run(h, 2) == 0
    assert _used() - before < (4 * 2 + 8 + 0.5) * plane
    for h in handles + [warm]:
        N.lib().amb_integrator_destroy(h)
    assert _used() - before < 0.5 * plane


def test_threads_run_handles_at_once():
    """Handles of a size that leases its workspace, run by several threads: each the bits of a run alone."""
    lib, shape, n = N.lib(), (900, 800), 4
    rng = np.random.default_rng(5)
    fields = [rng.normal(-0.4, 0.1, shape) for _ in range(n)]
    out = []
    for together in (True, False):
        handles = [_handle(f, N.AMB_F64, seed=i) for i, f in enumerate(fields)]
        rcs = []

        def work(h):
            for steps in (3, 1, 2, 5):
                rcs.append(lib.amb_integrator_run(h, steps))
        if together:
            threads = [threading.Thread(target=work, args=(h,)) for h in handles]
            for t in threads:
                t.start()
            for t in threads:
                t.join()
        else:
            for h in handles:
                work(h)
        assert rcs == [0] * (4 * n)
        out.append([])
        for h in handles:
            f = np.empty(shape)
            assert lib.amb_integrator_get_field(h, f.ctypes.data) == 0
            out[-1].append(f)
            lib.amb_integrator_destroy(h)
    assert all(np.array_equal(a, b) for a, b in zip(*out))
