"""FP64 runs of more steps than one launch takes: several launches give one launch's results, and leave other
streams their turn."""
import ctypes
import threading
import time

import numpy as np
import pytest

import oracle
from activemodelbplus.integrator import Integrator, Model, Stencil
from activemodelbplus.integrator import _native as N

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,steps", [((256, 200), 2800), ((16, 20), 3501), ((1200, 1000), 140)])
def test_same_bits_as_the_tile_kernel(shape, steps):
    """Three launches of 1347 (odd: the buffers swap), 1666 and 57 steps, Philox noise."""
    st, m = Stencil(1e-3, 1, 1), Model(-0.25, 0, 0.25, 1, -1, -4, 0.05)
    f = np.random.default_rng(1).normal(-0.4, 0.1, shape)
    a, b = Integrator(f, st, m, seed=4), Integrator(f, st, m, seed=4, kernel="tile")
    a.run(steps)
    b.run(steps)
    assert np.array_equal(a.field, b.field)


def test_injected_noise_of_every_launch():
    import torch
    ny, nx, steps = 9, 12, 1700
    rng = np.random.default_rng(2)
    f, xi = rng.normal(-0.4, 0.1, (ny, nx)), rng.standard_normal((steps, 2, ny, nx))
    p = oracle.Params(dt=1e-3, dx=1.0, dy=1.0, a=-0.25, b=0.0, c=0.25, kappa=1, lamb=-1, zeta=-4, T=0.05)
    a = torch.from_numpy(f.copy()).cuda()
    b, x = torch.empty_like(a), torch.from_numpy(xi).cuda()
    nbytes = N.lib().amb_step_workspace_bytes(N.AMB_F64, ny, nx)
    ws = torch.empty(nbytes, dtype=torch.uint8, device="cuda")
    s, m, where = N.stencil_struct(Stencil(1e-3, 1, 1)), N.model_struct(Model(-0.25, 0, 0.25, 1, -1, -4, 0.05)), ctypes.c_int()
    assert N.lib().amb_step_f64_ws(ctypes.byref(s), ctypes.byref(m), 0, ny, nx, a.data_ptr(), b.data_ptr(), 0, steps,
                                   x.data_ptr(), ws.data_ptr(), nbytes, torch.cuda.current_stream().cuda_stream,
                                   ctypes.byref(where)) == 0
    ref = oracle.run(f, p, steps, noise="injected", injected=xi)
    assert np.abs((b if where.value else a).cpu().numpy() - ref).max() <= 1e-11 * np.abs(ref).max()


def test_a_long_run_lets_others_through():
    """Ten steps of a 300^2 grid, whose CTAs fill the SMs, issued during a run of 300000 steps of a 64^2 grid (two
    seconds) on another stream: done within half a second."""
    import torch
    st, m = Stencil(1e-3, 1, 1), Model(-0.25, 0, 0.25, 1, -1, -4, 0.05)
    rng = np.random.default_rng(3)
    long_, short = (Integrator(rng.normal(-0.4, 0.1, (n, n)), st, m, seed=1) for n in (64, 300))
    sl, ss = torch.cuda.Stream(), torch.cuda.Stream()
    with torch.cuda.stream(ss):
        short.run(10)
    long_.run(10)
    torch.cuda.synchronize()

    def work():
        with torch.cuda.stream(sl):
            long_.run(300000)
    t = threading.Thread(target=work)
    begin = time.perf_counter()
    t.start()
    time.sleep(0.1)
    t0 = time.perf_counter()
    with torch.cuda.stream(ss):
        short.run(10)
    wait = time.perf_counter() - t0
    t.join()
    total = time.perf_counter() - begin
    assert total > 1.0  # the long run was under way
    assert wait < 0.5, (wait, total)


@pytest.mark.parametrize("shape,steps", [((810, 810), 2050), ((16, 20), 8100)])
def test_same_bits_of_persistent_fp32_launches(shape, steps):
    """Three launches of 983 (odd: the buffers swap) and of 4000 steps against one launch per step."""
    st, m = Stencil(1e-3, 1, 1), Model(-0.25, 0, 0.25, 1, -1, -4, 0.05)
    f = np.random.default_rng(6).normal(-0.4, 0.1, shape)
    fields = []
    for persistent in (True, False):
        sim = Integrator(f, st, m, seed=4, precision="f32c", kernel="tile", launch={"persistent": persistent, "pairs_per_cta": 1})
        sim.run(steps)
        fields.append(sim.field)
    assert np.array_equal(*fields)


@pytest.mark.parametrize("precision", ["f64", "f32c"])
def test_a_long_fp32_run_lets_others_through(precision):
    """Ten steps of a 512^2 grid, whose CTAs fill the SMs, issued during a run of 600000 steps of a 64^2 FP32 grid
    (almost two seconds) on another stream: done within half a second."""
    import torch
    st, m = Stencil(1e-3, 1, 1), Model(-0.25, 0, 0.25, 1, -1, -4, 0.05)
    rng = np.random.default_rng(3)
    long_ = Integrator(rng.normal(-0.4, 0.1, (64, 64)), st, m, seed=1, precision="f32c")
    short = Integrator(rng.normal(-0.4, 0.1, (512, 512)), st, m, seed=1, precision=precision)
    sl, ss = torch.cuda.Stream(), torch.cuda.Stream()
    with torch.cuda.stream(ss):
        short.run(10)
    long_.run(10)
    torch.cuda.synchronize()

    def work():
        with torch.cuda.stream(sl):
            long_.run(600000)
    t = threading.Thread(target=work)
    begin = time.perf_counter()
    t.start()
    time.sleep(0.1)
    t0 = time.perf_counter()
    with torch.cuda.stream(ss):
        short.run(10)
    wait = time.perf_counter() - t0
    t.join()
    total = time.perf_counter() - begin
    assert total > 1.0  # the long run was under way
    assert wait < 0.5, (wait, total)
