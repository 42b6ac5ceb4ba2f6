"""Device memory of an FP64 integrator: what its runs need beside the field is given back, and does without."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
SIDE = 2048
PLANE = SIDE * SIDE * 8


def _sim(**kw):
    from activemodelbplus.integrator import Integrator, Model, Stencil
    f = np.random.default_rng(5).normal(-0.4, 0.1, (SIDE, SIDE))
    return Integrator(f, Stencil(1e-3, 1, 1), Model(-0.25, 0, 0.25, 1, -1, -4, 0.05), seed=2, **kw)


@pytest.fixture
def room():
    """room(planes): what this process may allocate on the device beside what it holds, through torch."""
    import torch

    def limit(planes):
        torch.cuda.empty_cache()
        total = torch.cuda.get_device_properties(0).total_memory
        torch.cuda.set_per_process_memory_fraction((torch.cuda.memory_reserved() + planes * PLANE) / total)
    yield limit
    torch.cuda.set_per_process_memory_fraction(1.0)


def test_an_integrator_holds_its_field_only():
    """Two planes (the field and its successor) from construction on and between runs."""
    import torch
    torch.cuda.empty_cache()
    before = torch.cuda.memory_allocated()
    sims = _sim(), _sim()
    for n in (0, 1, 2):
        sims[0].run(n)
        assert torch.cuda.memory_allocated() - before < 4.1 * PLANE
    reserved = torch.cuda.memory_reserved()
    sims[1].run(2)  # with the same planes
    assert torch.cuda.memory_reserved() == reserved


def test_a_run_without_room_takes_the_tile_kernel(room):
    import torch
    sim, tile = _sim(), _sim(kernel="tile")
    room(4)
    sim.run(2)
    sim.run(1)
    tile.run(3)
    assert torch.equal(sim.field_tensor, tile.field_tensor)


def test_getters_need_ten_planes(room):
    """Room for the term planes and no more: every current and potential, the same bits as with room."""
    from activemodelbplus.integrator import _native as N
    free, tight = _sim(), _sim()
    names = ["current", "deterministic_current", "passive_current", "active_current", "lambda_current",
             "circulating_current", "random_current", "chemical_potential", "passive_chemical_potential",
             "active_chemical_potential"]
    names = [n for n in names if hasattr(type(free), n)]
    assert len(names) >= len(N.CURRENTS)
    want = {n: getattr(free, n) for n in names}
    del free
    room(10.5)
    for n in names:
        got = getattr(tight, n)
        assert np.array_equal(np.asarray(got), np.asarray(want[n])), n
