"""The sliding FP32 kernel at the edges of its windows: fewer rows than a y ring, one strip whose
window wraps round the row, segments shorter than the pipeline. Bitwise the tile kernel's field."""
import numpy as np
import pytest

from activemodelbplus.integrator import Ensemble, Integrator, Model, Stencil

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["f32", "f32c"])
@pytest.mark.parametrize("fused", [False, True])
@pytest.mark.parametrize("shape,seg_rows", [((1, 112), 1), ((2, 116), 1), ((3, 128), 2), ((8, 224), 3), ((9, 228), 9),
                                            ((17, 132), 5), ((40, 340), 7)])
def test_edges(shape, seg_rows, fused, precision):
    f = np.random.default_rng(5).normal(-0.4, 0.1, shape)
    m, st = Model(a=-0.25, b=0.1, c=0.25, kappa=1, lamb=-1, zeta=-4, T=0.05), Stencil(dt=1e-3, dx=1.0, dy=1.25)
    a = Integrator(f, st, m, precision=precision, seed=2, kernel="tile")
    b = Integrator(f, st, m, precision=precision, seed=2, kernel="sliding",
                   launch={"seg_rows": seg_rows, "pairs_per_cta": 1, "fused": fused})
    a.run(4)
    b.run(4)
    assert np.array_equal(a.field, b.field)


@pytest.mark.parametrize("precision", ["f32", "f32c"])
@pytest.mark.parametrize("fused", [False, True])
def test_ensemble_of_one_stencil(fused, precision):
    """Replicas that share a stencil read it from the launch; odd heights, one strip and several."""
    rng = np.random.default_rng(6)
    shapes, st = [(1, 112), (33, 116), (70, 340), (129, 228)], Stencil(dt=1e-3, dx=1.0, dy=1.25)
    fields = [rng.normal(-0.4, 0.1, s) for s in shapes]
    models = [Model(a=-0.25, b=0.1 * i, c=0.25, kappa=1 + i, lamb=-1, zeta=-4 + i, T=0.05 * i) for i in range(4)]
    ens = Ensemble(fields, st, models, precision=precision, seeds=list(range(4)), graph_steps=2)
    ens.fused = fused
    ens.run(5)
    for r in range(4):
        a = Integrator(fields[r], st, models[r], precision=precision, seed=r, kernel="tile")
        a.run(5)
        assert np.array_equal(a.field, ens.field(r)), r
    ens.close()
