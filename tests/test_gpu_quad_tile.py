"""The FP32 tile kernel on column quads: grids whose rows are not whole quads, narrower than a
tile or than the stencils, partial tiles, every tile shape and launch form."""
import numpy as np
import pytest

import oracle
from activemodelbplus.integrator import Integrator, Model, Stencil

pytestmark = pytest.mark.gpu

SHAPES = [(1, 1), (3, 5), (2, 12), (7, 33), (19, 30), (40, 61), (33, 64), (65, 130), (50, 257)]
STENCIL = Stencil(dt=1e-3, dx=1.0, dy=1.25)


def _run(f, T, precision, **launch):
    m = Model(a=-0.25, b=0.1, c=0.25, kappa=1, lamb=-1, zeta=-4, T=T)
    sim = Integrator(f, STENCIL, m, precision=precision, seed=4, kernel="tile", launch=launch)
    sim.run(3)
    return sim.field


@pytest.mark.parametrize("T,tol", [(0.0, 1e-6), (0.05, 1e-5)])
@pytest.mark.parametrize("shape", SHAPES)
def test_matches_oracle(shape, T, tol):
    """The tolerances are those of FP32 arithmetic on increments below 0.1 per step, and of the noise
    (normals 5e-5 from the oracle's, J_r = 10 xi, so 2e-6 per step)."""
    f = np.random.default_rng(6).normal(-0.4, 0.1, shape)
    p = oracle.Params(dt=1e-3, dx=1.0, dy=1.25, a=-0.25, b=0.1, c=0.25, kappa=1, lamb=-1, zeta=-4, T=T)
    ref = oracle.run(f.astype(np.float32), p, 3, noise="philox" if T else "none", seed=4)
    assert np.abs(_run(f, T, "f32c", persistent=True) - ref).max() < tol


@pytest.mark.parametrize("precision", ["f32", "f32c"])
@pytest.mark.parametrize("shape", SHAPES)
def test_every_shape_gives_the_same_bits(shape, precision):
    f = np.random.default_rng(7).normal(-0.4, 0.1, shape)
    want = _run(f, 0.05, precision)
    for cols in (32, 64):
        for rows in (1, 5, 28, 64):
            for groups in (1, 2):
                for persistent in (False, True):
                    got = _run(f, 0.05, precision, seg_rows=rows, tile_cols=cols, pairs_per_cta=groups,
                               persistent=persistent)
                    assert np.array_equal(got, want), (rows, cols, groups, persistent)
