"""A learned stepper's captured macro step and its residual check run one network, whatever happens to the
FluxNet that it was made from."""
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("check_first", [False, True])
def test_later_training_reaches_neither_step_nor_check(check_first):
    """Weights and biases changed in place (as an optimiser does) and refreshed after the first macro steps or
    check: the field and the residuals are bitwise those of a stepper whose network stays."""
    import torch
    from activemodelbplus import learned as L
    from activemodelbplus.integrator import Model, Stencil
    path = os.path.join(os.path.dirname(L.__file__), "weights", "fluxnet_k50.npz")
    field = -0.4 + 0.01 * np.random.default_rng(3).standard_normal((64, 128))
    model = Model(-0.25, 0, 0.25, 1, -1, -4, 0.05)
    out = []
    for change in (False, True):
        net = L.FluxNet.load(path)
        st = L.LearnedStepper(net, field, Stencil(1e-3, 1, 1), model, K=50, seed=5, check_every=3, max_check_every=3,
                              tol=1e9, residual_sigma=2.0)
        if check_first:
            st._check_step()
        else:
            st.advance(3)
        if change:
            for p in net.parameters():
                p.mul_(0.5).add_(0.01)
            net.refresh()
        st.advance(6)
        out.append((st.phi_q.clone(), list(st.residuals)))
    assert torch.equal(out[0][0], out[1][0])
    assert out[0][1] == out[1][1]
