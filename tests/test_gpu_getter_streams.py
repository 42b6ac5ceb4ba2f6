"""Getters of one state on several streams and threads."""
import threading
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_a_second_stream_waits_for_the_terms():
    """The terms are queued behind half a second of other work on one thread's stream; a getter on another thread
    and stream meanwhile gives the same currents."""
    import torch
    from activemodelbplus.integrator import Integrator, Model, Stencil
    f = np.random.default_rng(1).normal(-0.4, 0.1, (200, 300))
    sim = Integrator(f, Stencil(1e-3, 1, 1), Model(-0.25, 0, 0.25, 1, -1, -4, 0.05), seed=3)
    sim.run(2)
    streams = torch.cuda.Stream(), torch.cuda.Stream()
    for s in streams:  # nothing to allocate later, and the planes hold another step's terms
        with torch.cuda.stream(s):
            before = sim.current + [sim.chemical_potential]
    sim.run(1)
    got = {}

    def read(name, stream):
        with torch.cuda.stream(stream):
            if name == "first":
                torch.cuda._sleep(10 ** 9)  # cycles
            got[name] = sim.current + [sim.chemical_potential]
    threads = [threading.Thread(target=read, args=a) for a in zip(("first", "second"), streams)]
    torch.cuda.synchronize()
    threads[0].start()
    time.sleep(0.2)
    threads[1].start()
    for t in threads:
        t.join()
    for a, b in zip(got["first"], got["second"]):
        assert np.array_equal(a, b)
    assert np.array_equal(got["first"][0], sim.current[0]) and not np.array_equal(got["first"][0], before[0])
