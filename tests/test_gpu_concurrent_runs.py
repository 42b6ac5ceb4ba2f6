"""FP64 runs of small grids on several streams and threads at once: their own results, and a share of the GPU."""
import threading
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _sims(n, side):
    from activemodelbplus.integrator import Integrator, Model, Stencil
    rng = np.random.default_rng(side)
    fields = [rng.normal(-0.4, 0.1, (side, side)) for _ in range(n)]
    return [Integrator(f, Stencil(1e-3, 1, 1), Model(-0.25, 0, 0.25, 1, -1, -4, 0.05), seed=i) for i, f in enumerate(fields)]


def _run(sims, streams, steps):
    """Seconds until all have taken their steps, one thread and stream each."""
    import torch
    failed = []

    def work(sim, stream):
        try:
            with torch.cuda.stream(stream):
                sim.run(steps)
        except Exception as e:
            failed.append(e)
    torch.cuda.synchronize()
    threads = [threading.Thread(target=work, args=a) for a in zip(sims, streams)]
    t0 = time.perf_counter()
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert not failed, failed
    return time.perf_counter() - t0


@pytest.mark.parametrize("side", [64, 128, 129, 130, 250])
def test_results_are_those_of_runs_alone(side):
    """The same bits as one run after the other (129^2 and 130^2: on both sides of the CTA width's rule)."""
    import torch
    n, steps = 6, 40
    together, alone = _sims(n, side), _sims(n, side)
    _run(together, [torch.cuda.Stream() for _ in range(n)], steps)
    for s in alone:
        s.run(steps)
    for a, b in zip(together, alone):
        assert np.array_equal(a.field, b.field)


def test_small_runs_share_the_gpu():
    """Eight 128^2 runs at once take at most 85 % of the time of one after the other (70 % with two CTAs of
    different runs per SM; 95 % where one run takes every SM whole)."""
    import torch
    n, steps = 8, 2000
    sims, streams = _sims(n, 128), [torch.cuda.Stream() for _ in range(n)]
    _run(sims, streams, 10)
    one = min(_run(sims[:1], streams[:1], steps) for _ in range(3))
    all_ = min(_run(sims, streams, steps) for _ in range(3))
    assert all_ <= 0.85 * n * one, (all_ / n / steps, one / steps)


@pytest.mark.parametrize("side", [64, 128])
def test_small_fp32_runs_share_the_gpu(side):
    """Eight FP32 runs at once, of the shape that the autotuner takes, need at most 70 % of the time of one after the
    other (about 30 % on a quarter of the GPU's threads each, 97 % where one run takes them all), and give the bits
    of runs alone."""
    import torch
    n, steps = 8, 4000
    from activemodelbplus.integrator import Integrator, Model, Stencil
    rng = np.random.default_rng(side)
    fields = [rng.normal(-0.4, 0.1, (side, side)) for _ in range(n)]
    sims, alone = ([Integrator(f, Stencil(1e-3, 1, 1), Model(-0.25, 0, 0.25, 1, -1, -4, 0.05), precision="f32c", seed=i)
                    for i, f in enumerate(fields)] for _ in range(2))
    streams = [torch.cuda.Stream() for _ in range(n)]
    _run(sims, streams, 10)
    for s in alone:
        s.run(10)
    assert all(np.array_equal(a.field, b.field) for a, b in zip(sims, alone))
    one = min(_run(sims[:1], streams[:1], steps) for _ in range(3))
    all_ = min(_run(sims, streams, steps) for _ in range(3))
    assert all_ <= 0.7 * n * one, (all_ / n / steps, one / steps, sims[0].kernel_config)
