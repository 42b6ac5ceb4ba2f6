"""Radial binning with more edges than its shared histogram holds and with wave numbers out of FP32's range, and
the binning of a full power spectrum (amb_radial_spectrum)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _binned(power, shape, dx, dy, edges):
    ky, kx = (2 * np.pi * (np.fft.fftfreq(n) * n * (1.0 / (n * d))) for n, d in zip(shape, (dy, dx)))
    l = np.digitize(np.sqrt(kx[None, :] ** 2 + ky[:, None] ** 2), edges, right=True).ravel()
    n = len(edges)
    return np.bincount(l, weights=power.ravel(), minlength=n + 1)[:n], np.bincount(l, minlength=n + 1)[:n]


@pytest.mark.parametrize("nedges", [2048, 2049, 20000])
@pytest.mark.parametrize("d", [1.0, 1e-20, 1e20])
@pytest.mark.parametrize("shape", [(64, 96), (33, 70)])
def test_counts_and_sums(shape, nedges, d):
    """Counts are exact, sums to FP64 rounding of the transform (1e-9 of the largest)."""
    from activemodelbplus import analysis
    f = np.random.default_rng(nedges).standard_normal(shape)
    edges = np.linspace(0, 4.5, nedges + 1)[1:] / d
    k, S, c = analysis.structure_factor(f, dx=d, dy=d, edges=edges)
    p = np.abs(np.fft.fft2(f - f.mean()) * (d * d)) ** 2
    sums, counts = _binned(p, shape, d, d, edges)
    assert np.array_equal(c, counts[: len(k)])
    want = np.where(counts > 0, sums / np.maximum(counts, 1), 0)[: len(k)]
    assert np.abs(np.where(c > 0, S - want, 0)).max() <= 1e-9 * want.max()


def test_time_grows_with_the_logarithm_of_the_edges():
    """A bin is found by halving: 100000 edges (17 comparisons, and copies of 2.4 MB) take no more than eight
    times as long as 2000 (walking to the bin from the first one took seventy times as long)."""
    import torch
    from activemodelbplus import analysis
    f = torch.randn(1024, 1024, dtype=torch.float64, device="cuda")
    times = []
    for n in (2000, 100000):
        edges = np.linspace(0, 4.5, n + 1)[1:]
        analysis.structure_factor(f, edges=edges)
        best = 1e9
        for _ in range(5):
            a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            a.record()
            analysis.structure_factor(f, edges=edges)
            b.record()
            b.synchronize()
            best = min(best, a.elapsed_time(b))
        times.append(best)
    assert times[1] <= 8 * times[0], times


@pytest.mark.parametrize("shape", [(1, 1), (1, 9), (8, 1), (2, 2), (15, 33), (17, 65), (96, 50)])
@pytest.mark.parametrize("nedges", [7, 2048, 2049])
def test_power_spectrum(shape, nedges):
    """amb_radial_spectrum over every mode of a power spectrum: counts exact, sums to FP64 rounding."""
    import torch
    from activemodelbplus.integrator import _native as N
    power = np.random.default_rng(nedges).random(shape)
    edges = np.linspace(0, 4.0, nedges + 1)[1:]
    p, e = torch.from_numpy(power).cuda(), torch.from_numpy(edges).cuda()
    s = torch.full((nedges,), 7.0, dtype=torch.float64, device="cuda")
    c = torch.full((nedges,), 7, dtype=torch.int64, device="cuda")
    assert N.lib().amb_radial_spectrum(p.data_ptr(), *shape, 1.0, 1.25, e.data_ptr(), nedges, s.data_ptr(), c.data_ptr(),
                                       torch.cuda.current_stream().cuda_stream) == 0
    sums, counts = _binned(power, shape, 1.0, 1.25, edges)
    assert np.array_equal(c.cpu().numpy(), counts)
    assert np.abs(s.cpu().numpy() - sums).max() <= 1e-12 * max(sums.max(), 1.0)
