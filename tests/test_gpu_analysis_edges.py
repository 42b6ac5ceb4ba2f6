"""Radial binning and component labelling where their kernels can go wrong: odd and tiny grids, one
column or row, tile borders and their periodic images, empty and full sets, edges that modes meet."""
import numpy as np
import pytest

from oracle import analysis as ref

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(1, 1), (1, 9), (8, 1), (2, 2), (15, 33), (16, 64), (17, 65), (31, 130), (96, 50)])
@pytest.mark.parametrize("edges", [None, np.linspace(0, 6, 2100)[1:], 2 * np.pi * np.arange(0, 9) / 16])
def test_structure_factor(shape, edges):
    """Counts are exact, sums to FP64 rounding of the transform (1e-9 of the largest)."""
    from activemodelbplus import analysis
    f = np.random.default_rng(shape[1]).standard_normal(shape)
    ed = analysis.default_edges() if edges is None else edges
    k, S, c = analysis.structure_factor(f, edges=edges)
    ky, kx = (2 * np.pi * np.fft.fftfreq(n) for n in shape)
    l = np.digitize(np.sqrt(kx[None, :] ** 2 + ky[:, None] ** 2), ed, right=True).ravel()
    p = np.abs(np.fft.fft2(f - f.mean())).ravel() ** 2
    assert np.array_equal(c, np.bincount(l, minlength=len(ed) + 1)[: len(k)])
    want = np.bincount(l, weights=p, minlength=len(ed) + 1)[: len(k)] / np.maximum(c, 1)
    assert np.array_equal(np.isnan(S), c == 0)
    assert np.abs(np.where(c > 0, S - want, 0)).max() <= 1e-9 * max(want.max(), 1.0)


@pytest.mark.parametrize("shape", [(1, 1), (1, 70), (40, 1), (2, 2), (16, 64), (17, 65), (33, 129), (100, 200)])
@pytest.mark.parametrize("density", [0.0, 0.3, 0.6, 0.9, 1.0])
def test_labels(shape, density):
    from activemodelbplus import analysis
    f = (np.random.default_rng(shape[0]).random(shape) < density).astype(np.float32)
    labels, n = analysis.label_droplets(f, 0.5)
    assert n == ref.count_droplets(f, 0.5)
    lab = labels.cpu().numpy()
    assert np.array_equal(lab >= 0, f > 0.5)
    flat = lab.ravel()
    for r in np.unique(flat[flat >= 0]):  # the smallest site of its component
        assert np.flatnonzero(flat == r)[0] == r
    for axis in (0, 1):  # neighbours of the set share their label
        other, both = np.roll(lab, -1, axis), (lab >= 0) & (np.roll(lab, -1, axis) >= 0)
        assert np.array_equal(lab[both], other[both])
