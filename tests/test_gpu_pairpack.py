"""The one-atomic-per-pair histogram kernel at the sizes and inputs where it can go wrong.

Counts must equal the oracle's exactly; distance axes are within the 16-bit quantisation of the in-bin
offset (bin_width * 2^-15, twice the bound of a bin's mean).
"""
import numpy as np
import pytest

from ausaxs_b200 import hist, synth
from oracle import py as O

pytestmark = pytest.mark.gpu

Z_EXV = 18.0 * 0.334


def check(xyz, ff, waters, width, ctx, exv=None, grid=False):
    m = hist.Molecule(atoms=xyz, ff_types=ff, waters=waters, exv=exv, volume=18.0 * len(xyz))
    if grid:
        h = hist.HistogramManagerMTFFGrid(m, width, 8000, ctx).calculate_all()
    else:
        h = hist.HistogramManagerMTFFAvg(m, True, width, 8000, ctx).calculate_all()
    pack = lambda p, t: O.pack_points(p, np.full(len(p), t, np.int32) if np.isscalar(t) else t, True)
    o = O.hist_ff(2 if grid else 0, pack(xyz, ff), pack(waters, 1), pack(exv, 0) if grid else None, width, 8000, Z_EXV)
    assert h.max_bin == len(o.d_axis)
    # rows 0 are excluded-volume marginals, scaled in floating point
    np.testing.assert_array_equal(h.get_raw_aa_counts_by_ff()[1:, 1:], o.aa[1:, 1:])
    np.testing.assert_array_equal(h.get_raw_aw_counts_by_ff()[1:], o.aw[1:])
    np.testing.assert_array_equal(h.get_raw_ww_counts_by_ff(), o.ww)
    np.testing.assert_allclose(h.get_d_axis(), o.d_axis, rtol=0, atol=width * 2.0 ** -15)


@pytest.mark.parametrize("width", [0.25, 0.1])
@pytest.mark.parametrize("n,nw", [(1, 0), (2, 1), (3, 2), (4, 3), (5, 7), (63, 64), (255, 5), (256, 0), (257, 1), (511, 129),
                                  (513, 64), (1025, 255), (2311, 517)])
def test_sizes(n, nw, width, gpu_ctx):
    xyz, ff = synth.globule(n + 3, n)
    waters = np.random.default_rng(n).normal(0, 15, (nw, 3))
    check(xyz, ff, waters, width, gpu_ctx)


@pytest.mark.parametrize("types", [1, 2, 7, 13])
def test_types(types, gpu_ctx):
    xyz, _ = synth.globule(5, 1900)
    ff = (1 + np.random.default_rng(types).integers(0, types, len(xyz))).astype(np.int32)
    check(xyz, ff, xyz[::9] + 0.37, 0.25, gpu_ctx)


@pytest.mark.parametrize("width", [0.25, 1.0])
@pytest.mark.parametrize("spacing", [0.0, 0.5, 1.0, 1.37])
def test_few_distances(spacing, width, gpu_ctx):
    """Lattices (and coincident points): words fill within a few pairs, so segments fail their check, are
    taken back and end with two atomics per pair."""
    g = np.arange(12, dtype=np.float64) * spacing
    xyz = np.stack(np.meshgrid(g, g, g, indexing="ij"), -1).reshape(-1, 3)
    ff = np.where(np.arange(len(xyz)) % 3 == 0, 7, 3).astype(np.int32)
    check(xyz, ff, xyz[:200] + 0.25, width, gpu_ctx)


def test_types_sorted_by_index(gpu_ctx):
    """All atoms of a type together: every self tile of a list is crossed by the diagonal or empty."""
    xyz, ff = synth.globule(8, 3001)
    check(xyz, np.sort(ff), np.zeros((0, 3)), 0.25, gpu_ctx)


def test_grid_passes(gpu_ctx):
    xyz, ff = synth.globule(4, 700)
    waters = np.random.default_rng(1).normal(0, 14, (77, 3))
    x = np.random.default_rng(2).normal(0, 9, (1301, 3))  # off the lattice: dummy pairs through this kernel
    check(xyz, ff, waters, 0.1, gpu_ctx, x, True)


@pytest.mark.parametrize("classes", [1, 2, 4, 15, 16, 700])
@pytest.mark.parametrize("n,nw", [(5, 0), (257, 3), (1301, 300)])
def test_weights_by_class(classes, n, nw, gpu_ctx):
    """Weighted (Simple) histograms: up to 15 distinct weights go by class of weight, more by value.  A pair's
    weight product is kept to max|w|^2 2^-30."""
    rng = np.random.default_rng(classes)
    xyz, _ = synth.globule(n + 1, n)
    values = rng.uniform(-2, 16, classes)
    w = values[rng.integers(0, classes, n)]
    waters = rng.normal(0, 14, (nw, 3))
    ww = np.full(nw, 9.25)
    m = hist.Molecule(atoms=xyz, weights=w, waters=waters, water_weights=ww)
    h = hist.HistogramManagerMT(m, True, 0.25, 8000, gpu_ctx).calculate_all()
    sets = [hist.pack(xyz, w, False), hist.pack(waters, ww, False)]
    jobs = [(0, None, 1, 0)] + ([(0, 1, 1, 0), (1, None, 1, 1)] if nw else [])
    o = O.calculator(sets, jobs, 0.25, 8000)
    top = max(np.abs(w).max(), ww.max() if nw else 0.0) ** 2
    for got, key in ((h.get_aa_counts(), (0, 0)), (h.get_aw_counts(), (1, 0)), (h.get_ww_counts(), (0, 1))):
        if key not in o:
            assert not got.any()
            continue
        value, count, _ = o[key]
        k = len(got)
        # (the self diagonal in bin 0 is not quantised; its sum runs in another order)
        assert np.all(np.abs(got - value[:k]) <= count[:k] * top * 2.0 ** -30 + 1e-12 * np.abs(value[:k]))
        assert not value[k:].any() or not np.abs(value[k:]).max() > count[k:].max() * top * 2.0 ** -30
