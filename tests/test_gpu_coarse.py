"""Histograms of few bins: the one-atomic-per-pair kernel keeps several copies of its packed words there.  Counts equal
the oracle's exactly; distance axes are within the 16-bit quantisation of the in-bin offset (width * 2^-15)."""
import numpy as np
import pytest

from ausaxs_b200 import hist, synth
from oracle import py as O

pytestmark = pytest.mark.gpu


def check(xyz, ff, waters, width, ctx):
    m = hist.Molecule(atoms=xyz, ff_types=ff, waters=waters, volume=18.0 * len(xyz))
    h = hist.HistogramManagerMTFFAvg(m, True, width, 8000, ctx).calculate_all()
    o = O.hist_ff(0, O.pack_points(xyz, ff, True), O.pack_points(waters, np.ones(len(waters), np.int32), True), None, width, 8000,
                  18.0 * 0.334)
    assert h.max_bin == len(o.d_axis)
    np.testing.assert_array_equal(h.get_raw_aa_counts_by_ff()[1:, 1:], o.aa[1:, 1:])
    np.testing.assert_array_equal(h.get_raw_aw_counts_by_ff()[1:], o.aw[1:])
    np.testing.assert_array_equal(h.get_raw_ww_counts_by_ff(), o.ww)
    np.testing.assert_allclose(h.get_d_axis(), o.d_axis, rtol=0, atol=width * 2.0 ** -15)


@pytest.mark.parametrize("width", [0.5, 1.0, 1.5, 2.0, 4.0])
@pytest.mark.parametrize("types", [1, 2, 13])
@pytest.mark.parametrize("n,nw", [(257, 700), (1301, 260), (4099, 33)])
def test_few_bins(n, nw, types, width, gpu_ctx):
    xyz, _ = synth.globule(n, n)
    ff = (1 + np.random.default_rng(types).integers(0, types, n)).astype(np.int32)
    check(xyz, ff, np.random.default_rng(n).normal(0, 14, (nw, 3)), width, gpu_ctx)


@pytest.mark.parametrize("n", [9000, 20011])
def test_long_runs_between_flushes(n, gpu_ctx):
    """Enough tiles per CTA that the 16-bit counts of the fullest bins are flushed on the way."""
    xyz, _ = synth.globule(n, n)
    check(xyz, np.full(n, 3, np.int32), xyz[::40] + 3.3, 3.0, gpu_ctx)


@pytest.mark.parametrize("spacing", [0.01, 2.0, 4.0])
def test_few_distances(spacing, gpu_ctx):
    """Nearly all pairs in a few bins: segments are taken back at any number of copies, and end with two atomics
    per pair, many of them between two flushes."""
    g = np.arange(13, dtype=np.float64) * spacing
    xyz = np.stack(np.meshgrid(g, g, g, indexing="ij"), -1).reshape(-1, 3)
    check(xyz, np.where(np.arange(len(xyz)) % 3 == 0, 7, 3).astype(np.int32), xyz[:300] + 0.25, 4.0, gpu_ctx)
