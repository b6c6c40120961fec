"""Batches of structures of very different extents: one launch's rows are as wide as its widest structure, and the small
ones' copies of the packed words have to fit beside it.  Counts and bits are those of lone calls."""
import numpy as np
import pytest

from ausaxs_b200 import hist, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("width", [0.25, 1.0, 2.0])
@pytest.mark.parametrize("spread", [1.0, 6.0, 30.0])
def test_batch_of_different_extents(spread, width, gpu_ctx):
    molecules = []
    for i, n in enumerate((40, 300, 900, 60, 2000, 500)):
        xyz, ff = synth.globule(i + 1, n)
        xyz = xyz * (spread if i in (2, 3) else 1.0)
        molecules.append(hist.Molecule(atoms=xyz, ff_types=ff, waters=xyz[::6] + 2.7, volume=18.0 * n))
    q = np.linspace(0.01, 0.6, 60)
    b = hist.BatchedProfiles(molecules, bin_width=width, ctx=gpu_ctx)
    I = b.debye_transform(q)
    for i, m in enumerate(molecules):
        h = hist.HistogramManagerMTFFAvg(m, True, width, 8000, gpu_ctx).calculate_all()
        got = b.histogram(i)
        np.testing.assert_array_equal(got["aa"][1:, 1:], h.get_raw_aa_counts_by_ff()[1:, 1:])
        np.testing.assert_array_equal(got["aw"][1:], h.get_raw_aw_counts_by_ff()[1:])
        np.testing.assert_array_equal(got["ww"], h.get_raw_ww_counts_by_ff())
        np.testing.assert_array_equal(I[i], hist.profile(hist.HistogramManagerMTFFAvg(m, True, width, 8000, gpu_ctx), q))
    b.close()
