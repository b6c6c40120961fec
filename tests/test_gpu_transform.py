"""The FP64 Debye transform at the edges of its tilings: q values per CTA by the q count, chunks of bins."""
import numpy as np
import pytest

from ausaxs_b200 import hist, synth
from oracle import py as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", params=[1.0, 12.0], ids=["compact", "spread"])
def histogram(request, gpu_ctx):
    """(device histogram, oracle's): under a hundred bins, or more than any tiling's chunk but the widest."""
    xyz, ff = synth.globule(6, 400)
    xyz, waters = xyz * request.param, xyz[::7] * request.param + 2.9
    m = hist.Molecule(atoms=xyz, ff_types=ff, waters=waters, volume=18.0 * len(xyz))
    o = O.hist_ff(0, O.pack_points(xyz, ff, True), O.pack_points(waters, np.ones(len(waters), np.int32), True), None, 0.25,
                  8000, 18.0 * 0.334)
    return hist.HistogramManagerMTFFAvg(m, True, 0.25, 8000, gpu_ctx).calculate_all(), o


@pytest.mark.parametrize("nq", [1, 2, 3, 295, 296, 297, 592, 593, 2368, 2369, 2391])
def test_q_counts(nq, histogram):
    h, o = histogram
    q = np.linspace(0.004, 0.9, nq)
    I = h.debye_transform(q)[1]
    np.testing.assert_allclose(I, O.debye_ff(0, o, q)[0], rtol=1e-6)  # (the mean distances are quantised)
