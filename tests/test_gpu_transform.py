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


@pytest.mark.parametrize("spread", [1.0, 5.0, 9.0])
@pytest.mark.parametrize("k,nq", [(3, 200), (40, 100), (40, 200), (40, 600), (200, 30), (200, 300)])
def test_batches_equal_single_calls(spread, k, nq, gpu_ctx):
    """Batches choose their q values per CTA by all of their structures: the same bits as each alone."""
    molecules = []
    for i in range(k):
        xyz, ff = synth.globule(i, 40 + 7 * (i % 9))
        molecules.append(hist.Molecule(atoms=xyz * spread, ff_types=ff, waters=xyz[::8] * spread + 3.1, volume=18.0 * len(xyz)))
    q = np.linspace(0.005, 0.7, nq)
    b = hist.BatchedProfiles(molecules, ctx=gpu_ctx)
    I = b.debye_transform(q)
    b.close()
    for i in range(0, k, max(1, k // 9)):
        np.testing.assert_array_equal(I[i], hist.profile(hist.HistogramManagerMTFFAvg(molecules[i], True, 0.25, 8000, gpu_ctx), q))
