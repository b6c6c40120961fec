"""The last partners of a row in the reference's loops go through its scalar evaluator (fours first): contracted
products, ties away from zero.  On a line of points an eighth of a unit apart every odd separation is a tie between
two bins, so each such pair shows which evaluator took it."""
import numpy as np
import pytest

from ausaxs_b200 import hist
from oracle import py as O

pytestmark = pytest.mark.gpu

WIDTH = 0.25


def line(n, seed):
    """n points of a line in random order: lists and tiles see all separations."""
    xyz = np.zeros((n, 3))
    xyz[:, 0] = np.random.default_rng(seed).permutation(n) * (WIDTH / 2)
    return xyz


def compare(atoms, ff, waters, ctx):
    m = hist.Molecule(atoms=atoms, ff_types=ff, waters=waters, volume=18.0 * max(1, len(atoms)))
    h = hist.HistogramManagerMTFFAvg(m, True, WIDTH, 8000, ctx).calculate_all()
    o = O.hist_ff(0, O.pack_points(atoms, ff, True), O.pack_points(waters, np.ones(len(waters), np.int32), True), None, WIDTH,
                  8000, 18.0 * 0.334)
    np.testing.assert_array_equal(h.get_raw_aa_counts_by_ff()[1:, 1:], o.aa[1:, 1:])
    np.testing.assert_array_equal(h.get_raw_aw_counts_by_ff()[1:], o.aw[1:])
    np.testing.assert_array_equal(h.get_raw_ww_counts_by_ff(), o.ww)


# sizes about the inner tiles of 64 to 512 points: the last three points in one tile, or split one and two or two
# and one over the last two
@pytest.mark.parametrize("n", [255, 257, 258, 259, 260, 321, 513, 514, 515, 577, 769, 1025, 1026, 1027, 1537, 2049, 3073])
def test_waters(n, gpu_ctx):
    compare(line(9, 1), np.full(9, 3, np.int32), line(n, n), gpu_ctx)


@pytest.mark.parametrize("n", [257, 513, 769, 1025, 1026, 2049, 3073])
def test_atoms_of_one_type(n, gpu_ctx):
    compare(line(n, n), np.full(n, 3, np.int32), line(5, 2), gpu_ctx)


@pytest.mark.parametrize("n", [1027, 2051, 4101])
def test_atoms_of_two_types(n, gpu_ctx):
    """The type of the last three alone: its list has their tile to itself."""
    ff = np.full(n, 3, np.int32)
    ff[-n // 2:] = 11
    ff[::5] = 3
    ff[-3:] = 11
    compare(line(n, n), ff, line(5, 2), gpu_ctx)
