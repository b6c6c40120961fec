"""One-shot calls share a context's buffers and keep its last plan: calls in any order give what a context that
makes only the one call gives."""
import numpy as np
import pytest

import ausaxs_b200 as ab
from ausaxs_b200 import _capi, hist, synth
from oracle import py as O

pytestmark = pytest.mark.gpu

Q = np.linspace(0.01, 0.5, 40)
MANAGERS = {"ffavg": hist.HistogramManagerMTFFAvg, "ffexplicit": hist.HistogramManagerMTFFExplicit, "mt": hist.HistogramManagerMT}


def molecule(seed, n=600, nw=100):
    xyz, ff = synth.globule(seed, n)
    rng = np.random.default_rng(seed)
    ff = np.resize(np.array([3, 7, 11, 3], np.int32), n)  # the same types in every molecule of a size
    return ab.Molecule(atoms=xyz, ff_types=ff, weights=synth.ff_charge(ff), waters=rng.normal(0, 12, (nw, 3)),
                       water_weights=np.full(nw, 10.0), volume=18.0 * n)


def profile(kind, m, ctx):
    return ab.profile(MANAGERS[kind](m, True, 0.25, 8000, ctx), Q)


def alone(kind, m):
    ctx = _capi.Context(0)
    I = profile(kind, m, ctx)
    ctx.close()
    return I


def load_only(how, m, ctx):
    """A call that loads the molecule's points and makes no plan."""
    a, w, _ = m.compact_ff()
    if how == "grid":
        assert len(_capi.grid_exv(ctx, a, w)[0]) > 0
    else:
        bad = ab.Molecule(atoms=m.atoms, ff_types=np.full(len(m.atoms), 15, np.int32), waters=m.waters, volume=m.volume)
        with pytest.raises(_capi.AusaxsError) as e:
            profile("ffavg", bad, ctx)
        assert e.value.code == _capi.ERR_FORM_FACTOR


@pytest.mark.parametrize("how", ["grid", "rejected"])
@pytest.mark.parametrize("kind", list(MANAGERS))
def test_larger_load_between(kind, how):
    """The larger load moves the point buffers that the kept plan's tables point into."""
    ctx = _capi.Context(0)
    for n in (5000, 20000):
        first = molecule(3)
        np.testing.assert_array_equal(profile(kind, first, ctx), alone(kind, first))
        load_only(how, molecule(4, n, n // 5), ctx)
        again = molecule(5)
        np.testing.assert_array_equal(profile(kind, again, ctx), alone(kind, again))
    ctx.close()


@pytest.mark.parametrize("kind", list(MANAGERS))
def test_rejected_call_leaves_no_plan(kind):
    """A call whose bins do not fit on chip is refused however often it is made, and the calls around it are as ever."""
    ctx = _capi.Context(0)
    m = molecule(3)
    for _ in range(2):
        for _ in range(2):
            with pytest.raises(_capi.AusaxsError) as e:
                ab.profile(MANAGERS[kind](m, True, 5e-4, 400000, ctx), Q)
            assert e.value.code == _capi.ERR_CAPACITY
        np.testing.assert_array_equal(profile(kind, m, ctx), alone(kind, m))
    ctx.close()


@pytest.mark.parametrize("classes", [1, 5, 8, 15])
@pytest.mark.parametrize("n", [60, 301, 900])
def test_weighted_points_of_one_kind(classes, n):
    """Only atoms, or only waters, after a molecule of both: no rows of the missing kind are read.  The weights are
    whole numbers, so the sums are exact; a bin's mean is within the quantisation of its offsets."""
    ctx = _capi.Context(0)
    rng = np.random.default_rng(n + classes)
    w = (1.0 + np.arange(n) % classes)[rng.permutation(n)]
    xyz, none = synth.globule(n, n)[0], np.zeros((0, 3))
    both = ab.Molecule(atoms=xyz, weights=w, waters=xyz[::2] + 7.3, water_weights=w[::2])
    for atoms, waters in ((True, True), (True, False), (False, True)):
        m = ab.Molecule(atoms=both.atoms if atoms else none, weights=w if atoms else w[:0],
                        waters=both.waters if waters else none, water_weights=w[::2] if waters else w[:0])
        h = hist.HistogramManagerMT(m, True, 0.25, 8000, ctx).calculate_all()
        o = O.hist_simple(*m.compact_w(), 0.25, 8000)
        assert h.max_bin == len(o.tot)
        for got, want in ((h.get_aa_counts(), o.aa), (h.get_aw_counts(), o.aw), (h.get_ww_counts(), o.ww),
                          (h.get_counts(), o.tot)):
            np.testing.assert_array_equal(got, want)
        np.testing.assert_allclose(h.get_d_axis(), o.d_axis, rtol=0, atol=0.25 * 2.0 ** -15)
    ctx.close()


@pytest.mark.parametrize("classes", [(4, 4), (4, 9), (15, 15), (6, 40)])
def test_weights_change_between_calls(classes):
    """Molecules of one shape and other weights: the same number of classes with other values and shares, another
    number, and more than the route by class takes."""
    ctx = _capi.Context(0)
    n = 700
    xyz = synth.globule(2, n)[0]
    for k in range(4):
        c = classes[k % 2]
        rng = np.random.default_rng(10 * k + c)
        values = rng.permutation(60)[:c] - 9.0
        m = ab.Molecule(atoms=xyz + 0.01 * k, weights=values[np.concatenate([np.arange(c), rng.integers(0, 1 + c // 2, n - c)])],
                        waters=xyz[::5] + 6.1, water_weights=np.full(len(xyz[::5]), 10.0 + k))
        h = hist.HistogramManagerMT(m, True, 0.25, 8000, ctx).calculate_all()
        o = O.hist_simple(*m.compact_w(), 0.25, 8000)
        assert h.max_bin == len(o.tot)
        for got, want in ((h.get_aa_counts(), o.aa), (h.get_aw_counts(), o.aw), (h.get_ww_counts(), o.ww)):
            np.testing.assert_array_equal(got, want)
    ctx.close()


@pytest.mark.parametrize("n", [30, 119, 120, 121, 239, 240, 241, 700])
def test_weights_by_class_or_value(n):
    """15 classes (225 count rows): few points go by value, sooner in a one-shot call than in a kept structure.  The
    weights are whole numbers, so every route gives the oracle's sums."""
    rng = np.random.default_rng(n)
    xyz = synth.globule(5, n)[0]
    w = (1.0 + np.arange(n) % 15)[rng.permutation(n)]
    m = ab.Molecule(atoms=xyz, weights=w)
    ctx = _capi.Context(0)
    manager = hist.HistogramManagerMT(m, True, 0.25, 8000, ctx)
    h = manager.calculate_all()
    a, waters = m.compact_w()
    kept = _capi.Structure(ctx, a, waters, ff_typed=False)
    r, bufs = kept.histogram(manager.config(), 8000)
    o = O.hist_simple(a, waters, 0.25, 8000)
    assert h.max_bin == r.max_bin == len(o.tot)
    np.testing.assert_array_equal(h.get_aa_counts(), o.aa)
    np.testing.assert_array_equal(bufs["aa"][:r.max_bin], o.aa)
    kept.close()
    ctx.close()
