"""A context per host thread, calls of different sizes at the same time."""
import threading

import numpy as np
import pytest

import ausaxs_b200 as ab
from ausaxs_b200 import _capi, hist, synth

pytestmark = pytest.mark.gpu


def test_contexts_of_several_threads():
    q = np.linspace(0.01, 0.5, 20)
    molecules = []
    for k, spread in enumerate((1.0, 3.0, 9.0, 20.0)):  # bins, and so shared memory, of different sizes
        xyz, ff = synth.globule(k + 1, 500)
        molecules.append(ab.Molecule(atoms=xyz * spread, ff_types=ff, waters=xyz[::4] * spread + 3.0, volume=9000.0))
    want, failed = [None] * 4, []

    def profile(m, ctx):
        return ab.profile(hist.HistogramManagerMTFFAvg(m, True, 0.25, 8000, ctx), q)

    for k, m in enumerate(molecules):
        ctx = _capi.Context(0)
        want[k] = profile(m, ctx)
        ctx.close()

    def work(k):
        try:
            ctx = _capi.Context(0)
            for _ in range(100):
                np.testing.assert_array_equal(profile(molecules[k], ctx), want[k])
            ctx.close()
        except BaseException as e:
            failed.append((k, e))

    threads = [threading.Thread(target=work, args=(k,)) for k in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed, failed


def test_weighted_contexts_of_several_threads():
    """The same through the kernel that weighted points of many weights take."""
    molecules = []
    for k, spread in enumerate((1.0, 3.0, 9.0, 20.0)):
        xyz, _ = synth.globule(k + 1, 500)
        molecules.append(ab.Molecule(atoms=xyz * spread, weights=1.0 + np.arange(500) % 40))
    want, failed = [], []

    def counts(m, ctx):
        return hist.HistogramManagerMT(m, True, 0.25, 8000, ctx).calculate_all().get_aa_counts()

    for m in molecules:
        ctx = _capi.Context(0)
        want.append(counts(m, ctx))
        ctx.close()

    def work(k):
        try:
            ctx = _capi.Context(0)
            for _ in range(100):
                np.testing.assert_array_equal(counts(molecules[k], ctx), want[k])
            ctx.close()
        except BaseException as e:
            failed.append((k, e))

    threads = [threading.Thread(target=work, args=(k,)) for k in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed, failed
