"""The bins a plan accumulates from its largest distance (csrc/bins.cuh): the pair kernels leave out the clamp
to the overflow column only where the bins cover every distance."""
import math
import os
import subprocess

import numpy as np
import pytest

import ausaxs_b200 as ab
from ausaxs_b200 import _capi, hist

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SOURCE = r"""
#include <cstdio>
#include <cstdlib>
#include "bins.cuh"
int main(int, char** v) {
    const ausaxs_b200::BinSpan s = ausaxs_b200::bin_span(strtod(v[1], 0), strtof(v[2], 0), atoi(v[3]));
    std::printf("%d %d\n", s.bins, (int)s.covered);
}
"""


@pytest.fixture(scope="module")
def bin_span(tmp_path_factory):
    d = tmp_path_factory.mktemp("bins")
    (d / "main.cpp").write_text(SOURCE)
    subprocess.check_call(["g++", "-O3", "-std=c++17", "-x", "c++", "-I", os.path.join(ROOT, "ausaxs_b200", "csrc"),
                           str(d / "main.cpp"), "-o", str(d / "main")])
    return lambda dmax, inv_w, count: tuple(map(int, subprocess.check_output(
        [str(d / "main"), repr(float(dmax)), repr(float(inv_w)), str(count)]).split()))


@pytest.mark.parametrize("inv_w", [4.0, 10.0, 0.5])
@pytest.mark.parametrize("bin_count", [5, 11, 8000])
def test_distances_with_a_bin(bin_span, inv_w, bin_count):
    for dmax in (0.0, 1.0, 7.3, 100.0, 1999.4, 1999.6, 2e4, 1e6):
        need = max(math.ceil(dmax * inv_w) + 2, 11)
        assert bin_span(dmax, inv_w, bin_count) == (min(need, bin_count), int(need <= bin_count))


@pytest.mark.parametrize("dmax", [5.3e8, 5.4e8, 6e8, 1.7e9, 1e30, math.inf, math.nan])
@pytest.mark.parametrize("inv_w", [4.0, math.inf])
def test_distances_no_int_holds(bin_span, dmax, inv_w):
    """Finite coordinates of any size are accepted: from 2^31 bins on the bins cover nothing for certain."""
    assert bin_span(dmax, inv_w, 8000) == (8000, 0)


@pytest.mark.gpu
@pytest.mark.parametrize("far", [5.3e8, 6e8, 1.7e9, 1e30, 3e38])
def test_far_points_are_an_overflow(far, gpu_ctx):
    xyz = np.random.default_rng(1).normal(0, 5, (300, 3))
    xyz[::7, 0] = far
    m = ab.Molecule(atoms=xyz, ff_types=np.full(300, 3, np.int32), weights=np.full(300, 6.0), volume=5400.0)
    for manager in (hist.HistogramManagerMTFFAvg, hist.HistogramManagerMT):
        with pytest.raises(_capi.AusaxsError) as e:
            manager(m, True, 0.25, 8000, gpu_ctx).calculate_all()
        assert e.value.code == _capi.ERR_BIN_OVERFLOW
    calc = _capi.Calculator(gpu_ctx, 0.25, 8000)
    calc.enqueue_calculate_self(hist.pack(xyz, np.full(300, 6.0), False), 1, 0)
    with pytest.raises(_capi.AusaxsError) as e:
        calc.run()
    assert e.value.code == _capi.ERR_BIN_OVERFLOW
    calc.close()
