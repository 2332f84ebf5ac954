"""Host arrays of a call: small ones travel together through the handle's
host buffer, large ones by themselves.  Sizes on both sides of each
limit, against the oracle."""
import os

import numpy as np
import pytest

from crysplight_b200.params import TimeBinning
from cases import BOX_CSI, GRID, OP_CSI_TEFLON, TAU_CSI, TB80
from test_zz_no_alloc import _same

pytestmark = pytest.mark.gpu
NT = os.cpu_count() or 1


def _points(n, times):
    rng = np.random.default_rng(n)
    pts = (rng.uniform(0.02, 0.98, (n, 3)) * np.array(BOX_CSI.L)).astype(np.float32)
    return pts, rng.uniform(0.0, 50.0, n).astype(np.float32) if times else None


# 4,096 positions fill the inputs' 64 KB; 64 cells x 1,022 bins, first times and
# counters the outputs' 256 KB
@pytest.mark.parametrize("npos,nbins,times,records", [
    (1, 80, False, False), (3, 80, True, True), (4095, 1021, False, False), (4096, 1021, True, False),
    (4097, 1022, True, True), (4097, 40, False, False), (5, 1022, False, False)])
def test_point_sources(engine, oracle, npos, nbins, times, records):
    pts, t0 = _points(npos, times)
    tb = TimeBinning(100.0, nbins)
    kw = dict(n_photons=9001, seed=31, tau_ns=TAU_CSI, positions=pts, t0s=t0, return_records=records)
    d = engine.run_photons_ka(BOX_CSI, OP_CSI_TEFLON, GRID, tb, **kw)
    o = oracle.run_photons_ka(BOX_CSI, OP_CSI_TEFLON, GRID, tb, nthreads=NT, **kw)
    if records:
        for name in ("status", "idx", "t", "bounces"):
            assert np.array_equal(getattr(d[1], name), getattr(o[1], name)), name
        d, o = d[0], o[0]
    _same(d, o)


# 2,304 sources and 507 segments fit, 2,336 and 508 do not
@pytest.mark.parametrize("n_src,n_seg,times", [
    (1, 1, False), (2304, 507, True), (2304, 508, False), (2336, 507, False), (2336, 508, True)])
def test_segments(engine, oracle, n_src, n_seg, times):
    pts, t0 = _points(n_src, times)
    seg = np.arange(n_src) * n_seg // n_src
    kw = dict(sources=pts, photons_per_source=np.full(n_src, 3), segment_of_source=seg, n_segments=n_seg, t0s=t0,
              seed=8, tau_ns=TAU_CSI)
    d = engine.run_segments(BOX_CSI, OP_CSI_TEFLON, GRID, TB80, **kw)
    o = oracle.run_segments(BOX_CSI, OP_CSI_TEFLON, GRID, TB80, nthreads=NT, **kw)
    for name in ("maps", "tmin", "npe"):
        assert np.array_equal(getattr(d, name), o[name]), name
    assert d.counters == o["counters"]
