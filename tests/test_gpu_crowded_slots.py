"""Segment mode with many photons per (segment, SiPM) slot: a warp's detections
of a slot are added together (from 1,024 photons a slot on for grids of fewer
than 64 cells, from 4,096 on for others).  Same maps, times and moments on both
sides of the rule, and one slot that all photons share costs no more than many."""
import os
import time

import numpy as np
import pytest

from crysplight_b200.params import OpticalParams, Readout, SipmGrid, deg2rad_f32
from crysplight_b200.surrogate import scan_light
from cases import BOX_BGO, BOX_CSI, CENTRE_CSI, GRID, INF, OP_ALL, OP_BGO_ESR, OP_CSI_TEFLON, RO_ALL, TB80

pytestmark = pytest.mark.gpu
NT = os.cpu_count() or 1
ONE = SipmGrid(48.0, 1, 1)
# matched index, no bulk interaction: most photons leave on the first step
CLEAR = OpticalParams(1.79, 1.79, INF, INF, 0.99, False, True, deg2rad_f32(1.3), 1.0)


def _kw(n_seg, photons):
    pts = np.array(CENTRE_CSI, np.float32) + np.linspace(-9.0, 9.0, n_seg, dtype=np.float32)[:, None]
    return dict(sources=pts, photons_per_source=np.full(n_seg, photons, np.int64),
                segment_of_source=np.arange(n_seg, dtype=np.int32), n_segments=n_seg, seed=91, pid_offset=3,
                tau_ns=1000.0)


@pytest.mark.parametrize("box,op,ro,n_seg,photons", [
    (BOX_CSI, OP_CSI_TEFLON, Readout(ONE), 1, 1023), (BOX_CSI, OP_CSI_TEFLON, Readout(ONE), 1, 1024),
    (BOX_CSI, OP_CSI_TEFLON, Readout(SipmGrid(24.0, 2, 2)), 3, 4097),
    (BOX_CSI, CLEAR, Readout(SipmGrid(24.0, 2, 2)), 3, 50_001),
    (BOX_CSI, CLEAR, Readout(GRID), 1, 64 * 4096 - 1), (BOX_CSI, CLEAR, Readout(GRID), 1, 64 * 4096),
    (BOX_BGO, OP_BGO_ESR, Readout(SipmGrid(24.0, 2, 2), two_sided=True), 2, 9000),
    (BOX_CSI, OP_ALL, RO_ALL, 1, 64 * 4096 + 17), (BOX_CSI, OP_CSI_TEFLON, Readout(SipmGrid(1.5, 32, 32)), 1, 4097)])
def test_maps_and_records_equal_the_oracle(engine, oracle, box, op, ro, n_seg, photons):
    kw = _kw(n_seg, photons)
    ores, orec = oracle.run_segments(box, op, ro, TB80, nthreads=NT, return_records=True, **kw)
    dres, drec = engine.run_segments(box, op, ro, TB80, return_records=True, **kw)
    plain = engine.run_segments(box, op, ro, TB80, **kw)
    for name in ("status", "idx", "t", "bounces"):
        assert np.array_equal(getattr(drec, name), getattr(orec, name)), name
    for res in (dres, plain):
        assert np.array_equal(res.maps, ores["maps"])
        assert np.array_equal(res.tmin.view(np.uint32), ores["tmin"].view(np.uint32))
        assert np.array_equal(res.npe, ores["npe"]) and res.counters == ores["counters"]


@pytest.mark.parametrize("op", [OP_CSI_TEFLON, CLEAR, OP_ALL])
def test_moments_are_the_sums_of_smaller_batches(engine, op):
    """Integer sums: 4,096 photons in one slot are those of eight batches of 512,
    which take the other kernel."""
    pts = np.array([CENTRE_CSI], np.float32)
    kw = dict(points=pts, seed=5, tau_ns=1000.0)
    whole = scan_light(engine, BOX_CSI, op, Readout(ONE), photons_per_point=4096, **kw)
    parts = [scan_light(engine, BOX_CSI, op, Readout(ONE), photons_per_point=512, pid_offset=512 * i, **kw)
             for i in range(8)]
    for name in ("counts", "tsum", "tsum2"):
        assert np.array_equal(getattr(whole, name), sum(getattr(p, name) for p in parts)), name
    assert np.array_equal(whole.tmin, np.minimum.reduce([p.tmin for p in parts]))
    assert whole.counters == {k: sum(p.counters[k] for p in parts) for k in whole.counters}


def test_one_slot_costs_no_more_than_many(engine):
    """4M photons into one slot and into 16,384.  Added one by one, the first took
    2.4 times as long as the second; together it takes 0.8 of it."""
    def best(n_seg):
        kw = _kw(n_seg, 4_000_000 // n_seg)
        t = []
        for _ in range(6):
            t0 = time.perf_counter()
            engine.run_segments(BOX_CSI, CLEAR, Readout(ONE), TB80, **kw)
            t.append(time.perf_counter() - t0)
        return min(t)
    assert best(1) < 1.5 * best(16_384)
