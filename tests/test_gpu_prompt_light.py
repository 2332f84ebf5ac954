"""Point sources without a decay time: all detections fall into the first time bins,
and the histogram tile in shared memory takes them up to larger histograms (three
CTAs per SM instead of four).  Same counts on both sides of the rule, and a
histogram of 51 bins costs no more than one of 21."""
import os
import time

import numpy as np
import pytest

from crysplight_b200.params import OpticalParams, Readout, SipmGrid, TimeBinning, deg2rad_f32
from cases import BOX_BGO, BOX_CSI, CENTRE_BGO, CENTRE_CSI, GRID, INF, OP_BGO_ESR, OP_CSI_TEFLON

pytestmark = pytest.mark.gpu
NT = os.cpu_count() or 1
CLEAR = OpticalParams(1.79, 1.79, INF, INF, 0.99, False, True, deg2rad_f32(1.3), 1.0)


@pytest.mark.parametrize("box,op,pos,grid,bin_ns,nbins,tau,n", [
    (BOX_CSI, OP_CSI_TEFLON, CENTRE_CSI, GRID, 100.0, 50, 0.0, (1 << 17) - 1),
    (BOX_CSI, OP_CSI_TEFLON, CENTRE_CSI, GRID, 100.0, 50, 0.0, 1 << 17),
    (BOX_CSI, OP_CSI_TEFLON, CENTRE_CSI, GRID, 0.5, 114, 0.0, 140_000),      # the largest histogram with the tile,
    (BOX_CSI, OP_CSI_TEFLON, CENTRE_CSI, GRID, 0.5, 130, 0.0, 140_000),      # one without
    (BOX_CSI, CLEAR, CENTRE_CSI, SipmGrid(12.0, 4, 4), 10.0, 300, 79.0, 140_000),     # 128 slots,
    (BOX_CSI, CLEAR, CENTRE_CSI, SipmGrid(12.0, 4, 4), 10.0, 300, 80.0, 140_000),     # 144
    (BOX_BGO, OP_BGO_ESR, CENTRE_BGO, GRID, 1.0, 80, 0.0, 135_000)])
def test_counts_equal_the_oracle(engine, oracle, box, op, pos, grid, bin_ns, nbins, tau, n):
    tb = TimeBinning(bin_ns, nbins)
    kw = dict(n_photons=n, seed=41, pos=pos, tau_ns=tau)
    oacc, orec = oracle.run_photons_ka(box, op, grid, tb, return_records=True, nthreads=NT, **kw)
    dacc, drec = engine.run_photons_ka(box, op, grid, tb, return_records=True, **kw)
    plain = engine.run_photons_ka(box, op, grid, tb, **kw)
    assert np.array_equal(drec.status, orec.status) and np.array_equal(drec.idx, orec.idx)
    for acc in (dacc, plain):
        assert np.array_equal(acc.counts, oacc.counts) and acc.counters() == oacc.counters()
        assert np.array_equal(acc.first_ns.view(np.uint32), oacc.first_ns.view(np.uint32))


def test_prompt_light_costs_no_more_in_a_longer_histogram(engine):
    """4M photons of a clear crystal: 51 bins took 2.1 times as long as 21 on global
    atomics, and take as long with the tile."""
    def best(nbins):
        t = []
        for _ in range(6):
            t0 = time.perf_counter()
            engine.run_photons_ka(BOX_CSI, CLEAR, Readout(GRID), TimeBinning(100.0, nbins), n_photons=4_000_000,
                                  seed=3, pos=CENTRE_CSI, tau_ns=0.0)
            t.append(time.perf_counter() - t0)
        return min(t)
    assert best(50) < 1.5 * best(20)
