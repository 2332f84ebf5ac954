"""Bulk lengths that no crystal has (negative, zero) are accepted, and a photon's
path under them is still the reference's: a path length below zero competes with
the wall in a step (src/transport.jl:127-145), and not in a further UNIFIED try at
the same wall (src/optics.jl:54-78)."""
import os

import numpy as np
import pytest

from crysplight_b200.params import OpticalParams, Readout, deg2rad_f32
from cases import BOX_BGO, BOX_CSI, CENTRE_CSI, GRID, INF, RO_ALL, TB80

pytestmark = pytest.mark.gpu
NT = os.cpu_count() or 1
ROUGH = deg2rad_f32(35.0)      # many facet tries fail


@pytest.mark.parametrize("spec", [False, True])
@pytest.mark.parametrize("abs_len,ray_len", [(3115.0, -5.0), (INF, -40.0), (-5.0, 346.0), (-5.0, -7.0), (-3.0, INF),
                                             (0.0, 346.0), (3115.0, 0.0), (1e-38, 2.0), (-0.0, -0.0)])
def test_records_equal_the_oracle(engine, oracle, abs_len, ray_len, spec):
    op = OpticalParams(1.79, 1.45, abs_len, ray_len, 0.97, spec, True, ROUGH, 1.0)
    for box, ro, pos in ((BOX_CSI, Readout(GRID), CENTRE_CSI), (BOX_CSI, RO_ALL, (47.9, 0.1, 37.0)),
                         (BOX_BGO, Readout(GRID, two_sided=True), (0.0, 48.0, 0.0))):
        kw = dict(n_photons=20_000, seed=17, pos=pos, tau_ns=10.0, max_bounces=300)
        dacc, drec = engine.run_photons_ka(box, op, ro, TB80, return_records=True, **kw)
        oacc, orec = oracle.run_photons_ka(box, op, ro, TB80, return_records=True, nthreads=NT, **kw)
        for name in ("status", "idx", "bounces"):
            assert np.array_equal(getattr(drec, name), getattr(orec, name)), name
        assert np.array_equal(drec.t.view(np.uint32), orec.t.view(np.uint32))
        assert np.array_equal(dacc.counts, oacc.counts) and dacc.counters() == oacc.counters()
