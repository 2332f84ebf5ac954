"""Launch shapes chosen by size: few photons are spread thinly over the GPU
(some photons per warp), many are claimed in chunks; and the kernels that
evaluate the logs in place give the results of those that look them up."""
import os

import numpy as np
import pytest

from crysplight_b200 import _lib
from cases import (BOX_BGO, BOX_CSI, CENTRE_BGO, CENTRE_CSI, GRID, OP_ALL, OP_BGO_ESR, OP_CSI_TEFLON, RO_ALL, TAU_BGO,
                   TAU_CSI, TB, TB80)
from test_zz_no_alloc import _noalloc, _same

pytestmark = pytest.mark.gpu
NT = os.cpu_count() or 1


@pytest.mark.parametrize("n", [1, 2, 33, 1183, 1185, 37_887, 37_888])
def test_every_photon_is_transported_once(engine, oracle, n):
    kw = dict(n_photons=n, seed=77, tau_ns=TAU_CSI, pos=CENTRE_CSI)
    dacc, drec = engine.run_photons_ka(BOX_CSI, OP_CSI_TEFLON, GRID, TB80, return_records=True, **kw)
    oacc, orec = oracle.run_photons_ka(BOX_CSI, OP_CSI_TEFLON, GRID, TB80, return_records=True, nthreads=NT, **kw)
    for name in ("status", "idx", "t", "bounces"):
        assert np.array_equal(getattr(drec, name), getattr(orec, name)), name
    _same(dacc, oacc)


@pytest.mark.parametrize("box,op,ro,tb,pos,tau", [
    (BOX_BGO, OP_BGO_ESR, GRID, TB80, CENTRE_BGO, TAU_BGO), (BOX_BGO, OP_BGO_ESR, GRID, TB, CENTRE_BGO, TAU_BGO),
    (BOX_CSI, OP_CSI_TEFLON, GRID, TB, CENTRE_CSI, TAU_CSI), (BOX_CSI, OP_ALL, RO_ALL, TB80, CENTRE_CSI, 800.0)])
def test_evaluated_logs_equal_the_tables(engine, box, op, ro, tb, pos, tau):
    kw = dict(n_photons=20_000, seed=5, tau_ns=tau)
    rc, msg, got = _noalloc(box, op, ro, tb, positions=[pos], **kw)
    assert rc == _lib.CL_OK, msg
    _same(got, engine.run_photons_ka(box, op, ro, tb, pos=pos, **kw))
