"""A detection is booked inside the pixel grid whatever its pitch: x / pitch beyond
2^31 belongs to the last pixel (src/transport.jl:96-108 clamps the index)."""
import numpy as np
import pytest

from crysplight_b200.params import Box, Readout, SipmGrid
from cases import BOX_CSI, CENTRE_CSI, OP_CSI_TEFLON, TB

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("box,pitch", [(BOX_CSI, 1e-6), (BOX_CSI, 1e-8), (BOX_CSI, 1e-12), (BOX_CSI, 1e-38),
                                       (Box((3e12, 3e12, 37.2)), 6.0)])
def test_all_detections_in_the_last_pixel(engine, box, pitch):
    ro = Readout(SipmGrid(pitch, 5, 3))
    pos = tuple(float(v) / 2 for v in box.L)
    kw = dict(n_photons=20_000, seed=3, pos=pos, tau_ns=10.0, max_bounces=200)
    acc, rec = engine.run_photons_ka(box, OP_CSI_TEFLON, ro, TB, return_records=True, **kw)
    det = rec.status == 1
    assert acc.ndet == det.sum() > 100
    assert (rec.idx[det] == 15).all()
    assert acc.counts.reshape(5, 3, -1, order="F").sum(2)[4, 2] == acc.ndet
    res = engine.run_segments(box, OP_CSI_TEFLON, ro, TB, sources=np.array([pos], np.float32),
                              photons_per_source=[20_000], segment_of_source=[0], n_segments=1, seed=3, tau_ns=10.0,
                              max_bounces=200)
    assert res.maps[4, 2, 0] == res.maps.sum() == res.npe[0] == acc.ndet
