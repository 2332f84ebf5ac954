"""A site_light call that is refused half-way waits for its stream before its
temporaries go back to torch's allocator: the networks still write them."""
import os

import pytest

from crysplight_b200 import _lib
from crysplight_b200.params import Readout, SipmGrid

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def events():
    from crysplight_b200.fast_events import SurrogateEvents
    from crysplight_b200.surrogate import LightSurrogate
    root = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "crysplight_b200", "surrogates")
    ev = SurrogateEvents(LightSurrogate.load(os.path.join(root, "bgo_esr.npz")),
                         experts=[LightSurrogate.load(os.path.join(root, "bgo_esr_face.npz"))])
    yield ev
    ev.close()


@pytest.mark.parametrize("named_stream", [False, True])
def test_a_refused_call_leaves_its_stream_idle(events, named_stream):
    import torch
    ro = Readout(SipmGrid(6.0, 8, 8))
    L = torch.tensor([float(v) for v in events.sur.box_mm], device="cuda")
    # some milliseconds of networks between the first launch and the refusal (PDE above 1)
    xyz = torch.rand((400_000, 3), device="cuda") * L
    torch.cuda.synchronize()
    st = torch.cuda.Stream() if named_stream else torch.cuda.default_stream()
    handle = st.cuda_stream if named_stream else None
    with pytest.raises(_lib.CudaTransportError, match="cl_surrogate_combine"):
        events.site_light(xyz, ro=ro, pde=2.0, stream=handle)
    assert st.query()
    good = events.site_light(xyz[:2000], ro=ro, pde=0.4, stream=handle)
    again = events.site_light(xyz[:2000], ro=ro, pde=0.4)
    assert all(torch.equal(getattr(good, f), getattr(again, f)) for f in ("p", "tmean", "tsig", "spread", "flag"))
