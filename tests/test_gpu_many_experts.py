"""Any number of experts: one split serves 256, and the later ones take their sites
over, as a single split with all of them would."""
import os

import numpy as np
import pytest

from crysplight_b200.params import Readout, SipmGrid

pytestmark = pytest.mark.gpu
FIELDS = ("p", "tmean", "tsig", "spread", "flag")


@pytest.fixture(scope="module")
def events():
    from crysplight_b200.fast_events import SurrogateEvents
    from crysplight_b200.surrogate import LightSurrogate
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    main = LightSurrogate.load(os.path.join(root, "crysplight_b200", "surrogates", "bgo_esr.npz"))
    Lz = float(main.box_mm[2])
    slabs = [LightSurrogate(main.box_mm, main.y_mean, main.y_std, main.members[k:k + 1], z_range=r,
                            first_pass=main.first_pass)
             for k, r in enumerate(((0.2 * Lz, 0.7 * Lz), (0.5 * Lz, 0.9 * Lz), (0.6 * Lz, Lz)))]
    ev = SurrogateEvents(main, experts=slabs, max_batch=128)
    yield ev
    ev.close()


def _light(ev, n):
    import torch
    rng = np.random.default_rng(n)
    xyz = torch.from_numpy((rng.uniform(0, 1, (n, 3)) * ev.sur.box_mm).astype(np.float32)).cuda()
    out = ev.site_light(xyz, ro=Readout(SipmGrid(6.0, 8, 8)), pde=0.4)
    return [getattr(out, f).cpu().numpy() for f in FIELDS]


@pytest.mark.parametrize("n", [1, 700])
def test_more_experts_than_one_split_takes(events, n):
    three = events.experts
    want = _light(events, n)
    try:
        events.experts = [three[0]] * 255 + [three[1], three[2]]       # 257: the last one in a second split
        got = _light(events, n)
    finally:
        events.experts = three
    assert all(np.array_equal(a, b) for a, b in zip(got, want))


@pytest.mark.parametrize("per_split", [1, 2])
def test_later_splits_take_over(events, per_split):
    want = _light(events, 3001)
    try:
        events.EXPERTS_PER_SPLIT = per_split
        got = _light(events, 3001)
    finally:
        del events.EXPERTS_PER_SPLIT
    assert all(np.array_equal(a, b) for a, b in zip(got, want))
