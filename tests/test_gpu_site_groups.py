"""Sites shared out over several ensembles: overlapping slabs (the last one
serves), depths exactly on a slab's ends, groups that are empty or hold every
site, against each ensemble evaluated on all sites."""
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FIELDS = ("p", "tmean", "tsig", "spread", "flag")


@pytest.fixture(scope="module")
def parts():
    from crysplight_b200.fast_events import SurrogateEvents
    from crysplight_b200.surrogate import LightSurrogate
    from crysplight_b200.transport import Engine
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    main = LightSurrogate.load(os.path.join(root, "crysplight_b200", "surrogates", "bgo_esr.npz"))
    Lz = float(main.box_mm[2])
    slabs = [LightSurrogate(main.box_mm, main.y_mean, main.y_std, main.members[:k], z_range=r, first_pass=fp)
             for k, r, fp in ((3, (0.3 * Lz, 0.8 * Lz), main.first_pass), (2, (0.6 * Lz, Lz), None))]
    engine = Engine(0)
    alone = [SurrogateEvents(e, engine) for e in [main] + slabs]
    both = SurrogateEvents(main, engine, experts=slabs, expert_margin_mm=0.7)
    yield main, slabs, alone, both
    for se in alone + [both]:
        se.close()


@pytest.mark.parametrize("n,depths", [(1, "any"), (31, "any"), (33, "any"), (1000, "any"), (20_001, "any"),
                                      (70, "front"), (70, "readout"), (0, "any")])
def test_each_site_from_the_ensemble_that_serves_it(parts, n, depths):
    import torch
    from crysplight_b200.params import Readout, SipmGrid
    main, slabs, alone, both = parts
    L = [float(v) for v in main.box_mm]
    ends = [np.float32(v) for s in slabs for v in (s.z_range[0] + 0.7, s.z_range[1])]
    rng = np.random.default_rng(n + len(depths))
    z = rng.uniform(0.0, L[2], n) if depths == "any" else np.full(n, 0.1 if depths == "front" else 0.95 * L[2])
    xyz = np.stack([rng.uniform(0, L[0], n), rng.uniform(0, L[1], n), z], 1).astype(np.float32)
    if depths == "any":
        edge = [f(v) for v in ends for f in (lambda v: v, lambda v: np.nextafter(v, np.float32(0)),
                                             lambda v: np.nextafter(v, np.float32(99)))]
        m = min(n, len(edge))
        xyz[:m, 2] = np.minimum(edge[:m], np.float32(L[2]))
    d = torch.from_numpy(xyz).cuda()
    kw = dict(ro=Readout(SipmGrid(6.0, 8, 8)), pde=0.4)
    got = both.site_light(d, **kw)
    owner = np.zeros(n, int)
    for e, s in enumerate(slabs):
        owner[((d[:, 2] >= s.z_range[0] + 0.7) & (d[:, 2] <= s.z_range[1])).cpu().numpy()] = e + 1
    if n >= 1000:
        assert set(owner) == {0, 1, 2}
    each = [se.site_light(d, **kw) for se in alone]
    for name in FIELDS:
        a = getattr(got, name).cpu().numpy()
        for e in range(3):
            ref = getattr(each[e], name).cpu().numpy()
            assert np.array_equal(a[owner == e], ref[owner == e]), (name, e)


def test_split_refuses(parts):
    import ctypes as C
    import torch
    from crysplight_b200 import _lib
    lib = _lib.load()
    x = torch.zeros(4, 3, device="cuda")
    lists, cnt = torch.zeros(2, 4, dtype=torch.int32, device="cuda"), torch.zeros(2, dtype=torch.int32, device="cuda")
    lo, hi, count = (C.c_float * 1)(0.0), (C.c_float * 1)(1.0), (C.c_int32 * 2)()
    P = C.c_void_p

    def call(n=4, experts=1, xp=x.data_ptr(), low=lo):
        return lib.cl_surrogate_split(P(xp), n, experts, low, hi, P(lists.data_ptr()), P(cnt.data_ptr()), count, None)
    assert call(n=-1) == _lib.CL_ERR_ARG and call(experts=-1) == _lib.CL_ERR_ARG
    assert call(experts=257) == _lib.CL_ERR_ARG and call(xp=0) == _lib.CL_ERR_ARG and call(low=None) == _lib.CL_ERR_ARG
    assert call() == _lib.CL_OK and list(count) == [0, 4]
    assert call(n=0, xp=0) == _lib.CL_OK and list(count) == [0, 0]
