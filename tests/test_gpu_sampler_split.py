"""The sampler's sites per warp follow the number of sites: a site's draws and
times do not depend on them (its streams are keyed by its index), and its counts
add up."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SLOTS = 148 * 8 * 4          # warps resident at once


@pytest.fixture(scope="module")
def engine():
    from crysplight_b200.transport import Engine
    e = Engine(0)
    yield e
    e.close()


def _sample(engine, n):
    import torch
    from crysplight_b200.fast_events import SiteLight, sample_sites
    from crysplight_b200.params import Box, OpticalParams, Readout, SipmGrid, TimeBinning
    rng = np.random.default_rng(3)                       # rows of a longer list, in order
    m = 32 * SLOTS + 5
    p = rng.dirichlet(np.full(64, 0.2), m).astype(np.float32)[:n] * 0.4
    ph = rng.integers(0, 300, m)[:n]
    T = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    full = lambda v: torch.full((n, 64), v, device="cuda")
    light = SiteLight(T(p), full(0.8), full(0.3), torch.zeros(n, device="cuda"),
                      torch.zeros(n, dtype=torch.uint8, device="cuda"))
    op = OpticalParams(2.15, 1.45, 20000.0, 2222.0, 0.985, True, True, 0.0227, 0.4)
    (maps, tmin, npe, _, sampled), _ = sample_sites(
        engine, Box((48.0, 48.0, 22.4)), op, Readout(SipmGrid(6.0, 8, 8)), TimeBinning(100.0, 80),
        xyz=torch.zeros(n, 3, device="cuda"), t0=torch.zeros(n, device="cuda"), photons=T(ph.astype(np.int64)),
        segment=torch.arange(n, dtype=torch.int32, device="cuda"), n_segments=n, seed=11, tau_ns=300.0, light=light)
    maps = maps.cpu().numpy().reshape(n, 64)
    assert np.array_equal(npe.cpu().numpy(), maps.sum(1)) and sampled.cpu().tolist() == [ph.sum(), maps.sum()]
    assert (maps.sum(1) <= ph).all()
    return maps, tmin.cpu().numpy().reshape(n, 64).view(np.uint32)


@pytest.mark.parametrize("n", [1, 33, SLOTS, SLOTS + 1, 2 * SLOTS + 3, 4 * SLOTS + 1, 16 * SLOTS + 1])
def test_a_site_is_the_same_in_any_split(engine, n):
    maps, tmin = _sample(engine, n)
    ref_maps, ref_tmin = _sample(engine, 32 * SLOTS + 5)     # 32 sites per warp
    assert np.array_equal(maps, ref_maps[:n]) and np.array_equal(tmin, ref_tmin[:n])
