"""The transport's quick wall decision decides: nearly every step inside the crystal,
with the incidence cosine that the readout's Fresnel test takes (a decision that never
came would pass the comparisons of the decided ones)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
F = np.float32


@pytest.mark.parametrize("box", [(48.0, 48.0, 37.2), (48.0, 48.0, 22.4), (1.0, 1.0, 1.0), (3e-3, 5e4, 7.0)])
def test_nearly_every_step_is_decided(engine, box):
    rng = np.random.default_rng(11)
    n = 1_000_000
    L = np.asarray(box, F)
    p = (rng.uniform(0.001, 0.999, (n, 3)) * L).astype(F)
    u = rng.standard_normal((n, 3))
    u = (u / np.linalg.norm(u, axis=1, keepdims=True)).astype(F)
    # half of the steps start on a wall and leave it
    on, wall = rng.integers(0, 3, n), rng.random(n) < 0.5
    rows = np.nonzero(wall)[0]
    p[rows, on[rows]] = np.where(u[rows, on[rows]] > 0, F(0), L[on[rows]])
    x = np.hstack([p, u, np.broadcast_to(L, (n, 3))]).astype(F)
    o = engine.eval_step(12, x)
    quick = o[:, 0] != 0
    # what is left undecided: quotients within 2e-6 of each other, mantissas of ones
    assert quick.mean() > 0.9999
    assert np.array_equal(o[quick, 1].view(np.uint32), o[quick, 2].view(np.uint32))
    full = engine.eval_step(9, x)
    assert np.array_equal(full[:, 1], o[:, 0]) and np.array_equal(full[quick, 1], full[quick, 3])
    assert set(np.unique(o[:, 0])) >= ({1, 2, 5, 6} if box[1] > 1e3 else {1, 2, 3, 4, 5, 6})


def test_bulk_events_are_ruled_out_where_they_are_far(engine):
    """And the quick bulk test decides nearly every step of the run files' crystals."""
    rng = np.random.default_rng(12)
    n = 1_000_000
    u = (rng.integers(1, 2 ** 24 + 1, n) * 2.0 ** -24).astype(F)
    d = rng.uniform(0, 60, n).astype(F)
    for length in (20000.0, 3115.0, 2222.0, 346.0):
        o = engine.eval_step(11, np.stack([u, d, np.full(n, length, F)], 1))
        no_event = o[:, 1] > d
        assert (o[no_event, 0] == 1).mean() > 0.998       # within 2^-15 of the threshold it does not
