"""The transport loop decides the wall, the bulk competition and Fresnel from
bounded approximations and takes the exact expressions where those do not
decide.  Every decision, distance and correctly rounded helper is compared
here with the exact expression, at random operands and at the ones where the
approximations are worst (ties, corners, grazing directions, uniforms next to
the threshold)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
F = np.float32


def _bits(a):
    return np.ascontiguousarray(a, F).view(np.uint32)


@pytest.mark.parametrize("exponent", [-38, -1, 0, 3])
def test_root_and_reciprocal_of_every_mantissa(engine, exponent):
    m = np.arange(2 ** 23, dtype=np.uint32) | np.uint32(127 << 23)
    x = (m.view(F) * F(2.0 ** exponent)).astype(F)
    for s in (F(1), F(2)):
        got = engine.eval_step(7, (x * s)[:, None])[:, 0]
        assert np.array_equal(_bits(got), _bits(np.sqrt(x * s)))
        got = engine.eval_step(8, (x * s)[:, None])[:, 0]
        assert np.array_equal(_bits(got), _bits(F(1) / (x * s)))
    assert engine.eval_step(7, np.zeros((1, 1), F))[0, 0] == 0


def _directions(rng, n):
    u = rng.standard_normal((n, 3))
    u /= np.linalg.norm(u, axis=1, keepdims=True)
    u[: n // 8, 0] *= 10.0 ** rng.uniform(-12, 0, n // 8)      # grazing
    u[n // 8: n // 7, 1] = 0.0
    u[n // 7: n // 6, 2] = u[n // 7: n // 6, 0]                # equal components
    return u.astype(F)


@pytest.mark.parametrize("box", [(48.0, 48.0, 37.2), (48.0, 48.0, 22.4), (1.0, 1.0, 1.0), (3e-3, 5e4, 7.0)])
def test_wall_distance_and_face(engine, box):
    rng = np.random.default_rng(3)
    n = 4_000_000
    L = np.asarray(box, F)
    p = (rng.uniform(0, 1, (n, 3)) * L).astype(F)
    on = rng.integers(0, 3, n)
    wall = rng.random(n) < 0.7                                 # most steps start on a wall
    p[wall, on[wall]] = np.where(rng.random(wall.sum()) < 0.5, F(0), L[on[wall]])
    p[: n // 20] = L * rng.integers(0, 2, (n // 20, 3)).astype(F)          # corners
    p[n // 20: n // 15] = (L * F(0.5))                          # ties from the centre
    p[n // 15: n // 14] *= F(-1.5)                              # outside the crystal
    u = _directions(rng, n)
    u[n // 20: n // 15] = (rng.integers(0, 2, (n // 15 - n // 20, 3)) * 2 - 1) * F(0.57735026)
    o = engine.eval_step(9, np.hstack([p, u, np.broadcast_to(L, (n, 3))]))
    quick = o[:, 1] != 0
    assert np.array_equal(o[quick, 1], o[quick, 3])
    assert np.array_equal(_bits(o[quick, 0]), _bits(o[quick, 2]))
    bad = np.full((5, 9), np.nan, F)
    assert (engine.eval_step(9, bad)[:, 1] == 0).all()


@pytest.mark.parametrize("n1,n2", [(2.15, 1.45), (2.15, 1.0), (1.79, 1.0), (1.79, 1.45), (1.0, 1.8), (1.5, 1.5),
                                   (5e-4, 1.0)])
def test_fresnel_decision(engine, n1, n2):
    rng = np.random.default_rng(4)
    n = 2_000_000
    c = rng.uniform(0, 1, n)
    crit = np.sqrt(max(0.0, 1 - (n2 / n1) ** 2))
    c[: n // 4] = crit + 10.0 ** rng.uniform(-9, 0, n // 4)    # from the critical angle on
    c = np.clip(c, 1e-9, 1).astype(F)
    q = n1 / n2
    s2 = np.minimum(q * q * (1 - c.astype(np.float64) ** 2), 1.0)
    ct = np.sqrt(1 - s2)
    R = 0.5 * (((n1 * c - n2 * ct) / (n1 * c + n2 * ct)) ** 2 + ((n1 * ct - n2 * c) / (n1 * ct + n2 * c)) ** 2)
    k = np.rint(R * 2 ** 24) + rng.integers(-6, 7, n)          # uniforms next to R
    k = np.where(rng.random(n) < 0.3, rng.integers(1, 2 ** 24 + 1, n), k)
    u = (np.clip(k, 1, 2 ** 24) * 2.0 ** -24).astype(F)
    o = engine.eval_step(10, np.stack([np.full(n, n1, F), np.full(n, n2, F), c, u], 1))
    assert np.array_equal(o[:, 0], o[:, 1])


@pytest.mark.parametrize("length", [20000.0, 3115.0, 346.0, 30.0, 0.5, 1e9, 0.0, -5.0, np.inf])
def test_bulk_events_are_never_ruled_out_wrongly(engine, length):
    rng = np.random.default_rng(5)
    n = 2_000_000
    k = rng.integers(1, 2 ** 24 + 1, n)
    k[: n // 4] = 2 ** 24 - rng.integers(0, 300, n // 4)
    u = (k * 2.0 ** -24).astype(F)
    d = rng.uniform(0, 70, n).astype(F)
    if np.isfinite(length) and length > 0:
        near = -length * np.log(u.astype(np.float64))          # distances next to the path length
        e = 1 + rng.integers(-40, 41, n) * 2.0 ** -22
        d = np.where(rng.random(n) < 0.7, near * e, d).astype(F)
    d[:10] = [0.0, -0.0, np.inf, np.nan, -3.0, 1e-40, 1e38, 5.0, 1e-3, 60.0]
    o = engine.eval_step(11, np.stack([u, d, np.full(n, length, F)], 1))
    ruled_out = o[:, 0] == 1
    if np.isinf(length):
        return                                                 # no draw, the flag decides
    assert not (ruled_out & (o[:, 1] < d)).any()
    if length >= 300 and length < 1e8:
        far = np.isfinite(d) & (o[:, 1] > d * F(1.001) + F(1e-3) * F(length))
        assert ruled_out[far].mean() > 0.999                   # and the quick test does decide
