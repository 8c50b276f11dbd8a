"""The narrow phase ends a sub-test early only when the solver has no root in [0, 1] for it: the
rule of cubic_misses (ccc_geom.cuh), restated here, against the oracle's solver."""
import numpy as np
import pytest

EPS = 1e-16


def _misses(a, b, c, d):
    with np.errstate(all="ignore"):
        A, B, C, D = (np.abs(v).astype(np.float32) for v in (a, b, c, d))
        inv = np.float32(1) / A
        q = B * inv
        r3 = np.maximum(np.maximum(q * q * B, C * np.sqrt(C * inv)), D)
        m = (np.float32(1e-3) * r3 + np.float32(1e-6) * (A + B + C)).astype(np.float64)
        bern = np.stack([d, d + c / 3, d + (2 * c + b) / 3, (a + b) + (c + d)])
        return (np.abs(a) >= EPS) & ((bern > m).all(0) | (bern < -m).all(0))


def _cubics(family, n, g):
    s = g.choice([-1.0, 1.0], n) * 2.0 ** g.uniform(-40, 5, n)
    tiny = 2.0 ** g.uniform(-45, 0, n)
    if family == "free":
        return tuple(g.uniform(-1, 1, n) * 2.0 ** g.uniform(-50, 10, n) for _ in range(4))
    if family == "tetrahedra":
        v, w = 2.0 ** g.uniform(-10, 0, n), 2.0 ** g.uniform(-12, 0, n)
        return tuple(g.uniform(-1, 1, n) * k for k in (w ** 3, v * w * w, v * v * w, v ** 3))
    if family == "double roots at 1":
        r0, r1 = 1 + g.choice([-1.0, 1.0], n) * tiny, g.uniform(-2, 2, n)
        p, q = 2 * r0 + tiny, r0 * (r0 + tiny)
        return s, -s * (p + r1), s * (q + p * r1), -s * q * r1
    if family == "pairs near the axis":
        x, r1 = g.uniform(-1.5, 1.5, n), g.uniform(-1, 1, n) * 2.0 ** g.uniform(-3, 12, n)
        return s, -s * (2 * x + r1), s * (x * x + tiny * tiny + 2 * x * r1), -s * (x * x + tiny * tiny) * r1
    m, e, f = g.uniform(-2, 2, n), g.uniform(-1, 1, n) * tiny, g.uniform(-1, 1, n) * tiny[::-1]
    return s, -3 * s * m, s * (3 * m * m + f), s * (e - m ** 3 - f * m)          # f and g small


@pytest.mark.parametrize("family", ["free", "tetrahedra", "double roots at 1", "pairs near the axis", "triple roots"])
def test_no_cubic_that_is_dropped_has_a_root(oracle, family):
    n = 60000
    cubics = np.stack(_cubics(family, n, np.random.default_rng(len(family))))
    dropped = cubics[:, _misses(*cubics)]
    assert dropped.shape[1] > n // 50
    for a, b, c, d in dropped.T:
        roots = oracle.solve_cubic(a, b, c, d)
        assert not ((roots >= 0) & (roots <= 1)).any()
        # (rounded to single precision, as the float path keeps them)
        single = roots.astype(np.float32)
        assert not ((single >= 0) & (single <= 1)).any()


def test_what_cannot_be_told_is_solved():
    bad = np.array([np.nan, np.inf, 0.0, 1e-17])
    one = np.ones(4)
    assert not _misses(bad, one, one, one).any()
    assert not _misses(one, bad[:2].repeat(2), one, one).any()
    assert not _misses(one, one, bad[:2].repeat(2), one).any()
    assert not _misses(one, one, one, bad[:2].repeat(2)).any()
