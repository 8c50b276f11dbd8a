"""The narrow phase leaves out the solver for a sub-test only when none of the roots that it
would return passes the filter: the rule of roots_fail (ccc_geom.cuh), restated here for doubles,
against the oracle's solver and filter, and the kernel on calls large enough to apply it."""
from collections import Counter

import numpy as np
import pytest
import torch

f32 = np.float32


def _reach(v):
    return np.abs(v).sum(-1, dtype=f32)


def _fails(F, k, t, dt):
    a0, b0, c0, a1, b1, c1, size, pos = F
    ea, eb, ec = (dt * _reach(d) + pos for d in (a1, b1, c1))
    va, vb, vc = (x + y * t[:, None] for x, y in ((a0, a1), (b0, b1), (c0, c1)))
    la, lb, lc = _reach(va), _reach(vb), _reach(vc)
    n, gs, gp = np.cross(va, vb), np.cross(vc, vb), np.cross(vc, va)
    ln, ls, lp = _reach(n), _reach(gs), _reach(gp)
    en, es, ep = la * eb + lb * ea + ea * eb, lc * eb + lb * ec + eb * ec, lc * ea + la * ec + ea * ec
    low = f32(1e-13) * size ** 4 + f32(1e-30)
    s, p, det = (gs * n).sum(-1), (gp * n).sum(-1), (n * n).sum(-1)
    ms, mp, md = ls * en + ln * es + es * en + low, lp * en + ln * ep + ep * en + low, 2 * ln * en + en * en + low
    ee = k < 9
    out = (s < -ms) | np.where(ee, (p < -mp) | (s - det > ms + md) | (p - det > mp + md),
                               (p > mp) | ((s - p) - det > ms + mp + md))
    return out & (det > md) & (np.abs(s) + np.abs(p) + det < 1e30)


def _roots_fail(v, dv, k, cf):
    """v, dv (N, 4, 3), types k (N,), cubics cf (N, 4): the sub-tests that the kernel drops."""
    a, b, c, d = cf.T
    fa, fb, fc, fd = (x.astype(f32) for x in (a, b, c, d))
    A, B, C, D = map(np.abs, (fa, fb, fc, fd))
    r3 = np.maximum(np.maximum((B / A) ** 2 * B, C * np.sqrt(C / A)), D)
    X, Y, Z = b * b, a * c, a * a * d
    f, g = 3 * Y - X, b * (2 * X - 9 * Y) + 27 * Z
    three = g * g / 4 + f ** 3 < -1e-10 * (X ** 3 + np.abs(Y) ** 3 + Z * Z)
    total = A + B + C
    m = np.where(three, f32(1e-12), f32(1e-3)) * r3 + f32(1e-6) * total
    e1 = ((a + b) + (c + d)).astype(f32)
    zero = D <= m
    q3, q2, q1, q0 = np.where(zero, 0, fa), np.where(zero, fa, fb), np.where(zero, fb, fc), np.where(zero, fc, fd)
    qe = np.where(zero, ((a + b) + c).astype(f32), e1)
    s0, s1, s2 = q1, q1 + q2, 2 * q2 + 3 * q3 + q1
    mono = ((s0 < 0) == (s2 < 0)) & (zero | ((s0 < 0) == (s1 < 0)))
    slope = np.minimum(np.minimum(np.abs(s0), np.abs(s2)), np.where(zero, f32(3e38), np.abs(s1))) - f32(4e-6) * total
    crosses = (q0 < 0) != (qe < 0)
    mid = q1 / 2 + q0
    least = np.minimum(np.minimum(np.abs(q0), np.abs(qe)), np.abs(mid)) - f32(4e-6) * total
    definite = zero & ~crosses & ((q0 < 0) == (mid < 0)) & (least > 0)
    one = crosses & mono & (slope > 0) & (zero | ((D > m) & (np.abs(e1) > m)))
    q = lambda t: ((q3 * t + q2) * t + q1) * t + q0
    t = q0 / (q0 - qe)
    for _ in range(2):
        t = np.clip(t - q(t) / ((3 * q3 * t + 2 * q2) * t + q1), 0, 1).astype(f32)
    off = (np.abs(q(t)) + f32(4e-6) * (total + np.where(zero, 0, D))) / slope
    dt = np.where(one, np.where(zero, 2 * (m + D) / (slope * (t - off)) + off, m / slope + off), (m + D) / least)
    dt = (f32(1.0001) * dt + f32(1e-6)).astype(f32)
    ok = (np.abs(a) >= 1e-16) & (definite | (one & (t > off)))
    t = np.where(one, t, 0).astype(f32)
    w, u = ((x[:, :3] - x[:, 3:]).astype(f32) for x in (v, dv))
    ee, last = (k < 9)[:, None], (k >= 12)[:, None]
    pick = lambda w: (np.where(last, w[:, 1], w[:, 1] - w[:, 0]),
                      np.where(ee, -w[:, 2], np.where(last, w[:, 2], w[:, 2] - w[:, 0])),
                      np.where(ee, w[:, 2] - w[:, 0], np.where(last, w[:, 0], -w[:, 0])))
    V, U = pick(w), pick(u)
    size = sum(_reach(x) for x in V + U)
    pos = f32(1.2e-14) * np.maximum(np.abs(v[:, 3]).max(-1), np.abs(dv[:, 3]).max(-1)).astype(f32) + f32(2e-6) * size
    F = V + U + (size, pos)
    return ok & _fails(F, k, t, dt) & (~(one & zero) | _fails(F, k, np.zeros_like(t), dt))


def _tetrahedra(family, n, g):
    S = 2.0 ** g.uniform(-8, 3, (n, 1, 1))
    M = S * 2.0 ** g.uniform(-10, 2, (n, 1, 1))
    v, w = S * g.uniform(-1, 1, (n, 4, 3)), M * g.uniform(-1, 1, (n, 4, 3))
    k = g.integers(0, 15, n)
    if family == "flat":
        v[:, :, 1] = 0
    elif family == "offset":
        v += 2.0 ** g.uniform(0, 16, (n, 1, 1))
    elif family == "rigid":
        w = M * g.uniform(-1, 1, (n, 1, 3)) + M * 2.0 ** g.uniform(-20, -1, (n, 1, 1)) * w / M
    elif family == "parallel":
        v[:, 3] = v[:, 2] + (v[:, 1] - v[:, 0]) * g.uniform(0.7, 1.3, (n, 1)) + v[:, 3] * 2.0 ** g.uniform(-20, -1, (n, 1))
    elif family == "border":
        # at one time the edges meet, or the vertex is in the face's plane, next to the filter's border
        t, p = g.uniform(0, 1, (n, 1)), g.uniform(0, 1, (n, 1))
        e = g.choice([-1.0, 1.0], (n, 1)) * 2.0 ** g.uniform(-40, -2, (n, 1))
        s = np.where(g.random((n, 1)) < 0.5, e, 1 + e)
        P = v.copy()
        move = P[:, 0] + s * (P[:, 1] - P[:, 0]) - (P[:, 2] + p * (P[:, 3] - P[:, 2]))
        inv = (k >= 12)[:, None]
        f0, f1, f2 = (np.where(inv, P[:, i + 1], P[:, i]) for i in range(3))
        on = f0 + s * (f1 - f0) + p * (1 - s) * (f2 - f0)
        ee = (k < 9)[:, None]
        P[:, 0] = np.where(inv, on, P[:, 0])
        P[:, 2] = np.where(ee, P[:, 2] + move, P[:, 2])
        P[:, 3] = np.where(ee, P[:, 3] + move, np.where(inv, P[:, 3], on))
        v = P - t[:, None] * w
    return v, (v + w) - v, k


@pytest.mark.parametrize("family", ["free", "flat", "offset", "rigid", "parallel", "border"])
def test_no_subtest_that_is_dropped_passes(oracle, family):
    n = 20000
    v, dv, k = _tetrahedra(family, n, np.random.default_rng(len(family)))
    tets = np.concatenate([v.reshape(n, 12), dv.reshape(n, 12)], 1)
    cf = np.stack([oracle.cubic_coeffs(t) for t in tets])
    with np.errstate(all="ignore"):
        dropped = _roots_fail(v, dv, k, cf)
    with_root = 0
    for i in np.flatnonzero(dropped):
        roots = oracle.solve_cubic(*cf[i])
        roots = roots[(roots >= 0) & (roots <= 1)]
        with_root += len(roots) > 0
        assert not any(oracle.ccd_filter(tets[i], k[i], r) for r in roots)
    assert with_root > n // 200         # (the rule is about those)


def _mesh(name):
    from cccollisions_b200 import workloads as W
    if name == "fold":
        return W.jittered_fold(3, 90, 90)
    # a flat sheet that is crumpled within its grid's spacing: every sub-test starts coplanar
    g = np.random.default_rng(5)
    verts, faces = W.grid(90, 90)
    verts = np.concatenate([verts[:, :2], np.zeros((len(verts), 1))], 1)
    x0 = verts[faces]
    return x0, (verts + g.normal(0, 0.012, verts.shape))[faces], g.uniform(0.5, 2.0, (len(faces), 3))


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("name", ["fold", "sheet"])
def test_rows_of_large_calls(cuda, oracle, name, dtype):
    import cccollisions_b200 as C
    from cccollisions_b200 import _native as N
    x0, x1 = (a.astype(dtype) for a in _mesh(name)[:2])
    bb, tr = oracle.bvh(x0, x1)
    pairs = len(oracle.candidates(bb, tr))
    assert pairs >= 3 * 148 * 256       # a block's worth of pairs for every resident block
    er, et = oracle.ccd(bb, tr, x0, x1)
    X0, X1 = (torch.from_numpy(a[None]).to(cuda) for a in (x0, x1))
    with N.math_library(N.LIB_PORTABLE):
        boxes, tree = C.bvh_motion(X0, X1)
        rows, times = C.find_collisions_continuous(boxes, tree, X0, X1, pairs // len(x0) + 2, len(er) // len(x0) + 2)
    n = int((rows[0, :, 0] >= 0).sum())
    got = Counter(zip(map(tuple, rows[0, :n].tolist()), times[0, :n, 0].double().tolist()))
    assert got == Counter(zip(map(tuple, er.tolist()), map(float, et.tolist())))
