"""The device's own early ends of the narrow phase (cubic_misses, roots_fail) and short cuts of the
solver against the device's solver and filter, in both precisions and with both math libraries.
The rules have no tolerance: a sub-test that ends early has no row."""
import numpy as np
import pytest
import torch

from test_cubic_misses import _cubics
from test_gpu_math import _bits_equal, _col, _run
from test_gpu_reference import _stage
from test_roots_fail import _tetrahedra

pytestmark = pytest.mark.gpu
LIBS = [0, 1]                    # CUDA's elementary functions, the library's own
N = 1 << 20


@pytest.mark.parametrize("lib", LIBS)
@pytest.mark.parametrize("family", ["free", "tetrahedra", "double roots at 1", "pairs near the axis", "triple roots"])
def test_no_cubic_that_ends_early_has_a_root(cuda, family, lib):
    cubics = np.stack(_cubics(family, N, np.random.default_rng(len(family) + 10)), 1)
    out = _stage(5, lib, cubics, 4)
    for misses, roots in (out[:, :2].T, out[:, 2:].T):
        assert (misses > 0).sum() > N // 50
        assert not roots[misses > 0].any()


@pytest.mark.parametrize("lib", LIBS)
@pytest.mark.parametrize("family", ["free", "flat", "offset", "rigid", "parallel", "border"])
def test_no_subtest_that_ends_early_has_a_root_that_passes(cuda, family, lib):
    v, dv, k = _tetrahedra(family, N, np.random.default_rng(len(family) + 10))
    rows = np.concatenate([v.reshape(N, 12), dv.reshape(N, 12), k[:, None].astype(np.float64)], 1)
    out = _stage(6, lib, rows, 8)
    for misses, fails, roots, passing in (out[:, :4].T, out[:, 4:].T):
        assert not roots[misses > 0].any()
        assert not passing[fails > 0].any()
        assert ((fails > 0) & (roots > 0)).sum() > N // 1000          # (the rule is about those)
        assert passing.any()


def _wide(g, n):
    return g.choice([-1.0, 1.0], n) * g.uniform(1, 2, n) * 2.0 ** g.integers(-1074, 1023, n)


def test_solver_prefix_is_that_of_the_certified_products(cuda):
    g = np.random.default_rng(1)
    for family in ("free", "tetrahedra", "double roots at 1", "pairs near the axis", "triple roots"):
        cubics = np.stack(_cubics(family, N, g), 1)
        cls, gg, h = _stage(4, 1, cubics, 3).T
        plain = _run(10, cubics)
        solved = np.abs(cubics[:, 0]) >= 1e-16
        assert solved.sum() > N // 2
        assert _bits_equal(gg, plain[:, 1])[solved].all() and _bits_equal(h, plain[:, 2])[solved].all()
        assert np.array_equal(cls[solved] == 3, (h <= 0)[solved] & (cls != 2)[solved])
    # the classes that have no prefix
    few = _stage(4, 1, np.array([[0.0, 0, 1, 1], [0, 1, 1, 1], [1e-17, 1, 1, 1]]), 3)
    assert np.array_equal(few, [[0, 0, 0], [1, 0, 0], [1, 0, 0]])


def test_division_by_constants_is_the_division(cuda):
    g = np.random.default_rng(2)
    small = g.integers(1, 1 << 40, N) * 2.0 ** g.integers(-600, 600, N)
    x = np.concatenate([_wide(g, N), 3 * small, 27 * small, np.nextafter(27 * small, np.inf),
                        [0.0, -0.0, np.inf, -np.inf, np.nan, 5e-324, np.finfo(float).max]])
    got = _run(11, _col(x))
    assert _bits_equal(got[:, 0], x / 3.0).all()
    assert _bits_equal(got[:, 1], x / 27.0).all()


def test_sincos_has_the_bits_of_sin_and_cos(cuda):
    x = np.random.default_rng(3).uniform(0, 1.1, 4 * N)
    both = _run(12, _col(x))
    assert _bits_equal(both[:, 0], _run(9, _col(x))[:, 0]).all()
    assert _bits_equal(both[:, 1], _run(8, _col(x))[:, 0]).all()
