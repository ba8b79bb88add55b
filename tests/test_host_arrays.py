"""The library's checks and packing of host arrays against NumPy, on both sides of the
sizes where they take over and where their spans begin to use threads."""

import numpy as np
import pytest

import igl
from igl import _lib


@pytest.mark.parametrize("n", [0, 1, 4095, 4096, 4097, 131072, 262144, 300001, 1 << 20])
def test_checks(n):
    rng = np.random.default_rng(n)
    x = rng.normal(size=n)
    k = rng.integers(0, 1000, size=n)
    assert igl._all_finite(x) and igl._in_range(k, 1000)
    assert igl._equal(x, x) and igl._equal(x, x.copy()) and igl._equal(k, k.copy())
    if not n:
        assert igl._in_range(k, 0)
        return
    for at in {0, n // 2, n - 1}:
        for bad in (np.nan, np.inf, -np.inf, -np.nan):
            y = x.copy()
            y[at] = bad
            assert not igl._all_finite(y)
        for bad in (-1, 1000, np.iinfo(np.int64).min, np.iinfo(np.int64).max):
            y = k.copy()
            y[at] = bad
            assert not igl._in_range(y, 1000) and not igl._equal(y, k)
        y = x.copy()
        y[at] = np.finfo(np.float64).max
        assert igl._all_finite(y) and not igl._equal(y, x)
        z = x.copy()
        z[at], y[at] = 0.0, -0.0
        assert igl._equal(z, y)
    assert not igl._in_range(np.zeros(n, dtype=np.int64), 0)
    assert not igl._equal(x, x[:-1])


@pytest.mark.parametrize("nf", [0, 1, 511, 512, 513, 10922, 43690, 87382, 200003])
def test_soup(nf):
    rng = np.random.default_rng(nf)
    V, F = rng.normal(size=(997, 3)), rng.integers(0, 997, size=(nf, 3))
    want = V[F].transpose(1, 2, 0).reshape(9, nf)
    assert np.array_equal(igl._triangle_soa(V, F), want)
    assert np.array_equal(igl._triangle_soa(np.asfortranarray(V), np.asfortranarray(F)), want)
    if nf:
        for bad in (-1, 997, np.iinfo(np.int64).min):
            G = F.copy()
            G[nf // 2, 1] = bad
            with pytest.raises(IndexError):
                igl._triangle_soa(V, G)


def test_threads():
    """Several callers at once: nothing is shared between calls."""
    from concurrent.futures import ThreadPoolExecutor

    rng = np.random.default_rng(1)
    V = rng.normal(size=(5000, 3))
    faces = [rng.integers(0, 5000, size=(30000 + k, 3)) for k in range(8)]
    with ThreadPoolExecutor(8) as pool:
        for F, soup in zip(faces, pool.map(lambda F: igl._triangle_soa(V, F), faces)):
            assert np.array_equal(soup, V[F].transpose(1, 2, 0).reshape(9, len(F)))


def test_errors_of_large_inputs_are_the_small_ones():
    """Refused inputs of native size raise what small ones raise."""
    V, F = igl.synthetic.terrain_grid(80)
    O = np.zeros((2000, 3))
    for change, error in ((lambda V, F, O: V.__setitem__((5, 1), np.nan), ValueError),
                          (lambda V, F, O: F.__setitem__((7, 2), len(V)), IndexError),
                          (lambda V, F, O: F.__setitem__((7, 2), -1), IndexError),
                          (lambda V, F, O: O.__setitem__((1999, 0), np.inf), ValueError)):
        a = [V.copy(), F.copy(), O.copy()]
        change(*a)
        with pytest.raises(error):
            igl.winding_number(*a)
    tree = igl.AABB()
    tree.init(V, F)
    tree.squared_distance(V, F, O[:1])
    tree.squared_distance(V.astype(np.float64, order="F"), F.astype(np.int32), O[:1])
    other = V.copy()
    other[-1, 2] += 1.0
    with pytest.raises(ValueError, match="must match"):
        tree.squared_distance(other, F, O[:1])
    V[0, 0] = np.nan  # the arrays given to init, changed since
    with pytest.raises(ValueError, match="finite"):
        tree.squared_distance(V, F, O[:1])
    assert _lib.lib().wn_host_same(None, None, 0) == 1
