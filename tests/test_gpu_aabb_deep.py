"""Caller-made trees deeper than the library's own median split makes (leaves cut off one
face at a time), up to the deepest that wn_aabb_create accepts: every bit of distance, face
and point as the host's walk has it."""

import ctypes

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from igl import _lib, synthetic  # noqa: E402

pytestmark = pytest.mark.gpu


def _chain(V, F):
    """(boxes, nodes) of the tree whose level k splits off face k: len(F) levels."""
    tri = V[F]
    n = len(F)
    boxes, nodes = np.empty((2 * n - 1, 6)), np.empty((2 * n - 1, 4), np.int64)
    for k in range(n):
        rest = tri[k:].reshape(-1, 3)
        boxes[2 * k] = np.r_[rest.min(0), rest.max(0)]
        nodes[2 * k] = (2 * k + 1, 2 * k + 2, 0, 0) if k < n - 1 else (-1, -1, k, 1)
        if k < n - 1:
            boxes[2 * k + 1] = np.r_[tri[k].min(0), tri[k].max(0)]
            nodes[2 * k + 1] = (-1, -1, k, 1)
    return boxes, nodes


@pytest.mark.parametrize("depth", [2, 47, 48, 49, 62, 63])
def test_depths(depth):
    V, F = synthetic.bumpy_icosphere(2, seed=1)
    F = np.ascontiguousarray(F[np.argsort(V[F].mean(1)[:, 0])][:depth])
    boxes, nodes = _chain(V, F)
    order = np.arange(len(F))
    P = np.concatenate([V, synthetic.mixed_queries(V, F, 2000, seed=3, near_sigma=1e-2)])
    h, addr = _lib.lib(), _lib.addr
    tree = ctypes.c_void_p()
    assert h.wn_aabb_create(addr(V), len(V), addr(F), len(F), addr(boxes), addr(nodes),
                            addr(order), len(nodes), ctypes.byref(tree)) == 0, _lib.last_error(h)
    out = []
    for device in ("gpu", "cpu"):
        d, i, c = np.empty(len(P)), np.empty(len(P), np.int64), np.empty((len(P), 3))
        if device == "gpu":
            assert h.wn_aabb_squared_distance_host(tree, addr(P), len(P), addr(d), addr(i),
                                                   addr(c)) == 0, _lib.last_error(h)
        else:
            stack = np.empty(256, np.int64)
            h.mli_aabb_squared_distance(addr(P), addr(V), addr(F), addr(boxes), addr(nodes),
                                        addr(order), addr(d), addr(i), addr(c),
                                        stack.ctypes.data, len(P), len(nodes), 0, len(P))
        out.append((d, i, c))
    h.wn_aabb_destroy(tree)
    for a, b in zip(*out):
        assert a.tobytes() == b.tobytes()
