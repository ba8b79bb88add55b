"""Caller-made trees deeper than the library's own median split makes (leaves cut off a few
faces at a time), up to the deepest that wn_aabb_create accepts: every bit of distance, face
and point as the host's walk has it."""

import ctypes

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from igl import _lib, synthetic  # noqa: E402

pytestmark = pytest.mark.gpu


def _chain(V, F, depth):
    """(boxes, nodes) of the tree whose level k splits off the next faces: `depth` levels."""
    tri = V[F]
    each = len(F) // depth
    boxes, nodes = np.empty((2 * depth - 1, 6)), np.empty((2 * depth - 1, 4), np.int64)
    for k in range(depth):
        at = each * k
        rest = tri[at:].reshape(-1, 3)
        boxes[2 * k] = np.r_[rest.min(0), rest.max(0)]
        if k == depth - 1:
            nodes[2 * k] = (-1, -1, at, len(F) - at)
            break
        part = tri[at:at + each].reshape(-1, 3)
        nodes[2 * k] = (2 * k + 1, 2 * k + 2, 0, 0)
        boxes[2 * k + 1] = np.r_[part.min(0), part.max(0)]
        nodes[2 * k + 1] = (-1, -1, at, each)
    return boxes, nodes


@pytest.mark.parametrize("depth", [2, 47, 48, 49, 62, 63])
def test_depths(depth):
    V, F = synthetic.bumpy_icosphere(2, seed=1)
    F = np.ascontiguousarray(F[np.argsort(V[F].mean(1)[:, 0])])
    boxes, nodes = _chain(V, F, depth)
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


def _create(V, F, boxes, nodes, order):
    h, addr = _lib.lib(), _lib.addr
    tree = ctypes.c_void_p()
    assert h.wn_aabb_create(addr(V), len(V), addr(F), len(F), addr(boxes), addr(nodes),
                            addr(order), len(nodes), ctypes.byref(tree)) == 0, _lib.last_error(h)
    return tree


def _median_split(V, F):
    h, addr = _lib.lib(), _lib.addr
    n = h.wn_aabb_node_count(len(F), 8)
    boxes, nodes = np.empty((n, 6)), np.empty((n, 4), np.int64)
    order, stack = np.empty(len(F), np.int64), ctypes.c_int64(0)
    assert h.wn_aabb_build(addr(V), len(V), addr(F), len(F), 8, addr(boxes), addr(nodes),
                           addr(order), ctypes.byref(stack), 0) == 0
    return boxes, nodes, order


def _changed(boxes, nodes, kind):
    boxes, nodes = boxes.copy(), nodes.copy()
    if kind == "float32 boxes":  # some no longer hold their faces
        boxes = boxes.astype(np.float32).astype(np.float64)
    elif kind == "right first":  # children exchanged: the runs of faces change sides
        inner = nodes[:, 3] <= 0
        nodes[inner, :2] = nodes[inner, 1::-1]
    return boxes, nodes


@pytest.mark.parametrize("kind", ["float32 boxes", "right first"])
def test_caller_made_trees_keep_the_discs(kind):
    """Same bits as the host, and near the cost of the library's own tree (without the discs
    87,000 points in and around a 20,480-face sphere took 15 times as long)."""
    V, F = synthetic.bumpy_icosphere(5, seed=1)
    boxes, nodes, order = _median_split(V, F)
    P = np.ascontiguousarray(np.concatenate(
        [V[:2000], synthetic.mixed_queries(V, F, 85000, seed=3, near_sigma=1e-3)]))
    h, addr = _lib.lib(), _lib.addr
    n = len(P)
    p = torch.from_numpy(P).cuda()
    d, i, c = (torch.empty(s, dtype=t, device="cuda") for s, t in
               ((n, torch.float64), (n, torch.int64), ((n, 3), torch.float64)))
    cost = []
    for made in ((boxes, nodes), _changed(boxes, nodes, kind)):
        tree = _create(V, F, *made, order)
        times = []
        for _ in range(12):
            e = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
            e[0].record()
            assert h.wn_aabb_squared_distance_device(
                tree, p.data_ptr(), n, d.data_ptr(), i.data_ptr(), c.data_ptr(),
                ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
            e[1].record()
            torch.cuda.synchronize()
            times.append(e[0].elapsed_time(e[1]))
        cost.append(min(times[1:]))  # what other work on the host adds is no part of it
        h.wn_aabb_destroy(tree)
        few = P[:6000]
        ref = np.empty(len(few)), np.empty(len(few), np.int64), np.empty((len(few), 3))
        stack = np.empty(256, np.int64)
        h.mli_aabb_squared_distance(addr(few), addr(V), addr(F), addr(made[0]), addr(made[1]),
                                    addr(order), *(addr(x) for x in ref), stack.ctypes.data,
                                    len(few), len(nodes), 0, len(few))
        for a, b in zip((d, i, c), ref):
            assert a[:len(few)].cpu().numpy().tobytes() == b.tobytes()
    assert cost[1] < 8 * cost[0]
