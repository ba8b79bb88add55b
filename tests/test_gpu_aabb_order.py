"""The closest-point kernel's own walk order (csrc/wn_aabb.cu: the minimum first, then
the face that the reference's order keeps) against the host traversal, which is the
reference's walk: every bit of distance, face and point. The cases are those where the
two could part: ties at vertices, on edges and between duplicated faces (more than the
kernel keeps), box distances that tie, thin and collapsed faces, other leaf sizes,
caller-made boxes, single faces, distant and tiny coordinates, partial warps."""

import ctypes

import numpy as np
import pytest

torch = pytest.importorskip("torch")

import igl  # noqa: E402
from igl import _lib, synthetic  # noqa: E402

pytestmark = pytest.mark.gpu


def _query(V, F, P, leaf=8, boxes_hook=None):
    """(gpu, cpu) results of one tree through the C ABI."""
    h = _lib.lib()
    addr = _lib.addr
    nn = h.wn_aabb_node_count(len(F), leaf)
    boxes, nodes = np.empty((nn, 6)), np.empty((nn, 4), np.int64)
    order, stack = np.empty(len(F), np.int64), ctypes.c_int64(0)
    assert h.wn_aabb_build(addr(V), len(V), addr(F), len(F), leaf, addr(boxes), addr(nodes),
                           addr(order), ctypes.byref(stack), 0) == 0
    if boxes_hook:
        boxes_hook(boxes, nodes)
    tree = ctypes.c_void_p()
    assert h.wn_aabb_create(addr(V), len(V), addr(F), len(F), addr(boxes), addr(nodes),
                            addr(order), nn, ctypes.byref(tree)) == 0, _lib.last_error(h)
    out = []
    for device in ("gpu", "cpu"):
        d, i, c = np.empty(len(P)), np.empty(len(P), np.int64), np.empty((len(P), 3))
        if device == "gpu":
            assert h.wn_aabb_squared_distance_host(tree, addr(P), len(P), addr(d), addr(i),
                                                   addr(c)) == 0
        else:
            st = np.empty(stack.value + 64, np.int64)
            h.mli_aabb_squared_distance(addr(P), addr(V), addr(F), addr(boxes), addr(nodes),
                                        addr(order), addr(d), addr(i), addr(c), st.ctypes.data,
                                        len(P), nn, 0, len(P))
        out.append((d, i, c))
    h.wn_aabb_destroy(tree)
    return out


def _same(V, F, P, **kw):
    V, F, P = (np.ascontiguousarray(x) for x in (V, F, P))
    gpu, cpu = _query(V, F, P, **kw)
    for a, b in zip(gpu, cpu):
        assert a.tobytes() == b.tobytes()


def _points(V, F, n, seed):
    tri = V[F]
    return np.concatenate([V, tri.mean(1), 0.5 * (tri[:, 0] + tri[:, 1]),
                           1.5 * V, 0.5 * V, np.zeros((3, 3)),
                           synthetic.mixed_queries(V, F, n, seed, near_sigma=1e-3)])


@pytest.mark.parametrize("leaf", [1, 3, 8, 37])
@pytest.mark.parametrize("mesh", ["sphere", "open", "soup", "duplicates", "flat", "terrain"])
def test_meshes(mesh, leaf):
    V, F = synthetic.bumpy_icosphere(3, seed=4)
    if mesh == "open":
        F = synthetic.delete_faces(F, 0.2, seed=1)
    elif mesh == "soup":
        V, F = synthetic.unshare_vertices(V, F)
    elif mesh == "duplicates":  # up to twelve records of one face
        F = np.concatenate([F] + [F[:200]] * 10 + [F[:100, [1, 2, 0]]])
    elif mesh in ("flat", "terrain"):
        V, F = synthetic.terrain_grid(25)
        if mesh == "flat":
            V[:, 2] = 0.0
    P = _points(V, F, 3000, 7)
    if mesh == "flat":  # box distances that tie at every level
        g = np.random.default_rng(3).integers(-8, 56, size=(4000, 3)) * 0.5
        P = np.concatenate([P, g])
    _same(V, F, P, leaf=leaf)


@pytest.mark.parametrize("kind", ["thin", "needles", "collapsed", "far", "tiny", "one"])
def test_shapes(kind):
    rng = np.random.default_rng(5)
    V, F = synthetic.bumpy_icosphere(3, seed=6)
    if kind == "thin":  # flattened along z: faces of 1 : 100 and less
        V = V * [1.0, 1.0, 1e-2]
    elif kind == "needles":  # one in ten faces thinner than 1 : 10^4
        V = np.concatenate([V, V[F[::10, 0]] + 1e-6 * rng.normal(size=V[F[::10, 0]].shape)])
        k = len(F[::10])
        F = F.copy()
        F[::10, 1] = len(V) - k + np.arange(k)
    elif kind == "collapsed":
        F = np.concatenate([F, np.stack([F[:60, 0], F[:60, 0], F[:60, 1]], 1),
                            np.stack([F[:20, 0]] * 3, 1)])
    elif kind == "far":
        V = V + 1e7
    elif kind == "tiny":
        V = V * 1e-13
    elif kind == "one":
        F = F[:1]
    P = _points(V, F, 3000, 8)
    P = np.concatenate([P, (P[:50] - P.mean(0)) * 1e5, (P[:20] - P.mean(0)) * 1e18])
    _same(V, F, P)


def test_boxes_that_do_not_hold_their_faces():
    V, F = synthetic.bumpy_icosphere(3, seed=2)

    def shrink(boxes, nodes):
        boxes[:, 3:] = boxes[:, :3] + 0.9 * (boxes[:, 3:] - boxes[:, :3])

    _same(V, F, _points(V, F, 2000, 9), boxes_hook=shrink)


@pytest.mark.parametrize("n", [1, 31, 33, 127, 513, 16383, 16384, 20001])
def test_point_counts(n):
    V, F = synthetic.bumpy_icosphere(4, seed=3)
    _same(V, F, synthetic.mixed_queries(V, F, n, seed=n, near_sigma=1e-2))


def test_larger_mesh():
    V, F = synthetic.bumpy_icosphere(6, seed=3)
    P = np.concatenate([synthetic.mixed_queries(V, F, 60000, seed=1, near_sigma=1e-4),
                        0.2 * synthetic.box_points(V, 20000, seed=2), V[::4]])
    V, F, P = (np.ascontiguousarray(x) for x in (V, F, P))
    tree = igl.AABB()
    tree.init(V, F)
    for a, b in zip(tree.squared_distance(V, F, P, device="gpu"),
                    tree.squared_distance(V, F, P)):
        assert a.tobytes() == b.tobytes()
