"""Closest points on meshes far from the origin and in other units: the same bits as the
host's walk, at about the cost of the same mesh at the origin. (With bounds in FP32 world
coordinates, 10,000 points over a 243,602-face terrain in map coordinates took 67 times as
long as at the origin.)"""

import numpy as np
import pytest

torch = pytest.importorskip("torch")

import igl  # noqa: E402
from igl import distance, synthetic  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("move", [[1e3, -1e3, 0], [4.5e5, 5.2e6, 300], [1e9, 0, 1e9], [1e13, 1e13, 0]])
@pytest.mark.parametrize("mesh", ["sphere", "terrain"])
def test_offsets(mesh, move):
    V, F = synthetic.bumpy_icosphere(3, seed=2) if mesh == "sphere" else synthetic.terrain_grid(25)
    P = np.concatenate([synthetic.mixed_queries(V, F, 3000, 5, near_sigma=1e-3), 30 * V[:200]])
    _check(V + move, F, np.concatenate([P + move, P[:50]]))


@pytest.mark.parametrize("unit", [1e-160, 1e-118, 1e-30, 1e-17, 1e-6, 1e15, 1e40, 1e118, 1e140])
def test_units(unit):
    V, F = synthetic.bumpy_icosphere(3, seed=2)
    P = np.concatenate([synthetic.mixed_queries(V, F, 2000, 5, near_sigma=1e-3), 30 * V[:200]])
    _check(V * unit, F, P * unit)


def _check(V, F, P):
    tree = igl.AABB()
    tree.init(V, F)
    for a, b in zip(tree.squared_distance(V, F, P, device="gpu"),
                    tree.squared_distance(V, F, P)):
        assert a.tobytes() == b.tobytes()


def _ms(tree, P):
    p = torch.from_numpy(P).cuda()
    times = []
    for _ in range(12):
        e = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
        e[0].record()
        tree.query(p)
        e[1].record()
        torch.cuda.synchronize()
        times.append(e[0].elapsed_time(e[1]))
    return min(times[2:])  # what other work on the host adds is no part of it


@pytest.mark.parametrize("move, unit", [([4.5e5, 5.2e6, 300], 1.0), ([0, 0, 0], 1e16)])
def test_cost(move, unit):
    V, F = synthetic.terrain_grid(200)
    P = np.column_stack([np.random.default_rng(0).uniform(-10, 210, (10000, 2)),
                         np.random.default_rng(1).uniform(-5, 5, 10000)])
    at = [distance.DeviceAABB(v, F) for v in (V, (V + move) * unit)]
    assert _ms(at[1], (P + move) * unit) < 10 * _ms(at[0], P)


@pytest.mark.parametrize("bad", [np.inf, -np.inf, 1e200, np.nan])
def test_points_beyond_any_bound(bad):
    """They take the reference's walk alone (27 times the call's cost when the walk with
    bounds saw every face for them first), and the other points keep their results."""
    V, F = synthetic.bumpy_icosphere(4, seed=2)
    P = synthetic.mixed_queries(V, F, 4000, 5, near_sigma=1e-3)
    Q = P.copy()
    Q[::10, 1] = bad
    tree = distance.DeviceAABB(V, F)
    clean = [x.cpu().numpy() for x in tree.query(torch.from_numpy(P).cuda())]
    mixed = [x.cpu().numpy() for x in tree.query(torch.from_numpy(Q).cuda())]
    keep = np.arange(len(P)) % 10 != 0
    for a, b in zip(clean, mixed):
        assert a[keep].tobytes() == b[keep].tobytes()
    if abs(bad) != 1e200:
        assert (mixed[1][~keep] == -1).all()
    if not np.isnan(bad):  # the reference's walk visits every node for NaN
        assert _ms(tree, Q) < 8 * _ms(tree, P)


@pytest.mark.parametrize("level, every", [(6, 81920), (6, 10), (4, 5120), (4, 10)])
def test_thin_faces(level, every):
    """Meshes with thin faces take the reference's walk, the larger ones with few of them by
    the discs and the others by the slabs."""
    V, F = synthetic.bumpy_icosphere(level, seed=4)
    P = np.concatenate([synthetic.mixed_queries(V, F, 4000, 5, near_sigma=1e-3), 30 * V[:200]])
    at = F[::every, 0]
    F = F.copy()
    F[::every, 1] = len(V) + np.arange(len(at))
    V = np.concatenate([V, V[at] + 1e-6])
    _check(V, F, P)
    _check(V + [4.5e5, 5.2e6, 300], F, P + [4.5e5, 5.2e6, 300])


@pytest.mark.parametrize("spokes", [9, 40, 2000])
def test_many_faces_at_one_vertex(spokes):
    """A fan whose hub is the closest point of most points: every face ties."""
    a = np.linspace(0, 2 * np.pi, spokes + 1)[:-1]
    V = np.concatenate([[[0, 0, 1.0]], np.stack([np.cos(a), np.sin(a), 0 * a], 1)])
    k = np.arange(spokes)
    F = np.stack([0 * k, 1 + k, 1 + (k + 1) % spokes], 1)
    P = np.random.default_rng(1).normal(size=(3000, 3)) * 0.3 + [0, 0, 1.5]
    _check(V, F, np.concatenate([P, V[:50]]))


@pytest.mark.parametrize("faces", [1, 2, 63, 64, 65, 80])
def test_small_meshes(faces):
    """On both sides of the size from which the walk has an order of its own."""
    V, F = synthetic.bumpy_icosphere(1, seed=1)
    P = np.concatenate([V, synthetic.mixed_queries(V, F, 3000, 5, near_sigma=1e-2)])
    _check(V, np.ascontiguousarray(F[:faces]), P)
