"""The device's mesh edges (wn_edges.cu) against the general tensor operations on the CPU:
boundary edges are the same bits in the same order; sides welded by position give the
same gradients. The welded bar, 2e-5 of the largest entry, is the mixed adjoint's (FP32
pairs): the two sides differ only in the orientation and order of the welded edges."""

import numpy as np
import pytest

torch = pytest.importorskip("torch")

import igl  # noqa: E402
from igl import autograd as wa  # noqa: E402

pytestmark = pytest.mark.gpu


def _mesh(name):
    V, F = igl.synthetic.bumpy_icosphere(3, seed=5)
    rng = np.random.default_rng(7)
    if name == "one face":
        return V[:3], np.array([[0, 1, 2]])
    if name == "closed":
        return V, F
    if name == "open":
        return V, igl.synthetic.delete_faces(F, 0.1, seed=6)
    if name == "soup":
        return igl.synthetic.unshare_vertices(V, F)
    if name == "open soup":
        return igl.synthetic.unshare_vertices(V, igl.synthetic.delete_faces(F, 0.1, seed=6))
    if name == "random":  # sides met many times, zero-length ones, unused vertices
        return rng.normal(size=(256, 3)), rng.integers(0, 16, size=(4097, 3))
    if name == "last vertex":  # every bit of a vertex number set
        return rng.normal(size=(256, 3)), np.array([[255, 254, 253], [255, 254, 0], [255] * 3])
    if name == "points":  # no side has a length
        return np.zeros((6, 3)), np.array([[0, 1, 2], [3, 4, 5]])
    V = rng.integers(-1, 2, size=(300, 3)) * 0.5  # positions shared at random, both zeros
    V[::3] = np.where(V[::3] == 0.0, -0.0, V[::3])
    return V, rng.integers(0, 300, size=(1001, 3))


NAMES = ["one face", "closed", "open", "soup", "open soup", "random", "last vertex", "points",
         "shared positions"]


@pytest.mark.parametrize("index", [torch.int64, torch.int32])
@pytest.mark.parametrize("name", NAMES)
def test_boundary_edges(name, index):
    V, F = _mesh(name)
    Vt, Ft = torch.from_numpy(V), torch.from_numpy(F).to(index)
    edges, ne, ends = wa.boundary_edges(Vt, Ft)
    got, n, got_ends = wa.boundary_edges(Vt.cuda(), Ft.cuda())
    assert n == ne and got.shape == edges.shape
    assert torch.equal(got.cpu(), edges) and torch.equal(got_ends.cpu(), ends)


@pytest.mark.parametrize("name", NAMES)
def test_gathered_edges(name):
    V, F = _mesh(name)
    Vt, Ft = torch.from_numpy(V).cuda(), torch.from_numpy(F).cuda()
    found = wa.boundary_edges(Vt, Ft)
    O = torch.from_numpy(np.random.default_rng(3).uniform(-2, 2, size=(65, 3))).cuda()
    g = O[:, 0].contiguous()
    dV, dO = wa.backward_edges(Vt, Ft, O, g, found)
    eV, eO = wa.backward_edges(Vt, Ft, O, g, tuple(found))  # summed through the vertex list
    assert torch.equal(dV, eV) and torch.equal(dO, eO)


@pytest.mark.parametrize("name", NAMES)
def test_welded_sides(name):
    V, F = _mesh(name)
    Vt, Ft = torch.from_numpy(V).cuda(), torch.from_numpy(F).cuda()
    rng = np.random.default_rng(4)
    O = torch.from_numpy(rng.uniform(-2.0, 2.0, size=(129, 3))).cuda()
    g = torch.from_numpy(rng.normal(size=129)).cuda()
    want = wa.welded_edges(Vt, Ft)
    weld = wa._weld(Vt, Ft)
    assert isinstance(weld, wa._Weld) and weld[1] == want[1]
    assert weld.cancelled == int((want[0][6, :want[1]] == 0).sum())
    if name == "closed":  # its gradient is zero: nothing but rounding to compare
        return
    dV, dO = wa.backward_welded_edges(Vt, Ft, O, g)
    eV, eO = wa.backward_welded_edges(Vt, Ft, O, g, want)
    for a, b in ((dV, eV), (dO, eO)):
        assert torch.isfinite(a).all()
        assert float((a - b).abs().max()) <= 2e-5 * max(float(b.abs().max()), 1e-12)
    again = wa.backward_welded_edges(Vt, Ft, O, g)
    assert torch.equal(dV, again[0]) and torch.equal(dO, again[1])


@pytest.mark.parametrize("index", [-1, 3])
def test_bad_index_is_left_to_the_general_path(index):
    V = torch.eye(3, dtype=torch.float64).cuda()
    F = torch.tensor([[0, 1, index]]).cuda()
    assert wa._boundary_edges_device(V, F) is None
