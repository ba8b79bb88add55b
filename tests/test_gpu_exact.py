"""The FP64 winding number through near faces, boundary edges and an integer
(csrc/wn_exact.cu) against the all-pairs FP64 kernel, at the sizes and meshes where it
can go wrong: remainders of leaves and warps, every number of lanes per query, queries
on vertices, edges and faces, boundaries as fans and as single edges, faces that share
positions but not indices, duplicated, flipped and collapsed faces, queries that only
the all-pairs fallback can do. Bar: the plain path's own (1e-12 per query)."""

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from igl import autograd as wa, synthetic  # noqa: E402

pytestmark = pytest.mark.gpu


def _both(V, F, O):
    Vt, Ft, Ot = (torch.from_numpy(np.ascontiguousarray(x)).cuda() for x in (V, F, O))
    tri, ld, nf = wa.triangle_soa(Vt, Ft)
    got = wa.forward_exact(tri, ld, nf, Ot)
    return got, wa.forward_fp64(tri, ld, nf, Ot)


def _check(V, F, O):
    got, ref = _both(V, F, O)
    assert got is not None
    assert float((got - ref).abs().max()) <= 1e-12


@pytest.mark.parametrize("faces, queries", [(36631, 4096), (36632, 4097), (20479, 17000),
                                            (20473, 70001), (5119, 40031), (1281, 262147),
                                            (1024, 150001)])
@pytest.mark.parametrize("cut", [0.0, 0.08])
def test_sizes(faces, queries, cut):
    level = 3 if faces < 1300 else 4 if faces < 5200 else 5 if faces < 21000 else 6
    V, F = synthetic.bumpy_icosphere(level, seed=faces)
    # The lowest faces (the generator's own order is not local) leave one long boundary;
    # `cut` deletes single faces too.
    F = F[np.argsort(V[F][:, :, 2].max(1), kind="stable")]
    F = synthetic.delete_faces(F[:faces], cut, seed=3)
    F = F if len(F) >= 1024 else F[np.arange(1024) % len(F)]
    queries = max(queries, int(1.5e8 / len(F)) + 1)
    _check(V, F, synthetic.mixed_queries(V, F, queries, seed=5))


def _degenerate(V, F):
    extra = np.concatenate([F[:700], F[:300, ::-1],
                            np.stack([F[:200, 0], F[:200, 0], F[:200, 1]], 1)])
    return V, np.concatenate([F, extra])


@pytest.mark.parametrize("mesh", ["closed", "open", "soup", "degenerate", "signed_zero", "grid",
                                  "far", "tiny"])
def test_queries_on_the_mesh(mesh):
    V, F = synthetic.bumpy_icosphere(5, seed=9)
    if mesh == "open":
        F = synthetic.delete_faces(F, 0.2, seed=4)  # holes that meet, loops of every length
    elif mesh == "soup":
        V, F = synthetic.unshare_vertices(V, F)
    elif mesh == "degenerate":
        V, F = _degenerate(V, F)
    elif mesh == "signed_zero":
        V = np.where(np.abs(V) < 0.05, 0.0, V)  # flattened, collapsed and repeated faces
        V, F = synthetic.unshare_vertices(V, F)
        V[::2] = np.where(V[::2] == 0.0, -0.0, V[::2])
    elif mesh == "grid":
        V, F = synthetic.terrain_grid(101)
    elif mesh == "far":
        V = V + 1e5
    elif mesh == "tiny":
        V = V * 1e-30
    tri = V[F]
    O = np.concatenate([V[::3], tri.mean(1)[::3], 0.5 * (tri[:, 0] + tri[:, 1])[::3],
                        0.9 * tri[::5, 1] + 0.1 * tri[::5, 2],
                        synthetic.mixed_queries(V, F, 3000, seed=6)])
    _check(V, F, O)


def test_distant_and_nonfinite_queries():
    V, F = synthetic.bumpy_icosphere(5, seed=2)
    F = synthetic.delete_faces(F, 0.05, seed=2)
    O = synthetic.mixed_queries(V, F, 12000, seed=3)
    O[5] = [1e12, 0.0, 0.0]  # beyond the FP32 walk's range: the fallback's
    O[6] = [-3e40, 1e40, 0.0]
    O[7] = [np.nan, 0.0, 0.0]
    O[8:40] *= 1e4
    got, ref = _both(V, F, O)
    assert bool(torch.isnan(got[7])) and bool(torch.isnan(ref[7]))
    keep = torch.ones(len(O), dtype=torch.bool, device="cuda")
    keep[7] = False
    assert float((got - ref)[keep].abs().max()) <= 1e-12


def test_calls_left_to_the_all_pairs_kernels():
    rng = np.random.default_rng(1)
    O = rng.normal(size=(20000, 3))
    V = rng.normal(size=(30000, 3))
    F = np.arange(30000).reshape(-1, 3)
    assert _both(V, F, O)[0] is None  # no edge has a partner
    V, F = synthetic.bumpy_icosphere(5, seed=2)
    assert _both(V, F, O[:1000])[0] is None  # too few queries
    V[7, 1] = 1e80
    assert _both(V, F, O)[0] is None  # products of such coordinates may overflow


def test_under_capture_the_all_pairs_kernel_runs():
    V, F = synthetic.bumpy_icosphere(5, seed=2)
    O = synthetic.mixed_queries(V, F, 20000, seed=3)
    Vt, Ft, Ot = (torch.from_numpy(np.ascontiguousarray(x)).cuda() for x in (V, F, O))
    tri, ld, nf = wa.triangle_soa(Vt, Ft)
    ref = wa.forward_fp64(tri, ld, nf, Ot)
    assert wa.forward_exact(tri, ld, nf, Ot) is not None
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        assert wa.forward_exact(tri, ld, nf, Ot) is None
        w = wa.forward_fp64(tri, ld, nf, Ot)
    graph.replay()
    assert torch.equal(w, ref)


def test_reduced_precision_results_and_faces_adjoint():
    """float32 queries take the FP64 path too; the per-face adjoint prepares its mesh in
    the backward pass then."""
    V, F = synthetic.bumpy_icosphere(4, seed=3)
    F = synthetic.delete_faces(F, 0.05, seed=3)
    O = synthetic.mixed_queries(V, F, 40000, seed=4)
    grads = {}
    for adjoint in ("faces", "edges"):
        Vt = torch.tensor(V, dtype=torch.float32, device="cuda", requires_grad=True)
        Ot = torch.tensor(O, dtype=torch.float32, device="cuda", requires_grad=True)
        W = wa.winding_number_torch(Vt, torch.tensor(F, device="cuda"), Ot, adjoint=adjoint)
        tri, ld, nf = wa.triangle_soa(Vt.detach(), torch.tensor(F, device="cuda"))
        ref = wa.forward_fp64(tri, ld, nf, Ot.detach()).to(torch.float32)
        assert float((W - ref).abs().max()) <= 2.0 ** -22  # one rounding to float32 each
        grads[adjoint] = torch.autograd.grad((W * W).sum(), (Vt, Ot))
    for a, b in zip(grads["faces"], grads["edges"]):
        assert float((a - b).abs().max()) <= 1e-4 * float(b.abs().max())
