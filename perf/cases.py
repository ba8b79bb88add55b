"""The calls that users of this package make, for timing: sizes, inputs, one pass, exact values.

Every case goes through the package's public Python entry points on seeded
synthetic meshes: bumpy icospheres of subdivision ``level`` (20*4^level faces,
``cut`` of them deleted) and terrain grids (2*(n-1)^2 faces), with queries half
in the 1.2x bounding box and half near the surface, as in ``igl.synthetic``.

kind         a pass
wn           igl.winding_number(V, F, O, device="gpu"), host arrays in and out, FP64
forward      winding_number_torch(V, F, O) on device tensors, no gradient
grad         the same and its gradients dL/dV, dL/dO
batch        Batch.replay(): forward and adjoint of uneven meshes from one CUDA graph
closest      AABB.squared_distance(..., device="gpu"), host arrays, tree kept
query        DeviceAABB.query(P) on device tensors, tree kept
signed       DeviceAABB.signed_distance(P, precision="fast"), tree kept
normals      DeviceNormals.evaluate(V, weighting), topology kept
"""

import functools
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                                "mojo-libigl_b200", "python"))

import igl  # noqa: E402
from igl import synthetic  # noqa: E402


def listed():
    return [
        # One point against a small mesh (an interactive inside test): the smallest call.
        {"name": "wn_point", "kind": "wn", "mesh": "sphere", "level": 3, "cut": 0.08, "queries": 1},
        # The reference's own winding-number benchmark: grid(120) x 1024 queries.
        {"name": "wn_grid120", "kind": "wn", "mesh": "grid", "n": 120, "queries": 1024},
        # The plain FP64 drop-in at size: open subdivision-5 mesh x 2^20 queries.
        {"name": "wn_open_1m", "kind": "wn", "mesh": "sphere", "level": 5, "cut": 0.08,
         "queries": 1 << 20},
        # The headline workload with float32 tensors (mixed precision is their default).
        {"name": "forward_f32_1m", "kind": "forward", "mesh": "sphere", "level": 7, "cut": 0.0,
         "queries": 1 << 20, "near": 1e-4, "dtype": "float32", "soup": False},
        # The gradient workload: open subdivision-5 mesh, near-surface queries, float32.
        {"name": "grad_f32", "kind": "grad", "mesh": "sphere", "level": 5, "cut": 0.08,
         "queries": 262144, "near": 1e-3, "dtype": "float32", "soup": False},
        # The same in float64 (FP64 forward and adjoint), an odd number of queries.
        {"name": "grad_f64", "kind": "grad", "mesh": "sphere", "level": 5, "cut": 0.08,
         "queries": 100003, "near": 1e-3, "dtype": "float64", "soup": False},
        # Triangle soup as read from an STL file (no shared vertices), float32.
        {"name": "grad_soup_f32", "kind": "grad", "mesh": "sphere", "level": 5, "cut": 0.0,
         "queries": 131072, "near": 1e-3, "dtype": "float32", "soup": True},
        # Uneven meshes with uneven query sets, one graph replay per step.
        {"name": "batch_16", "kind": "batch", "meshes": 16, "max_level": 6,
         "max_queries": 1 << 16},
        # The reference's own closest-point benchmark: grid(350) x 10,000 points.
        {"name": "closest_grid350", "kind": "closest", "mesh": "grid", "n": 350,
         "queries": 10000},
        # Closest points of a million points on the headline mesh.
        {"name": "query_1m", "kind": "query", "mesh": "sphere", "level": 7, "cut": 0.0,
         "queries": 1 << 20, "near": 1e-4},
        # Signed distance samples (hierarchical sign), e.g. for training a distance field.
        {"name": "signed_250k", "kind": "signed", "mesh": "sphere", "level": 6, "cut": 0.0,
         "queries": 250000, "near": 1e-2},
        # Vertex normals of a deforming mesh, topology prepared once.
        {"name": "normals_1m", "kind": "normals", "mesh": "sphere", "level": 8, "cut": 0.0,
         "weighting": 1},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["wn", "wn", "forward", "grad", "grad", "batch", "closest", "query",
                       "signed", "normals"])
    if kind == "batch":
        return {"kind": kind, "meshes": rng.randint(2, 24), "max_level": rng.randint(4, 6),
                "max_queries": _log_int(rng, 1 << 12, 1 << 16)}
    case = {"kind": kind}
    if kind in ("wn", "closest") and rng.random() < 0.5:
        case.update(mesh="grid", n=_log_int(rng, 12, 350))
        nf = 2 * (case["n"] - 1) ** 2
    else:
        level = rng.randint(5, 8) if kind == "normals" else rng.randint(3, 7)
        case.update(mesh="sphere", level=level,
                    cut=0.0 if rng.random() < 0.4 else round(rng.uniform(0.0, 0.1), 3))
        nf = 20 * 4 ** level
    if kind == "normals":
        case["weighting"] = rng.randint(0, 3)
        return case
    # At most this many pairs, so that no drawn case costs more than the largest listed one.
    most = {"wn": 2e10, "forward": 3e11, "grad": 5e9}.get(kind, math.inf)
    hi = 1 << 20
    if kind == "grad":
        case["soup"] = rng.random() < 0.3
        hi = 1 << 18
    case["queries"] = _log_int(rng, 1 if kind == "wn" else 512, max(1024, min(hi, most / nf)))
    if kind in ("forward", "grad"):
        case["dtype"] = rng.choice(["float32", "float32", "float64"])
        case.setdefault("soup", False)
        if case["dtype"] == "float64" and kind == "forward":
            case["queries"] = min(case["queries"], int(4e10 / nf))
    if kind not in ("wn", "closest"):
        case["near"] = rng.choice([1e-4, 1e-3, 1e-2])
    # Open where a closed mesh would leave nothing but rounding to return: W of a few
    # points that may all lie outside, and the gradients (zero on a closed indexed mesh).
    if case.get("cut") == 0.0 and ((kind == "wn" and case["queries"] < 64)
                                   or (kind == "grad" and not case["soup"])):
        case["cut"] = 0.05
    return case


@functools.lru_cache(maxsize=None)
def _unit_sphere(level):
    V, F = synthetic.icosahedron()
    for _ in range(level):
        V, F = synthetic._subdivide(V, F)
    return V, F


def _sphere(level, cut, seed):
    """synthetic.bumpy_icosphere with the subdivision kept between seeds."""
    V, F = _unit_sphere(level)
    rng = np.random.default_rng(seed)
    a = rng.uniform(0.0, 0.02, size=8)
    k = rng.normal(size=(8, 3))
    k *= rng.uniform(1.0, 6.0, size=(8, 1)) / np.linalg.norm(k, axis=1, keepdims=True)
    phi = rng.uniform(0.0, 2.0 * np.pi, size=8)
    V = V * (1.0 + (a * np.sin(V @ k.T + phi)).sum(1))[:, None]
    return V, synthetic.delete_faces(F, cut, seed + 1)


def _mesh(case, seed):
    if case["mesh"] == "grid":
        V, F = synthetic.terrain_grid(case["n"])
        rng = np.random.default_rng(seed)
        V[:, 2] += rng.normal(0.0, 0.01, size=len(V))
        return V, F
    return _sphere(case["level"], case["cut"], seed)


def _points(case, V, F, seed):
    n = case["queries"]
    if case["mesh"] == "grid":  # the reference benchmarks' query boxes
        rng = np.random.default_rng(seed + 5)
        margin, height = (0.0, 2.0) if case["kind"] == "wn" else (10.0, 5.0)
        top = case["n"] - 1 + margin
        return np.column_stack([rng.uniform(-margin, top, size=(n, 2)),
                                rng.uniform(-height, height, size=n)])
    near = case.get("near", 1e-3)
    if case["kind"] == "grad":
        return synthetic.near_surface_points(V, F, n, seed + 5, near)
    return synthetic.mixed_queries(V, F, n, seed + 5, near_sigma=near)


def _batch(case, seed):
    sizes = np.random.default_rng(case["meshes"])  # the same sizes for every seed
    meshes, queries = [], []
    for i in range(case["meshes"]):
        level = int(sizes.integers(2, case["max_level"] + 1)) if i else case["max_level"]
        V, F = _sphere(level, float(sizes.uniform(0.01, 0.1)), seed + 100 * i + 7)
        n = case["max_queries"]
        n = int(math.exp(sizes.uniform(math.log(1024), math.log(n)))) if i else n
        meshes.append((V, F))
        queries.append(synthetic.mixed_queries(V, F, n, seed + 100 * i + 9))
    rng = np.random.default_rng(seed)
    gW = [rng.normal(size=len(q)) for q in queries]
    return meshes, queries, gW


def _tensors(case, seed):
    V, F = _mesh(case, seed)
    O = _points(case, V, F, seed)
    if case["soup"]:
        V, F = synthetic.unshare_vertices(V, F)
    dtype = getattr(torch, case["dtype"])
    rng = np.random.default_rng(seed + 11)
    return (torch.tensor(V, dtype=dtype, device="cuda"), torch.tensor(F, device="cuda"),
            torch.tensor(O, dtype=dtype, device="cuda"),
            torch.tensor(rng.normal(size=len(O)), dtype=dtype, device="cuda"))


def prepare(case, seed):
    kind = case["kind"]
    state = {"kind": kind}
    if kind == "batch":
        from igl.batched import Batch

        meshes, queries, gW = _batch(case, seed)
        batch = Batch(meshes, queries)
        batch.gW.copy_(torch.from_numpy(np.concatenate(gW)))
        batch.capture()
        state["batch"] = batch
    elif kind in ("forward", "grad"):
        V, F, O, gW = _tensors(case, seed)
        if kind == "grad":
            V.requires_grad_(True)
            O.requires_grad_(True)
        state.update(V=V, F=F, O=O, gW=gW)
    else:
        V, F = _mesh(case, seed)
        if kind == "normals":
            from igl.normals import DeviceNormals

            state.update(normals=DeviceNormals(F, len(V)), V=torch.from_numpy(V).cuda(),
                         weighting=case["weighting"])
            return state
        P = _points(case, V, F, seed)
        if kind == "wn":
            # One query is a (3,) point, and the answer a float.
            state.update(V=V, F=F, O=P[0] if len(P) == 1 else P)
        elif kind == "closest":
            tree = igl.AABB()
            tree.init(V, F)
            tree.squared_distance(V, F, P[:1], device="gpu")  # uploads the tree
            state.update(V=V, F=F, P=P, tree=tree)
        else:
            from igl.distance import DeviceAABB

            tree = DeviceAABB(V, F)
            if kind == "signed":
                tree.fast_winding()
            state.update(tree=tree, P=torch.from_numpy(P).cuda())
    return state


def run(state):
    kind = state["kind"]
    if kind == "wn":
        return igl.winding_number(state["V"], state["F"], state["O"], device="gpu")
    if kind == "forward":
        with torch.no_grad():
            return igl.autograd.winding_number_torch(state["V"], state["F"], state["O"])
    if kind == "grad":
        W = igl.autograd.winding_number_torch(state["V"], state["F"], state["O"])
        dV, dO = torch.autograd.grad(W, (state["V"], state["O"]), state["gW"])
        return [W.detach(), dV, dO]
    if kind == "batch":
        batch = state["batch"]
        batch.replay()
        return [batch.W, batch.dV, batch.dQ]
    if kind == "closest":
        return list(state["tree"].squared_distance(state["V"], state["F"], state["P"],
                                                   device="gpu"))
    if kind == "query":
        return list(state["tree"].query(state["P"]))
    if kind == "signed":
        return list(state["tree"].signed_distance(state["P"], precision="fast"))
    return state["normals"].evaluate(state["V"], state["weighting"])


def _sizes(case):
    """(faces, vertices, queries) of a case."""
    if case["kind"] == "batch":
        nf = 20 * 4 ** case["max_level"]
        return 2 * nf, nf, 2 * case["max_queries"]
    if case["mesh"] == "grid":
        nf, nv = 2 * (case["n"] - 1) ** 2, case["n"] ** 2
    else:
        nf, nv = 20 * 4 ** case["level"], 10 * 4 ** case["level"] + 2
        nf -= int(round(case["cut"] * nf))
    if case.get("soup"):
        nv = 3 * nf
    return nf, nv, case.get("queries", 0)


def work(case):
    """Inputs read once, outputs written once; every face and query takes part in at
    least one pair term (62 flops). The sum over all pairs defines the winding number
    but bounds no method that computes it."""
    kind = case["kind"]
    nf, nv, nq = _sizes(case)
    size = 4 if case.get("dtype") == "float32" else 8
    mesh = 24 * nf + 3 * size * nv
    if kind == "normals":
        return {"bytes": 24 * nf + 48 * nv, "flops": 30 * nf}
    if kind in ("closest", "query", "signed"):
        out = 48 if kind == "signed" else 40
        return {"bytes": mesh + (24 + out) * nq, "flops": 62 * nq}
    moved = mesh + 4 * size * nq
    if kind in ("grad", "batch"):
        moved += 3 * size * nv + 4 * size * nq
    return {"bytes": moved, "flops": 62 * (nf + nq)}


# ---- exact values: plain torch in 64 bits -----------------------------------

_CHUNK = 1 << 23  # pairs per evaluation


def _solid_angles(tri, q):
    """Winding numbers of q against tri (nf, 3, 3) in one piece."""
    r = tri[None] - q[:, None, None, :]
    a, b, c = r.unbind(2)
    la, lb, lc = (x.square().sum(-1).sqrt() for x in (a, b, c))
    det = (a * torch.linalg.cross(b, c)).sum(-1)
    denom = la * lb * lc + (a * b).sum(-1) * lc + (b * c).sum(-1) * la + (c * a).sum(-1) * lb
    return torch.atan2(det, denom).sum(1) / (2.0 * math.pi)


def _exact_winding(V, F, O):
    tri = V[F]
    W = torch.zeros(len(O), dtype=torch.float64, device=V.device)
    step = max(1, min(len(tri), _CHUNK // max(1, min(len(O), 4096))))
    rows = max(1, _CHUNK // step)
    for i in range(0, len(O), rows):
        for j in range(0, len(tri), step):
            W[i:i + rows] += _solid_angles(tri[j:j + step], O[i:i + rows])
    return W


def _exact_gradient(V, F, O, gW):
    """(W, dL/dV, dL/dO) by torch.autograd over blocks of pairs."""
    V = V.clone().requires_grad_(True)
    O = O.clone().requires_grad_(True)
    W = torch.zeros(len(O), dtype=torch.float64, device=V.device)
    dV, dO = torch.zeros_like(V), torch.zeros_like(O)
    step = max(1, min(len(F), _CHUNK // max(1, min(len(O), 4096))))
    rows = max(1, _CHUNK // step)
    for i in range(0, len(O), rows):
        for j in range(0, len(F), step):
            o = O[i:i + rows]
            w = _solid_angles(V[F[j:j + step]], o)
            gv, go = torch.autograd.grad(w, (V, O), gW[i:i + rows])
            W[i:i + rows] += w.detach()
            dV += gv
            dO += go
    return W, dV, dO


def _exact_closest(V, F, P):
    """Squared distances by brute force: inside the face's prism, else the nearest side."""
    tri = V[F]
    best = torch.full((len(P),), math.inf, dtype=torch.float64, device=V.device)
    step = max(1, (_CHUNK // 2) // max(1, len(P)))
    for j in range(0, len(tri), step):
        A, B, C = tri[j:j + step].unbind(1)
        n = torch.linalg.cross(B - A, C - A)
        n = n / n.square().sum(-1, keepdim=True).sqrt()
        inside, d2 = None, None
        for S, T in ((A, B), (B, C), (C, A)):
            e = T - S
            p = P[:, None] - S
            t = ((p * e).sum(-1) / e.square().sum(-1)).clamp(0.0, 1.0)
            side = (p - t[..., None] * e).square().sum(-1)
            left = (torch.linalg.cross(n, e) * p).sum(-1) >= 0
            d2 = side if d2 is None else torch.minimum(d2, side)
            inside = left if inside is None else inside & left
        plane = ((P[:, None] - A) * n).sum(-1).square()
        best = torch.minimum(best, torch.where(inside, plane, d2).amin(1))
    return best


def _exact_normals(V, F, weighting):
    A, B, C = V[F].unbind(1)
    n = torch.linalg.cross(B - A, C - A)
    length = n.square().sum(-1, keepdim=True).sqrt()
    u = n / length
    N = torch.zeros_like(V)
    for k, (p, q, r) in enumerate(((A, B, C), (B, C, A), (C, A, B))):
        if weighting == 0:
            w = 1.0
        elif weighting == 2:
            e, f = q - p, r - p
            cosine = (e * f).sum(-1) / (e.square().sum(-1) * f.square().sum(-1)).sqrt()
            w = torch.acos(cosine.clamp(-1.0, 1.0))[:, None]
        else:
            w = length
        N.index_add_(0, F[:, k], u * w)
    size = N.square().sum(-1, keepdim=True).sqrt()
    return torch.where(size > 1e-30, N / size, N)


def exact(case, seed):
    kind = case["kind"]
    nf, nv, nq = _sizes(case)
    if kind == "signed":
        return None  # the hierarchical W approximates: plain sums give another number
    if kind == "batch":
        meshes, queries, gW = _batch(case, seed)
        if sum(len(F) * len(q) for (_, F), q in zip(meshes, queries)) > 1.5e10:
            return None
        got = [_exact_gradient(*(torch.from_numpy(x).cuda() for x in (V, F, q, g)))
               for (V, F), q, g in zip(meshes, queries, gW)]
        return [torch.cat(x) for x in zip(*got)]
    if kind in ("forward", "grad"):
        if nf * nq > (6e10 if kind == "forward" else 1.5e10):
            return None
        V, F, O, gW = _tensors(case, seed)
        if kind == "forward":
            return _exact_winding(V.double(), F, O.double())
        W, dV, dO = _exact_gradient(V.double(), F, O.double(), gW.double())
        return [W, dV, dO if case["cut"] else None]  # a closed soup's dL/dO is zero
    V, F = _mesh(case, seed)
    Vd, Fd = torch.from_numpy(V).cuda(), torch.from_numpy(F).cuda()
    if kind == "normals":
        return _exact_normals(Vd, Fd, case["weighting"])
    if nf * nq > 6e10:
        return None
    P = torch.from_numpy(_points(case, V, F, seed)).cuda()
    if kind == "wn":
        W = _exact_winding(Vd, Fd, P)
        return float(W[0]) if len(P) == 1 else W.cpu().numpy()
    return [_exact_closest(Vd, Fd, P), None, None]  # ties leave face and point open
