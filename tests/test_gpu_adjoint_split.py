"""The boundary-edge adjoints at the edges of their splits (edges per thread and tile,
queries per chunk and group, groups per finishing slice) against torch.autograd of the
solid-angle sum in 64 bits. Bars: 1e-9 of the largest entry in FP64, 2e-5 in mixed
precision (FP32 pairs, 24 bits, a few hundred to a sum)."""

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from igl import autograd as wa  # noqa: E402

pytestmark = pytest.mark.gpu


def _strip(n):
    """A fan of n faces about a bent line: n + 2 boundary edges."""
    t = np.linspace(0.0, 4.0, n + 2)
    V = np.stack([np.cos(t) * (1 + 0.3 * (np.arange(n + 2) % 2)), np.sin(t), 0.2 * t], 1)
    F = np.stack([np.arange(n), np.arange(n) + 1, np.arange(n) + 2], 1)
    F[1::2] = F[1::2][:, [0, 2, 1]]
    return V, F


def _autograd(V, F, O, g):
    V = V.clone().requires_grad_(True)
    O = O.clone().requires_grad_(True)
    r = V[F][None] - O[:, None, None, :]
    a, b, c = r.unbind(2)
    la, lb, lc = (x.norm(dim=-1) for x in (a, b, c))
    det = (a * torch.linalg.cross(b, c)).sum(-1)
    den = la * lb * lc + (a * b).sum(-1) * lc + (b * c).sum(-1) * la + (c * a).sum(-1) * lb
    W = torch.atan2(det, den).sum(1) / (2 * np.pi)
    return torch.autograd.grad(W, (V, O), g)


@pytest.mark.parametrize("precision, bar", [("fp64", 1e-9), ("mixed", 2e-5)])
@pytest.mark.parametrize("faces, queries", [(1, 1), (2, 63), (61, 64), (62, 65), (63, 15),
                                            (254, 513), (255, 129), (510, 2049), (511, 17),
                                            (770, 4100)])
def test_split_edges(faces, queries, precision, bar):
    V, F = _strip(faces)
    rng = np.random.default_rng(faces)
    O = torch.from_numpy(rng.uniform(-2.0, 2.0, size=(queries, 3))).cuda()
    g = torch.from_numpy(rng.normal(size=queries)).cuda()
    Vt, Ft = torch.from_numpy(V).cuda(), torch.from_numpy(F).cuda()
    dV, dO = wa.backward_edges(Vt, Ft, O, g, precision=precision)
    eV, eO = _autograd(Vt, Ft, O, g)
    assert float((dV - eV).abs().max()) <= bar * float(eV.abs().max())
    assert float((dO - eO).abs().max()) <= bar * float(eO.abs().max())


@pytest.mark.parametrize("faces, queries", [(1, 3), (21, 31), (22, 33), (85, 65), (341, 2050)])
def test_split_welded(faces, queries):
    rng = np.random.default_rng(faces)
    V = rng.normal(size=(3 * faces, 3))
    F = np.arange(3 * faces).reshape(-1, 3)
    O = torch.from_numpy(rng.uniform(-3.0, 3.0, size=(queries, 3))).cuda()
    g = torch.from_numpy(rng.normal(size=queries)).cuda()
    Vt, Ft = torch.from_numpy(V).cuda(), torch.from_numpy(F).cuda()
    dV, dO = wa.backward_welded_edges(Vt, Ft, O, g)
    eV, eO = _autograd(Vt, Ft, O, g)
    assert float((dV - eV).abs().max()) <= 2e-5 * float(eV.abs().max())
    assert float((dO - eO).abs().max()) <= 2e-5 * float(eO.abs().max())
